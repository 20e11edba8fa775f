"""SpMV on the edge-cut engine is no further from 64-bit sums than on the row engine: the same rows and values are swept
by both, the row engine in a graph below 65,536 edges, the other in one that holds one long row more. Rows of every
length class of the row engine that fits such a graph, and mixed.

Bound: the row engine's own error on the same sums (root mean square over all rows of five draws of values, each row's
error relative to the sum of its terms' sizes)."""
import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu

CLASSES = {
    "light": (2, 32),
    "around_a_group": (33, 140),
    "medium": (33, 400),
    "long": (300, 3000),
    "mixed": (1, 600),
}


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("name", sorted(CLASSES))
def test_error_against_64_bits(gbx, cuda_device, name, positive):
    lo, hi = CLASSES[name]
    rng = np.random.default_rng(hi)
    rows = []
    while sum(rows) + hi < 65_000:
        rows.append(int(rng.integers(lo, hi + 1)))
    n, V = len(rows), 40_000
    errors = {}
    off, src = base.csr(rows + [70_000], V, 2, True)
    E = int(off[n])
    small = off.copy()
    small[n + 1:] = E
    for engine, (o, s) in {"rows": (small, src[:E]), "edges": (off, src)}.items():
        assert (len(s) < 65_536) == (engine == "rows")
        total = 0.0
        with base.graph(gbx, o, s, V) as g:
            for seed in range(5):
                r = np.random.default_rng(100 + seed)
                val = (1.0 - r.random(len(src))).astype(np.float32)[:len(s)]
                x = r.uniform(0 if positive else -1, 1, V).astype(np.float32)
                terms = val.astype(np.float64) * x.astype(np.float64)[s]
                y = gbx.spmv(g, x, values=val)[:n]
                total += np.sum(((y - base.row_sums(terms, o)[:n]) / base.row_sums(np.abs(terms), o)[:n]) ** 2)
        errors[engine] = np.sqrt(total / (5 * n))
    print(name, positive, errors["edges"] / errors["rows"])
    assert errors["edges"] <= errors["rows"], errors
