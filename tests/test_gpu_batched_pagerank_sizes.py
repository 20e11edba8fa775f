"""Batched PageRank against 64-bit sums at the sizes where its kernel changes: batches whose largest graph allows
two contribution buffers in shared memory (46,976 / 2 vertices), one (46,976) or none; ids around the 15 bits of a
16-bit word (32,768); vertex counts around 32 (the place of a contribution), edge counts around a group (256) and
around 32 warps' groups; one row with all edges, rows of one edge, graphs without edges.

Tolerance: ranks are sums of positive terms, added in trees of at most 8 + 5 levels, rounded once more by the
recurrence's two operations and its division, and the recurrence damps what an iteration adds by 0.85:
16 * 2^-24 / 0.15 = 6.4e-6 at the very worst, 2e-6 for what roundings do on average."""
import numpy as np
import pytest

import graphblox_gb300 as gg

pytestmark = pytest.mark.gpu

BASE, DAMP = 1.0 - float(np.float32(0.85)), float(np.float32(0.85))


def graph(V, E, shape, seed):
    rng = np.random.default_rng(seed)
    src = (rng.random(E) ** 3 * V).astype(np.uint32)
    if shape == "hub":
        dst = np.full(E, V // 2, np.uint32)
    elif shape == "chain":
        src = np.arange(min(E, V - 1), dtype=np.uint32)
        dst = src + 1
    else:
        dst = (rng.random(E) ** 2 * V).astype(np.uint32)
    return V, src, dst


def reference(V, src, dst, iterations, epsilon):
    out = np.bincount(src, minlength=V).astype(np.float64)
    order = np.argsort(dst, kind="stable")
    off = np.zeros(V + 1, np.int64)
    off[1:] = np.cumsum(np.bincount(dst, minlength=V))
    rows, s = np.flatnonzero(np.diff(off)), src[order]
    r = np.full(V, BASE)
    for it in range(iterations):
        c = np.divide(r, out, out=np.zeros(V), where=out > 0)
        sums = np.zeros(V)
        if len(rows):
            sums[rows] = np.add.reduceat(c[s], off[rows])
        nxt = BASE + DAMP * sums
        moved = np.abs(nxt - r).max()
        r = nxt
        if epsilon and moved < epsilon:
            return r / V, it
    return r / V, iterations


SMALL = [(1, 0, "any"), (1, 5, "any"), (31, 255, "any"), (32, 256, "any"), (33, 257, "any"), (5, 300, "hub"), (300, 299, "chain"),
         (1000, 8191, "any"), (1000, 8192, "any"), (1000, 8193, "any"), (1024, 60_000, "hub"), (9000, 8999, "chain")]
BATCHES = {
    "two_buffers": SMALL + [(23_488, 200_000, "any"), (23_457, 50_000, "hub")],
    "one_buffer": SMALL + [(23_489, 200_000, "any"), (32_767, 300_000, "any"), (32_768, 300_000, "any"), (32_769, 300_000, "any"),
                           (46_976, 100_000, "any"), (40_000, 39_999, "chain")],
    "no_buffer": SMALL + [(46_977, 300_000, "any"), (32_768, 70_000, "hub"), (100_000, 500_000, "hub"), (100_000, 99_999, "chain")],
}


@pytest.mark.parametrize("name", sorted(BATCHES))
@pytest.mark.parametrize("iterations,epsilon", [(0, 0.0), (1, 0.0), (2, 0.0), (3, 0.0), (30, 0.0), (80, 1e-3)])
def test_batched_pagerank_sizes(gbx, cuda_device, name, iterations, epsilon):
    graphs = [graph(V, E, shape, 11 + i) for i, (V, E, shape) in enumerate(BATCHES[name])]
    packed = gg.pack_graphs(graphs)
    base = packed.vertex_base.astype(np.int64)
    with gg.GraphBatch(packed) as b:
        first, res = b.page_rank(iterations, epsilon)
        second, again = b.page_rank(iterations, epsilon)
    np.testing.assert_array_equal(first, second)  # a fixed order of additions
    np.testing.assert_array_equal(res["iterations"], again["iterations"])
    for g, (V, src, dst) in enumerate(graphs):
        want, count = reference(V, src, dst, iterations, epsilon)
        # a vertex within rounding of epsilon may end the run an iteration earlier or later
        assert abs(int(res["iterations"][g]) - count) <= (1 if epsilon else 0)
        tol = 2e-6 * want + (2 * epsilon / V if epsilon else 0.0)
        assert np.all(np.abs(first[base[g]:base[g + 1]] - want) <= tol), (g, V)
