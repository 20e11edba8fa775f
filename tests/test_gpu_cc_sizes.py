"""Connected components where the phases' work changes: vertex counts around a warp's 32 and the 1,024 sampled
labels, components of equal size (the sampled label decides nothing but speed), long chains (deep trees), rows
longer than a warp, isolated vertices, with and without an inverse CSR. Labels equal the oracle's."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_parity import host_views

pytestmark = pytest.mark.gpu


def pairs(V):
    a = np.arange(0, V - 1, 2)
    return a, a + 1


def shuffled_chain(V, seed):
    p = np.random.default_rng(seed).permutation(V)
    return p[:-1], p[1:]


def two_halves(V):
    rng = np.random.default_rng(2)
    a = rng.integers(0, V // 2, 3 * V)
    b = rng.integers(0, V // 2, 3 * V)
    return np.concatenate([a, a + V // 2]), np.concatenate([b, b + V // 2])


GRAPHS = {
    "one": lambda: (1, np.zeros(0, int), np.zeros(0, int)),
    "31": lambda: (31, *shuffled_chain(31, 1)),
    "33": lambda: (33, *pairs(33)),
    "1023": lambda: (1023, *shuffled_chain(1023, 3)),
    "1025": lambda: (1025, *two_halves(1025)),
    "no_edges": lambda: (5000, np.zeros(0, int), np.zeros(0, int)),
    "pairs": lambda: (100_003, *pairs(100_003)),
    "chain": lambda: (200_001, *shuffled_chain(200_001, 4)),
    "two_halves": lambda: (60_000, *two_halves(60_000)),
    "stars": lambda: (90_000, np.repeat(np.arange(30) * 3000 + 2999, 2999), np.concatenate([np.arange(2999) + 3000 * k for k in range(30)])),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("directed", [True, False])
def test_labels(gbx, cuda_device, name, directed):
    V, src, dst = GRAPHS[name]()
    if not directed:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    el = gbx.EdgeList(V, src.astype(np.uint32), dst.astype(np.uint32))
    g = gbx.graph_csr_preprocessing(el, sort=1, dedup=False, directed=directed, keep_weights=False)
    host, pull = host_views(g)
    want = po.cc(host, 1, pull)
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        for variant in (1, 0):
            comp, _ = gbx.connected_components(dg, variant)
            np.testing.assert_array_equal(np.asarray(comp), want, err_msg=f"variant {variant}")
