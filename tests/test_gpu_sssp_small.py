"""SSSP at the sizes where one CTA takes it: around 24,576 edges and 24,576 vertices, rows long enough for the whole
CTA and more of them than its list holds, chains, unweighted graphs, fractional weights (truncated at every step),
zero weights, unreachable vertices. Distances equal the oracle's bit for bit."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_parity import host_views

pytestmark = pytest.mark.gpu


def random_edges(V, E, seed):
    rng = np.random.default_rng(seed)
    return (rng.random(E) ** 3 * V).astype(np.int64), (rng.random(E) ** 2 * V).astype(np.int64)


def wheel(V, hubs, spokes):
    h = np.arange(1, hubs + 1)
    src = np.concatenate([np.zeros(hubs, np.int64), np.repeat(h, spokes)])
    return src, np.concatenate([h, (np.arange(hubs * spokes) * 7 + hubs) % V])


GRAPHS = {
    "one_vertex": (1, lambda: (np.zeros(0, np.int64),) * 2),
    "tiny": (33, lambda: random_edges(33, 100, 1)),
    "edges_24575": (3000, lambda: random_edges(3000, 24_575, 2)),
    "edges_24576": (3000, lambda: random_edges(3000, 24_576, 3)),
    "edges_24577": (3000, lambda: random_edges(3000, 24_577, 4)),
    "vertices_24576": (24_576, lambda: random_edges(24_576, 20_000, 5)),
    "vertices_24577": (24_577, lambda: random_edges(24_577, 20_000, 6)),
    "chain": (1500, lambda: (np.arange(1499), np.arange(1, 1500))),
    "long_rows": (5000, lambda: wheel(5000, 100, 200)),
    "row_of_all": (20_000, lambda: (np.zeros(20_000, np.int64), np.arange(20_000))),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("weights", ["int", "fraction", "zero", None])
def test_small_sssp(gbx, cuda_device, name, weights):
    V, make = GRAPHS[name]
    src, dst = make()
    rng = np.random.default_rng(9)
    w = None
    if weights:
        w = {"int": rng.integers(1, 256, len(src)), "fraction": rng.random(len(src)) * 3, "zero": rng.integers(0, 2, len(src))}[weights]
        w = w.astype(np.float32)
    el = gbx.EdgeList(V, src.astype(np.uint32), dst.astype(np.uint32), w)
    g = gbx.graph_csr_preprocessing(el, sort=1, dedup=False, directed=True, keep_weights=w is not None)
    host, _ = host_views(g)
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        for root in sorted({0, V // 2, V - 1}):
            want = po.sssp(host, root, 64, use_weights=w is not None)
            for delta in (0, 7):
                st = gbx.sssp(dg, root, delta)
                np.testing.assert_array_equal(np.asarray(st.distances), want)
                reached = want != 0xFFFFFFFF // 2
                assert st.reached == int(reached.sum())
                assert st.edges_traversed == int(g.out_degree[reached].sum())
