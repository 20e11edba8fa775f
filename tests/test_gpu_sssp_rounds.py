"""SSSP rounds of the persistent kernel: rows on both sides of its hub line (256), more hubs side by side than a warp
stages (32), rounds on both sides of the scan line, bucket moves, ragged vertex counts. Distances equal the oracle's
bit for bit."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_parity import host_views

pytestmark = pytest.mark.gpu


def layers(V, hubs, spokes):
    """Vertex 0 reaches `hubs` vertices side by side, which together reach as many others side by side, `spokes` edges
    each; those reach the whole graph, `spokes` edges each."""
    first, second = np.arange(1, hubs + 1), np.arange(hubs + 1, 2 * hubs + 1)
    k = np.arange(hubs * spokes)
    src = np.concatenate([np.zeros(hubs, np.int64), np.repeat(first, spokes), np.repeat(second, spokes)])
    return src, np.concatenate([first, second[k % hubs], (k * 13 + 7) % V])


def skewed(V, E, seed):
    rng = np.random.default_rng(seed)
    return (rng.random(E) ** 4 * V).astype(np.int64), (rng.random(E) ** 2 * V).astype(np.int64)


GRAPHS = {
    "hubs_257": (100_001, lambda: layers(100_001, 3000, 257)),
    "no_hubs_256": (100_001, lambda: layers(100_001, 3000, 256)),
    "few_hubs": (50_003, lambda: layers(50_003, 33, 2500)),
    "skewed": (60_000, lambda: skewed(60_000, 1_500_000, 1)),
    "sparse": (300_007, lambda: skewed(300_007, 500_000, 2)),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("weights", ["int", "fraction", None])
def test_sssp_rounds(gbx, cuda_device, name, weights):
    V, make = GRAPHS[name]
    src, dst = make()
    rng = np.random.default_rng(3)
    w = None
    if weights:
        w = (rng.integers(1, 256, len(src)) if weights == "int" else rng.random(len(src)) * 5).astype(np.float32)
    el = gbx.EdgeList(V, src.astype(np.uint32), dst.astype(np.uint32), w)
    g = gbx.graph_csr_preprocessing(el, sort=1, dedup=False, directed=True, keep_weights=w is not None)
    host, _ = host_views(g)
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        for root in (0, 1, V // 3):
            want = po.sssp(host, root, 64, use_weights=w is not None)
            reached = want != 0xFFFFFFFF // 2
            for delta in (0, 16, 5000):
                st = gbx.sssp(dg, root, delta)
                np.testing.assert_array_equal(np.asarray(st.distances), want)
                assert st.reached == int(reached.sum())
                assert st.edges_traversed == int(g.out_degree[reached].sum())
