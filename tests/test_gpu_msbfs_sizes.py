"""Multi-source BFS where its passes change: source counts around each mask width (1, 2, 4, 8 words) and off a multiple
of four, traversals of 8, 9, 16, 17 and more than 32 levels (3 or 4 planes, the general pass), vertex counts off a
warp's group, output rows off a 16-byte boundary, hubs among few sources, sources that die early or reach nothing,
more than 255 vertices per warp and out-degree sums. Distances and counters equal single-source BFS by the oracle."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_parity import host_views

pytestmark = pytest.mark.gpu


def build(gbx, V, src, dst):
    el = gbx.EdgeList(V, np.asarray(src, np.uint32), np.asarray(dst, np.uint32))
    return gbx.graph_csr_preprocessing(el, sort=1, dedup=False, directed=True, keep_weights=False)


def ladder(levels, width):
    """`levels` levels of `width` vertices, each joined to all of the next."""
    a = np.arange(levels - 1)[:, None, None] * width
    src = (a + np.arange(width)[None, :, None]) + np.zeros((1, 1, width), int)
    dst = (a + width + np.arange(width)[None, None, :]) + np.zeros((1, width, 1), int)
    return levels * width, src.ravel(), dst.ravel()


def random_graph(V, E, seed):
    rng = np.random.default_rng(seed)
    return V, (rng.random(E) ** 3 * V).astype(int), (rng.random(E) ** 2 * V).astype(int)


GRAPHS = {
    "random": lambda: random_graph(1001, 8000, 1),
    "random_large": lambda: random_graph(300_003, 1_500_000, 2),
    "levels_8": lambda: ladder(8, 9),
    "levels_9": lambda: ladder(9, 9),
    "levels_16": lambda: ladder(16, 5),
    "levels_17": lambda: ladder(17, 5),
    "levels_40": lambda: ladder(40, 3),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 66, 127, 130, 255, 256])
def test_multisource_sizes(gbx, cuda_device, name, n):
    import torch

    V, src, dst = GRAPHS[name]()
    g = build(gbx, V, src, dst)
    host, pull = host_views(g)
    rng = np.random.default_rng(n)
    roots = rng.integers(0, V, n)
    roots[0] = 0
    roots[n // 2] = int(np.argmax(g.out_degree))
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        room = torch.full((V * n + 1,), -7, dtype=torch.int32, device=cuda_device)
        for offset in (0, 1):
            out = room[offset:offset + V * n].view(V, n)
            _, res = gbx.bfs_multisource(dg, roots, distances=out)
            d = out.cpu().numpy().view(np.uint32)
            for i in sorted({0, 1 % n, n // 2, n - 1}):
                want, _, proc, _ = po.bfs(host, int(roots[i]), pull)
                np.testing.assert_array_equal(d[:, i], want)
                reached = want > 0
                reached[roots[i]] = True
                assert res["processed_nodes"][i] == proc == int(reached.sum())
                assert res["edges_traversed"][i] == int(g.out_degree[reached].sum(dtype=np.int64))
                assert res["depth"][i] == int(want.max())
