"""BFS at the sizes where one CTA takes a traversal: around 65,536 edges (one source) and 8 x 65,536 (trials with
outputs of their own), around 65,536 vertices, rows long enough for the whole CTA and more of them than its list
holds, chains of one vertex per level, sources without out-edges, graphs without an inverse. Levels,
processed_nodes, iteration and edges traversed equal the oracle's; parents form a BFS tree."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_bfs_trials import _check_parents
from test_gpu_parity import host_views

pytestmark = pytest.mark.gpu


def build(gbx, V, src, dst, directed=True):
    if not directed:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    el = gbx.EdgeList(V, src.astype(np.uint32), dst.astype(np.uint32))
    return gbx.graph_csr_preprocessing(el, sort=1, dedup=False, directed=directed, keep_weights=False)


def random_edges(V, E, seed):
    rng = np.random.default_rng(seed)
    return (rng.random(E) ** 3 * V).astype(np.int64), (rng.random(E) ** 2 * V).astype(np.int64)


def wheel(V, hubs):
    """Vertex 0 reaches `hubs` vertices, each of which reaches 200 others."""
    h = np.arange(1, hubs + 1)
    src = np.concatenate([np.zeros(hubs, np.int64), np.repeat(h, 200)])
    dst = np.concatenate([h, (np.arange(hubs * 200) * 7 + hubs) % V])
    return src, dst


GRAPHS = {
    "one_vertex": lambda: (1, np.zeros(0, np.int64), np.zeros(0, np.int64)),
    "tiny": lambda: (33, *random_edges(33, 100, 1)),
    "edges_65535": lambda: (9000, *random_edges(9000, 65_535, 2)),
    "edges_65536": lambda: (9000, *random_edges(9000, 65_536, 3)),
    "edges_65537": lambda: (9000, *random_edges(9000, 65_537, 4)),
    "trial_limit": lambda: (30_000, *random_edges(30_000, 3 * 65_536, 5)),
    "vertices_65536": lambda: (65_536, *random_edges(65_536, 60_000, 6)),
    "vertices_65537": lambda: (65_537, *random_edges(65_537, 60_000, 7)),
    "chain": lambda: (900, np.arange(899), np.arange(1, 900)),
    "many_long_rows": lambda: (20_000, *wheel(20_000, 300)),
    "more_long_rows_than_listed": lambda: (40_000, *wheel(40_000, 1500)),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("directed", [True, False])
def test_small_traversals(gbx, cuda_device, name, directed):
    import torch

    V, src, dst = GRAPHS[name]()
    g = build(gbx, V, src, dst, directed)
    host, pull = host_views(g)
    roots = [0, V - 1, V // 2, V // 3][: min(V, 4)]
    n = len(roots)
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        for mode in (2, 0, 1):
            dist = torch.full((n * V,), -7, dtype=torch.int32, device=cuda_device)
            par = torch.full((n * V,), -7, dtype=torch.int32, device=cuda_device)
            trials = gbx.breadth_first_search_trials(dg, roots, mode, distances=dist, parents=par, out_stride=V)
            bare = gbx.breadth_first_search_trials(dg, roots, mode)
            d_all, p_all = dist.cpu().numpy().view(np.uint32).reshape(n, V), par.cpu().numpy().reshape(n, V)
            for i, r in enumerate(roots):
                s = gbx.breadth_first_search(dg, r, mode)
                d, _, proc, it = po.bfs(host, r, pull)
                np.testing.assert_array_equal(s.distances, d)
                np.testing.assert_array_equal(d_all[i], d)
                _check_parents(g, r, d, np.asarray(s.parents))
                _check_parents(g, r, d, p_all[i])
                for t in (s, trials[i], bare[i]):
                    assert t.processed_nodes == proc
                    if mode == 2:
                        assert t.iteration == it
                    assert (t.iteration, t.depth, t.edges_traversed) == (s.iteration, s.depth, s.edges_traversed)


def test_many_trials_at_once(gbx, cuda_device):
    """More trials than one launch takes, strided wider than the graph; the gaps stay untouched."""
    import torch

    V, src, dst = GRAPHS["edges_65536"]()
    g = build(gbx, V, src, dst)
    host, pull = host_views(g)
    roots = [int(r) for r in np.random.default_rng(1).integers(0, V, 150)]
    stride = V + 5
    dist = torch.full((len(roots) * stride,), -7, dtype=torch.int32, device=cuda_device)
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        trials = gbx.breadth_first_search_trials(dg, roots, distances=dist, out_stride=stride)
    got = dist.cpu().numpy().reshape(len(roots), stride)
    assert np.all(got[:, V:] == -7)
    for i in range(0, len(roots), 13):
        d, _, proc, it = po.bfs(host, roots[i], pull)
        np.testing.assert_array_equal(got[i, :V].view(np.uint32), d)
        assert (trials[i].processed_nodes, trials[i].iteration) == (proc, it)
