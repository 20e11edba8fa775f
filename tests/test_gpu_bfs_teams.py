"""BFS trials taken by teams of CTAs: fewer and more trials than teams, team counts on both sides of the lines in
edges, rows that are hubs, a long chain (many steps per trial), one output or none, gaps between outputs, roots
without out-edges. Levels, processed_nodes and iteration equal the oracle's; parents form a BFS tree; the counts
equal one traversal's."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_bfs_small import build, random_edges
from test_gpu_bfs_trials import _check_parents
from test_gpu_parity import host_views

pytestmark = pytest.mark.gpu


def chain_with_hubs(V):
    """A chain over all vertices; every 3,000th vertex also reaches 2,500 others."""
    hubs = np.arange(0, V - 1, 3000)
    src = np.concatenate([np.arange(V - 1), np.repeat(hubs, 2500)])
    dst = np.concatenate([np.arange(1, V), (np.arange(len(hubs) * 2500) * 11 + 5) % (V // 8)])
    return src, dst


GRAPHS = {
    "over_the_small_limit": lambda: (30_001, *random_edges(30_001, 3 * 65_536 + 1, 1)),
    "64_teams": lambda: (50_000, *random_edges(50_000, 1_250_000, 2)),
    "32_teams": lambda: (50_000, *random_edges(50_000, 1_250_001, 3)),
    "16_teams_by_vertices": lambda: (700_003, *random_edges(700_003, 900_000, 4)),
    "chain_with_hubs": lambda: (70_000, *chain_with_hubs(70_000)),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("n", [2, 3, 9, 70])
def test_trials_by_teams(gbx, cuda_device, name, n):
    import torch

    V, src, dst = GRAPHS[name]()
    g = build(gbx, V, src, dst)
    host, pull = host_views(g)
    rng = np.random.default_rng(n)
    roots = [int(r) for r in rng.integers(V - 400 if name == "chain_with_hubs" else 0, V, n)]
    roots[0] = int(np.argmax(g.out_degree))
    roots[-1] = int(np.argmin(g.out_degree))
    stride = V + 3
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        for mode in (2, 0, 1) if n == 3 else (2,):
            dist = torch.full((n * stride,), -7, dtype=torch.int32, device=cuda_device)
            par = torch.full((n * stride,), -7, dtype=torch.int32, device=cuda_device)
            trials = gbx.breadth_first_search_trials(dg, roots, mode, distances=dist, parents=par, out_stride=stride)
            only = torch.full((n * stride,), -7, dtype=torch.int32, device=cuda_device)
            levels_only = gbx.breadth_first_search_trials(dg, roots, mode, distances=only, out_stride=stride)
            bare = gbx.breadth_first_search_trials(dg, roots, mode)
            assert torch.equal(dist, only)
            last = torch.full((V,), -7, dtype=torch.int32, device=cuda_device)
            gbx.breadth_first_search_trials(dg, roots[::-1], mode, distances=last)
            assert torch.equal(last, dist[:V])
            d_all, p_all = dist.cpu().numpy().reshape(n, stride), par.cpu().numpy().reshape(n, stride)
            assert np.all(d_all[:, V:] == -7) and np.all(p_all[:, V:] == -7)
            for i in sorted({0, 1, n // 2, n - 1}):
                s = gbx.breadth_first_search(dg, roots[i], mode)
                d, _, proc, it = po.bfs(host, roots[i], pull)
                np.testing.assert_array_equal(d_all[i, :V].view(np.uint32), d)
                _check_parents(g, roots[i], d, p_all[i, :V])
                for t in (trials[i], levels_only[i], bare[i]):
                    assert t.processed_nodes == proc
                    if mode == 2:
                        assert t.iteration == it
                    assert (t.iteration, t.depth, t.edges_traversed) == (s.iteration, s.depth, s.edges_traversed)
