"""Multi-source BFS where there is memory for the masks of the levels that a sweep has, but not for those that are
allocated ahead of it: from the first step on, and after a first batch of eight levels."""
import numpy as np
import pytest

from memory_pool import limited_pool

pytestmark = pytest.mark.gpu

SOURCES = 256


def symmetric(gbx, V, a, b):
    """The graph with edges a - b."""
    s, d = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.lexsort((d, s))
    s, d = s[order], d[order]
    off = np.searchsorted(s, np.arange(V + 1)).astype(np.uint32)
    return gbx.DeviceGraph.from_offsets(V, off, d.astype(np.uint32))


@pytest.mark.parametrize("limit_mb", [112, 1024])
def test_star(gbx, cuda_device, limit_mb):
    """A hub and 2^19 leaves: four masks of 16 MB and the seen bits; eleven masks when eight levels are enqueued ahead."""
    import torch

    V = 1 << 19
    leaves = np.arange(1, V)
    with symmetric(gbx, V, np.zeros(V - 1, np.int64), leaves) as g:
        d = torch.empty(V, SOURCES, dtype=torch.int32, device=cuda_device)
        sources = np.arange(SOURCES, dtype=np.uint32)
        with limited_pool(limit_mb << 20):
            _, r = gbx.bfs_multisource(g, sources, distances=d)
        want = torch.full((V, SOURCES), 2, dtype=torch.int32, device=cuda_device)
        want[:, 0] = 1
        want[0, :] = 1
        want[torch.arange(SOURCES), torch.arange(SOURCES)] = 0
        assert torch.equal(d, want)
        np.testing.assert_array_equal(r["processed_nodes"], V)
        np.testing.assert_array_equal(r["edges_traversed"], 2 * (V - 1))


@pytest.mark.parametrize("limit_mb", [192, 1024])
def test_path_and_star(gbx, cuda_device, limit_mb):
    """A path of eight vertices and a star at its end: nine levels, so that the first batch of eight steps leaves one. With
    the seen bits ten masks of 16 MB; four more where the second batch allocates ahead."""
    import torch

    n, V = 8, 1 << 19
    path = np.arange(n - 1)
    a = np.concatenate([path, np.full(V - n, n - 1)])
    b = np.concatenate([path + 1, np.arange(n, V)])
    with symmetric(gbx, V, a, b) as g:
        d = torch.empty(V, SOURCES, dtype=torch.int32, device=cuda_device)
        with limited_pool(limit_mb << 20):
            _, r = gbx.bfs_multisource(g, np.zeros(SOURCES, np.uint32), distances=d)
        want = torch.cat([torch.arange(n), torch.full((V - n,), n)]).int().to(cuda_device)
        assert torch.equal(d, want[:, None].expand(V, SOURCES))
        np.testing.assert_array_equal(r["depth"], n)
