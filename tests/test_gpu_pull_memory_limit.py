"""SpMV and PageRank where memory is short: a graph that has its layout is swept without any allocation, and one whose
layout finds no room is swept by rows. Values are small whole numbers and sums exact: equality."""
import numpy as np
import pytest

import test_gpu_pull_layout as base
from memory_pool import limited_pool

pytestmark = pytest.mark.gpu


def inputs(gbx, device, name):
    import torch

    rows, V = base.SHAPES[name]
    off, src = base.csr(rows, V, 4, True)
    x = np.random.default_rng(3).integers(-3, 4, V).astype(np.float32)
    want = base.row_sums(x.astype(np.float64)[src], off)
    return (base.graph(gbx, off, src, V), V, torch.from_numpy(x).to(device), torch.ones(len(src), device=device),
            torch.zeros(V, device=device), want)


def test_no_memory_once_the_layout_is_there(gbx, cuda_device):
    import torch

    g, V, x, val, y, want = inputs(gbx, cuda_device, "hubs_between_small")
    with g:
        gbx.spmv(g, x, values=val, y=y)
        ranks, again = torch.empty(V, device=cuda_device), torch.empty(V, device=cuda_device)
        with limited_pool(4 << 20, full=True):
            gbx.spmv(g, x, values=val, y=y.zero_(), iterations=70)
            gbx.page_rank(g, 7, 0.0, ranks=ranks)
        np.testing.assert_array_equal(y.cpu().numpy(), 70 * want)
        gbx.page_rank(g, 7, 0.0, ranks=again)
        assert torch.equal(ranks, again)


def test_no_room_for_the_layout(gbx, cuda_device):
    g, V, x, val, y, want = inputs(gbx, cuda_device, "large")  # 63 MB of words
    with g:
        with limited_pool(32 << 20):
            for _ in range(3):
                gbx.spmv(g, x, values=val, y=y.zero_())
                np.testing.assert_array_equal(y.cpu().numpy(), want)
        gbx.spmv(g, x, values=val, y=y.zero_())
    np.testing.assert_array_equal(y.cpu().numpy(), want)
