"""A captured SpMV works whatever call came to the graph first, and gives the bits that the same call gives uncaptured;
its working memory outlives the call that captured it. Values and sources are small integers, so that every sum is exact
in 32 bits and any order of additions must give it: the checks are for equality."""
import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu


def whole(off, src, x):
    return base.row_sums(x.astype(np.float64)[src], off)


def first_calls(gbx, g, how, x, val, y):
    if how == "one_sweep":
        gbx.spmv(g, x, values=val, y=y)
    elif how == "four_sweeps":
        gbx.spmv(g, x, values=val, y=y, iterations=4)
    else:
        gbx.page_rank(g, 20, 0.0)


@pytest.mark.parametrize("how", ["one_sweep", "four_sweeps", "page_rank"])
@pytest.mark.parametrize("name", ["hubs_between_small", "under_the_limit"])
def test_capture_after(gbx, cuda_device, name, how):
    import torch

    rows, V = base.SHAPES[name]
    off, src = base.csr(rows, V, 8, True)
    rng = np.random.default_rng(2)
    val = torch.ones(len(src), device=cuda_device)
    x = torch.from_numpy(rng.integers(-3, 4, V).astype(np.float32)).to(cuda_device)
    y = torch.zeros(V, device=cuda_device)
    with base.graph(gbx, off, src, V) as g:
        first_calls(gbx, g, how, x, val, y)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        cg = torch.cuda.CUDAGraph()
        with torch.cuda.graph(cg, stream=stream):
            gbx.spmv(g, x, values=val, y=y, iterations=2, stream=torch.cuda.current_stream().cuda_stream)
        spare = [torch.full((1 << 20,), float("nan"), device=cuda_device) for _ in range(8)]  # over freed memory
        for seed in range(2):
            xh = np.random.default_rng(seed).integers(-3, 4, V).astype(np.float32)
            x.copy_(torch.from_numpy(xh))
            y.zero_()
            cg.replay()
            torch.cuda.synchronize()
            captured = y.cpu().numpy()
            np.testing.assert_array_equal(captured, 2 * whole(off, src, xh))
            alone = gbx.spmv(g, x, values=val, y=torch.zeros(V, device=cuda_device), iterations=2)
            np.testing.assert_array_equal(alone.cpu().numpy(), captured)
        del spare


@pytest.mark.parametrize("iterations", [63, 64, 65, 130])
def test_more_sweeps_than_cursors(gbx, cuda_device, iterations):
    rows, V = base.SHAPES["hubs_between_small"]
    off, src = base.csr(rows, V, 9, True)
    x = np.random.default_rng(3).integers(-3, 4, V).astype(np.float32)
    with base.graph(gbx, off, src, V) as g:
        y = gbx.spmv(g, x, default_value=1.0, iterations=iterations)
    np.testing.assert_array_equal(y, iterations * whole(off, src, x))
