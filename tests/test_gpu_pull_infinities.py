"""SpMV on the edge-cut engine with infinities: a row holds what plain 32-bit addition gives -- the infinity, or NaN
where infinities of both signs or a NaN meet -- whatever its length: within a group of 128 edges, over several, cut
into units. The other rows are whole numbers below 2^24 and exact."""
import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu

LENGTHS = [5, 100, 129, 300, 700, 3000, 5000, 70_000, 3, 40, 300_000]


@pytest.mark.parametrize("at", ["first", "middle", "last"])
def test_infinite_values(gbx, cuda_device, at):
    import torch

    # every length four times: finite, +inf, -inf, both signs (NaN)
    rows = [n for n in LENGTHS for _ in range(4)] + [1] * 300
    V = len(rows) + 50
    off, src = base.csr(rows, V, 6, False)
    o = off.astype(np.int64)
    val = np.ones(len(src), np.float32)
    x = np.ones(V, np.float32)
    want = np.diff(o).astype(np.float64)
    for r in range(4 * len(LENGTHS)):
        b, e = o[r], o[r + 1]
        i = {"first": b, "middle": (b + e) // 2, "last": e - 1}[at]
        if r % 4 == 1:
            val[i], want[r] = np.inf, np.inf
        elif r % 4 == 2:
            val[i], want[r] = -np.inf, -np.inf
        elif r % 4 == 3:
            val[i], val[b + (i - b + 1) % (e - b)], want[r] = np.inf, -np.inf, np.nan
    with base.graph(gbx, off, src, V) as g:
        y = gbx.spmv(g, torch.from_numpy(x).to(cuda_device), values=torch.from_numpy(val).to(cuda_device),
                     y=torch.zeros(V, device=cuda_device)).cpu().numpy()
    np.testing.assert_array_equal(y, want)


def test_overflow(gbx, cuda_device):
    """Sums past the largest 32-bit number are infinite, as in plain addition."""
    rows = [n for n in LENGTHS if n > 3] + [1] * 300
    V = len(rows) + 50
    off, src = base.csr(rows, V, 6, False)
    y = None
    with base.graph(gbx, off, src, V) as g:
        y = gbx.spmv(g, np.ones(V, np.float32), values=np.full(len(src), 2e38, np.float32))
    n = np.diff(off.astype(np.int64))
    np.testing.assert_array_equal(y, np.where(n > 1, np.inf, np.where(n == 1, np.float32(2e38), 0)).astype(np.float32))
