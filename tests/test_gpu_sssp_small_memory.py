"""SSSP on small graphs works in the graph's scratch memory: a second call allocates nothing and passes where the device
is full, into device and host memory."""
import numpy as np
import pytest

from memory_pool import limited_pool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 33, 1000, 24_576])
def test_second_call_needs_no_memory(gbx, cuda_device, V):
    import torch

    off = np.minimum(np.arange(V + 1), V - 1).astype(np.uint32)  # a path
    with gbx.DeviceGraph.from_offsets(V, off, np.arange(1, V, dtype=np.uint32), np.full(V - 1, 3, np.float32)) as g:
        first = gbx.sssp(g, 0).distances
        d = torch.empty(V, dtype=torch.int32, device=cuda_device)
        with limited_pool(4 << 20, full=True):
            host = gbx.sssp(g, 0).distances
            gbx.sssp(g, 0, distances=d)
    want = 3 * np.arange(V)
    for got in (first, host, d.cpu().numpy()):
        np.testing.assert_array_equal(got, want)
