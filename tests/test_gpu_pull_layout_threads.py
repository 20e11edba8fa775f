"""The first sweep of one graph does not wait for the first sweep of another: building a graph's layout waits for its own
stream only. A second of work is queued on the first graph's stream; the second graph, from another thread and stream,
is swept to the end meanwhile."""
import threading

import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu


def test_another_graph_does_not_wait(gbx, cuda_device):
    import torch

    rows, V = base.SHAPES["hubs_between_small"]
    off, src = base.csr(rows, V, 4, True)
    want = base.row_sums(np.ones(len(src)), off)
    x, val = torch.ones(V, device=cuda_device), torch.ones(len(src), device=cuda_device)
    out = [torch.zeros(V, device=cuda_device) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    started, late = threading.Event(), []
    with base.graph(gbx, off, src, V) as warm, base.graph(gbx, off, src, V) as g, base.graph(gbx, off, src, V) as h:
        gbx.spmv(warm, x, values=val, y=torch.zeros(V, device=cuda_device))  # kernels loaded, memory in the pool
        torch.cuda.synchronize()

        def first():
            with torch.cuda.stream(streams[0]):
                torch.cuda._sleep(2_000_000_000)
            started.set()
            gbx.spmv(g, x, values=val, y=out[0], stream=streams[0].cuda_stream)

        t = threading.Thread(target=first)
        t.start()
        started.wait()
        for _ in range(3):
            gbx.spmv(h, x, values=val, y=out[1], stream=streams[1].cuda_stream)
        streams[1].synchronize()
        late.append(streams[0].query())
        t.join()
        torch.cuda.synchronize()
    assert late == [False]  # the first stream's second of work was still under way
    np.testing.assert_array_equal(out[0].cpu().numpy(), want)
    np.testing.assert_array_equal(out[1].cpu().numpy(), 3 * want)
