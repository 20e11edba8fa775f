"""Calls on different graphs from several host threads, each on its own stream: launches that need little shared memory
beside launches that need much. A kernel's limit on dynamic shared memory belongs to the process, so a small call must
not lower it under a large one. Values are small whole numbers, sums are exact: equality."""
import threading

import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu


def run_all(jobs):
    failed = []

    def guarded(job):
        try:
            job()
        except Exception as e:  # reported by the test's own thread
            failed.append(e)

    threads = [threading.Thread(target=guarded, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_spmv_and_pagerank(gbx, cuda_device):
    import torch

    def job(rows, V, calls):
        off, src = base.csr(rows, V, 4, True)
        want = base.row_sums(np.ones(len(src)), off)
        stream = torch.cuda.Stream()
        x, val = torch.ones(V, device=cuda_device), torch.ones(len(src), device=cuda_device)
        y = torch.zeros(V, device=cuda_device)
        torch.cuda.synchronize()

        def go():
            with base.graph(gbx, off, src, V) as g:
                ranks = None
                for _ in range(calls):
                    with torch.cuda.stream(stream):
                        y.zero_()
                    gbx.spmv(g, x, values=val, y=y, iterations=3, stream=stream.cuda_stream)
                    r = gbx.page_rank(g, 2, 0.0, stream=stream.cuda_stream).pageRanks
                    ranks = r if ranks is None else ranks
                    np.testing.assert_array_equal(r, ranks)
                stream.synchronize()
                np.testing.assert_array_equal(y.cpu().numpy(), 3 * want)

        return go

    small, large = base.SHAPES["at_the_limit"], base.SHAPES["large"]  # slots for a few and for 20,000 sources
    run_all([job(*small, 1500), job(*large, 400), job(*small, 1500)])


def test_batched_pagerank(gbx, cuda_device):
    rng = np.random.default_rng(1)

    def job(V, E, calls):
        s, d = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)

        def go():
            with gbx.GraphBatch(gbx.pack_graphs([(V, s, d)] * 2)) as b:
                first, _ = b.page_rank(2, 0.0)
                for _ in range(calls):
                    np.testing.assert_array_equal(b.page_rank(2, 0.0)[0], first)

        return go

    run_all([job(100, 1000, 1500), job(46_000, 200_000, 400), job(100, 1000, 1500)])
