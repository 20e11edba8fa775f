"""Equal SpMV and PageRank calls give equal bits, whatever was called on the graph before: which engine sweeps a graph
depends on the graph alone. The engine is read off the launch count of a call: a sweep on the edge-cut engine is
preceded by the gather of the slots' values. Shapes on both sides of the rule, and one of 62M edges, whose units end in
a tail of shorter ones with a cut row among them.

Tolerance of the large shape: small integers as values, every sum exact in 32 bits: equality."""
import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu

LAYOUT = {
    "at_the_limit": base.SHAPES["at_the_limit"],
    "hubs_between_small": base.SHAPES["hubs_between_small"],
    "row_3072": ([2] * 40_000 + [3072], 70_000),
    "large": base.SHAPES["large"],
}
ROWS = {
    "under_the_limit": base.SHAPES["under_the_limit"],
    "row_3071": ([2] * 40_000 + [3071], 70_000),
    "many_short": base.SHAPES["many_short"],
}


def launches(gbx, g, x, val, y):
    before = gbx.load().gbx_kernel_launches()
    gbx.spmv(g, x, values=val, y=y)
    return gbx.load().gbx_kernel_launches() - before


@pytest.mark.parametrize("name", sorted(LAYOUT) + sorted(ROWS))
def test_equal_calls_equal_bits(gbx, cuda_device, name):
    import torch

    rows, V = {**LAYOUT, **ROWS}[name]
    off, src = base.csr(rows, V, 3, True)
    rng = np.random.default_rng(5)
    val = torch.from_numpy((1.0 - rng.random(len(src))).astype(np.float32)).to(cuda_device)
    x = torch.from_numpy(rng.uniform(-1, 1, V).astype(np.float32)).to(cuda_device)
    zeros = lambda: torch.zeros(V, device=cuda_device)  # noqa: E731
    with base.graph(gbx, off, src, V) as g, base.graph(gbx, off, src, V) as h:
        y = [gbx.spmv(g, x, values=val, y=zeros()).cpu().numpy() for _ in range(6)]
        y += [gbx.spmv(h, x, values=val, y=zeros(), iterations=1).cpu().numpy()]
        for other in y[1:]:
            np.testing.assert_array_equal(other, y[0])
        # one launch a sweep by rows; by edges one more for the slots' values
        assert launches(gbx, g, x, val, zeros()) == (2 if name in LAYOUT else 1)
    for iterations in (1, 3, 9):
        with base.graph(gbx, off, src, V) as g:
            first = gbx.page_rank(g, iterations, 0.0).pageRanks
            gbx.page_rank(g, 20, 0.0)
            np.testing.assert_array_equal(gbx.page_rank(g, iterations, 0.0).pageRanks, first)


def test_tail_units(gbx, cuda_device):
    import torch

    V = 3_000_000
    deg = torch.full((V,), 22, dtype=torch.int64, device=cuda_device)
    deg[::7] = 0
    deg[1::1000] = 900
    deg[-200_000] = 3_500_000
    deg[-50_000] = 4_000
    off = torch.zeros(V + 1, dtype=torch.int64, device=cuda_device)
    torch.cumsum(deg, 0, out=off[1:])
    E = int(off[-1])
    assert 60_000_000 < E < 64_000_000
    gen = torch.Generator(device=cuda_device).manual_seed(4)
    src = (torch.rand(E, device=cuda_device, generator=gen) ** 4 * V).long().clamp_(max=V - 1)
    x = torch.randint(-1, 2, (V,), device=cuda_device, generator=gen).float()
    want = torch.segment_reduce(x.double()[src], "sum", offsets=off, initial=0.0)
    row = torch.repeat_interleave(torch.arange(V, device=cuda_device), deg)
    order = torch.argsort(src, stable=True)
    foff = torch.zeros(V + 1, dtype=torch.int64, device=cuda_device)
    torch.cumsum(torch.bincount(src, minlength=V), 0, out=foff[1:])
    with gbx.DeviceGraph.from_offsets(V, foff.int(), row[order].int(), None, off.int(), src.int(), None) as g:
        for _ in range(2):
            y = gbx.spmv(g, x, values=torch.ones(E, device=cuda_device), y=torch.zeros(V, device=cuda_device))
            assert torch.equal(y.double(), want)
