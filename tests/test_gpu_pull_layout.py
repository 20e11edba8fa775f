"""PageRank and SpMV on the hot-table pull engine against 64-bit sums, at the places where its layout changes:
rows around one group (128) and one unit of edges (up to 3,072, and a quarter of that at the end), rows of many units, rows that start or end on a unit's first edge,
graphs around the smallest that gets a layout (65,536 edges), sources beyond the slots, empty rows, and value arrays off a
16-byte boundary. SpMV uses the row engine for a graph's first three sweeps and this engine after them; both
must agree within the rounding of 32-bit sums.

Tolerance: a sum of n products in 32 bits, added as trees of at most 8 levels with a compensated running sum,
is within (8 + 3) * 2^-24 of the sum of the products' sizes: 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-6


def csr(rows, V, seed, skew):
    """Offsets and sources of the given row lengths; skewed sources make some vertices hot."""
    rng = np.random.default_rng(seed)
    deg = np.zeros(V, np.int64)
    deg[:len(rows)] = rows
    off = np.zeros(V + 1, np.int64)
    off[1:] = np.cumsum(deg)
    E = int(off[-1])
    src = (rng.random(E) ** (4 if skew else 1) * V).astype(np.int64)
    return off.astype(np.uint32), src.astype(np.uint32)


def graph(gbx, off, src, V):
    """A graph whose pull CSR is (off, src) and whose forward CSR is its transpose."""
    dst = np.repeat(np.arange(V, dtype=np.uint32), np.diff(off.astype(np.int64)))
    order = np.argsort(src, kind="stable")
    foff = np.zeros(V + 1, np.uint32)
    foff[1:] = np.cumsum(np.bincount(src, minlength=V))
    return gbx.DeviceGraph.from_offsets(V, foff, dst[order].copy(), None, off, src, None)


def row_sums(x, off):
    o = off.astype(np.int64)
    sums = np.zeros(len(o) - 1)
    rows = np.flatnonzero(o[1:] > o[:-1])
    sums[rows] = np.add.reduceat(x, o[rows])
    return sums


SHAPES = {
    "under_the_limit": ([65_535], 5),
    "at_the_limit": ([65_536], 5),
    "under_a_unit": ([127, 0, 128, 129, 1, 0, 0, 255, 256, 257] * 60, 2000),
    "around_a_span": ([3071, 3072, 3073, 1, 6143, 6144, 6145, 0, 3, 767, 768, 769] * 20, 70_000),
    "one_hub": ([300_000, 1, 2, 3], 100_000),
    "hubs_between_small": (([5] * 100 + [50_000] + [0] * 50 + [1] * 31) * 8, 90_000),
    "many_short": (list(range(0, 40)) * 5000, 300_000),
    "only_ones": ([1] * 200_000, 200_001),
    "large": ([30] * 520_000 + [200_000], 600_003),
}


@pytest.mark.parametrize("name", sorted(SHAPES))
@pytest.mark.parametrize("skew", [False, True])
def test_spmv(gbx, cuda_device, name, skew):
    import torch

    rows, V = SHAPES[name]
    off, src = csr(rows, V, 3, skew)
    rng = np.random.default_rng(5)
    E = len(src)
    val = (1.0 - rng.random(E)).astype(np.float32)
    x = rng.uniform(-1, 1, V).astype(np.float32)
    terms = val.astype(np.float64) * x.astype(np.float64)[src]
    want, size = row_sums(terms, off), row_sums(np.abs(terms), off)
    ones, ones_size = row_sums(x.astype(np.float64)[src], off), row_sums(np.abs(x.astype(np.float64)[src]), off)
    with graph(gbx, off, src, V) as g:
        xd = torch.from_numpy(x).to(cuda_device)
        for offset in (0, 1, 2, 0, 3, 0):  # three sweeps of one engine, three of the other
            vd = torch.zeros(E + offset, device=cuda_device)
            vd[offset:] = torch.from_numpy(val)
            y = gbx.spmv(g, xd, values=vd[offset:], y=torch.zeros(V, device=cuda_device)).cpu().numpy()
            assert np.all(np.abs(y - want) <= TOL * size), np.abs(y - want).max()
            again = gbx.spmv(g, xd, values=vd[offset:], y=torch.zeros(V, device=cuda_device)).cpu().numpy()
            assert np.all(np.abs(again - want) <= TOL * size)
        two = [gbx.spmv(g, xd, values=vd, y=torch.zeros(V, device=cuda_device)).cpu().numpy() for _ in range(2)]
        np.testing.assert_array_equal(two[0], two[1])  # a fixed order of additions
        y = gbx.spmv(g, x, default_value=1.0, iterations=2)
        assert np.all(np.abs(y - 2 * ones) <= 2 * TOL * ones_size)


@pytest.mark.parametrize("name", sorted(SHAPES))
@pytest.mark.parametrize("iterations,epsilon", [(1, 0.0), (2, 0.0), (4, 0.0), (21, 0.0), (60, 1e-4)])
def test_pagerank(gbx, cuda_device, name, iterations, epsilon):
    rows, V = SHAPES[name]
    off, src = csr(rows, V, 4, True)
    out = np.bincount(src, minlength=V).astype(np.float64)
    base, damp = 1.0 - float(np.float32(0.85)), float(np.float32(0.85))
    r, count = np.full(V, base), iterations
    for it in range(iterations):
        c = np.divide(r, out, out=np.zeros(V), where=out > 0)
        nxt = base + damp * row_sums(c[src], off)
        moved = np.abs(nxt - r).max()
        r = nxt
        if epsilon and moved < epsilon:
            count = it
            break
    with graph(gbx, off, src, V) as g:
        for _ in range(2):
            st = gbx.page_rank(g, iterations, epsilon)
            # a vertex within rounding of epsilon may end the run an iteration earlier or later
            assert abs(st.iterations - count) <= (1 if epsilon else 0)
            tol = 2 * epsilon / V if epsilon else 0.0
            assert np.all(np.abs(st.pageRanks * 1.0 - r / V) <= tol + 2e-6 * np.abs(r / V))


def test_infinite_and_nan_values_stay_in_their_rows(gbx, cuda_device):
    import torch

    rows, V = SHAPES["under_a_unit"]
    off, src = csr(rows, V, 6, False)
    val = np.ones(len(src), np.float32)
    o = off.astype(np.int64)
    val[o[2] + 5] = np.inf
    val[o[4]] = np.nan
    x = np.full(V, 0.5, np.float32)
    with graph(gbx, off, src, V) as g:
        for _ in range(5):
            y = gbx.spmv(g, torch.from_numpy(x).to(cuda_device), values=torch.from_numpy(val).to(cuda_device),
                         y=torch.zeros(V, device=cuda_device)).cpu().numpy()
            bad = ~np.isfinite(y)
            assert set(np.flatnonzero(bad)) == {2, 4}
            np.testing.assert_array_equal(y[~bad], 0.5 * np.diff(o)[~bad])


def test_spmv_under_stream_capture(gbx, cuda_device):
    """A captured call keeps to the row engine and replays on new inputs."""
    import torch

    rows, V = SHAPES["hubs_between_small"]
    off, src = csr(rows, V, 8, True)
    val = torch.ones(len(src), device=cuda_device)
    x = torch.rand(V, device=cuda_device)
    y = torch.zeros(V, device=cuda_device)
    with graph(gbx, off, src, V) as g:
        gbx.spmv(g, x, values=val, y=y)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        cg = torch.cuda.CUDAGraph()
        with torch.cuda.graph(cg, stream=stream):
            for _ in range(3):
                gbx.spmv(g, x, values=val, y=y, stream=torch.cuda.current_stream().cuda_stream)
        y.zero_()
        x.fill_(0.25)
        cg.replay()
        torch.cuda.synchronize()
        want = 0.75 * np.diff(off.astype(np.int64))
        np.testing.assert_allclose(y.cpu().numpy(), want, rtol=TOL)
