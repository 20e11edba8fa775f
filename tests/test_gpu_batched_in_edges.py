"""Batched PageRank with an in-edge CSR that is not the forward one's transpose: graphs with far more or far fewer
in-edges than out-edges, as when the two were filtered apart. The in-edge words of a graph are as many as its in-edges,
so its neighbours' words and the end of the array stay clear whatever the out-edges are.

Tolerance: every term is positive, so an iteration's sums (trees of at most 8 + 5 levels) and its two operations and
division add at most 16 * 2^-24 of the rank; twelve iterations 1.2e-5."""
import numpy as np
import pytest

import graphblox_gb300 as gg

pytestmark = pytest.mark.gpu

BASE, DAMP = 1.0 - float(np.float32(0.85)), float(np.float32(0.85))


def packed(graphs, lead, seed):
    """graphs: (V, out-edges, in-edges); lead: in-edges before the first graph's, which nobody owns."""
    rng = np.random.default_rng(seed)
    base = np.concatenate([[0], np.cumsum([g[0] for g in graphs])]).astype(np.uint32)

    def csr(k):
        deg, ids = [], []
        for g in graphs:
            deg.append(np.bincount(rng.integers(0, g[0], g[k]), minlength=g[0]))
            ids.append(rng.integers(0, g[0], g[k]))
        return np.concatenate([[0], np.cumsum(np.concatenate(deg))]).astype(np.uint32), np.concatenate(ids).astype(np.uint32)

    (off, dest), (in_off, in_src) = csr(1), csr(2)
    in_off, in_src = in_off + np.uint32(lead), np.concatenate([np.zeros(lead, np.uint32), in_src])
    in_src = np.concatenate([in_src, np.zeros(max(0, len(dest) - len(in_src)), np.uint32)])
    assert in_off[-1] <= len(dest)
    return gg.PackedGraphs(base, off, dest, in_off, in_src)


def reference(p, g, iterations):
    lo, hi = int(p.vertex_base[g]), int(p.vertex_base[g + 1])
    out = np.diff(p.offsets[lo:hi + 1].astype(np.int64)).astype(np.float64)
    io = p.in_offsets[lo:hi + 1].astype(np.int64)
    src, rows = p.in_src[io[0]:io[-1]], np.flatnonzero(np.diff(io))
    r = np.full(hi - lo, BASE)
    for _ in range(iterations):
        c = np.divide(r, out, out=np.zeros(hi - lo), where=out > 0)
        sums = np.zeros(hi - lo)
        if len(rows):
            sums[rows] = np.add.reduceat(c[src], io[rows] - io[0])
        r = BASE + DAMP * sums
    return r / (hi - lo)


BATCHES = {
    "swapped": ([(40, 10, 300), (40, 300, 10)], 0),
    "swapped_back": ([(40, 300, 10), (40, 10, 300)], 0),
    "none_against_many": ([(100, 0, 5000), (33, 6000, 0), (1000, 0, 1000)], 0),
    "in_edges_start_late": ([(50, 400, 700), (50, 900, 300), (7, 100, 0)], 300),
    "wide_words": ([(33_000, 1000, 90_000), (500, 100_000, 2000), (47_000, 30_000, 30_000)], 0),
    "many": ([(30 + i, 257 * (i % 5), 257 * ((4 - i) % 5)) for i in range(400)], 0),
}


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_ranks(gbx, cuda_device, name):
    p = packed(*BATCHES[name], seed=7)
    with gg.GraphBatch(p) as b:
        ranks, _ = b.page_rank(12, 0.0)
        again, _ = b.page_rank(12, 0.0)
    np.testing.assert_array_equal(ranks, again)
    for g in range(p.num_graphs):
        want = reference(p, g, 12)
        got = ranks[int(p.vertex_base[g]):int(p.vertex_base[g + 1])]
        assert np.all(np.abs(got - want) <= 1.2e-5 * want), (name, g)
