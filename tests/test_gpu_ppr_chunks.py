"""Personalised PageRank at the lengths where its rows are cut: 64 edges in graphs of up to 1,000,000, 128 above, rows of
one less, as many and one more, many pieces, and edge counts on either side of the line.

Tolerances as in test_gpu_ppr: ranks against FP64 run for the same sweeps, relative L1 <= 1e-6 per column; the size-
independent identities L = <dL/dT, T> within 1e-5 of sum |dL/dT T| and, per vertex, sum over its edges of w dL/dw = 0
within 1e-4 of sum |w dL/dw| plus 1e-6 of the largest such sum."""
import numpy as np
import pytest

from graphblox_gb300 import graph as gg
from oracle import ppr_oracle as pp
from test_gpu_ppr import D, TOL, _csr, _device, _rel_l1_cols

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 63, 64, 65, 127, 128, 129, 191, 192, 193, 40, 7]


def rows(V, E, seed):
    """V rows whose lengths run through LENGTHS, then one row that brings the edges to E; some vertices are hit often."""
    rng = np.random.default_rng(seed)
    n = np.resize(LENGTHS, V - 1)
    n = np.append(n, E - n.sum())
    assert n[-1] >= 0
    src = np.repeat(np.arange(V), n)
    return _csr(V, src, (rng.random(E) ** 2.5 * V).astype(np.int64))


@pytest.mark.parametrize("V,E", [(300, 30_000), (10_000, 1_000_000), (10_000, 1_000_001)])
@pytest.mark.parametrize("K", [32, 128])
def test_ppr_chunks(gbx, cuda_device, V, E, K):
    off, dst = rows(V, E, 1)
    rng = np.random.default_rng(2)
    w = rng.lognormal(size=E).astype(np.float32)
    T = pp.seeds_teleport(V, K, 32, rng)
    W = rng.standard_normal((V, K)).astype(np.float32)
    with _device(V, off, dst) as dg:
        st = gg.ppr_forward(dg, w, T, D, TOL)
        adj = gg.ppr_adjoint(dg, w, st.ranks, W, D, TOL)
    R64, _, _ = pp.forward_iter(off, dst, w, T, D, iterations=st.iterations)
    assert _rel_l1_cols(st.ranks.astype(np.float64), R64) <= 1e-6
    terms = adj.grad_teleport.astype(np.float64) * T
    loss = float((W.astype(np.float64) * R64).sum())
    assert abs(terms.sum() - loss) <= 1e-5 * np.abs(terms).sum()
    per_edge = w.astype(np.float64) * adj.grad_weights
    src = np.repeat(np.arange(V), np.diff(off.astype(np.int64)))
    total, size = np.bincount(src, per_edge, V), np.bincount(src, np.abs(per_edge), V)
    assert np.all(np.abs(total) <= 1e-4 * size + 1e-6 * size.max())
