"""Triangle count at the lines between its membership tests: pivots above the bitmap range (32,768 ids) whose lists
N+(v) hold 511 to 2,050 ids, 127 to 130 of them above the range, with few and with many upper neighbours, and pivots
within the range with long lists. The count equals the oracle's, the first time and the later times a graph is
counted."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_gpu_parity import host_views

pytestmark = pytest.mark.gpu

RANGE = 32_768


def graph(gbx, low, high, uppers, first_pivot):
    """Six pivots, each with `low` neighbours below the range and `high` above it (both below the pivot), and `uppers`
    common upper neighbours that share part of the pivots' lists; a sparse random rest."""
    rng = np.random.default_rng(low * 7 + high * 3 + uppers)
    V = 37_003
    pairs = [rng.integers(0, V, (30_000, 2))]
    for i in range(6):
        v = first_pivot + 5 * i
        ids = np.concatenate([rng.choice(RANGE - 2000, low, replace=False),
                              RANGE + rng.choice(1000, high, replace=False)])
        pairs.append(np.stack([np.full(len(ids), v), ids], 1))
        for u in range(35_000, 35_000 + uppers):
            shared = rng.choice(ids, 9, replace=False)
            pairs.append(np.stack([np.full(10, u), np.append(shared, v)], 1))
    e = np.concatenate(pairs)
    e = e[e[:, 0] != e[:, 1]]
    e = np.unique(np.concatenate([e, e[:, ::-1]]), axis=0)
    el = gbx.EdgeList(V, e[:, 0].astype(np.uint32), e[:, 1].astype(np.uint32))
    return gbx.graph_csr_preprocessing(el, sort=1, dedup=False, directed=False, keep_weights=False)


@pytest.mark.parametrize("low,high,first_pivot", [
    (382, 129, 34_000), (383, 129, 34_000), (383, 130, 34_000), (600, 127, 34_000), (600, 128, 34_000),
    (600, 129, 34_000), (1919, 128, 34_000), (1920, 128, 34_000), (1921, 128, 34_000), (0, 128, 34_000),
    (0, 129, 34_000), (2040, 0, 32_700), (2049, 0, 32_740), (3000, 0, 33_900)])
@pytest.mark.parametrize("uppers", [3, 300])
def test_triangle_lists(gbx, cuda_device, low, high, first_pivot, uppers):
    g = graph(gbx, low, high, uppers, first_pivot)
    host, _ = host_views(g)
    want = po.triangle_count(host)
    with gbx.DeviceGraph.from_graph_csr(g) as dg:
        for _ in range(3):
            assert gbx.triangle_count(dg) == want
