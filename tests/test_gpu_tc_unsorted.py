"""Triangle counts ask for sorted rows. A graph whose rows are not is counted on the path that searches rows within their
bounds, never on the one whose tables are sized by sorted rows: the call returns, repeats, and leaves the device and the
sorted graph's count as they should be."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def graph(V, E, seed, descending):
    rng = np.random.default_rng(seed)
    a, b = (rng.random(E) ** 2 * V).astype(np.int64), rng.integers(0, V, E)
    key = np.unique(np.concatenate([a * V + b, b * V + a])[np.concatenate([a != b, a != b])])
    s, d = key // V, key % V
    off = np.searchsorted(s, np.arange(V + 1)).astype(np.uint32)
    if descending:
        d = d[np.lexsort((-d, s))]
    else:  # one row out of order
        r = int(np.argmax(np.diff(off.astype(np.int64))))
        d[off[r]:off[r + 1]] = rng.permutation(d[off[r]:off[r + 1]])
    return V, off, d.astype(np.uint32), (key % V).astype(np.uint32)


@pytest.mark.parametrize("descending", [False, True])
@pytest.mark.parametrize("V,E", [(300, 3000), (40_000, 600_000), (500_000, 3_000_000)])
def test_rows_out_of_order(gbx, cuda_device, V, E, descending):
    V, off, shuffled, ascending = graph(V, E, 3, descending)
    with gbx.DeviceGraph.from_offsets(V, off, shuffled) as g:
        assert gbx.triangle_count(g) == gbx.triangle_count(g)
    with gbx.DeviceGraph.from_offsets(V, off, ascending) as g:
        deg = np.diff(off.astype(np.int64)).astype(np.uint32)
        want = po.triangle_count(po.HostCSR(V, deg, off[:-1].copy(), ascending))
        assert gbx.triangle_count(g) == want
