"""SpMV without values on the edge-cut engine: a default value that is infinite or NaN reaches the rows with edges and
no others, and no edge of a neighbouring unit (whose words a group of 128 holds beside its own) counts."""
import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.0])
def test_default_value(gbx, cuda_device, value):
    rows = [127, 0, 128, 129, 1, 0, 255, 256, 257, 3, 2] * 60 + [3073, 6145, 5]
    V = 2000
    off, src = base.csr(rows, V, 6, False)
    n = np.diff(off.astype(np.int64))
    with base.graph(gbx, off, src, V) as g:
        y = gbx.spmv(g, np.ones(V, np.float32), default_value=value)
    np.testing.assert_array_equal(y, np.where(n > 0, value * np.maximum(n, 1), 0).astype(np.float32))
