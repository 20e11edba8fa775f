"""The BFS step trace tells a step that waits for one warp from one that keeps all busy: a bottom-up step in which a
single row of 400,000 in-edges is scanned to its end by one warp, in one CTA of 24 warps, while every other warp has next
to nothing to do. The mean over the grid's thousands of warps is then far below a thousandth of the longest; if a warp's
time held its wait for the rest of its CTA, the mean would be over a two-hundredth."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu


def traverse():
    import graphblox_gb300 as gbx

    V, long_row = 70_000, 400_000
    rng = np.random.default_rng(0)
    deg = np.zeros(V, np.int64)
    deg[1], deg[5] = 1, long_row
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    src = np.concatenate([[0], rng.integers(100, V, long_row)]).astype(np.uint32)
    with base.graph(gbx, off, src, V) as g:
        for _ in range(3):
            st = gbx.breadth_first_search(g, 0, 0)
    assert st.processed_nodes == 2


def test_busy_time_is_the_warps_own(gbx, cuda_device):
    env = dict(os.environ, GBX_TRACE="1")
    code = "import sys; sys.path[:0] = %r; import test_gpu_bfs_trace as t; t.traverse()" % [
        os.path.dirname(os.path.abspath(__file__)), os.path.dirname(os.path.dirname(os.path.abspath(__file__)))]
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    steps = re.findall(r"\| BU +\| *\d+ *\| *[\d.]+ *\| *([\d.]+) *\| *([\d.]+) *\|", r.stderr)
    assert len(steps) == 6, r.stderr
    for longest, mean in steps[2:]:  # the first traversal's come with cold caches
        assert float(longest) > 200 and float(mean) < float(longest) / 1000, steps
