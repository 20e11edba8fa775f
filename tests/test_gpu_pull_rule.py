"""The pull engines' dispatch: graphs of fewer than 12M edges get the hot-table layout when their longest row has 3,072
in-edges or more. The shapes and checks are test_gpu_pull_layout's, with the longest row on either side of that line
beside rows of every other kind."""
import numpy as np
import pytest

import test_gpu_pull_layout as base

pytestmark = pytest.mark.gpu

LONG = {
    "row_3071": ([2] * 40_000 + [3071], 70_000),
    "row_3072": ([2] * 40_000 + [3072], 70_000),
    "units_and_long": ([127, 0, 128, 129, 1, 0, 0, 255, 256, 257] * 60 + [3073], 2000),
    "short_and_long": (list(range(0, 40)) * 5000 + [9000], 300_001),
    "ones_and_long": ([3072] + [1] * 200_000, 200_001),
    "all_even": ([6] * 2_000_000, 2_000_000),
}


@pytest.fixture(autouse=True)
def shapes(monkeypatch):
    monkeypatch.setattr(base, "SHAPES", LONG)


@pytest.mark.parametrize("name", sorted(LONG))
@pytest.mark.parametrize("skew", [False, True])
def test_spmv(gbx, cuda_device, name, skew):
    base.test_spmv(gbx, cuda_device, name, skew)


@pytest.mark.parametrize("name", sorted(LONG))
@pytest.mark.parametrize("iterations,epsilon", [(3, 0.0), (21, 0.0), (60, 1e-4)])
def test_pagerank(gbx, cuda_device, name, iterations, epsilon):
    base.test_pagerank(gbx, cuda_device, name, iterations, epsilon)


def test_infinite_and_nan_values(gbx, cuda_device, monkeypatch):
    monkeypatch.setattr(base, "SHAPES", {"under_a_unit": LONG["units_and_long"]})
    base.test_infinite_and_nan_values_stay_in_their_rows(gbx, cuda_device)
