"""The binary32 column filter of the probability build: the binary64 maxima of
the direct backend equal the host build's (the reference CPU's operations) bit
for bit on both pair tilings, at ragged sizes, and where the filter has to step
aside (columns of near-equal contributions, constant columns, values whose
squares or weights leave binary32)."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu

GPU_FN = {"l2": uha.compute_l2_importance_probabilities_gpu,
          "l1": uha.compute_l1_importance_probabilities_gpu}


def _equal(metric, rows):
    got = GPU_FN[metric](rows).probabilities
    want = uha.compute_importance_probabilities_host(metric, rows)
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("metric", ["l2", "l1"])
@pytest.mark.parametrize("rows, d", [(2, 1), (8, 31), (9, 33), (31, 7), (33, 257), (65, 513),
                                     (256, 37), (300, 129), (1536, 37), (1601, 66)])
def test_sizes_around_the_tiles(metric, rows, d):
    rng = np.random.default_rng([rows, d])
    m = rng.normal(size=(rows, d)).astype(np.float32)
    m[:, d // 2] = 1.5 if d > 1 else m[:, 0]  # a constant column
    _equal(metric, m)


@pytest.mark.parametrize("metric", ["l2", "l1"])
def test_near_equal_contributions(metric):
    # two values a column, so thousands of pairs lie within a few ulps of the
    # largest contribution and the binary64 roundings decide
    rng = np.random.default_rng(3)
    m = rng.integers(0, 2, size=(90, 400)).astype(np.float32)
    m += rng.integers(0, 3, size=m.shape).astype(np.float32) * np.float32(2.0 ** -22)
    _equal(metric, m)


@pytest.mark.parametrize("metric", ["l2", "l1"])
@pytest.mark.parametrize("scale", [1e-38, 1e-30, 1e-16, 1e16, 1e30, 1e38])
def test_values_outside_the_filter_range(metric, scale):
    rng = np.random.default_rng(4)
    m = (rng.uniform(-1, 1, size=(40, 130)) * scale).astype(np.float32)
    _equal(metric, m)
    # ordinary columns beside tiny ones, whose filter products underflow
    m[:, ::2] = rng.normal(size=(40, 65)).astype(np.float32)
    _equal(metric, m)
