"""Rows whose fixed-point value is past binary32 (w (x - o) overflows) on L1 batches
past 8 queries: wherever such a row lies, the answers are the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu

ROWS = 5000


def _check(oracle_module, rows, queries, weights, expected_row):
    index = uha.CudaDenseL1ScanIndex(rows, weights)
    ws = index.make_query_workspace(queries.shape[0])
    dist = np.zeros(queries.shape[0])
    got = index.query_batch(queries, queries.shape[0], None, ws, distances=dist)
    if weights is None:
        expected, edist = oracle_module.exact("l1", rows, queries)
    else:
        expected, edist = oracle_module.weighted_l1(rows, weights, queries)
    assert (expected == expected_row).all()
    assert np.array_equal(got, expected)
    np.testing.assert_allclose(dist, edist, rtol=1e-5)


@pytest.mark.parametrize("at", [20, 63, 64, 127, 128, ROWS - 1])
@pytest.mark.parametrize("columns", [6, 100])
def test_column_range_past_binary32(oracle_module, at, columns):
    # row `at` is 5e38 and 3.5e38 above the smallest values of its columns: past
    # binary32, so its second value takes the last of the 65,536 levels
    rng = np.random.default_rng(at)
    rows = np.zeros((ROWS, columns), np.float32)
    rows[:, :2] = rng.uniform(-2e38, -1e38, (ROWS, 2))
    rows[0, :2] = -2e38
    rows[10] = 0
    rows[at, :2] = 3e38, 1.5e38
    queries = np.zeros((16, columns), np.float32)
    queries[:, :2] = rng.uniform(1.29e38, 1.31e38, (16, 2))
    _check(oracle_module, rows, queries, None, at)


@pytest.mark.parametrize("at", [20, 64, ROWS - 1])
def test_weighted_range_past_binary32(oracle_module, at):
    rng = np.random.default_rng(at)
    rows = np.zeros((ROWS, 6), np.float32)
    rows[:, :2] = rng.uniform(-1e38, -0.6e38, (ROWS, 2))
    rows[0, :2] = -1e38
    rows[300, :2] = 1e38, -1e38         # the step: 6e38 / 65,535
    rows[10, :2] = -0.5e38, 0.6e38
    rows[at, :2] = 0, 1e38              # 2 * 2e38 above the smallest value
    weights = np.array([3, 2, 1, 1, 1, 1], np.float32)
    queries = np.zeros((16, 6), np.float32)
    queries[:, 0] = rng.uniform(-1e36, 1e36, 16)
    queries[:, 1] = 0.6e38
    _check(oracle_module, rows, queries, weights, at)


@pytest.mark.parametrize("columns", [32000, 32001])
def test_both_epilogues(oracle_module, columns):
    rng = np.random.default_rng(columns)
    rows = np.zeros((300, columns), np.float32)
    rows[:, :2] = rng.uniform(-2e38, -1e38, (300, 2))
    rows[0, :2] = -2e38
    rows[10] = 0
    rows[200, :2] = 3e38, 1.5e38
    queries = np.zeros((40, columns), np.float32)
    queries[:, :2] = 1.3e38
    _check(oracle_module, rows, queries, None, 200)


@pytest.mark.parametrize("count", [(1 << 24) - 256, (1 << 24) - 200, 1 << 24, (1 << 24) + 1])
def test_most_rows(count):
    # around the most rows the fixed-point scan takes; past 2^24 the binary32 scan
    torch = pytest.importorskip("torch")
    torch.manual_seed(count)
    rows = torch.rand(count, 4, device="cuda")
    at = torch.linspace(0, count - 1, 12, dtype=torch.float64).long().cuda()
    rows[at] += 100 * torch.arange(1, 13, device="cuda")[:, None]
    queries = (rows[at] + 0.25).contiguous()
    torch.cuda.synchronize()
    index = uha.CudaExactL1Index(rows)
    ws = index.make_query_workspace(12)
    dist = np.zeros(12)
    out = np.zeros(12, np.uint64)
    index.query_device_batch(queries.data_ptr(), 12, out, ws, distances=dist)
    assert np.array_equal(out, at.cpu().numpy().astype(np.uint64))
    # 0.25 in each of four columns, up to the rounding of the query
    np.testing.assert_allclose(dist, 1.0, rtol=4 * 1200 * 2.0 ** -24)
