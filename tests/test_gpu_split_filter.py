"""The filter form of the certified split scan (8,192 rows and more, at most 512
columns: estimates stay in the tensor cores' accumulators, rows below a sampled
threshold are listed in the epilogue): every tile width (64, 128 and 256 queries)
and 1 to 8 stages in one accumulator, ragged last row tiles, ties, lists that
overflow, and queries whose norm the error bound does not cover."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha
from ultrahigh_ann_b200 import synthetic

pytestmark = pytest.mark.gpu


def _check(oracle_module, rows, queries, rtol):
    expected, edist = oracle_module.exact("l2", rows, queries)
    index = uha.CudaExactL2Index(rows)
    n = queries.shape[0]
    ws = index.make_query_workspace(n)
    dist = np.zeros(n)
    got = index.query_batch(queries, n, None, ws, distances=dist)
    assert np.array_equal(got, expected)
    np.testing.assert_allclose(dist, edist, rtol=rtol)


# rows, columns (1, 2, 3, 5, 7, 8 stages), queries
SHAPES = [(8193, 64, 40), (20000, 128, 100), (8320, 130, 300), (12345, 257, 129),
          (9001, 448, 257), (8193, 512, 65)]


@pytest.mark.parametrize("rows, d, batch", SHAPES)
def test_answers_at_the_tile_widths_and_stages(oracle_module, rows, d, batch):
    ds = synthetic.row_dataset(rows=rows, classes=7, queries=batch, d=d, seed=rows + batch)
    # settled: a binary64 sum
    _check(oracle_module, ds.rows, ds.queries, 1e-10)


@pytest.mark.parametrize("rows, d, batch", SHAPES)
def test_ties_and_overflowing_lists(oracle_module, rows, d, batch):
    rng = np.random.default_rng(d)
    x = rng.standard_normal((rows, d)).astype(np.float32)
    queries = rng.standard_normal((batch, d)).astype(np.float32)
    x[rows - 20:] = x[rows - 700]       # ties that reach past the last whole tile
    queries[3] = x[rows - 1]
    _check(oracle_module, x, queries, 1e-10)
    x[2000:2100] = x[17]                # more equal rows than a list holds
    queries[5] = x[17]
    _check(oracle_module, x, queries, 1e-5)


@pytest.mark.parametrize("rows, d, batch", SHAPES)
@pytest.mark.parametrize("value", [1e11, 1e13, 1e20, 3e38])
def test_queries_past_the_bound(oracle_module, rows, d, batch, value):
    rng = np.random.default_rng(d)
    x = rng.standard_normal((rows, d)).astype(np.float32)
    queries = rng.standard_normal((batch, d)).astype(np.float32)
    queries[batch - 2] = 0
    queries[batch - 2, 1] = value
    queries[4] *= np.float32(value / 8)
    _check(oracle_module, x, queries, 1e-5)


@pytest.mark.parametrize("value", [1.0, 1e20])
def test_hierarchy(oracle_module, value):
    ds = synthetic.row_dataset(rows=8300, classes=5, queries=150, d=3000, seed=11)
    probs = uha.compute_l2_importance_probabilities_gpu(ds.rows[:100]).probabilities
    index = uha.CudaHierarchicalL2AnnIndex(ds.rows, 16, 70, uha.MT19937_64(3),
                                           importance_probabilities=probs)
    queries = ds.queries.copy()
    queries[7] *= np.float32(value)
    ws = index.make_query_workspace(150)
    dist = np.zeros(150)
    got = index.query_batch(queries, 150, None, ws, distances=dist)
    cs = index.coordinate_sample
    expected, edist = oracle_module.hierarchical("l2", ds.rows, cs.source_columns,
                                                 index.projection, queries)
    assert np.array_equal(got, expected)
    np.testing.assert_allclose(dist, edist, rtol=1e-12)
