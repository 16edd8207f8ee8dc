"""The bitmap median scan of L1 hierarchies (median_bits.cu): answers and
distances are the oracle's at the edges of its chunks, column groups and query
blocks, with values outside the boundaries' sample, ties, constant columns, and
where lists overflow and the binary32 passes answer."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha
from ultrahigh_ann_b200 import synthetic

pytestmark = pytest.mark.gpu


def _index(rows, p, T=8, seed=3):
    probs = uha.compute_l1_importance_probabilities_gpu(rows[:60]).probabilities
    return uha.CudaHierarchicalL1AnnIndex(rows, T, p, uha.MT19937_64(seed),
                                          importance_probabilities=probs)


def _check(oracle_module, index, rows, queries, rtol=1e-12):
    n = queries.shape[0]
    ws = index.make_query_workspace(n)
    dist = np.zeros(n)
    got = index.query_batch(queries, n, None, ws, distances=dist)
    cs = index.coordinate_sample
    expected, edist = oracle_module.hierarchical("l1", rows, cs.source_columns,
                                                 index.projection, queries)
    assert np.array_equal(got, expected)
    # the reference's own binary64 medians (rtol 1e-5 where the binary32 passes
    # answer)
    np.testing.assert_allclose(dist, edist, rtol=rtol, atol=1e-300)


@pytest.mark.parametrize("rows, p, batch", [
    (1024, 1, 5), (1025, 2, 8), (1500, 7, 127), (2047, 8, 128), (2048, 9, 129), (3000, 16, 40),
    (4096, 33, 1), (5000, 64, 300), (9217, 65, 17), (2500, 255, 64), (1100, 256, 130),
])
def test_answers_at_the_edges(oracle_module, rows, p, batch):
    ds = synthetic.row_dataset(rows=rows, classes=7, queries=batch, d=1500, seed=rows + p)
    _check(oracle_module, _index(ds.rows, p), ds.rows, ds.queries)


def test_values_outside_the_boundaries_and_ties(oracle_module):
    rng = np.random.default_rng(2)
    rows = rng.standard_normal((3000, 400)).astype(np.float32)
    rows[7] *= 1e4            # far outside the sampled quantiles
    rows[2900:2910] = rows[40]  # ties: the lowest row wins
    queries = np.vstack([rows[7], rows[40], 1e6 * rows[3], np.zeros((1, 400)),
                         rng.standard_normal((20, 400))]).astype(np.float32)
    _check(oracle_module, _index(rows, 32), rows, queries)


def test_constant_and_few_valued_columns(oracle_module):
    rng = np.random.default_rng(4)
    rows = rng.integers(0, 3, (2200, 200)).astype(np.float32)
    queries = rng.integers(0, 3, (30, 200)).astype(np.float32)
    _check(oracle_module, _index(rows, 48, T=64), rows, queries)


def test_overflowing_lists_are_answered_by_the_binary32_passes(oracle_module):
    rng = np.random.default_rng(5)
    rows = rng.standard_normal((4000, 300)).astype(np.float32)
    rows[1500:] = rows[11]      # 2,501 equal rows: more than a list holds
    queries = np.vstack([rows[11], rng.standard_normal((15, 300))]).astype(np.float32)
    index = _index(rows, 24)
    _check(oracle_module, index, rows, queries, rtol=1e-5)
    plain = rng.standard_normal((16, 300)).astype(np.float32)
    batch = uha.QueryBatch([(index, 16)])
    cs = index.coordinate_sample
    for q in (queries, plain, queries):
        want, _ = oracle_module.hierarchical("l1", rows, cs.source_columns, index.projection, q)
        assert np.array_equal(batch.run([q])[0][0], want)


@pytest.mark.parametrize("scale", [1e-30, 1e-12, 1e12, 1e25])
def test_scales(oracle_module, scale):
    rng = np.random.default_rng(6)
    rows = (rng.standard_normal((2000, 300)) * scale).astype(np.float32)
    queries = (rng.standard_normal((40, 300)) * scale).astype(np.float32)
    _check(oracle_module, _index(rows, 40), rows, queries)


def test_non_finite_queries_are_refused():
    rng = np.random.default_rng(7)
    rows = rng.standard_normal((1200, 300)).astype(np.float32)
    index = _index(rows, 16, T=64)
    ws = index.make_query_workspace(20)
    column = int(index.coordinate_sample.source_columns[0])
    for bad in (np.nan, np.inf):
        queries = rows[:20].copy()
        queries[3, column] = bad
        with pytest.raises(uha.InvalidArgument):
            index.query_batch(queries, 20, None, ws)
    assert np.array_equal(index.query_batch(rows[:20], 20, None, ws), np.arange(20))
