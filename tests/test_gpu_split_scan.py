"""The certified split scan (tensor-core estimates of centred BF16 parts, binary64
settlement) of direct L2 batches past 8 queries: the answers are the oracle's at
the edges of its tiles and stages, and where the estimates cannot decide (ties,
lists that overflow, values outside the bound's range) the answers and errors
are those of the binary32 scan."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha
from ultrahigh_ann_b200 import synthetic

pytestmark = pytest.mark.gpu


def _check(oracle_module, rows, queries, index=None, emulated=False, rtol=1e-10):
    expected, edist = oracle_module.exact("l2", rows, queries)
    index = index or uha.CudaExactL2Index(rows)
    n = queries.shape[0]
    ws = index.make_query_workspace(n)
    ws.set_replay(emulated)
    dist = np.zeros(n)
    got = index.query_batch(queries, n, None, ws, distances=dist)
    assert np.array_equal(got, expected)
    # the settled distance is a binary64 sum (emulated: binary32 within its
    # certified bound, or float-float)
    np.testing.assert_allclose(dist, edist, rtol=1e-5 if emulated else rtol, atol=1e-300)
    return ws.last_stats()


@pytest.mark.parametrize("rows, d, batch", [
    (2, 32769, 9), (127, 4099, 63), (128, 4160, 64), (129, 4097, 65), (257, 3001, 128),
    (300, 2047, 129), (511, 8191, 255), (640, 1031, 256), (1000, 515, 257), (2049, 130, 513),
    (20000, 64, 40),
])
@pytest.mark.parametrize("emulated", [False, True])
def test_answers_at_the_tile_edges(oracle_module, rows, d, batch, emulated):
    ds = synthetic.row_dataset(rows=rows, classes=min(rows, 7), queries=batch, d=d,
                               seed=rows + batch)
    _check(oracle_module, ds.rows, ds.queries, emulated=emulated)


@pytest.mark.parametrize("scale", [1e-30, 1e-15, 1.0, 1e10, 1e15])
@pytest.mark.parametrize("offset", [0.0, 1000.0])
def test_scales_and_offsets(oracle_module, scale, offset):
    # an offset shared by every value leaves the centred products small; the
    # rows' norms are scaled near 1
    rng = np.random.default_rng(5)
    rows = ((rng.standard_normal((600, 700)) + offset) * scale).astype(np.float32)
    queries = ((rng.standard_normal((70, 700)) + offset) * scale).astype(np.float32)
    _check(oracle_module, rows, queries)


def test_ties_and_overflowing_lists(oracle_module):
    rng = np.random.default_rng(6)
    rows = rng.standard_normal((400, 300)).astype(np.float32)
    rows[200:210] = rows[17]            # ties: the lowest row wins
    rows[211] = np.nextafter(rows[17], np.float32(np.inf))
    queries = np.vstack([rows[17], rows[211], rng.standard_normal((30, 300))]).astype(np.float32)
    st = _check(oracle_module, rows, queries)
    assert st["replayed_queries"] >= 1
    # 181 equal rows: more than a list holds, so the call is answered by the
    # binary32 scan (distances within 1e-5)
    rows[230:] = rows[17]
    _check(oracle_module, rows, queries, rtol=1e-5)


def test_zero_rows_and_queries(oracle_module):
    rows = np.zeros((130, 256), np.float32)
    rows[5:] = np.random.default_rng(7).standard_normal((125, 256)).astype(np.float32)
    queries = np.zeros((12, 256), np.float32)
    queries[3:] = rows[20:29]
    _check(oracle_module, rows, queries)


def test_non_finite_query_is_refused():
    rows = np.random.default_rng(8).standard_normal((300, 500)).astype(np.float32)
    index = uha.CudaExactL2Index(rows)
    ws = index.make_query_workspace(40)
    for bad in (np.nan, np.inf, -np.inf):
        queries = rows[:40].copy()
        queries[11, 3] = bad
        with pytest.raises(uha.InvalidArgument):
            index.query_batch(queries, 40, None, ws)
    queries = rows[:40].copy()
    assert np.array_equal(index.query_batch(queries, 40, None, ws), np.arange(40))


@pytest.mark.parametrize("rows, p, batch", [(129, 16, 9), (700, 63, 64), (1500, 65, 200),
                                            (3000, 256, 300)])
def test_hierarchies(oracle_module, rows, p, batch):
    ds = synthetic.row_dataset(rows=rows, classes=5, queries=batch, d=3000, seed=p)
    probs = uha.compute_l2_importance_probabilities_gpu(ds.rows[:100]).probabilities
    index = uha.CudaHierarchicalL2AnnIndex(ds.rows, 16, p, uha.MT19937_64(3),
                                           importance_probabilities=probs)
    ws = index.make_query_workspace(batch)
    dist = np.zeros(batch)
    got = index.query_batch(ds.queries, batch, None, ws, distances=dist)
    cs = index.coordinate_sample
    expected, edist = oracle_module.hierarchical("l2", ds.rows, cs.source_columns,
                                                 index.projection, ds.queries)
    assert np.array_equal(got, expected)
    np.testing.assert_allclose(dist, edist, rtol=1e-12)


def test_batch_whose_list_overflows_answers_again(oracle_module):
    rng = np.random.default_rng(9)
    rows = rng.standard_normal((500, 400)).astype(np.float32)
    rows[100:] = rows[3]
    queries = rng.standard_normal((20, 400)).astype(np.float32)
    queries[0] = rows[3]
    index = uha.CudaExactL2Index(rows)
    batch = uha.QueryBatch([(index, 20)])
    expected, _ = oracle_module.exact("l2", rows, queries)
    plain = rng.standard_normal((20, 400)).astype(np.float32)
    for q in (queries, plain, queries):
        want, _ = oracle_module.exact("l2", rows, q)
        assert np.array_equal(batch.run([q])[0][0], want)


@pytest.mark.parametrize("positive", [True, False])
def test_estimate_error_is_within_the_bound(positive):
    """One chunk of the estimate against binary64 on BF16 values: the tensor
    core's error is below the 2^-19 per instruction that the bound assumes."""
    rng = np.random.default_rng(10)
    rows = rng.uniform(0 if positive else -1, 1, (512, 64)).astype(np.float32)
    queries = rng.uniform(0 if positive else -1, 1, (64, 64)).astype(np.float32)
    # exponents spread, so products are shifted out against the largest
    rows *= np.exp2(rng.integers(-12, 1, rows.shape)).astype(np.float32)
    torch = pytest.importorskip("torch")
    bf = [torch.from_numpy(x).bfloat16().float().numpy() for x in (rows, queries)]
    index = uha.CudaExactL2Index(bf[0])
    ws = index.make_query_workspace(64)
    scores, _ = index.precision_scores(bf[1], 64, ws)
    r64, q64 = bf[0].astype(np.float64), bf[1].astype(np.float64)
    magnitude = np.abs(q64) @ np.abs(r64).T
    error = np.abs(scores - q64 @ r64.T) / magnitude
    assert error.max() <= 4 * 2.0 ** -19
