"""The certified fixed-point scan (16-bit integer estimates, binary64 settlement)
of direct L1 batches past 8 queries: the answers are the oracle's at the edges of
its tiles and stages, weighted and sampled, for queries outside the rows' range,
and where the estimates cannot decide (ties, lists that overflow, a step too
coarse for the rows) the answers are those of the binary32 scan."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha
from ultrahigh_ann_b200 import synthetic

pytestmark = pytest.mark.gpu


def _run(index, queries):
    n = queries.shape[0]
    ws = index.make_query_workspace(n)
    dist = np.zeros(n)
    got = index.query_batch(queries, n, None, ws, distances=dist)
    return got, dist, ws.last_stats()


def _check(oracle_module, rows, queries, weights=None, rtol=1e-10):
    # a settled distance is a binary64 sum in another order; the binary32 scan's
    # own distances are within 1e-5
    index = uha.CudaDenseL1ScanIndex(rows, weights)
    got, dist, stats = _run(index, queries)
    if weights is None:
        expected, edist = oracle_module.exact("l1", rows, queries)
    else:
        expected, edist = oracle_module.weighted_l1(rows, weights, queries)
    assert np.array_equal(got, expected)
    np.testing.assert_allclose(dist, edist, rtol=rtol, atol=1e-300)
    return stats


@pytest.mark.parametrize("rows, d, batch", [
    (2, 32769, 9), (127, 4099, 63), (128, 4160, 64), (129, 4097, 65), (257, 3001, 128),
    (300, 2047, 33), (511, 8191, 255), (1000, 515, 257), (2049, 130, 513), (20000, 64, 32),
    (40, 70001, 17),
])
@pytest.mark.parametrize("weighted", [False, True])
def test_answers_at_the_tile_edges(oracle_module, rows, d, batch, weighted):
    ds = synthetic.row_dataset(rows=rows, classes=min(rows, 7), queries=batch, d=d,
                               seed=rows + batch)
    weights = None
    if weighted:
        weights = np.random.default_rng(d).uniform(0, 3, d).astype(np.float32)
        weights[::5] = 0
    _check(oracle_module, ds.rows, ds.queries, weights)


@pytest.mark.parametrize("reps", [16, 64])
def test_sampled_columns(oracle_module, reps):
    ds = synthetic.row_dataset(rows=9000, classes=33, queries=100, d=5003, seed=reps)
    probs = oracle_module.probabilities("l1", ds.rows[:500])
    index = uha.CudaSampledCoordinateL1AnnIndex(ds.rows, probs, reps, uha.MT19937_64(2))
    cs = index.coordinate_sample
    expected, edist = oracle_module.flat("l1", ds.rows, cs.source_columns, cs.multiplicities,
                                         cs.inverse_probabilities, ds.queries)
    got, dist, _ = _run(index, ds.queries)
    assert np.array_equal(got, expected)
    np.testing.assert_allclose(dist, edist, rtol=1e-10)


@pytest.mark.parametrize("scale", [1e-25, 1e-6, 1.0, 1e12, 1e30])
@pytest.mark.parametrize("offset", [0.0, 1000.0])
def test_scales_offsets_and_queries_outside_the_range(oracle_module, scale, offset):
    rng = np.random.default_rng(5)
    rows = ((rng.uniform(-1, 1, (600, 700)) + offset) * scale).astype(np.float32)
    rows[:, 11] = np.float32(7 * scale)     # a constant column
    queries = ((rng.uniform(-1, 1, (40, 700)) + offset) * scale).astype(np.float32)
    queries[3, 5] = 1e5 * scale             # one value far outside
    _check(oracle_module, rows, queries, rtol=1e-10)
    # all values outside: the estimates decide nothing, so the lists overflow
    _check(oracle_module, rows, queries * np.float32(40), rtol=1e-5)


def test_ties_and_overflowing_lists(oracle_module):
    rng = np.random.default_rng(6)
    rows = rng.standard_normal((400, 300)).astype(np.float32)
    rows[200:210] = rows[17]            # ties: the lowest row wins
    rows[211] = np.nextafter(rows[17], np.float32(np.inf))
    queries = np.vstack([rows[17], rows[211], rng.standard_normal((30, 300))]).astype(np.float32)
    st = _check(oracle_module, rows, queries)
    assert st["replayed_queries"] >= 1
    # 181 equal rows: more than a list holds
    rows[230:] = rows[17]
    _check(oracle_module, rows, queries, rtol=1e-5)


def test_steps_too_coarse_for_the_rows(oracle_module):
    # one column's range hides the others: the index keeps the binary32 scan
    rng = np.random.default_rng(7)
    rows = rng.standard_normal((500, 256)).astype(np.float32)
    rows[:, 9] *= 1e6
    rows[:, 9] = np.sort(rows[:, 9])
    queries = (rows[100:130] + 0.1 * rng.standard_normal((30, 256))).astype(np.float32)
    _check(oracle_module, rows, queries, rtol=1e-5)
    # equal rows, and rows of zeros
    rows[:] = rows[0]
    _check(oracle_module, rows, queries, rtol=1e-5)
    _check(oracle_module, np.zeros((300, 64), np.float32), np.zeros((9, 64), np.float32))


def test_non_finite_query_is_refused():
    rows = np.random.default_rng(8).standard_normal((300, 500)).astype(np.float32)
    index = uha.CudaExactL1Index(rows)
    ws = index.make_query_workspace(40)
    for bad in (np.nan, np.inf, -np.inf):
        queries = rows[:40].copy()
        queries[11, 3] = bad
        with pytest.raises(uha.InvalidArgument):
            index.query_batch(queries, 40, None, ws)
    queries = rows[:40].copy()
    assert np.array_equal(index.query_batch(queries, 40, None, ws), np.arange(40))


def test_captured_batches_answer_new_queries(oracle_module):
    rng = np.random.default_rng(9)
    rows = rng.standard_normal((500, 400)).astype(np.float32)
    rows[100:] = rows[3]
    near = rng.standard_normal((20, 400)).astype(np.float32)
    near[0] = rows[3]                   # 401 equal rows: answered again
    batch = uha.QueryBatch([(uha.CudaExactL1Index(rows), 20)])
    plain = rng.standard_normal((20, 400)).astype(np.float32)
    for q in (near, plain, near):
        want, _ = oracle_module.exact("l1", rows, q)
        assert np.array_equal(batch.run([q])[0][0], want)


@pytest.mark.parametrize("d", [32000, 32001])
def test_both_widths_of_the_epilogue(d):
    # 444 tiles fill the chip at one column split; the binary32 scan (FP64-free
    # settlement) answers the same queries
    torch = pytest.importorskip("torch")
    torch.manual_seed(d)
    rows = torch.rand(444 * 128 - 5, d, device="cuda")
    queries = torch.rand(64, d, device="cuda")
    queries[:32] = rows[1000:57000:1750][:32] + 0.02 * torch.rand(32, d, device="cuda")
    torch.cuda.synchronize()
    index = uha.CudaExactL1Index(rows)
    answers = []
    for emulated in (False, True):
        ws = index.make_query_workspace(64)
        ws.set_replay(emulated)
        dist = np.zeros(64)
        out = np.zeros(64, np.uint64)
        index.query_device_batch(queries.data_ptr(), 64, out, ws, distances=dist)
        answers.append((out, dist))
    assert np.array_equal(answers[0][0], answers[1][0])
    assert np.array_equal(answers[0][0][:32], np.arange(1000, 57000, 1750)[:32])
    np.testing.assert_allclose(answers[0][1], answers[1][1], rtol=1e-5)
