"""Queries that the estimating scans leave open (more equal rows than a list holds,
values past the estimates' range): they alone are answered by the binary32 scans,
every other query of the call keeps its settled binary64 distance, and calls or
captured batches whose queries are mostly open stop paying for the estimates."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu

ROWS, D = 3000, 1100
KINDS = ["exact_l2", "exact_l1", "flat_l2", "flat_l1", "hier_l2", "hier_l1"]


def _case(oracle_module, kind, seed, count, opened):
    """An index of 1,500 equal rows among others, queries of which `opened` are
    that row, and the oracle's answers."""
    rng = np.random.default_rng(seed)
    rows = rng.standard_normal((ROWS, D)).astype(np.float32)
    rows[1000:2500] = rows[70]
    queries = rng.standard_normal((count, D)).astype(np.float32)
    queries[opened] = rows[70]
    metric = kind[-2:]
    l2 = metric == "l2"
    if kind.startswith("exact"):
        index = (uha.CudaExactL2Index if l2 else uha.CudaExactL1Index)(rows)
        return index, queries, oracle_module.exact(metric, rows, queries)
    probs = np.full(D, 0.02)
    if kind.startswith("flat"):
        cls = (uha.CudaSampledCoordinateL2AnnIndex if l2
               else uha.CudaSampledCoordinateL1AnnIndex)
        index = cls(rows, probs, 16, uha.MT19937_64(1))
        cs = index.coordinate_sample
        return index, queries, oracle_module.flat(metric, rows, cs.source_columns,
                                                  cs.multiplicities, cs.inverse_probabilities,
                                                  queries)
    cls = uha.CudaHierarchicalL2AnnIndex if l2 else uha.CudaHierarchicalL1AnnIndex
    index = cls(rows, 16, 33, uha.MT19937_64(3), importance_probabilities=probs)
    cs = index.coordinate_sample
    return index, queries, oracle_module.hierarchical(metric, rows, cs.source_columns,
                                                      index.projection, queries)


def _compare(got, dist, expected, edist, opened):
    assert np.array_equal(got, expected)
    settled = np.ones(got.size, bool)
    settled[opened] = False
    # binary64 sums of the same terms; the binary32 scan's distances
    np.testing.assert_allclose(dist[settled], edist[settled], rtol=1e-10)
    np.testing.assert_allclose(dist[opened], edist[opened], rtol=1e-5, atol=1e-30)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("opened", [[0], [5, 6, 7, 20], list(range(0, 90, 9)), [99]])
@pytest.mark.parametrize("device", [False, True])
def test_only_open_queries_are_answered_again(oracle_module, kind, opened, device):
    torch = pytest.importorskip("torch")
    index, queries, (expected, edist) = _case(oracle_module, kind, 1, 100, opened)
    held = torch.from_numpy(queries).cuda()
    torch.cuda.synchronize()
    source = held.data_ptr() if device else queries
    for batch in (100, 45):
        for _ in range(2):
            # (one that has just left queries open may answer by the binary32 scan)
            ws = index.make_query_workspace(batch)
            dist = np.zeros(100)
            out = np.zeros(100, np.uint64)
            index.query_many(source, 100, batch, out, ws, distances=dist, on_device=device)
            _compare(out, dist, expected, edist, opened)
            st = ws.last_stats()
            assert st["query_count"] == 100
            assert st["replayed_queries"] + st["certified_queries"] == 100
            assert st["replayed_queries"] >= len(opened)
        # without distances
        out[:] = 0
        index.query_many(source, 100, batch, out, ws, on_device=device)
        assert np.array_equal(out, expected)


@pytest.mark.parametrize("kind", KINDS)
def test_mostly_open_calls_stop_estimating(oracle_module, kind):
    index, queries, (expected, edist) = _case(oracle_module, kind, 2, 40, slice(0, 36))
    rng = np.random.default_rng(3)
    plain = rng.standard_normal(queries.shape).astype(np.float32)
    ws = index.make_query_workspace(40)

    def launches(q):
        out = index.query_batch(q, 40, None, ws)
        if q is queries:
            assert np.array_equal(out, expected)
        return ws.last_stats()["kernel_launches"]

    ordinary = launches(plain)
    both = launches(queries)
    assert both > ordinary              # the estimates and the open queries
    alone = launches(queries)
    assert alone < both                 # one call by the binary32 scan
    assert launches(queries) == both    # tried again,
    assert launches(queries) == alone   # then two calls
    assert launches(plain) == alone
    assert launches(plain) == ordinary
    assert launches(plain) == ordinary


@pytest.mark.parametrize("kind", ["exact_l2", "exact_l1", "hier_l2", "hier_l1"])
def test_captured_batches(oracle_module, kind):
    index, queries, (expected, edist) = _case(oracle_module, kind, 4, 40, [3, 39])
    mostly, (_, many, (mexpected, medist)) = list(range(30)), _case(
        oracle_module, kind, 4, 40, list(range(30)))
    _, plain, (pexpected, pedist) = _case(oracle_module, kind, 4, 40, [])
    other, oqueries, (oexpected, oedist) = _case(oracle_module, "hier_l2", 5, 25, [])
    batch = uha.QueryBatch([(index, 40), (other, 25)])

    def run(q, expected, edist, opened):
        got = batch.run([q, oqueries])
        _compare(got[0][0], got[0][1], expected, edist, opened)
        _compare(got[1][0], got[1][1], oexpected, oedist, [])
        return batch.stats()["kernel_launches"]

    first = run(plain, pexpected, pedist, [])
    assert run(queries, expected, edist, [3, 39]) == first
    assert run(plain, pexpected, pedist, []) == first
    assert run(many, mexpected, medist, mostly) == first
    assert run(many, mexpected, medist, mostly) == first
    # captured anew on the binary32 scans, whose distances are within 1e-5 (a
    # hierarchy's are binary64 all the same)
    every = [] if kind.startswith("hier") else list(range(40))
    binary32 = run(many, mexpected, medist, every or mostly)
    if kind != "hier_l2":               # six launches either way
        assert binary32 != first
    for _ in range(62):
        batch.run([plain, oqueries])
    assert run(queries, expected, edist, every or [3, 39]) == binary32
    # and after 64 runs on the estimates
    assert run(queries, expected, edist, [3, 39]) == first


@pytest.mark.parametrize("kind", ["hier_l2", "hier_l1"])
def test_projections_past_the_bound(oracle_module, kind):
    index, queries, _ = _case(oracle_module, kind, 6, 60, [])
    cs = index.coordinate_sample
    queries[11] *= np.float32(1e30)
    rng = np.random.default_rng(6)
    rows = rng.standard_normal((ROWS, D)).astype(np.float32)
    rows[1000:2500] = rows[70]
    expected, edist = oracle_module.hierarchical(kind[-2:], rows, cs.source_columns,
                                                 index.projection, queries)
    ws = index.make_query_workspace(60)
    dist = np.zeros(60)
    out = index.query_batch(queries, 60, None, ws, distances=dist)
    _compare(out, dist, expected, edist, [11])


@pytest.mark.parametrize("kind", KINDS)
def test_skipped_calls_report_binary64_distances(oracle_module, kind):
    index, queries, (expected, edist) = _case(oracle_module, kind, 7, 40, slice(0, 36))
    _, plain, (pexpected, pedist) = _case(oracle_module, kind, 7, 40, [])
    ws = index.make_query_workspace(40)
    estimated = np.zeros(40)
    index.query_batch(plain, 40, None, ws, distances=estimated)
    for _ in range(2):                  # left open; the next call skips the estimates
        dist = np.zeros(40)
        assert np.array_equal(index.query_batch(queries, 40, None, ws, distances=dist), expected)
        np.testing.assert_allclose(dist, edist, rtol=1e-10, atol=1e-30)
    index.query_batch(queries, 40, None, ws)
    dist = np.zeros(40)                 # skipped
    assert np.array_equal(index.query_batch(plain, 40, None, ws, distances=dist), pexpected)
    np.testing.assert_allclose(dist, pedist, rtol=1e-10)
    np.testing.assert_allclose(dist, estimated, rtol=1e-13)
