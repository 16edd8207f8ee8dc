"""Autotuning batches that the filter form of the split scan answers: one shape, but
a measured one, which replaces what an earlier tuning kept."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["exact", "hierarchy"])
@pytest.mark.parametrize("batch", [12, 100, 300])
def test_report_and_answers(oracle_module, kind, batch):
    rng = np.random.default_rng(batch)
    rows = rng.standard_normal((9000, 200)).astype(np.float32)
    queries = rng.standard_normal((batch, 200)).astype(np.float32)
    if kind == "exact":
        index = uha.CudaExactL2Index(rows)
        expected, edist = oracle_module.exact("l2", rows, queries)
    else:
        index = uha.CudaHierarchicalL2AnnIndex(rows, 16, 40, uha.MT19937_64(2),
                                               importance_probabilities=np.full(200, 0.05))
        cs = index.coordinate_sample
        expected, edist = oracle_module.hierarchical("l2", rows, cs.source_columns,
                                                     index.projection, queries)
    ws = index.make_query_workspace(batch)

    def answer(rtol):
        dist = np.zeros(batch)
        assert np.array_equal(index.query_batch(queries, batch, None, ws, distances=dist),
                              expected)
        np.testing.assert_allclose(dist, edist, rtol=rtol)
        return ws.last_stats()["kernel_launches"]

    if kind == "exact":
        ws.set_replay(True)             # keeps, and tunes, the binary32 scan
        assert ws.autotune(batch)["kernel"] in ("stream", "tile")
        tuned = answer(1e-5)
        ws.set_replay(False)
    report = ws.autotune(batch)
    assert report["kernel"] == "tensor" and report["candidates"] == 1
    assert report["tile_queries"] in (64, 128, 256) and report["splits"] == 1
    assert 0 < report["best_ms"] == report["default_ms"]
    filtered = answer(1e-10)
    assert kind != "exact" or filtered > tuned
    batched = uha.QueryBatch([(index, batch)], autotune=True)
    assert batched.tuning(0)["kernel"] == "tensor"
    assert np.array_equal(batched.run([queries])[0][0], expected)
