"""Batches past 8 queries with the FP64-free settlement (set_replay(True)): the
estimating scans form norms and sums in binary64, so these batches take the
binary32 scan and its emulated settlement."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["exact_l2", "exact_l1", "flat_l2", "flat_l1"])
@pytest.mark.parametrize("batch", [9, 70])
def test_launches_are_the_binary32_scan_s(oracle_module, kind, batch):
    rng = np.random.default_rng(batch)
    rows = rng.standard_normal((3000, 3000)).astype(np.float32)
    queries = rng.standard_normal((batch, 3000)).astype(np.float32)
    metric = kind[-2:]
    if kind.startswith("exact"):
        index = (uha.CudaExactL2Index if metric == "l2" else uha.CudaExactL1Index)(rows)
        expected, edist = oracle_module.exact(metric, rows, queries)
    else:
        cls = (uha.CudaSampledCoordinateL2AnnIndex if metric == "l2"
               else uha.CudaSampledCoordinateL1AnnIndex)
        index = cls(rows, np.full(3000, 0.02), 8, uha.MT19937_64(1))
        cs = index.coordinate_sample
        expected, edist = oracle_module.flat(metric, rows, cs.source_columns,
                                             cs.multiplicities, cs.inverse_probabilities,
                                             queries)
    launches = []
    for emulated in (True, False, True):
        ws = index.make_query_workspace(batch)
        ws.set_replay(emulated)
        dist = np.zeros(batch)
        got = index.query_batch(queries, batch, None, ws, distances=dist)
        assert np.array_equal(got, expected)
        np.testing.assert_allclose(dist, edist, rtol=1e-5 if emulated else 1e-10)
        launches.append(ws.last_stats()["kernel_launches"])
    # preparation, scan and certified argmin; the estimating scans launch more
    assert launches[0] == launches[2] == 3 < launches[1]


def test_autotune_keeps_the_binary32_scan(oracle_module):
    rng = np.random.default_rng(3)
    rows = rng.standard_normal((500, 2000)).astype(np.float32)
    queries = rng.standard_normal((40, 2000)).astype(np.float32)
    expected, _ = oracle_module.exact("l2", rows, queries)
    index = uha.CudaExactL2Index(rows)
    ws = index.make_query_workspace(40)
    ws.set_replay(True)
    assert ws.autotune(40)["kernel"] in ("stream", "tile")
    assert np.array_equal(index.query_batch(queries, 40, None, ws), expected)
    ws.set_replay(False)
    assert np.array_equal(index.query_batch(queries, 40, None, ws), expected)
