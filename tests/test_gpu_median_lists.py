"""The row lists of the bitmap median scan on indexes of many rows: more equal
rows than a list of fewer rows' indexes holds, and more than any list holds (the
call is answered again), give the oracle's answers, lowest row on ties."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, equal", [(16384, 1000), (16384, 1500), (16385, 1500),
                                         (17500, 4000), (17500, 4500)])
def test_many_equal_rows(oracle_module, rows, equal):
    rng = np.random.default_rng(rows + equal)
    data = rng.standard_normal((rows, 60)).astype(np.float32)
    data[rows - equal:] = data[5]
    queries = (data[rng.integers(0, rows, 40)] +
               0.1 * rng.standard_normal((40, 60))).astype(np.float32)
    queries[3] = data[5]
    index = uha.CudaHierarchicalL1AnnIndex(
        data, 16, 24, uha.MT19937_64(3),
        coordinate_sample=uha.CoordinateSample(list(range(60)), [1] * 60, [1.0] * 60))
    ws = index.make_query_workspace(40)
    dist = np.zeros(40)
    got = index.query_batch(queries, 40, None, ws, distances=dist)
    expected, edist = oracle_module.hierarchical(
        "l1", data, index.coordinate_sample.source_columns, index.projection, queries)
    assert np.array_equal(got, expected)
    assert got[3] == 5
    np.testing.assert_allclose(dist, edist, rtol=1e-12)
