"""The gathering binary64 projection of query batches: every split of the
coordinates over lanes, warps and rounds, and remainders of its query groups and
column chunks, give the oracle's answers (L2 hierarchies, whose scan starts with
it at any number of rows)."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p, k, batch", [(1, 1, 9), (31, 127, 17), (33, 129, 40), (64, 300, 33),
                                         (65, 8, 16), (129, 257, 21), (257, 40, 12),
                                         (513, 130, 10)])
def test_projections(oracle_module, p, k, batch):
    rng = np.random.default_rng(p)
    rows = rng.standard_normal((150, 900)).astype(np.float32)
    queries = (rows[rng.integers(0, 150, batch)] +
               0.3 * rng.standard_normal((batch, 900))).astype(np.float32)
    columns = np.sort(rng.choice(900, k, replace=False)).astype(np.uint32)
    index = uha.CudaHierarchicalL2AnnIndex(
        rows, 16, p, uha.MT19937_64(3),
        coordinate_sample=uha.CoordinateSample(list(columns), [1] * k, [1.0] * k))
    ws = index.make_query_workspace(batch)
    dist = np.zeros(batch)
    got = index.query_batch(queries, batch, None, ws, distances=dist)
    cs = index.coordinate_sample
    expected, edist = oracle_module.hierarchical("l2", rows, cs.source_columns,
                                                 index.projection, queries)
    assert np.array_equal(got, expected)
    np.testing.assert_allclose(dist, edist, rtol=1e-12)
