"""Rows whose distances from a query differ by far less than the split estimates'
error: the error bound has to list them all for the nearest to be among them. 40 rows
a query, their squared distances within 1e-7 of the query's squared norm of one
another (the estimates' measured errors, relative to the centred norms, are 3e-7 to
8e-6, their bound 2e-5 to 2e-4), in the slab and the filter form, at every tile width
and 1 to 8 stages in one accumulator."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu

NEAR = 40


@pytest.mark.parametrize("rows, d, batch", [
    (3000, 64, 40), (3000, 700, 100), (3000, 2111, 257), (1000, 16011, 64),
    (8200, 64, 40), (8200, 128, 100), (8200, 256, 200), (8200, 450, 64), (8200, 512, 129)])
@pytest.mark.parametrize("positive", [False, True])
def test_the_nearest_of_near_ties(oracle_module, rows, d, batch, positive):
    rng = np.random.default_rng(rows + d)

    def draw(*shape):
        return rng.uniform(0, 2, shape) if positive else rng.standard_normal(shape)

    picks = 12                          # queries with near ties, spread over the batch
    queries = draw(batch, d).astype(np.float32)
    x = draw(rows, d).astype(np.float32)
    at = rng.permutation(rows)[:picks * NEAR].reshape(picks, NEAR)
    which = np.linspace(0, batch - 1, picks).astype(int)
    for q, slots in zip(which, at):
        # the query plus steps in random directions, of lengths that differ by a few
        # rounding errors of the values
        step = rng.standard_normal((NEAR, d))
        step *= 0.05 * np.sqrt(d) / np.linalg.norm(step, axis=1, keepdims=True)
        x[slots] = (queries[q] + step).astype(np.float32)
    expected, edist = oracle_module.exact("l2", x, queries)
    # as near as the file's comment says
    for q, slots in zip(which, at):
        near = ((x[slots].astype(np.float64) - queries[q]) ** 2).sum(1)
        norm = (queries[q].astype(np.float64) ** 2).sum()
        assert near.max() - near.min() < 1e-7 * norm and np.unique(near).size > 30
        assert expected[q] in slots
    index = uha.CudaExactL2Index(x)
    ws = index.make_query_workspace(batch)
    dist = np.zeros(batch)
    got = index.query_batch(queries, batch, None, ws, distances=dist)
    assert np.array_equal(got, expected)
    # settled, not answered by the binary32 scan
    np.testing.assert_allclose(dist, edist, rtol=1e-10)
