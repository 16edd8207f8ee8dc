"""Column maxima over several launches: a build of more than 2^39 pairs times
columns, split into up to three launches a pass, has the same probabilities, bit for
bit, however many launches are allowed."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("maxima", ["binary64", "binary32"])
@pytest.mark.parametrize("metric", ["l2", "l1"])
def test_probabilities_do_not_depend_on_the_launches(metric, maxima):
    torch = pytest.importorskip("torch")
    torch.manual_seed(5)
    rows, d = 4509, 55001
    assert rows * rows / 2 * d > 2.0 ** 39
    x = torch.rand(rows, d, device="cuda")
    x[4400] = x[3]                      # a pair at distance zero
    # columns whose largest contribution lies in the first, a middle and the last
    # rows: far apart in one pair only
    far = [(0, 1), (2000, 2100), (rows - 2, rows - 1), (0, rows - 1), (31, 32)]
    for column, (a, b) in enumerate(far):
        x[:, column] = 0.5
        x[a, column], x[b, column] = 40.0, -40.0
    torch.cuda.synchronize()
    fn = (uha.compute_l2_importance_probabilities_gpu if metric == "l2"
          else uha.compute_l1_importance_probabilities_gpu)
    one = fn(x, pair_chunks=1, maxima=maxima)
    assert one.pair_chunks == 1
    for chunks in (2, 3, 128):
        got = fn(x, pair_chunks=chunks, maxima=maxima)
        assert got.pair_chunks == chunks
        assert got.probabilities.tobytes() == one.probabilities.tobytes()
    # each such pair's ratio: 80 (or its square) over the pair's distance
    for column, (a, b) in enumerate(far):
        diff = (x[a].double() - x[b].double()).abs()
        ratio = ((diff[column].square() / diff.square().sum()) if metric == "l2"
                 else diff[column] / diff.sum()).item()
        np.testing.assert_allclose(one.probabilities[column], ratio,
                                   rtol=1e-12 if maxima == "binary64" else 3e-7)
