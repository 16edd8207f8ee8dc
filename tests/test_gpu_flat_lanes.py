"""The fused query of small batches on both sides of its split rules: rows short
enough to be copied into shared memory and rows read directly, launches alone
and launches that share the chip, answer as the oracle does."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["l2", "l1"])
@pytest.mark.parametrize("rows, d", [(700, 124), (5001, 128), (5000, 129), (2311, 520),
                                     (40001, 131)])
def test_alone_and_beside_others(oracle_module, metric, rows, d):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(rows + d)
    data = rng.standard_normal((rows, d)).astype(np.float32)
    data[rows - 1] = data[3]                     # a tie: the lower row wins
    queries = rng.standard_normal((43, d)).astype(np.float32)
    queries[7] = data[3]
    expected, _ = oracle_module.exact(metric, data, queries)
    index = (uha.CudaExactL2Index if metric == "l2" else uha.CudaExactL1Index)(data)
    device = torch.from_numpy(queries).cuda()
    torch.cuda.synchronize()
    for batch in (1, 5, 8):
        ws = index.make_query_workspace(batch)
        out = np.zeros(43, np.uint64)
        index.query_many(device.data_ptr(), 43, batch, out, ws, uha.QueryStrategy.direct,
                         None, on_device=True)
        assert np.array_equal(out, expected)
        got = index.query_batch(queries[:batch], batch, None, ws)
        assert np.array_equal(got, expected[:batch])
