"""Host queries of sampled indexes cross PCIe as their sampled values alone:
answers equal the device-resident queries' for every index kind and batch form,
only sampled columns are validated, and the status words of a failed call do not
reach the next one."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha
from ultrahigh_ann_b200 import synthetic

pytestmark = pytest.mark.gpu

S = uha.QueryStrategy


def _indexes(rows, T):
    probs = np.full(rows.shape[1], 0.02)
    rng = uha.MT19937_64
    yield uha.CudaSampledCoordinateL2AnnIndex(rows, probs, T, rng(1)), S.direct
    yield uha.CudaSampledCoordinateL2AnnIndex(rows, probs, T, rng(1)), S.gemm
    yield uha.CudaSampledCoordinateL2AnnIndex(rows, probs, T, rng(1)), S.gemm_bf16_rerank
    yield uha.CudaSampledCoordinateL1AnnIndex(rows, probs, T, rng(2)), S.direct
    yield uha.CudaHierarchicalL2AnnIndex(rows, T, 24, rng(3),
                                         importance_probabilities=probs), S.direct
    yield uha.CudaHierarchicalL1AnnIndex(rows, T, 24, rng(4),
                                         importance_probabilities=probs), S.direct


# T = 1 and 4 sample below an eighth of the columns (gathered on the host), T = 40
# above it (whole vectors)
@pytest.mark.parametrize("T", [1, 4, 40])
@pytest.mark.parametrize("batch", [1, 7, 64])
def test_host_queries_answer_as_device_queries(T, batch):
    torch = pytest.importorskip("torch")
    ds = synthetic.row_dataset(rows=1500, classes=6, queries=90, d=2000, seed=T)
    device = torch.from_numpy(ds.queries).cuda()
    torch.cuda.synchronize()
    for index, strategy in _indexes(ds.rows, T):
        ws = index.make_query_workspace(batch)
        host, dev = np.zeros(90), np.zeros(90)
        a = index.query_many(ds.queries, 90, batch, None, ws, strategy, host)
        b = index.query_many(device.data_ptr(), 90, batch, None, ws, strategy, dev,
                             on_device=True)
        assert np.array_equal(a, b)
        assert np.array_equal(host, dev)


def test_only_sampled_columns_are_validated_and_errors_do_not_stick():
    ds = synthetic.row_dataset(rows=300, classes=6, queries=20, d=2000, seed=9)
    for index, strategy in _indexes(ds.rows, 2):
        ws = index.make_query_workspace(20)
        sampled = index.coordinate_sample.source_columns
        other = np.setdiff1d(np.arange(2000), sampled)
        want = index.query_batch(ds.queries, 20, None, ws, strategy)
        queries = ds.queries.copy()
        queries[:, other] = np.nan
        assert np.array_equal(index.query_batch(queries, 20, None, ws, strategy), want)
        queries[5, int(sampled[0])] = np.inf
        with pytest.raises(uha.InvalidArgument):
            index.query_batch(queries, 20, None, ws, strategy)
        assert np.array_equal(index.query_batch(ds.queries, 20, None, ws, strategy), want)
