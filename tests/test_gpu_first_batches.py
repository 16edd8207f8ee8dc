"""Row forms and scan buffers: built and sized by need, beside the rows and the
query buffer where they are small, and answering the oracle's rows whatever order
the calls come in (growing and shrinking batches, several workspaces, a large index
whose first small batches do not pay for its form)."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu


def _index(kind, rows, d):
    if kind.startswith("exact"):
        return (uha.CudaExactL2Index if kind == "exact_l2" else uha.CudaExactL1Index)(rows)
    cls = (uha.CudaHierarchicalL2AnnIndex if kind == "hier_l2"
           else uha.CudaHierarchicalL1AnnIndex)
    return cls(rows, 16, 40, uha.MT19937_64(3), importance_probabilities=np.full(d, 0.02))


def _oracle(oracle_module, kind, index, rows, queries):
    if kind.startswith("exact"):
        return oracle_module.exact(kind[-2:], rows, queries)
    cs = index.coordinate_sample
    return oracle_module.hierarchical(kind[-2:], rows, cs.source_columns, index.projection,
                                      queries)


KINDS = ["exact_l2", "exact_l1", "hier_l2", "hier_l1"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows, d", [(1500, 1030), (9000, 130)])
def test_batches_of_every_size_in_turn(oracle_module, kind, rows, d):
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, d)).astype(np.float32)
    queries = rng.standard_normal((600, d)).astype(np.float32)
    index = _index(kind, x, d)
    expected, edist = _oracle(oracle_module, kind, index, x, queries)
    for most in (600, 64):
        ws = index.make_query_workspace(most)
        for n in (9, 64, 10, 65, 300, 8, 600, 17, 129, 600):
            if n > most:
                continue
            dist = np.zeros(n)
            got = index.query_batch(queries[:n], n, None, ws, distances=dist)
            assert np.array_equal(got, expected[:n])
            np.testing.assert_allclose(dist, edist[:n],
                                       rtol=1e-5 if n == 8 and kind[:5] == "exact" else 1e-10)


@pytest.mark.parametrize("metric", ["l2", "l1"])
def test_a_large_form_is_built_when_it_pays(metric):
    # 100 million values: the form is larger than the place beside the rows, and 9
    # queries save less than it costs
    torch = pytest.importorskip("torch")
    torch.manual_seed(4)
    rows = torch.rand(50000, 2000, device="cuda")
    at = torch.arange(100, 50000, 499, device="cuda")[:64]
    queries = rows[at] + 0.01 * torch.rand(64, 2000, device="cuda")
    torch.cuda.synchronize()
    index = (uha.CudaExactL2Index if metric == "l2" else uha.CudaExactL1Index)(rows)
    d = (rows[at].double() - queries.double())
    exact = (d.square() if metric == "l2" else d.abs()).sum(1).cpu().numpy()
    ws = index.make_query_workspace(64)
    launches, first = [], None
    for n in [9] * 12 + [64]:
        out, dist = np.zeros(n, np.uint64), np.zeros(n)
        index.query_device_batch(queries.data_ptr(), n, out, ws, distances=dist)
        assert np.array_equal(out, at[:n].cpu().numpy().astype(np.uint64))
        np.testing.assert_allclose(dist, exact[:n], rtol=1e-10)
        launches.append(ws.last_stats()["kernel_launches"])
        first = dist if first is None else first
    # preparation, scan, argmin and the winners' distances; then the estimating scan,
    # for good, with the same bits
    assert launches[0] == 4 and launches[-2] > 4
    assert np.array_equal(first, dist[:9])
    changes = [a != b for a, b in zip(launches[:-1], launches[1:-1])]
    assert sum(changes) == 1


@pytest.mark.parametrize("kind", KINDS)
def test_threads_share_a_new_form(oracle_module, kind):
    rng = np.random.default_rng(9)
    x = rng.standard_normal((3000, 700)).astype(np.float32)
    queries = rng.standard_normal((6, 40, 700)).astype(np.float32)
    index = _index(kind, x, 700)
    expected = [_oracle(oracle_module, kind, index, x, q)[0] for q in queries]
    failures = []

    def answer(i):
        try:
            ws = index.make_query_workspace(40)
            for _ in range(5):
                got = index.query_batch(queries[i], 40, None, ws)
                if not np.array_equal(got, expected[i]):
                    failures.append(i)
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=answer, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
