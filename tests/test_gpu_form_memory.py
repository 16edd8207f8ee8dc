"""Device memory of the row forms: a form of its own leaves as much free as it
takes, and one that no call uses is given back when another allocation finds no
room, so what fitted on the device without the forms fits with them."""
from __future__ import annotations

import numpy as np
import pytest

import ultrahigh_ann_b200 as uha

pytestmark = pytest.mark.gpu

ROWS, D = 20000, 20001
FORM = ROWS * D * 4                     # bytes of the rows, and of their split form


@pytest.fixture
def torch():
    module = pytest.importorskip("torch")
    module.cuda.empty_cache()
    yield module
    module.cuda.empty_cache()


def _fill(torch, leave):
    """Holds all free memory but about `leave` bytes."""
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def _data(torch):
    torch.manual_seed(1)
    rows = torch.rand(ROWS, D, device="cuda")
    at = torch.arange(70, ROWS, 290, device="cuda")[:64]
    queries = rows[at] + 0.01 * torch.rand(64, D, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return rows, at.cpu().numpy().astype(np.uint64), queries


def _ask(index, queries, expected):
    """The launches of one call of 64 queries on a new workspace."""
    ws = index.make_query_workspace(64)
    out = np.zeros(64, np.uint64)
    index.query_device_batch(queries.data_ptr(), 64, out, ws)
    assert np.array_equal(out, expected)
    return ws.last_stats()["kernel_launches"]


def test_an_idle_form_makes_room(torch):
    kind = uha.CudaExactL2Index
    rows, expected, queries = _data(torch)
    first = kind(rows)
    assert _ask(first, queries, expected) > 3     # the estimating scan
    # no room for a second index beside the first one's form, but in its place
    held = _fill(torch, FORM - (FORM >> 2))
    try:
        second = kind(rows)
        assert _ask(second, queries, expected) == 3   # and none for a form
        assert _ask(first, queries, expected) == 3
        del second
    finally:
        del held
    torch.cuda.empty_cache()
    third = kind(rows)
    assert _ask(third, queries, expected) > 3


def test_a_form_in_use_stays(torch):
    rows, expected, queries = _data(torch)
    index = uha.CudaExactL2Index(rows)
    batch = uha.QueryBatch([(index, 64)], autotune=False)
    held = _fill(torch, FORM - (FORM >> 2))
    try:
        with pytest.raises(uha.CudaRuntimeError):
            uha.CudaExactL2Index(rows)
        # the captured scan still reads it
        got = batch.run([queries.data_ptr()], on_device=True)[0][0]
        assert np.array_equal(got, expected)
        del batch
        other = uha.CudaExactL2Index(rows)        # now it is given back
    finally:
        del held
    torch.cuda.empty_cache()
    assert _ask(other, queries, expected) > 3


def test_a_form_takes_at_most_half_of_what_is_free(torch):
    rows, expected, queries = _data(torch)
    index = uha.CudaExactL2Index(rows)
    held = _fill(torch, 2 * FORM - (FORM >> 2))
    try:
        assert _ask(index, queries, expected) == 3
    finally:
        del held
    torch.cuda.empty_cache()
    # decided once per index
    assert _ask(index, queries, expected) == 3
    other = uha.CudaExactL2Index(rows)
    assert _ask(other, queries, expected) > 3


def test_a_call_takes_its_own_form_s_room(torch):
    # many queries: beside the form there is no room for their sums, by either scan;
    # without it there is for the binary32 scan's (one split of the columns)
    torch.manual_seed(2)
    rows = torch.rand(40000, 8000, device="cuda")
    at = torch.arange(70, 40000, 590, device="cuda")[:64]
    queries = rows[at] + 0.01 * torch.rand(64, 8000, device="cuda")
    many = queries.repeat(313, 1)[:20000].contiguous()
    expected = at.cpu().numpy().astype(np.uint64)
    index = uha.CudaExactL2Index(rows)
    for _ in range(4):
        launches = _ask(index, queries, expected)
    assert launches > 3
    ws = index.make_query_workspace(20000)
    form, sums = 40000 * 8000 * 4, 20000 * 40000 * 4
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = _fill(torch, sums - (form >> 1))
    try:
        out = np.zeros(20000, np.uint64)
        index.query_device_batch(many.data_ptr(), 20000, out, ws)
        assert np.array_equal(out, np.tile(expected, 313)[:20000])
        assert ws.last_stats()["kernel_launches"] == 3
    finally:
        del held


# MB beside the estimates' buffers (about 340): with 160 the binary32 scan's sums of
# all queries, 480 MB, just fit in their place
@pytest.mark.parametrize("spare", [400, 160])
@pytest.mark.parametrize("captured", [False, True])
def test_open_queries_need_little_room(torch, captured, spare):
    # every query open
    rows, _, _ = _data(torch)
    rows[:500] = rows[0]
    index = uha.CudaExactL2Index(rows)
    queries = rows[0] + 0.001 * torch.rand(2000, D, device="cuda")
    plain = torch.rand(2000, D, device="cuda")
    torch.cuda.synchronize()
    if captured:
        batch = uha.QueryBatch([(index, 2000)], autotune=False)

        def ask(q):
            return batch.run([q.data_ptr()], on_device=True)[0][0]
    else:
        ws = index.make_query_workspace(2000)

        def ask(q):
            out = np.zeros(2000, np.uint64)
            index.query_device_batch(q.data_ptr(), 2000, out, ws)
            return out
    first = ask(plain)                          # the form and the buffers are there
    torch.cuda.empty_cache()
    held = _fill(torch, spare << 20)
    try:
        assert (ask(queries) == 0).all()
        assert (ask(queries) == 0).all()
        assert np.array_equal(ask(plain), first)
    finally:
        del held
