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
    second = kind(rows)
    assert _ask(second, queries, expected) == 3   # and none for a form
    assert _ask(first, queries, expected) == 3
    del held, second
    torch.cuda.empty_cache()
    third = kind(rows)
    assert _ask(third, queries, expected) > 3


def test_a_form_in_use_stays(torch):
    rows, expected, queries = _data(torch)
    index = uha.CudaExactL2Index(rows)
    batch = uha.QueryBatch([(index, 64)], autotune=False)
    held = _fill(torch, FORM - (FORM >> 2))
    with pytest.raises(uha.CudaRuntimeError):
        uha.CudaExactL2Index(rows)
    # the captured scan still reads it
    assert np.array_equal(batch.run([queries.data_ptr()], on_device=True)[0][0], expected)
    del batch
    other = uha.CudaExactL2Index(rows)            # now it is given back
    del held
    torch.cuda.empty_cache()
    assert _ask(other, queries, expected) > 3


def test_a_form_takes_at_most_half_of_what_is_free(torch):
    rows, expected, queries = _data(torch)
    index = uha.CudaExactL2Index(rows)
    held = _fill(torch, 2 * FORM - (FORM >> 2))
    assert _ask(index, queries, expected) == 3
    del held
    torch.cuda.empty_cache()
    # decided once per index
    assert _ask(index, queries, expected) == 3
    other = uha.CudaExactL2Index(rows)
    assert _ask(other, queries, expected) > 3
