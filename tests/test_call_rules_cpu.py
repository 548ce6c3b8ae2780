"""Rules of the Python layer that hold without a GPU."""
import copy
import gc
import io
import threading
import weakref

import pytest
import torch


def _table(n=50, k=4):
    from hgcalml_b200 import _capi as C
    idx, order = torch.zeros((n, k), dtype=torch.int32), torch.randperm(n).to(torch.int32)
    C.set_order(idx, order)
    return C, idx, order


def test_a_noted_order_that_was_written_to_is_not_used():
    """A caller may do with the sorting as they like, for instance add an offset to it: what is left is no order of
    the table's rows, and its entries lie outside it."""
    C, idx, order = _table()
    note = C.noted_order(idx)
    assert C.order_of(idx, 50) is order
    order += 1000
    assert C.order_of(idx, 50) is None
    assert C.row_order(note, idx, 50) is None  # as a backward pass asks


def test_a_table_with_notes_can_be_saved_and_copied():
    C, idx, order = _table()
    idx._hgc_lists = C.BackwardLists(idx)
    file = io.BytesIO()
    torch.save(idx, file)
    file.seek(0)
    for other in (torch.load(file, weights_only=True), copy.deepcopy(idx)):
        assert torch.equal(other, idx)
        assert C.noted_order(other) is None and C.order_of(other, 50) is None and C.noted_lists(other) is None


def test_backward_lists_belong_to_the_table_as_the_search_left_it():
    C, idx, order = _table()
    idx._hgc_lists = C.BackwardLists(idx)
    assert C.noted_lists(idx) is idx._hgc_lists
    idx[:, 2] = -1
    assert C.noted_lists(idx) is None


def test_pipelines_given_up_by_the_garbage_collector_wait_for_nothing(monkeypatch):
    """A collection may start at any allocation, also at one that taking streams from the pool makes; the pipelines that
    it finalises give their streams to the same pool from the same thread."""
    from hgcalml_b200 import pipeline as P
    monkeypatch.setattr(P, "_idle_streams", {})
    monkeypatch.setattr(torch.cuda, "Stream", lambda device: object())

    class Pipeline:
        def __init__(self, key):
            self.me = self  # only a collection finds it
            weakref.finalize(self, P._give_streams, key, P._take_streams(key)).atexit = False

    taken = []

    def use():
        threshold = gc.get_threshold()
        gc.set_threshold(1)
        try:
            for key in ["a", "b", "c"] * 20:
                Pipeline(key)
                taken.append(P._take_streams(key + "x"))
        finally:
            gc.set_threshold(*threshold)

    thread = threading.Thread(target=use, daemon=True)
    thread.start()
    thread.join(20.)
    assert not thread.is_alive() and len(taken) == 60
    gc.collect()
    idle = [s for pool in P._idle_streams.values() for s in pool]
    assert len(set(map(id, idle))) == len(idle)  # no triple is there twice


@pytest.mark.parametrize("precision", ["tf32", "ieee", "none"])
@pytest.mark.parametrize("where", [torch.backends, torch.backends.cuda.matmul], ids=["everywhere", "products"])
def test_a_precision_chosen_by_the_caller_is_no_error(where, precision):
    """Asked about a layer, the host binding leaves it to the tensor operations and raises nothing."""
    from hgcalml_b200 import _capi as C
    before = where.fp32_precision
    try:
        where.fp32_precision = precision
        got, rc = C.native.dense(torch.ones((8, 4)), torch.ones((4, 4)), None, True)
    finally:
        where.fp32_precision = before
    assert got is None and rc == C.NOT_TAKEN
