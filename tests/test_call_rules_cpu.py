"""Rules of the Python layer that hold without a GPU."""
import copy
import io

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
    assert C.order_of(idx, 50, note) is None  # as a backward pass asks


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
