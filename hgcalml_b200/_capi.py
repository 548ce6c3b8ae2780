"""ctypes binding of libhgcalml_b200.so (the C ABI declared in include/hgcalml_b200.h).

There is no fallback: if the shared library is missing the import of any op fails with a clear
error, and every entry point raises when the library reports a non-zero status.
"""
from __future__ import annotations

import collections
import ctypes
import os
from ctypes import c_int, c_size_t, c_void_p

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libhgcalml_b200.so")

HGC_OK = 0
NOT_TAKEN = 1  # of the host binding: the arguments want the tensor operations
STATUS_BITS = {1: "bin index out of range", 2: "flat bin index overflow",
               4: "gathered index out of range", 8: "iteration cap reached"}


class HgcError(RuntimeError):
    pass


def _load():
    if not os.path.exists(LIB_PATH):
        raise ImportError(
            f"{LIB_PATH} not found: build it with `make -C {os.path.join(_HERE, 'csrc')}` "
            "(or __graft_entry__.build()); hgcalml_b200 has no CPU or eager fallback")
    lib = ctypes.CDLL(LIB_PATH)
    P, I, S = c_void_p, c_int, c_size_t
    sig = {
        "hgc_strerror": (ctypes.c_char_p, [I]),
        "hgc_last_cuda_error": (ctypes.c_char_p, []),
        "hgc_version": (I, []),
        "hgc_launch_count": (ctypes.c_ulonglong, []),
        "hgc_workspace_status": (I, [P, P, ctypes.POINTER(ctypes.c_uint)]),
        "hgc_bin_by_coordinates_workspace_bytes": (S, [I, I, I, I]),
        "hgc_bin_by_coordinates": (I, [P, P, P, P, P, P, P, I, I, I, I, I, P, S, P]),
        "hgc_binned_select_knn_workspace_bytes": (S, [I, I, I, I]),
        "hgc_binned_select_knn": (I, [P] * 9 + [I] * 7 + [P, S, P]),
        "hgc_binned_select_knn_static": (I, [P] * 9 + [I] * 7 + [P]),
        "hgc_binned_select_knn_static_status": (I, [P, ctypes.POINTER(ctypes.c_uint)]),
        "hgc_index_replacer": (I, [P, P, P, I, I, P, P]),
        "hgc_accumulate_knn": (I, [P] * 5 + [I] * 6 + [P]),
        "hgc_accumulate_knn_ordered": (I, [P] * 5 + [I] * 6 + [P, P]),
        "hgc_accumulate_knn_exp": (I, [P] * 5 + [I] * 5 + [ctypes.c_float, P, P]),
        "hgc_gravnet_collect": (I, [P, P, I, I, I, P, P, I, P, I, I, ctypes.c_float, I, P, P]),
        "hgc_dense": (I, [P] * 4 + [I] * 4 + [P]),
        "hgc_bias_act": (I, [P, P, I, I, I, P]),
        "hgc_copy_columns": (I, [P, P, I, I, I, P]),
        "hgc_binned_select_knn_ragged_workspace_bytes": (S, [I] * 6),
        "hgc_binned_select_knn_ragged": (I, [P] * 6 + [I] * 8 + [P, S, P]),
        "hgc_build_and_assign_condensates_workspace_bytes": (S, [I] * 4),
        "hgc_build_and_assign_condensates": (I, [P] * 11 + [I] * 3 + [ctypes.c_float] * 2 + [I] * 2 + [P, S, P]),
        "hgc_merge_noise_workspace_bytes": (S, [I, I]),
        "hgc_merge_noise": (I, [P] * 12 + [I, I] + [P, S, P]),
        "hgc_local_distance": (I, [P, P, P, I, I, I, I, P]),
        "hgc_push_knn": (I, [P, P, P, P, I, I, I, P, S, P]),
        "hgc_push_knn_ordered": (I, [P, P, P, P, I, I, I, P, P, S, P]),
        "hgc_push_knn_grad": (I, [P] * 6 + [I] * 3 + [P]),
        "hgc_push_knn_grad_ordered": (I, [P] * 6 + [I] * 3 + [P, P]),
        "hgc_knn_grad_workspace_bytes": (S, [I, I]),
        "hgc_accumulate_knn_grad_workspace_bytes": (S, [I] * 4),
        "hgc_select_knn_grad_workspace_bytes": (S, [I, I]),
        "hgc_push_knn_workspace_bytes": (S, [I] * 3),
        "hgc_accumulate_knn_grad": (I, [P] * 7 + [I] * 6 + [P, S, P]),
        "hgc_accumulate_knn_grad_ordered": (I, [P] * 7 + [I] * 6 + [P, P, S, P]),
        "hgc_select_knn_grad": (I, [P] * 5 + [I] * 3 + [P, S, P]),
        "hgc_select_knn_grad_ordered": (I, [P] * 5 + [I] * 3 + [P, P, S, P]),
        "hgc_select_knn_grad_after": (I, [P] * 5 + [I] * 3 + [P, P, S, P]),
        "hgc_binned_assign_to_condensates_workspace_bytes": (S, [I] * 4),
        "hgc_binned_assign_to_condensates": (I, [I, I] + [P] * 4 + [P] + [P] * 2 + [P] * 4 + [P] * 4 + [P] * 3
                                             + [P, I, I, I, I] + [P, S, P]),
    }
    for name, (res, args) in sig.items():
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    return lib


lib = _load()

try:
    from . import _native as native  # noqa: F401  (host binding of the most frequent ops, links against `lib`)
except ImportError as e:
    raise ImportError(f"{os.path.join(_HERE, '_native.so')} cannot be loaded ({e}): build it with "
                      f"`make -C {os.path.join(_HERE, 'csrc')}` (or __graft_entry__.build())") from e

EXPORTED = [n for n in dir(lib) if n.startswith("hgc_")]


def check(rc: int, what: str) -> None:
    if rc != HGC_OK:
        msg = lib.hgc_strerror(rc).decode()
        if rc == -4:
            msg += ": " + lib.hgc_last_cuda_error().decode()
        raise HgcError(f"{what}: {msg} ({rc})")


def ptr(t):
    """Device pointer of a tensor (None -> NULL)."""
    return None if t is None else t.data_ptr()


_raw_stream = torch._C._cuda_getCurrentRawStream if hasattr(torch._C, "_cuda_getCurrentRawStream") else \
    lambda index: torch.cuda.current_stream(index).cuda_stream


def check_device(t: torch.Tensor) -> int:
    """The library launches on the calling thread's current device, so that device must be the tensor's."""
    index = t.get_device()
    if index != torch.cuda.current_device():
        raise HgcError(f"tensors live on {t.device} but the current CUDA device is "
                       f"cuda:{torch.cuda.current_device()}: call torch.cuda.set_device (or use "
                       "torch.cuda.device) before calling hgcalml_b200 ops")
    return index


def stream_of(t: torch.Tensor):
    """The current stream of the tensor's device."""
    return _raw_stream(check_device(t))


def workspace(nbytes: int, device) -> torch.Tensor:
    return torch.empty((max(int(nbytes), 256),), dtype=torch.uint8, device=device)


def read_status(ws: torch.Tensor, raise_on_flag: bool = True) -> int:
    """Synchronising read of the status word a call left in its workspace."""
    out = ctypes.c_uint(0)
    rc = lib.hgc_workspace_status(ptr(ws), stream_of(ws), ctypes.byref(out))
    if rc not in (0, -5):
        check(rc, "hgc_workspace_status")
    if out.value and raise_on_flag:
        names = [v for k, v in STATUS_BITS.items() if out.value & k]
        raise HgcError("device status: " + ", ".join(names))
    return out.value


def _as(t, dtype, device):
    # the usual argument is a dense tensor of the right type and needs no call into torch
    if isinstance(t, torch.Tensor) and t.dtype is dtype and t.is_contiguous() and (device is None or t.device == device):
        return t
    return torch.as_tensor(t, device=device).to(dtype).contiguous()


def f32(t, device=None):
    return _as(t, torch.float32, device)


def i32(t, device=None):
    return _as(t, torch.int32, device)


def version_of(t: torch.Tensor):
    """Counts the changes made to a tensor in place; None where they are not counted (inference tensors)."""
    return None if t.is_inference() else t._version


class _Note:
    """Something kept in an attribute of a neighbour table.  Copies and files of a tensor take its attributes along; of
    a note they get an empty dictionary, which every reader of tensor files accepts and the lookups below ignore."""
    __slots__ = ()

    def __reduce_ex__(self, protocol):
        return collections.OrderedDict, ()


def _noted(idx, name: str, kind):
    note = getattr(idx, name, None)
    return note if type(note) is kind else None


class RowOrder(_Note):
    """An order noted with a neighbour table."""
    __slots__ = ("order", "n", "device", "version", "stream")

    def __init__(self, order: torch.Tensor):
        self.order, self.n, self.device, self.version = order, order.shape[0], order.device, version_of(order)
        self.stream = _raw_stream(order.get_device()) if order.is_cuda else None

    def get(self, idx, n: int):
        """The order, unless it belongs to other rows or has been written to since it was noted.  A caller that uses
        the table on a second stream can see to the table's memory but not to the order's, so that is done here."""
        order = self.order
        if self.n != n or idx.shape[0] != n or idx.device != self.device or \
                self.version is not None and self.version != order._version:
            return None
        if self.stream is not None and _raw_stream(self.device.index) != self.stream:
            order.record_stream(torch.cuda.current_stream(self.device))
        return order


def set_order(idx: torch.Tensor, order: torch.Tensor):
    """Notes with a neighbour table the order in which its rows are best processed (the search's sorting of the
    hits).  Ops that gather or scatter along the table look it up when the caller names no order; results do
    not depend on it, and a table without one (a slice, a copy) is processed row by row."""
    idx._hgc_order = RowOrder(order)


def noted_order(idx):
    """What set_order noted, for a backward pass, which sees another view of the table."""
    return _noted(idx, "_hgc_order", RowOrder)


def order_of(idx, n: int):
    note = noted_order(idx)
    return None if note is None else note.get(idx, n)


def row_order(order, idx, n: int):
    """The processing order the caller names (backward passes name the note of the forward pass), else the one noted
    with the neighbour table, if any."""
    if order is None:
        return order_of(idx, n)
    if type(order) is RowOrder:
        return order.get(idx, n)
    require_cuda(order)
    if order.numel() != n or order.device != idx.device:
        raise HgcError(f"order must be a permutation of the {n} hits on {idx.device}, not {order.numel()} entries on "
                       f"{order.device}")
    return i32(order)


class BackwardLists(_Note):
    """Hands the transposed neighbour table from one backward op to a later one of the same backward pass.
    One such object belongs to one differentiable search call and is noted with its table; an op whose forward pass got
    that table, unchanged, joins it (autograd itself sees to it that the table stays as it was from then on).  The
    lists are good on the stream they were built on; the autograd engine empties the object when the pass ends."""
    __slots__ = ("version", "ws", "stream")

    def __init__(self, idx):
        self.version = version_of(idx)
        self.clear()

    def clear(self):
        self.ws = self.stream = None

    def put(self, ws):
        try:
            torch.autograd.Variable._execution_engine.queue_callback(self.clear)
        except RuntimeError:
            return  # not inside a backward pass
        self.ws, self.stream = ws, stream_of(ws)

    def take(self):
        ws, stream = self.ws, self.stream
        self.clear()
        return ws if ws is not None and stream == stream_of(ws) else None


def noted_lists(idx):
    """The lists of the search that this table came from, unless it was written to since."""
    lists = _noted(idx, "_hgc_lists", BackwardLists)
    return lists if lists is not None and lists.version is not None and lists.version == version_of(idx) else None


def require_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise HgcError("hgcalml_b200 ops take CUDA tensors; there is no CPU path")
