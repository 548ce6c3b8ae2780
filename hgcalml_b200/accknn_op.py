"""Host-side mirror of HGCalML's ``modules/accknn_op.py`` on torch CUDA tensors."""
from __future__ import annotations

import torch

from . import _capi as C


def _prepare(weights, features, indices):
    C.require_cuda(weights, features, indices)
    weights, features, indices = C.f32(weights), C.f32(features), C.i32(indices)
    n, k = indices.shape
    f = features.shape[1]
    if features.shape[0] != n or weights.shape[0] != n:
        raise C.HgcError("AccumulateKnnOp expects first dimensions of all inputs to match.")
    if weights.shape[1] != k:
        raise C.HgcError("AccumulateKnnOp expects second dimension of distance and neighbour index "
                         "tensor to match")
    C.check_device(features)
    return weights, features, indices


def AccumulateLinKnn(weights, features, indices, mean_and_max=True, force_tf=False, with_max_idxs=True, order=None):
    """Accumulates neighbour features with linear weights: the registered op ``AccumulateKnn``
    as is (modules/accknn_op.py:17-36, modules/compiled/accumulate_knn_module.cc:7-14).
    Returns ``(out_features [N, 2F or F], out_max_idxs [N, F])``."""
    del force_tf
    w, feat, idx = _prepare(weights, features, indices)
    out, maxidx, rc = C.native.accumulate(w, feat, idx, C.row_order(order, indices, idx.shape[0]), bool(mean_and_max),
                                          bool(with_max_idxs), False, 1.)
    C.check(rc, "AccumulateKnn")
    return out, maxidx


def AccumulateKnn(distances, features, indices, mean_and_max=True, force_tf=False, with_max_idxs=True,
                  order=None, distance_scale=1.):
    """modules/accknn_op.py:39-58: weights are ``exp(-distances)``, computed inside the kernel.

    Indices may be padded with trailing -1.  ``order`` (optional int32 permutation of the hits) only
    sets the order in which rows are processed; the bin-sorting permutation of BinnedSelectKnn keeps
    neighbouring hits together and makes the feature gather cache-friendly.  ``distance_scale`` is
    multiplied into the distances inside the kernel (``AccumulateKnn(10.*distsq, ..)`` of GravNet is
    ``distance_scale=10`` on the raw squared distances, without the extra elementwise pass)."""
    del force_tf
    d, feat, idx = _prepare(distances, features, indices)
    out, maxidx, rc = C.native.accumulate(d, feat, idx, C.row_order(order, indices, idx.shape[0]), bool(mean_and_max),
                                          bool(with_max_idxs), True, float(distance_scale))
    C.check(rc, "AccumulateKnn")
    return out, maxidx


def AccumulateKnnGrad(grad_from_out_features, distances, features, neigh_indices, max_feat_indices, order=None,
                      _lists=None):
    """The registered op ``AccumulateKnnGrad`` (modules/compiled/accumulate_knn_grad_module.cc:7-15), the
    gradient the reference attaches to the op ``AccumulateKnn`` (modules/accknn_op.py:71-90).
    ``distances`` are the forward op's weights.  ``order`` (optional int32 permutation of the hits, e.g.
    the sorting of ``BinnedSelectKnn``) only sets the order in which hits are processed.
    Returns ``(grad_distances [N,K], grad_features [N,F])``;
    mean-and-max mode is detected from the width of the incoming gradient, as in the reference."""
    C.require_cuda(grad_from_out_features, distances, features, neigh_indices)
    g, w, feat = C.f32(grad_from_out_features), C.f32(distances), C.f32(features)
    idx = C.i32(neigh_indices)
    n, k = idx.shape
    f = feat.shape[1]
    mean_and_max = g.shape[1] > f
    if mean_and_max:
        C.require_cuda(max_feat_indices)
        maxidx = C.i32(max_feat_indices)
    else:
        maxidx = None
    C.check_device(feat)
    gw, gf, ws, rc = C.native.accumulate_grad(g, w, feat, idx, maxidx, C.row_order(order, neigh_indices, n))
    C.check(rc, "AccumulateKnnGrad")
    if _lists is not None and n > 0 and k > 0:
        _lists.put(ws)
    return gw, gf


class _AccumulateLinKnnFunction(torch.autograd.Function):
    """AccumulateLinKnn with the reference's gradient wired into torch autograd."""

    @staticmethod
    def forward(ctx, weights, features, indices, mean_and_max, order):
        out, maxidx = AccumulateLinKnn(weights, features, indices, mean_and_max=mean_and_max, order=order)
        ctx.save_for_backward(weights, features, indices, maxidx)
        ctx.order = C.noted_order(indices) if order is None else order
        ctx.lists = C.noted_lists(indices) if ctx.needs_input_grad[0] else None  # else no search comes after
        ctx.mark_non_differentiable(maxidx)
        ctx.set_materialize_grads(False)  # no zeros for the arg-max output
        return out, maxidx

    @staticmethod
    def backward(ctx, grad_out, _grad_maxidx):
        if grad_out is None:
            return None, None, None, None, None
        weights, features, indices, maxidx = ctx.saved_tensors
        gw, gf = AccumulateKnnGrad(grad_out, weights, features, indices, maxidx, order=ctx.order, _lists=ctx.lists)
        return gw, gf, None, None, None


def AccumulateKnnDifferentiable(distances, features, indices, mean_and_max=True, order=None):
    """``AccumulateKnn`` as the reference's training path sees it: ``exp(-distances)`` as a
    differentiable tensor op, then the op with its registered gradient (modules/accknn_op.py:52-57,71-90).
    ``order``: optional processing order for the backward pass (see ``AccumulateKnnGrad``)."""
    return _AccumulateLinKnnFunction.apply(torch.exp(-distances), features, indices, mean_and_max, order)
