"""Host-side mirror of HGCalML's ``modules/local_distance_op.py`` on torch CUDA tensors."""
from __future__ import annotations

import torch

from . import _capi as C
from .binned_select_knn_op import SelectKnnGrad


def _local_distance(neighbour_idxs, coordinates):
    idx, coords = C.i32(neighbour_idxs), C.f32(coordinates)
    C.check_device(coords)
    out, rc = C.native.local_distance(idx, coords)
    C.check(rc, "LocalDistance")
    return out


class _LocalDistanceFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, coordinates, neighbour_idxs):
        dist = _local_distance(neighbour_idxs, coordinates)
        ctx.save_for_backward(coordinates, neighbour_idxs, dist)
        ctx.order = C.noted_order(neighbour_idxs)
        return dist

    @staticmethod
    def backward(ctx, grad_dist):
        coords, idx, dist = ctx.saved_tensors
        # the reference registers SelectKnnGrad as the gradient (modules/local_distance_op.py:27-40)
        return SelectKnnGrad(grad_dist, idx, dist, coords, order=ctx.order), None


def LocalDistance(coords, neighbour_idxs):
    """modules/local_distance_op.py:11-18: squared distances ``[V, K]`` from every hit to its listed
    neighbours (0 for -1 and for the hit itself), differentiable with respect to the coordinates
    through SelectKnnGrad as in the reference (:25-40)."""
    C.require_cuda(coords, neighbour_idxs)
    return _LocalDistanceFunction.apply(C.f32(coords), C.i32(neighbour_idxs))
