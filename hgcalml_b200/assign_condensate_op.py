"""Host-side mirror of HGCalML's ``modules/assign_condensate_op.py`` on torch CUDA tensors."""
from __future__ import annotations

import math

import torch

from . import _capi as C
from .bin_by_coordinates_op import BinByCoordinates


def _BinnedAssignToCondensates(ccoords, dist, beta, no_condensation_mask, bins_flat, bin_splits,
                               indices_to_filtered, original_indices, row_splits, n_bins, bin_widths,
                               ccoords_h, dist_h, beta_h, no_condensation_mask_h, row_splits_h,
                               beta_threshold=0., assign_by_max_beta=True):
    """The registered op ``BinnedAssignToCondensates``
    (modules/compiled/binned_assign_to_condensates_module.cc:7-31), inputs in bin-sorted order.
    Returns ``assigned_h, assigned, alpha_indices, association, n_condensates``."""
    del beta_threshold, bins_flat  # attributes / inputs the reference kernel never reads
    C.require_cuda(ccoords, dist, beta, ccoords_h)
    ccoords, ccoords_h = C.f32(ccoords), C.f32(ccoords_h)
    dev = ccoords.device
    n, dims = ccoords.shape
    dist, dist_h, beta_h = C.f32(dist).reshape(-1), C.f32(dist_h).reshape(-1), C.f32(beta_h).reshape(-1)
    mask, mask_h = C.i32(no_condensation_mask).reshape(-1), C.i32(no_condensation_mask_h).reshape(-1)
    itf, orig_h = C.i32(indices_to_filtered), C.i32(original_indices)
    row_splits, row_splits_h = C.i32(row_splits, dev), C.i32(row_splits_h, dev)
    bin_splits, n_bins, bin_widths = C.i32(bin_splits), C.i32(n_bins, dev), C.f32(bin_widths, dev)
    nh = beta_h.shape[0]
    num_rows = row_splits.shape[0] - 1
    assigned_h = torch.empty((nh,), dtype=torch.int32, device=dev)
    assigned = torch.empty((n,), dtype=torch.int32, device=dev)
    alpha = torch.empty((nh,), dtype=torch.int32, device=dev)
    asso = torch.empty((n,), dtype=torch.int32, device=dev)
    ncond = torch.empty((num_rows + 1,), dtype=torch.int32, device=dev)
    ws = C.workspace(C.lib.hgc_binned_assign_to_condensates_workspace_bytes(n, nh, num_rows, dims), dev)
    C.check(C.lib.hgc_binned_assign_to_condensates(
        dims, n_bins.shape[0], C.ptr(ccoords_h), C.ptr(dist_h), C.ptr(beta_h), C.ptr(mask_h),
        C.ptr(assigned_h), C.ptr(orig_h), C.ptr(row_splits_h), C.ptr(ccoords), C.ptr(dist), C.ptr(mask),
        C.ptr(itf), C.ptr(assigned), C.ptr(asso), C.ptr(ncond), C.ptr(alpha), C.ptr(bin_splits),
        C.ptr(n_bins), C.ptr(bin_widths), C.ptr(row_splits), num_rows, n, nh,
        int(bool(assign_by_max_beta)), C.ptr(ws), ws.numel(), C.stream_of(ccoords)),
        "BinnedAssignToCondensates")
    return assigned_h, assigned, alpha, asso, ncond


def merge_noise_as_indiv_cp(assignment, asso_idx, alpha_idx, is_cond, n_condensates, row_splits):
    """modules/assign_condensate_op.py:16-44: every noise hit (assignment < 0) becomes a condensation
    point of its own.  Per event the noise hits take the shower numbers 0..n_noise-1 in hit order and
    the real showers are shifted up by n_noise; ``alpha_idx`` lists, per event, the noise hits first
    and then the condensates; noise hits are associated to themselves and flagged as condensates."""
    C.require_cuda(assignment, asso_idx, alpha_idx, is_cond, n_condensates)
    dev = assignment.device
    assignment, asso_idx, alpha_idx = C.i32(assignment).reshape(-1), C.i32(asso_idx, dev), C.i32(alpha_idx, dev)
    is_cond = is_cond.to(dev, torch.bool).contiguous().reshape(-1)
    n_condensates, row_splits = C.i32(n_condensates, dev), C.i32(row_splits, dev)
    n, n_rs = assignment.shape[0], row_splits.shape[0]
    if asso_idx.numel() != n or is_cond.numel() != n:
        raise C.HgcError("merge_noise_as_indiv_cp: assignment, asso_idx and is_cond must have one entry per hit")
    if n_condensates.shape[0] != n_rs:
        raise C.HgcError("merge_noise_as_indiv_cp: n_condensates must have an entry per row split")
    counts = n_condensates.cpu()  # the kernels go by them
    if (counts[1:] < counts[:-1]).any() or counts[-1] - counts[0] > min(alpha_idx.numel(), n):
        raise C.HgcError("merge_noise_as_indiv_cp: n_condensates must ascend, up to the length of alpha_idx")
    return _merge_noise(assignment, asso_idx, alpha_idx, is_cond, n_condensates, row_splits)


def _merge_noise(assignment, asso, alpha, is_cond, n_condensates, row_splits):
    # alpha may be longer than the list of condensates: its length is n_condensates[-1]
    C.check_device(assignment)
    new, cond, n_cond, n_alpha, rc = C.native.merge_noise(assignment, asso, alpha, is_cond, n_condensates, row_splits)
    C.check(rc, "merge_noise_as_indiv_cp")
    if n_alpha < 0:
        raise C.HgcError("merge_noise_as_indiv_cp: the row splits must ascend and cover all hits")
    return new[0][:, None], new[1], new[2:].reshape(-1)[:n_alpha], cond[:, None], n_cond


def _segment_ids_to_row_splits(ids, num_segments):
    counts = torch.bincount(ids.to(torch.int64), minlength=num_segments)
    return torch.cat([torch.zeros(1, dtype=torch.int64, device=ids.device), counts.cumsum(0)]).to(torch.int32)


def BuildAndAssignCondensatesBinned(ccoords, betas, dist, row_splits, beta_threshold,
                                    no_condensation_mask=None, distance_threshold=1.,
                                    assign_by_max_beta=False, nbin_dims=3, keep_noise=False):
    """modules/assign_condensate_op.py:210-373.

    Returns ``assignment [N,1], association [N], alpha_idx, is_cond [N,1], n_condensates`` with the
    reference's meaning.  Everything up to ``keep_noise`` is one library call
    (``hgc_build_and_assign_condensates``: threshold scaling, shift, binning, stable sort by bin,
    high-beta filter, the op, mapping back); the ``keep_noise`` renumbering is a second one."""
    assert 1 <= nbin_dims <= 6
    assert 0. <= beta_threshold <= 1.
    assert distance_threshold > 0.
    ccoords = C.f32(ccoords)
    C.require_cuda(ccoords)
    dev = ccoords.device
    n, dims = ccoords.shape
    betas = C.f32(betas, dev).reshape(-1)
    dist = C.f32(dist, dev).reshape(-1)
    row_splits = C.i32(row_splits, dev)
    n_rs = row_splits.shape[0]
    if betas.shape[0] != n or dist.shape[0] != n:
        raise C.HgcError("BuildAndAssignCondensatesBinned: ccoords, betas and dist must have one row per hit")
    mask = None
    if no_condensation_mask is not None:
        mask = C.i32(no_condensation_mask, dev).reshape(-1)
    C.check_device(ccoords)
    # the number of condensates is not needed in between when the noise comes after
    assignment, asso, alpha, is_cond, n_condensates, n_alpha, rc = C.native.condensates(
        ccoords, betas, dist, mask, row_splits, float(beta_threshold), float(distance_threshold), bool(assign_by_max_beta),
        nbin_dims, not keep_noise)
    C.check(rc, "BuildAndAssignCondensatesBinned")
    if keep_noise:
        return _merge_noise(assignment, asso, alpha, is_cond, n_condensates, row_splits)
    return assignment[:, None], asso, alpha[:n_alpha], is_cond[:, None], n_condensates


def BuildAndAssignCondensatesBinnedStepwise(ccoords, betas, dist, row_splits, beta_threshold,
                                            no_condensation_mask=None, distance_threshold=1.,
                                            assign_by_max_beta=False, nbin_dims=3, keep_noise=False):
    """The same function with the reference's tensor glue (modules/assign_condensate_op.py:245-310)
    spelled out step by step on CUDA tensors around the registered op ``_BinnedAssignToCondensates``;
    kept as the readable statement of what the one-call version does."""
    assert 1 <= nbin_dims <= 6
    assert 0. <= beta_threshold <= 1.
    assert distance_threshold > 0.
    ccoords = C.f32(ccoords)
    C.require_cuda(ccoords)
    dev = ccoords.device
    betas = C.f32(betas, dev).reshape(-1, 1)
    dist = C.f32(dist, dev).reshape(-1, 1) / distance_threshold
    row_splits = C.i32(row_splits, dev)
    num_rows = row_splits.shape[0] - 1
    n = ccoords.shape[0]
    if no_condensation_mask is None:
        no_condensation_mask = torch.zeros((n, 1), dtype=torch.int32, device=dev)
    mask = C.i32(no_condensation_mask, dev).reshape(-1, 1)

    rs_host = row_splits.cpu()
    nvertmax = int(rs_host[-1] - rs_host[0])
    n_bins_sc = max(4, min(int(math.ceil(math.pow(nvertmax / 5, 1 / 3))), 25))
    ccoords = ccoords - ccoords.min(dim=0, keepdim=True).values
    ccoords_2 = ccoords[:, 0:min(ccoords.shape[1], nbin_dims)].contiguous()
    _, bins_flat, n_bins, bin_width = BinByCoordinates(ccoords_2, row_splits, n_bins=n_bins_sc,
                                                       calc_n_per_bin=False, pre_normalized=True)
    sorting = torch.sort(bins_flat, stable=True).indices
    sorting_back = torch.empty_like(sorting)
    sorting_back[sorting] = torch.arange(n, device=dev)
    ccoords, betas, dist, mask = ccoords[sorting], betas[sorting], dist[sorting], mask[sorting]
    bins_flat = bins_flat[sorting]
    orig = sorting.to(torch.int32)
    total_bins = int(torch.prod(n_bins.cpu().to(torch.int64))) * num_rows
    bin_splits = _segment_ids_to_row_splits(bins_flat, total_bins)

    high = torch.logical_or(betas > beta_threshold, mask > 0)[:, 0]
    seg = torch.repeat_interleave(torch.arange(num_rows, device=dev),
                                  (row_splits[1:] - row_splits[:-1]).to(torch.int64))
    row_splits_h = _segment_ids_to_row_splits(seg[high], num_rows)
    betas_h, ccoords_h, dist_h = betas[high], ccoords[high], dist[high]
    mask_h, orig_h = mask[high], orig[high]
    nh = int(betas_h.shape[0])
    itf = torch.full((n,), -1, dtype=torch.int32, device=dev)
    itf[high] = torch.arange(nh, dtype=torch.int32, device=dev)

    _, assignment, alpha, asso, n_condensates = _BinnedAssignToCondensates(
        ccoords=ccoords, dist=dist, beta=betas, no_condensation_mask=mask, bins_flat=bins_flat,
        bin_splits=bin_splits, indices_to_filtered=itf, original_indices=orig_h, row_splits=row_splits,
        n_bins=n_bins, bin_widths=bin_width, ccoords_h=ccoords_h, dist_h=dist_h, beta_h=betas_h,
        no_condensation_mask_h=mask_h, row_splits_h=row_splits_h, beta_threshold=beta_threshold,
        assign_by_max_beta=assign_by_max_beta)

    assignment = assignment[sorting_back]
    asso = asso[sorting_back]
    alpha_idx = alpha[alpha != -1]
    is_cond = torch.zeros((n,), dtype=torch.bool, device=dev)
    is_cond[alpha_idx.to(torch.int64)] = True
    out = (assignment[:, None], asso, alpha_idx, is_cond[:, None], n_condensates)
    if keep_noise:
        out = merge_noise_as_indiv_cp(*out, row_splits)
    return out
