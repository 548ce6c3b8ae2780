"""Transposed neighbour lists and the kernels over them where they change shape: list lengths around the sizes
sorted in registers, hubs with thousands of incoming edges, feature widths around the slabs, K that is no power of
two, and a processing order.  Bit for bit against the CPU checker."""
import numpy as np
import pytest
import torch

from conftest import bits
from test_ops_gpu import T, N

pytestmark = pytest.mark.gpu


def _table(n, K, seed):
    """Random neighbours; some hits get exactly 0, 1, 31 .. 129 and thousands of incoming edges."""
    rng = np.random.default_rng(seed)
    idx = rng.integers(40, n, (n, K)).astype(np.int32)
    idx[rng.random((n, K)) < 0.1] = -1
    flat = idx.reshape(-1)
    at = rng.permutation(flat.size)
    for m, count in enumerate([0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 300, min(5000, flat.size // 3)]):
        flat[at[:count]] = m
        at = at[count:]
    idx[::7, 0] = np.arange(n)[::7]
    idx[::7, K - 1] = np.arange(n)[::7]  # the hit itself a second time
    return idx, rng


@pytest.mark.parametrize("n,K,F,mm", [(2500, 16, 64, True), (2500, 12, 65, True), (1500, 9, 130, True), (1500, 8, 31, True),
                                      (1500, 33, 33, False), (800, 1, 4, True)])
def test_accumulate_knn_grad(cuda, oracle, n, K, F, mm):
    from hgcalml_b200.accknn_op import AccumulateKnnGrad, AccumulateLinKnn
    idx, rng = _table(n, max(K, 2), n + K)
    idx = np.ascontiguousarray(idx[:, :K])
    feat = rng.standard_normal((n, F), dtype=np.float32)
    w = rng.random((n, K), dtype=np.float32)
    out, maxidx = AccumulateLinKnn(T(w, cuda), T(feat, cuda), T(idx, cuda), mean_and_max=mm)
    g = rng.standard_normal(tuple(out.shape), dtype=np.float32)
    rw, rf = oracle.op_accumulate_knn_grad(g, w, feat, idx, N(maxidx))
    order = T(rng.permutation(n).astype(np.int32), cuda)
    for o in (None, order):
        gw, gf = AccumulateKnnGrad(T(g, cuda), T(w, cuda), T(feat, cuda), T(idx, cuda), maxidx, order=o)
        assert np.array_equal(bits(N(gw)), bits(rw)) and np.array_equal(bits(N(gf)), bits(rf))


@pytest.mark.parametrize("n,K,F", [(2500, 16, 32), (1200, 7, 70), (600, 40, 3)])
def test_push_knn_and_gradients(cuda, oracle, n, K, F):
    from hgcalml_b200.push_knn_op import PushKnn, PushKnnGrad
    from hgcalml_b200.binned_select_knn_op import SelectKnnGrad
    idx, rng = _table(n, K, n)
    w = rng.random((n, K), dtype=np.float32)
    f, g = (rng.standard_normal((n, F), dtype=np.float32) for _ in range(2))
    c = rng.standard_normal((n, 4), dtype=np.float32)
    table = T(idx, cuda)
    order = T(rng.permutation(n).astype(np.int32), cuda)
    for o in (None, order):
        if o is not None:
            from hgcalml_b200 import _capi
            _capi.set_order(table, o)
        assert np.array_equal(bits(N(PushKnn(T(w, cuda), T(f, cuda), table))), bits(oracle.op_push_knn(w, f, idx)))
        rw, rf = oracle.op_push_knn_grad(g, w, f, idx)
        gw, gf = PushKnnGrad(T(g, cuda), T(w, cuda), T(f, cuda), table)
        assert np.array_equal(bits(N(gw)), bits(rw)) and np.array_equal(bits(N(gf)), bits(rf))
        ref = oracle.op_select_knn_grad(w, idx, c)
        assert np.array_equal(bits(N(SelectKnnGrad(T(w, cuda), table, None, T(c, cuda)))), bits(ref))


def test_search_notes_its_order(cuda):
    from hgcalml_b200 import _capi
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn, BinnedSelectKnnDifferentiable
    c = torch.rand((3000, 3), device=cuda)
    rs = torch.tensor([0, 3000], dtype=torch.int32, device=cuda)
    idx, _, sorting = BinnedSelectKnn(8, c, rs, return_sorting=True)
    assert torch.equal(_capi.order_of(idx, 3000), sorting)
    assert _capi.order_of(idx[:2000], 2000) is None and _capi.order_of(idx, 2999) is None
    idx, _ = BinnedSelectKnnDifferentiable(8, c.requires_grad_(True), rs)
    assert torch.equal(_capi.order_of(idx, 3000), sorting)


def test_backward_ops_share_lists_within_a_pass_only(cuda):
    """Gradients through both ops equal those of the ops called alone, pass after pass, also when the table changes
    hands between passes; nothing is kept after a pass."""
    from hgcalml_b200.accknn_op import AccumulateKnnDifferentiable, AccumulateKnnGrad
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnnDifferentiable, SelectKnnGrad
    g = torch.Generator(device=cuda).manual_seed(3)
    c = torch.rand((3000, 3), generator=g, device=cuda).requires_grad_(True)
    f = torch.randn((3000, 12), generator=g, device=cuda).requires_grad_(True)
    rs = torch.tensor([0, 1800, 3000], dtype=torch.int32, device=cuda)
    go = torch.randn((3000, 24), generator=g, device=cuda)
    idx, d2 = BinnedSelectKnnDifferentiable(14, c, rs)
    out, arg = AccumulateKnnDifferentiable(10. * d2, f, idx)
    w = torch.exp(-(10. * d2)).detach()
    gw, gf = AccumulateKnnGrad(go, w, f.detach(), idx, arg)
    gc = SelectKnnGrad(gw * -w * 10., idx, d2.detach(), c.detach())
    for _ in range(2):
        rc, rf = torch.autograd.grad(out, (c, f), go, retain_graph=True)
        assert torch.equal(rf, gf) and torch.allclose(rc, gc, rtol=1e-5, atol=1e-6)
        assert idx._hgc_lists.ws is None
    (rf,) = torch.autograd.grad(out, (f,), go, retain_graph=True)  # the search's gradient does not run
    assert torch.equal(rf, gf) and idx._hgc_lists.ws is None


@pytest.mark.parametrize("K", [3, 64])
def test_incoming_lists_around_the_longest_a_warp_sorts(cuda, oracle, K):
    """Lists of up to 256 and 512 edges are sorted by a warp, longer ones by a block; the gradient adds in list order."""
    from hgcalml_b200.binned_select_knn_op import SelectKnnGrad
    rng = np.random.default_rng(K)
    counts = [127, 128, 129, 255, 256, 257, 258, 511, 512, 513, 514, 1000, 2049]
    n = 9000 // K + 40
    flat = np.full(n * K, -1, np.int32)
    at = rng.permutation(flat.size)
    for m, count in enumerate(counts):
        flat[at[:count]] = m
        at = at[count:]
    flat[at[::3]] = rng.integers(len(counts), n, at[::3].size)
    idx = flat.reshape(n, K)
    assert (np.bincount(idx[idx >= 0], minlength=n)[:len(counts)] == counts).all()
    g, c = rng.standard_normal((n, K), dtype=np.float32), rng.standard_normal((n, 4), dtype=np.float32)
    got = SelectKnnGrad(T(g, cuda), T(idx, cuda), None, T(c, cuda))
    assert np.array_equal(bits(N(got)), bits(oracle.op_select_knn_grad(g, idx, c)))


@pytest.mark.parametrize("F", [1, 15, 16, 17])
def test_push_knn_grad_around_the_narrow_rows(cuda, oracle, F):
    from hgcalml_b200.push_knn_op import PushKnnGrad
    n, K = 900, 11
    idx, rng = _table(n, K, F)
    w = rng.random((n, K), dtype=np.float32)
    f, g = (rng.standard_normal((n, F), dtype=np.float32) for _ in range(2))
    rw, rf = oracle.op_push_knn_grad(g, w, f, idx)
    for o in (None, T(rng.permutation(n).astype(np.int32), cuda)):
        gw, gf = PushKnnGrad(T(g, cuda), T(w, cuda), T(f, cuda), T(idx, cuda), order=o)
        assert np.array_equal(bits(N(gw)), bits(rw)) and np.array_equal(bits(N(gf)), bits(rf))


@pytest.mark.parametrize("K", [8, 11])
@pytest.mark.parametrize("F", [2, 4, 16, 20, 36, 66, 68, 128])
def test_rows_of_whole_and_of_part_vectors(cuda, oracle, K, F):
    """Lanes per target change with the width (16, 32, 64); rows that are no whole vectors, lie off a 16-byte boundary or are
    divided by a K that is no power of two are copied first."""
    from hgcalml_b200.accknn_op import AccumulateKnnGrad, AccumulateLinKnn
    from hgcalml_b200.push_knn_op import PushKnn, PushKnnGrad
    n = 700
    idx, rng = _table(n, K, F)
    feat, grad = rng.standard_normal((n, F), dtype=np.float32), rng.standard_normal((n, 2 * F), dtype=np.float32)
    w = rng.random((n, K), dtype=np.float32)

    def shifted(a):
        flat = torch.empty(a.size + 1, dtype=torch.float32, device=cuda)
        return flat[1:].view(a.shape).copy_(T(a, cuda))
    table = T(idx, cuda)
    for put in (lambda a: T(a, cuda), shifted):
        _, maxidx = AccumulateLinKnn(T(w, cuda), T(feat, cuda), table)
        gw, gf = AccumulateKnnGrad(put(grad), put(w), put(feat), table, maxidx)
        rw, rf = oracle.op_accumulate_knn_grad(grad, w, feat, idx, N(maxidx))
        assert np.array_equal(bits(N(gw)), bits(rw)) and np.array_equal(bits(N(gf)), bits(rf))
        assert np.array_equal(bits(N(PushKnn(put(w), put(feat), table))), bits(oracle.op_push_knn(w, feat, idx)))
        g1 = np.ascontiguousarray(grad[:, :F])
        rw, rf = oracle.op_push_knn_grad(g1, w, feat, idx)
        gw, gf = PushKnnGrad(put(g1), put(w), put(feat), table)
        assert np.array_equal(bits(N(gw)), bits(rw)) and np.array_equal(bits(N(gf)), bits(rf))


@pytest.mark.parametrize("K", [1, 6, 8])
def test_select_knn_grad_over_the_range_of_floats(cuda, oracle, K):
    """Differences whose double is no float any more, subnormal ones, and gradients at both ends and of zero."""
    from hgcalml_b200.binned_select_knn_op import SelectKnnGrad
    n = 600
    rng = np.random.default_rng(K)
    idx = rng.integers(-1, n, (n, K)).astype(np.int32)
    powers = np.float32(2.) ** rng.integers(-149, 128, (2, n, max(K, 4))).astype(np.float32)
    c = (powers[0, :, :4] * rng.uniform(-1., 1., (n, 4))).astype(np.float32)
    c[::5], c[1::5] = np.float32(1.6e38), np.float32(-1.6e38)
    g = (powers[1, :, :K] * rng.uniform(-1., 1., (n, K))).astype(np.float32)
    g[::3] *= np.float32(1e-30)
    g[1::3] = 0.
    ref = oracle.op_select_knn_grad(g, idx, c)
    assert np.isfinite(ref).any() and (ref != 0.).any()
    got = N(SelectKnnGrad(T(g, cuda), T(idx, cuda), None, T(c, cuda)))
    nan = np.isnan(ref)
    assert np.array_equal(nan, np.isnan(got)) and np.array_equal(bits(got[~nan]), bits(ref[~nan]))


def _check_sums(cuda, oracle, idx, F, rng):
    from hgcalml_b200.accknn_op import AccumulateKnnGrad, AccumulateLinKnn
    from hgcalml_b200.push_knn_op import PushKnn
    n, K = idx.shape
    feat, grad = rng.standard_normal((n, F), dtype=np.float32), rng.standard_normal((n, 2 * F), dtype=np.float32)
    w = rng.random((n, K), dtype=np.float32)
    table, order = T(idx, cuda), T(rng.permutation(n).astype(np.int32), cuda)
    _, arg = AccumulateLinKnn(T(w, cuda), T(feat, cuda), table)
    for g, a in ((grad, arg), (np.ascontiguousarray(grad[:, F:]), None)):
        rw, rf = oracle.op_accumulate_knn_grad(g, w, feat, idx, N(arg))
        for o in (None, order):
            gw, gf = AccumulateKnnGrad(T(g, cuda), T(w, cuda), T(feat, cuda), table, a, order=o)
            assert np.array_equal(bits(N(gw)), bits(rw)) and np.array_equal(bits(N(gf)), bits(rf))
    assert np.array_equal(bits(N(PushKnn(T(w, cuda), T(feat, cuda), table))), bits(oracle.op_push_knn(w, feat, idx)))


def _hits(cuda, few):
    """On either side of the number of targets that fill the chip with two rows in flight each."""
    return 1300 if few else 2 * 16 * torch.cuda.get_device_properties(cuda).multi_processor_count + 17


@pytest.mark.parametrize("K,F", [(5, 16), (21, 64), (30, 32), (64, 6), (200, 66)])
@pytest.mark.parametrize("few", [True, False])
def test_sums_over_lists_that_whole_blocks_work_on(cuda, oracle, K, F, few):
    """Lists of more than 80, 127, five or six times K and 512 edges among shorter ones; the other targets of a block are dealt
    out again."""
    n, rng = _hits(cuda, few), np.random.default_rng(K)
    counts = [31, 80, 81, 5 * K, 5 * K + 1, 112, 113, 511, 512, 513, 527, 528, 529, 700]
    flat = rng.integers(-1, n, n * K).astype(np.int32)
    flat[np.isin(flat, rng.choice(n, n // 2, replace=False))] = -1  # half of the hits are nobody's neighbours
    flat[(flat >= 40) & (flat < 40 + 7 * len(counts))] = -1
    at = rng.permutation(flat.size)
    for i, count in enumerate(counts):  # between hits with short lists
        flat[at[:count]] = 40 + 7 * i
        at = at[count:]
    idx = flat.reshape(n, K)
    idx[40, 0] = idx[40, K - 1] = 40  # the hit itself twice
    _check_sums(cuda, oracle, idx, F, rng)


@pytest.mark.parametrize("K,F,every", [(40, 16, 4), (16, 32, 10), (16, 64, 6), (64, 64, 12), (64, 20, 12), (64, 16, 60), (24, 70, 50)])
@pytest.mark.parametrize("few", [True, False])
def test_sums_where_few_hits_are_neighbours(cuda, oracle, K, F, every, few):
    """Wide lists of both kinds, more of them than blocks, and blocks with few targets that have edges."""
    n, rng = _hits(cuda, few), np.random.default_rng(K + F)
    idx = rng.integers(0, n // every, (n, K)).astype(np.int32) * every
    idx[rng.random(idx.shape) < 0.05] = -1
    _check_sums(cuda, oracle, idx, F, rng)


@pytest.mark.parametrize("K", [1, 5, 8, 24])
@pytest.mark.parametrize("F", [3, 16, 30, 64, 70])
def test_no_op_leaves_its_workspace(cuda, oracle, K, F):
    from hgcalml_b200 import _capi as C
    from hgcalml_b200.accknn_op import AccumulateLinKnn
    n, L = 2100, C.lib
    idx, rng = _table(n, max(K, 2), F)
    idx = np.ascontiguousarray(idx[:, :K])
    feat, grad, w = (rng.standard_normal(s, dtype=np.float32) for s in ((n, F), (n, 2 * F), (n, K)))
    x, go, wt, table = T(feat, cuda), T(grad, cuda), T(w, cuda), T(idx, cuda)
    g1 = go[:, :F].contiguous()
    _, arg = AccumulateLinKnn(wt, x, table)
    coords = T(grad[:, :2].copy(), cuda)

    def call(need, fn, *outs):
        ws = torch.full((need + 4096,), 0xa5, dtype=torch.uint8, device=cuda)
        outs = [torch.empty(s, device=cuda) for s in outs]
        C.check(fn(ws, need, *[C.ptr(o) for o in outs], C.stream_of(ws)), "op")
        assert (ws[need:] == 0xa5).all()
        return [N(o) for o in outs]
    for mm, g in ((1, go), (0, g1)):
        gw, gf = call(L.hgc_accumulate_knn_grad_workspace_bytes(n, K, F, mm), lambda ws, b, gw, gf, s: L.hgc_accumulate_knn_grad(
            C.ptr(g), C.ptr(wt), C.ptr(x), C.ptr(arg) if mm else None, C.ptr(table), gw, gf, n, K, F, g.shape[1], 0, mm, C.ptr(ws), b, s), (n, K), (n, F))
        rw, rf = oracle.op_accumulate_knn_grad(N(g), w, feat, idx, N(arg))
        assert np.array_equal(bits(gw), bits(rw)) and np.array_equal(bits(gf), bits(rf))
    (out,) = call(L.hgc_push_knn_workspace_bytes(n, K, F), lambda ws, b, o, s: L.hgc_push_knn(
        C.ptr(wt), C.ptr(x), C.ptr(table), o, n, K, F, C.ptr(ws), b, s), (n, F))
    assert np.array_equal(bits(out), bits(oracle.op_push_knn(w, feat, idx)))
    (gc,) = call(L.hgc_select_knn_grad_workspace_bytes(n, K), lambda ws, b, o, s: L.hgc_select_knn_grad(
        C.ptr(wt), C.ptr(table), None, C.ptr(coords), o, n, K, 2, C.ptr(ws), b, s), (n, 2))
    assert np.array_equal(bits(gc), bits(oracle.op_select_knn_grad(w, idx, N(coords))))
