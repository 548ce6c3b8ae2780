"""What the Python layer must refuse or leave alone before it hands raw pointers to the library."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrong", ["host", "short", "long"])
def test_an_order_that_does_not_fit_the_table_is_refused(cuda, wrong):
    from hgcalml_b200 import _capi as C
    from hgcalml_b200.accknn_op import AccumulateKnn, AccumulateKnnDifferentiable, AccumulateKnnGrad, AccumulateLinKnn
    from hgcalml_b200.binned_select_knn_op import SelectKnnGrad
    from hgcalml_b200.GravNetLayersRagged import collect_neighbours
    from hgcalml_b200.push_knn_op import PushKnnGrad
    n, k, f = 100, 4, 8
    idx = torch.randint(0, n, (n, k), dtype=torch.int32, device=cuda)
    w, x, c = torch.rand((n, k), device=cuda), torch.randn((n, f), device=cuda), torch.randn((n, 3), device=cuda)
    good = torch.randperm(n, device=cuda).to(torch.int32)
    order = {"host": good.cpu(), "short": good[:n - 1], "long": torch.cat([good, good[:1]])}[wrong]
    _, arg = AccumulateLinKnn(w, x, idx)
    calls = [lambda o: AccumulateKnn(w, x, idx, order=o), lambda o: AccumulateLinKnn(w, x, idx, order=o),
             lambda o: AccumulateKnnDifferentiable(w, x, idx, order=o),
             lambda o: AccumulateKnnGrad(torch.cat([x, x], 1), w, x, idx, arg, order=o),
             lambda o: SelectKnnGrad(w, idx, None, c, order=o), lambda o: PushKnnGrad(x, w, x, idx, order=o),
             lambda o: collect_neighbours(x, idx, w, order=o)]
    for call in calls:
        with pytest.raises(C.HgcError):
            call(order)
        call(good[:, None])  # any shape that holds the n entries is taken


def test_a_sorting_whose_changes_are_not_counted_is_not_noted(cuda):
    from hgcalml_b200 import _capi as C
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn
    c, rs = torch.rand((300, 3), device=cuda), torch.tensor([0, 300], dtype=torch.int32, device=cuda)
    with torch.inference_mode():
        idx, _, sorting = BinnedSelectKnn(8, c, rs, return_sorting=True)
        assert C.order_of(idx, 300) is None
        idx, _ = BinnedSelectKnn(8, c, rs)  # no one else has it
        assert torch.equal(C.order_of(idx, 300), sorting)
    idx, _, sorting = BinnedSelectKnn(8, c, rs, return_sorting=True)
    assert C.order_of(idx, 300) is not None
    sorting += 300
    assert C.order_of(idx, 300) is None


def test_a_noted_order_lives_as_long_as_another_stream_needs_it(cuda):
    """The table goes out of use on the host while a second stream has yet to read it: the memory of the order that was
    noted with it must not be handed out on the first stream before that."""
    from hgcalml_b200.accknn_op import AccumulateKnn
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn
    n = 300001  # a size that nothing else here allocates
    c, rs = torch.rand((n, 3), device=cuda), torch.tensor([0, n], dtype=torch.int32, device=cuda)
    x = torch.randn((n, 8), device=cuda)
    idx, d2, sorting = BinnedSelectKnn(8, c, rs, return_sorting=True)
    want = AccumulateKnn(d2, x, idx)[0]
    where = sorting.data_ptr()
    del sorting
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)  # about 0.1 s
        got, _ = AccumulateKnn(d2, x, idx)
        for t in (idx, d2, x):
            t.record_stream(side)
    del idx, d2
    new = [torch.empty((n,), dtype=torch.int32, device=cuda) for _ in range(8)]
    assert not side.query() and where not in [t.data_ptr() for t in new]
    side.synchronize()
    assert torch.equal(got, want)


def test_backward_lists_are_of_the_table_that_the_search_made(cuda):
    """The accumulation runs on a table that was written to, and what both ops saved comes back as copies of that time:
    the lists of the changed table are not those of the search."""
    from hgcalml_b200.accknn_op import AccumulateKnnDifferentiable
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnnDifferentiable, SelectKnnGrad
    g = torch.Generator(device=cuda).manual_seed(5)
    c = torch.rand((4000, 3), generator=g, device=cuda).requires_grad_(True)
    f = torch.randn((4000, 8), generator=g, device=cuda)
    rs = torch.tensor([0, 4000], dtype=torch.int32, device=cuda)
    go = torch.randn((4000, 16), generator=g, device=cuda)
    with torch.autograd.graph.save_on_cpu():
        idx, d2 = BinnedSelectKnnDifferentiable(9, c, rs)
        found = idx.clone()
        idx[:, 4] = -1
        out, _ = AccumulateKnnDifferentiable(10. * d2, f, idx)
        d2.retain_grad()
        out.backward(go)
    assert torch.equal(c.grad, SelectKnnGrad(d2.grad, found, None, c.detach()))


def test_no_lists_are_kept_where_no_search_takes_them(cuda):
    from hgcalml_b200 import _capi as C
    from hgcalml_b200.accknn_op import AccumulateKnnDifferentiable
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnnDifferentiable
    c, rs = torch.rand((500, 3), device=cuda), torch.tensor([0, 500], dtype=torch.int32, device=cuda)
    f = torch.randn((500, 8), device=cuda, requires_grad=True)
    idx, d2 = BinnedSelectKnnDifferentiable(8, c, rs)
    assert C.noted_lists(idx) is None
    idx, d2 = BinnedSelectKnnDifferentiable(8, c.requires_grad_(True), rs)
    out, _ = AccumulateKnnDifferentiable(d2.detach(), f, idx)
    assert C.noted_lists(idx) is not None and out.grad_fn.lists is None


def test_merge_noise_refuses_what_its_kernels_could_not_read(cuda):
    from hgcalml_b200 import _capi as C
    from hgcalml_b200.assign_condensate_op import BuildAndAssignCondensatesBinned, merge_noise_as_indiv_cp
    g = torch.Generator(device=cuda).manual_seed(7)
    x, beta = torch.rand((900, 3), generator=g, device=cuda), torch.rand((900, 1), generator=g, device=cuda)
    rs, dist = torch.tensor([0, 400, 900], dtype=torch.int32, device=cuda), torch.full((900, 1), .1, device=cuda)
    call = lambda **kw: BuildAndAssignCondensatesBinned(x, beta, dist, rs, .9, assign_by_max_beta=True, **kw)
    args = [*call(), rs]
    got = merge_noise_as_indiv_cp(*args)
    for a, b in zip(got, call(keep_noise=True)):
        assert torch.equal(a, b)
    assert len(args[2]) > 2

    def refused(at, value):
        with pytest.raises((C.HgcError, RuntimeError)):
            merge_noise_as_indiv_cp(*[value if k == at else a for k, a in enumerate(args)])

    refused(1, args[1][:-1])                                   # associations of fewer hits
    refused(3, args[3][:-1])
    refused(2, args[2][:-1])                                   # fewer condensates than are counted
    refused(4, args[4][:-1])
    refused(4, args[4].flip(0))                                # counts that descend
    refused(5, rs - torch.tensor([0, 0, 1], dtype=torch.int32, device=cuda))  # a hit in no event
    refused(4, args[4].cpu())


@pytest.mark.parametrize("splits", [[0, 400, 899], [1, 400, 900], [0, 901, 900], [0] * 400 + [500, 300, 900]])
def test_kept_noise_needs_events_that_are_all_hits(cuda, splits):
    """The renumbering is by event; hits in none were refused by the tensor operations, and are."""
    from hgcalml_b200 import _capi as C
    from hgcalml_b200.assign_condensate_op import BuildAndAssignCondensatesBinned
    x, beta = torch.rand((900, 3), device=cuda), torch.rand((900, 1), device=cuda)
    rs, dist = torch.tensor(splits, dtype=torch.int32, device=cuda), torch.full((900, 1), .1, device=cuda)
    with pytest.raises(C.HgcError):
        BuildAndAssignCondensatesBinned(x, beta, dist, rs, .9, assign_by_max_beta=True, keep_noise=True)


def test_tensors_of_more_dimensions_are_refused(cuda):
    from hgcalml_b200 import _capi as C
    from hgcalml_b200.accknn_op import AccumulateKnn, AccumulateKnnGrad
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn, SelectKnnGrad
    from hgcalml_b200.push_knn_op import PushKnn, PushKnnGrad
    c, rs = torch.rand((40, 3), device=cuda), torch.tensor([0, 40], dtype=torch.int32, device=cuda)
    idx, d2 = BinnedSelectKnn(5, c, rs)
    x = torch.randn((40, 4), device=cuda)
    for call in (lambda: BinnedSelectKnn(5, c[:, :, None].repeat(1, 1, 2), rs), lambda: BinnedSelectKnn(5, c[:, 0], rs),
                 lambda: BinnedSelectKnn(5, c, rs, direction=rs), lambda: SelectKnnGrad(d2, idx[:, :, None], None, c),
                 lambda: AccumulateKnn(d2, x, idx[:, :, None]), lambda: PushKnn(d2, x, idx[:, :, None]),
                 lambda: AccumulateKnnGrad(x, d2, x, idx[:, :, None], None), lambda: PushKnnGrad(x, d2, x, idx[:, :, None])):
        with pytest.raises((C.HgcError, ValueError, IndexError, RuntimeError)):
            call()
