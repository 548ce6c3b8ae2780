"""The wrapper-level neighbour search (tiles of queries over boxed chunks) against the CPU checker where its
shapes change: list lengths, chunk / super-chunk / sort-tile remainders, many events, direction, bins that do
not fit the sort key, lists of chunks that do not fit the tile, and points that coincide."""
import numpy as np
import pytest

from conftest import assert_knn_equal
from hgcalml_b200 import synth
from test_ops_gpu import T, N

pytestmark = pytest.mark.gpu


def _check(cuda, oracle, K, c, rs, direction=None, **kw):
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn
    d = None if direction is None else T(direction, cuda)
    gi, gd, sorting = BinnedSelectKnn(K, T(c, cuda), T(rs, cuda), direction=d, return_sorting=True, **kw)
    ri, rd = oracle.BinnedSelectKnn(K, c, rs, direction=direction, **kw)
    assert_knn_equal(N(gi), N(gd), ri, rd)
    assert np.array_equal(np.sort(N(sorting)), np.arange(len(c)))
    return N(sorting)


@pytest.mark.parametrize("K", [1, 2, 32, 33, 34, 64, 65, 66, 129, 257, 513])
def test_list_lengths(cuda, oracle, K):
    c, _, rs = synth.shower_batch([1500, 40], dims=4, n_feat=0, seed=11, with_features=False)
    _check(cuda, oracle, K, c, rs)


@pytest.mark.parametrize("dims", [2, 3, 5, 6, 7, 8, 9, 13])
def test_coordinate_counts(cuda, oracle, dims):
    c, _, rs = synth.shower_batch([900, 33, 700], dims=dims, with_features=False, seed=dims)
    _check(cuda, oracle, 17, c, rs)


@pytest.mark.parametrize("sizes", [[31], [32], [33, 1, 0, 31], [1023, 1025], [1024], [2047, 2049, 2048, 5], [4097]])
def test_event_sizes(cuda, oracle, sizes):
    c, _, rs = synth.shower_batch(sizes, dims=3, with_features=False, seed=len(sizes))
    _check(cuda, oracle, 20, c, rs)


def test_many_small_events(cuda, oracle):
    sizes = np.random.default_rng(5).integers(0, 25, 700)
    rng = np.random.default_rng(6)
    rs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    _check(cuda, oracle, 12, rng.random((int(rs[-1]), 3), dtype=np.float32), rs)


@pytest.mark.parametrize("kw", [dict(n_bins=80), dict(n_bins=12, max_bin_dims=5), dict(n_bins=39, max_bin_dims=3)])
def test_bins_beyond_the_sort_key(cuda, oracle, kw):
    c, _, rs = synth.shower_batch([3000, 500], dims=5, with_features=False, seed=9)
    sorting = _check(cuda, oracle, 10, c, rs, **kw)
    assert np.array_equal(np.sort(sorting[:3000]), np.arange(3000))  # events stay together


def test_sorting_is_by_bin(cuda, oracle):
    from hgcalml_b200.bin_by_coordinates_op import BinByCoordinates
    c, _, rs = synth.shower_batch([5000, 70, 2500], dims=4, with_features=False, seed=19)
    sorting = _check(cuda, oracle, 8, c, rs, n_bins=9)
    _, flat, _, _, _ = BinByCoordinates(T(c[:, :3], cuda), T(rs, cuda), n_bins=9)
    assert (np.diff(N(flat)[sorting]) >= 0).all()


def test_direction_over_chunks(cuda, oracle):
    c, _, rs = synth.shower_batch([2100, 64], dims=4, with_features=False, seed=23)
    d = np.random.default_rng(24).integers(0, 4, len(c)).astype(np.int32)
    d[:1200] = 1  # whole chunks without a possible neighbour
    _check(cuda, oracle, 25, c, rs, direction=d)


def test_more_chunks_than_the_list_holds(cuda, oracle):
    rng = np.random.default_rng(31)
    c = rng.random((36000, 6), dtype=np.float32)
    _check(cuda, oracle, 40, c, np.array([0, 36000], np.int32))


@pytest.mark.parametrize("K", [16, 64])
def test_coinciding_points(cuda, oracle, K):
    rng = np.random.default_rng(41)
    c = rng.integers(0, 3, (2500, 3)).astype(np.float32)
    c[:400] = 1.5
    _check(cuda, oracle, K, c, np.array([0, 1300, 2500], np.int32))


@pytest.mark.parametrize("dims", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("sizes", [[1], [33, 0, 479], [512], [513], [2049, 1, 30], [4096], [100, 8000, 92], [1, 8190, 0, 1], [100] * 31, [264] * 31])
def test_small_batches_have_the_order_of_large_ones(cuda, dims, sizes):
    """Batches of up to 8192 hits in 31 events are ordered by one kernel; the same hits in front of others, which leave the
    range of the batch as it is, by the chain of kernels for any size."""
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn
    rng = np.random.default_rng(dims + len(sizes))
    n = sum(sizes)
    c = rng.standard_normal((n, dims), dtype=np.float32)
    more = c[rng.integers(0, n, 9000)]
    rs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    kw = dict(n_bins=7, return_sorting=True)
    i0, d0, s0 = BinnedSelectKnn(9, T(c, cuda), T(rs, cuda), **kw)
    i1, d1, s1 = BinnedSelectKnn(9, T(np.concatenate([c, more]), cuda), T(np.append(rs, n + 9000).astype(np.int32), cuda), **kw)
    assert np.array_equal(N(s0), N(s1)[:n])
    assert np.array_equal(N(i0), N(i1)[:n]) and np.array_equal(N(d0).view(np.uint32), N(d1)[:n].view(np.uint32))


def test_a_large_event_in_five_dimensions(cuda, oracle):
    """Parts of 256 hits are split into chunks where events hold 150k hits and more; brute force for a sample."""
    from hgcalml_b200.binned_select_knn_op import BinnedSelectKnn
    import torch
    n, K = 150211, 20
    c, _, rs = synth.shower_batch([n], dims=5, n_feat=0, with_features=False, seed=3)
    idx, d2, sorting = BinnedSelectKnn(K, T(c, cuda), T(rs, cuda), return_sorting=True)
    assert torch.equal(sorting.sort().values, torch.arange(n, dtype=torch.int32, device=cuda))
    x = T(c, cuda)
    rows = torch.arange(0, n, 997, device=cuda)
    d = torch.zeros((len(rows), n), device=cuda)
    for k in range(5):  # in coordinate order, unfused, as the op sums
        t = x[rows, k][:, None] - x[:, k][None]
        d = d + t * t
    d[torch.arange(len(rows), device=cuda), rows] = -1.
    want, _ = torch.topk(d, K, largest=False)
    assert torch.equal(want.sort(dim=1).values[:, 1:], d2[rows][:, 1:]) and torch.equal(idx[rows, 0].long(), rows)
    assert torch.equal(torch.gather(d, 1, idx[rows].long())[:, 1:], d2[rows][:, 1:])
