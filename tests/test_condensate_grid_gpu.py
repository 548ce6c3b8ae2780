"""The one-call condensate wrapper against the CPU checker where its passes change shape: dimensions, radii from
tiny to spanning the event, equal betas, masks of both signs, sort-tile remainders, many events, more high-beta hits
than a word of open bits holds per thread, and the noise renumbering."""
import numpy as np
import pytest

from test_ops_gpu import T, N, COND_KEYS

pytestmark = pytest.mark.gpu


def _check(cuda, oracle, cc, beta, d, rs, thr=0.1, mask=None, modes=(True, False), **kw):
    from hgcalml_b200.assign_condensate_op import BuildAndAssignCondensatesBinned
    m = None if mask is None else T(mask, cuda)
    for amb in modes:
        ref = oracle.BuildAndAssignCondensatesBinned(cc, beta, d, rs, thr, no_condensation_mask=mask,
                                                     assign_by_max_beta=amb, **kw)
        got = BuildAndAssignCondensatesBinned(T(cc, cuda), T(beta, cuda), T(d, cuda), T(rs, cuda), thr,
                                              no_condensation_mask=m, assign_by_max_beta=amb, **kw)
        for g, r, key in zip(got, ref, COND_KEYS):
            assert np.array_equal(N(g), r), (key, amb)


def _batch(sizes, dims, seed, spread=3.):
    rng = np.random.default_rng(seed)
    rs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    n = int(rs[-1])
    centres = rng.uniform(-spread, spread, (max(4, n // 200), dims))
    cc = (centres[rng.integers(0, len(centres), n)] + 0.1 * rng.standard_normal((n, dims))).astype(np.float32)
    return cc, rng.beta(0.5, 5., (n, 1)).astype(np.float32), rs, rng


@pytest.mark.parametrize("dims", [1, 2, 3, 4, 7, 8])
@pytest.mark.parametrize("radius", [0.01, 0.5, 20.])
def test_dimensions_and_radii(cuda, oracle, dims, radius):
    cc, beta, rs, rng = _batch([3000, 0, 2049], dims, dims)
    _check(cuda, oracle, cc, beta, (radius * rng.uniform(0.5, 1., beta.shape)).astype(np.float32), rs, modes=(dims % 2 == 0,))


def test_one_large_radius_among_small(cuda, oracle):
    cc, beta, rs, rng = _batch([4000], 3, 5)
    d = np.full_like(beta, 0.2)
    d[rng.integers(0, 4000, 5)] = 50.
    _check(cuda, oracle, cc, beta, d, rs)


@pytest.mark.parametrize("levels", [1, 3])
def test_equal_betas_fall_to_the_order_by_bin(cuda, oracle, levels):
    cc, beta, rs, rng = _batch([2500, 2500], 3, 6 + levels)
    beta = (0.2 + 0.1 * rng.integers(0, levels, beta.shape)).astype(np.float32)
    _check(cuda, oracle, cc, beta, np.full_like(beta, 0.3), rs)


@pytest.mark.parametrize("first", [0, 1, -1])
def test_masks_of_both_signs(cuda, oracle, first):
    cc, beta, rs, rng = _batch([2300, 1700], 3, 11)
    mask = rng.choice([0, 0, 0, 1, -1, 2], beta.shape).astype(np.int32)
    mask[:400] = first  # some of these come first in the order by bin, where the reference looks
    _check(cuda, oracle, cc, beta, np.full_like(beta, 0.4), rs, mask=mask)


def test_many_events(cuda, oracle):
    sizes = np.random.default_rng(3).integers(0, 40, 300)
    cc, beta, rs, _ = _batch(sizes, 3, 13)
    _check(cuda, oracle, cc, beta, np.full_like(beta, 0.5), rs)


def test_more_high_hits_than_a_word_holds(cuda, oracle):
    n = 280000
    rng = np.random.default_rng(17)
    cc = rng.uniform(-3, 3, (n, 3)).astype(np.float32)
    beta = rng.uniform(0.5, 1., (n, 1)).astype(np.float32)
    _check(cuda, oracle, cc, beta, np.full_like(beta, 0.9), np.array([0, n], np.int32), modes=(True,))


@pytest.mark.parametrize("sizes", [[2048], [5000, 0, 2049, 3]])
def test_noise_kept(cuda, oracle, sizes):
    cc, beta, rs, rng = _batch(sizes, 3, 19)
    mask = rng.choice([0, 0, 0, 0, 1, -1], beta.shape).astype(np.int32)
    _check(cuda, oracle, cc, beta, np.full_like(beta, 0.2), rs, thr=0.3, mask=mask, keep_noise=True)
    beta[:] = 0.  # nothing but noise
    _check(cuda, oracle, cc, beta, np.full_like(beta, 0.2), rs, thr=0.3, keep_noise=True)


@pytest.mark.parametrize("dims,radius", [(3, 1.2), (3, 1.7), (4, 0.8), (4, 1.), (5, 1.2), (8, 0.7)])
def test_few_cells_with_masks(cuda, oracle, dims, radius):
    """Around the numbers of cells at which claims go from windows to the grid, and hits from all condensates to those
    of the cells around them."""
    cc, beta, rs, rng = _batch([2600, 0, 1500], dims, 23 + dims)
    mask = rng.choice([0, 0, 0, 0, 1, -1], beta.shape).astype(np.int32)
    radii = np.full_like(beta, radius) if dims == 4 else (radius * rng.uniform(0.7, 1., beta.shape)).astype(np.float32)
    _check(cuda, oracle, cc, beta, radii, rs, mask=mask)


@pytest.mark.parametrize("dims", [3, 7])
def test_a_block_per_event(cuda, oracle, dims):
    """More events than clusters of eight blocks find room, one of them with more high hits than a thread's word holds."""
    sizes = np.random.default_rng(29).integers(0, 700, 40)
    sizes[7] = 36000
    cc, beta, rs, rng = _batch(sizes, dims, 31)
    cc *= 2.
    beta[:] = rng.uniform(0.05, 1., beta.shape)  # nearly all are high
    mask = rng.choice([0] * 30 + [1, -1], beta.shape).astype(np.int32)
    _check(cuda, oracle, cc, beta, np.full_like(beta, 0.5), rs, mask=mask, modes=(True,))


@pytest.mark.parametrize("n_events", [1, 4, 18, 19])
def test_events_without_high_hits(cuda, oracle, n_events):
    """Nothing to settle: the blocks of an event's cluster must still leave together."""
    cc, beta, rs, rng = _batch([300] * n_events, 3, 37)
    beta *= 0.05
    beta[:300:100] = 0.9 if n_events > 1 else 0.  # the first of several events has some
    for _ in range(20):
        _check(cuda, oracle, cc, beta, np.full_like(beta, 0.2), rs, thr=0.3, modes=(True,))
