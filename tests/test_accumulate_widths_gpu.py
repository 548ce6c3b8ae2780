"""AccumulateKnn at the widths and alignments where the kernel's loads change, at hit counts around its tiles: bit for
bit against the CPU checker."""
import numpy as np
import pytest
import torch

from conftest import bits
from test_ops_gpu import T, N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", [1, 2, 3, 6, 15, 16, 17, 18, 22, 31, 33, 34, 63, 65, 66, 127, 129, 130, 254, 258])
def test_widths(cuda, oracle, F):
    from hgcalml_b200.accknn_op import AccumulateLinKnn
    rng = np.random.default_rng(F)
    for n, K, pad in ((1, 1, False), (97, 9, True), (1500, 32, False), (700, 41, True)):
        feat = rng.standard_normal((n, F), dtype=np.float32)
        w = rng.random((n, K), dtype=np.float32)
        idx = rng.integers(0, n, (n, K)).astype(np.int32)
        if pad:
            idx[rng.random((n, K)) < 0.2] = -1
        for mm in (True, False):
            ro, ra = oracle.op_accumulate_knn(w, feat, idx, mean_and_max=mm)
            go, ga = AccumulateLinKnn(T(w, cuda), T(feat, cuda), T(idx, cuda), mean_and_max=mm)
            assert np.array_equal(bits(N(go)), bits(ro))
            if mm:
                assert np.array_equal(N(ga), ra)


@pytest.mark.parametrize("F,shift", [(64, 1), (64, 2), (12, 3), (20, 4)])
def test_unaligned_features(cuda, oracle, F, shift):
    from hgcalml_b200.accknn_op import AccumulateLinKnn
    rng = np.random.default_rng(F + shift)
    n, K = 900, 24
    feat = rng.standard_normal((n, F), dtype=np.float32)
    w = rng.random((n, K), dtype=np.float32)
    idx = rng.integers(0, n, (n, K)).astype(np.int32)
    buf = torch.zeros(n * F + shift, device=cuda)
    view = buf[shift:].view(n, F)
    view.copy_(T(feat, cuda))
    ro, ra = oracle.op_accumulate_knn(w, feat, idx)
    go, ga = AccumulateLinKnn(T(w, cuda), view, T(idx, cuda))
    assert np.array_equal(bits(N(go)), bits(ro)) and np.array_equal(N(ga), ra)
