"""When the dense layers may put bias and activation on in place: never where the tensor operations would do more."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(cuda, activation="relu", n_in=6, n_out=8):
    from hgcalml_b200.GravNetLayersRagged import _Dense
    g = torch.Generator(device=cuda).manual_seed(11)
    layer = _Dense(n_in, n_out, activation).to(cuda)
    with torch.no_grad():
        layer.bias.copy_(torch.randn(n_out, generator=g, device=cuda))
    return layer, torch.randn((40, n_in), generator=g, device=cuda)


@pytest.mark.parametrize("activation", ["relu", None])
def test_a_trainable_bias_on_a_frozen_kernel_gets_its_gradient(cuda, activation):
    layer, x = _layer(cuda, activation)
    layer.kernel.requires_grad_(False)
    y = layer(x)
    assert y.requires_grad
    y.sum().backward()
    z = x @ layer.kernel + layer.bias.detach()
    want = (z > 0).sum(0).float() if activation else torch.full((8,), 40., device=cuda)
    assert torch.equal(layer.bias.grad, want)
    with torch.no_grad():
        assert torch.equal(layer(x), y)


def test_a_bias_that_is_no_dense_row_beside_the_result(cuda):
    layer, x = _layer(cuda)
    with torch.no_grad():
        want = torch.relu(x @ layer.kernel + layer.bias[0])
        whole = layer.bias.clone()
        layer.bias = torch.nn.Parameter(whole[:1].clone())  # broadcast
        assert torch.equal(layer(x), want)
        layer.bias = torch.nn.Parameter(whole.cpu())
        with pytest.raises(RuntimeError):
            layer(x)


def test_forward_mode_vmap_and_modes_see_the_operations(cuda):
    from torch.utils.flop_counter import FlopCounterMode
    from hgcalml_b200.GravNetLayersRagged import _copy_columns
    layer, x = _layer(cuda)
    layer.requires_grad_(False)
    t = torch.randn(x.shape, generator=torch.Generator(device=cuda).manual_seed(2), device=cuda)
    z = x @ layer.kernel + layer.bias
    y, dy = torch.func.jvp(layer, (x,), (t,))
    assert torch.equal(y, torch.relu(z)) and torch.allclose(dy, (t @ layer.kernel) * (z > 0), rtol=1e-5, atol=1e-6)
    with torch.autograd.forward_ad.dual_level():
        out = torch.zeros((40, 9), device=cuda)
        dual = torch.autograd.forward_ad.make_dual(x, t)
        dy = torch.autograd.forward_ad.unpack_dual(layer(dual)).tangent
        assert torch.allclose(dy, (t @ layer.kernel) * (z > 0), rtol=1e-5, atol=1e-6)
        _copy_columns(dual, out, 3)
        assert torch.equal(torch.autograd.forward_ad.unpack_dual(out).tangent[:, 3:], t)
    assert torch.equal(torch.func.vmap(layer)(x.reshape(5, 8, 6)).reshape(40, 8), torch.relu(z))
    assert torch.equal(torch.jit.trace(layer, x, check_trace=False)(2. * x), layer(2. * x))
    with FlopCounterMode(display=False) as f:
        assert torch.equal(layer(x), torch.relu(z))
    assert f.get_total_flops() == 2 * 40 * 6 * 8


def test_the_activation_that_the_layer_has_now_is_used(cuda):
    layer, x = _layer(cuda)
    with torch.no_grad():
        z = x @ layer.kernel + layer.bias
        assert torch.equal(layer(x), torch.relu(z))
        layer.activation = torch.tanh
        assert torch.equal(layer(x), torch.tanh(z))


def test_the_sign_of_zero_is_that_of_the_operations(cuda):
    layer, _ = _layer(cuda, n_in=4, n_out=4)
    with torch.no_grad():
        layer.kernel.fill_(-0.)
        layer.bias.copy_(torch.tensor([-0., 0., 1., -1.]))
        x = torch.zeros((3, 4), device=cuda)
        want = torch.relu(x @ layer.kernel + layer.bias)
        got = layer(x)
    assert torch.equal(got, want) and torch.equal(torch.signbit(got), torch.signbit(want))
    from hgcalml_b200 import _capi as C
    for relu in (0, 1):
        y, b = torch.tensor([[-0., 0., -0., float("nan")]], device=cuda), torch.tensor([-0., -0., 0., 1.], device=cuda)
        want = torch.relu(y + b) if relu else y + b
        C.check(C.lib.hgc_bias_act(C.ptr(y), C.ptr(b), 1, 4, relu, C.stream_of(y)), "bias_act")
        assert torch.equal(torch.signbit(y)[:, :3], torch.signbit(want)[:, :3]) and y[0, 3].isnan(), (relu, y, want)


@pytest.mark.parametrize("n", [1, 31, 33, 127, 2049, 49153])
@pytest.mark.parametrize("n_in,n_out", [(4, 1), (12, 4), (64, 5), (132, 8), (16, 9), (20, 16), (48, 17), (32, 32), (36, 33), (64, 64), (192, 65), (512, 130)])
def test_dense_kernel_at_the_edges_of_its_tiles(cuda, n, n_in, n_out):
    from hgcalml_b200 import _capi as C
    g = torch.Generator(device=cuda).manual_seed(n + n_in)
    x, w = torch.randn((n, n_in), generator=g, device=cuda), torch.randn((n_in, n_out), generator=g, device=cuda)
    b = torch.randn(n_out, generator=g, device=cuda)
    for bias, relu in ((None, 0), (b, 0), (b, 1)):
        y = torch.full((n + 1, n_out), 7., device=cuda)
        C.check(C.lib.hgc_dense(C.ptr(x), C.ptr(w), C.ptr(bias), C.ptr(y), n, n_in, n_out, relu, C.stream_of(x)), "dense")
        want = x.double() @ w.double()
        size = x.double().abs() @ w.double().abs()
        if bias is not None:
            want, size = want + b, size + b.abs()
        if relu:
            want = want.clamp_min(0.)
        # n_in fused multiply-adds and one addition, each off by half an ulp of at most the sum of the terms' sizes
        assert ((y[:n].double() - want).abs() <= (n_in + 1) * 2. ** -24 * size).all()
        assert (y[n] == 7.).all()


def test_precisions_that_the_caller_chose_are_the_library_s(cuda):
    layer, x = _layer(cuda, n_in=64, n_out=64)
    layer.requires_grad_(False)
    x = torch.randn((3000, 64), generator=torch.Generator(device=cuda).manual_seed(2), device=cuda)
    want = torch.relu(x @ layer.kernel + layer.bias)
    assert torch.equal(layer(x), want)
    with torch.autocast("cuda", dtype=torch.float16):
        half = layer(x)
        assert torch.equal(half, torch.relu(x @ layer.kernel + layer.bias))
    assert not torch.equal(half.float(), want)
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        assert torch.equal(layer(x), torch.relu(x @ layer.kernel + layer.bias))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = False


@pytest.mark.parametrize("setting", ["ieee", "tf32", "tf32 everywhere", "high"])
def test_precisions_chosen_through_any_of_torch_s_settings(cuda, setting):
    layer, _ = _layer(cuda, n_in=64, n_out=64)
    layer.requires_grad_(False)
    x = torch.randn((3000, 64), generator=torch.Generator(device=cuda).manual_seed(2), device=cuda)
    plain = torch.relu(x @ layer.kernel + layer.bias)
    try:
        if setting == "high":
            torch.set_float32_matmul_precision("high")
        elif setting == "tf32 everywhere":
            torch.backends.fp32_precision = "tf32"
        else:
            torch.backends.cuda.matmul.fp32_precision = setting
        want, got = torch.relu(x @ layer.kernel + layer.bias), layer(x)
        layer.requires_grad_(True)
        trained = layer(x)
    finally:
        torch.set_float32_matmul_precision("highest")
        torch.backends.fp32_precision = "none"
        torch.backends.cuda.matmul.fp32_precision = "none"
    assert torch.equal(got, want) and torch.equal(trained, want)
    assert torch.equal(want, plain) == (setting == "ieee")


def test_a_failed_launch_is_no_reason_for_the_library(cuda, monkeypatch):
    from hgcalml_b200 import _capi as C
    layer, x = _layer(cuda)
    native = C.native

    class Failing:
        def __getattr__(self, name):
            return getattr(native, name)

        def dense(self, *args):
            return None, -4  # HGC_ERR_CUDA
    monkeypatch.setattr(C, "native", Failing())
    with torch.no_grad(), pytest.raises(C.HgcError):
        layer(x)


@pytest.mark.parametrize("n,n_in,n_out,own", [(3000, 64, 64, 1), (20, 64, 64, 1), (3000, 22, 8, 0), (3000, 512, 512, 0)])
def test_which_layers_take_the_kernel(cuda, n, n_in, n_out, own):
    """The kernel alone where it is taken; elsewhere the library's product and one pass for bias and activation."""
    from hgcalml_b200 import _capi as C
    layer, _ = _layer(cuda, n_in=n_in, n_out=n_out)
    x = torch.randn((n, n_in), generator=torch.Generator(device=cuda).manual_seed(4), device=cuda)
    with torch.no_grad():
        before = C.lib.hgc_launch_count()
        y, rc = C.native.dense(x, layer.kernel, layer.bias, True)
        assert C.lib.hgc_launch_count() - before == own and rc == (C.HGC_OK if own else C.NOT_TAKEN)
        before = C.lib.hgc_launch_count()
        z = layer(x)
        assert C.lib.hgc_launch_count() - before == 1
        if own:
            assert torch.equal(y, z)
            shifted = torch.empty(x.numel() + 1, device=cuda)[1:].view(x.shape).copy_(x)
            assert C.native.dense(shifted, layer.kernel, layer.bias, True)[1] == C.NOT_TAKEN
            assert torch.allclose(layer(shifted), z, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("n", [50, 49200])
@pytest.mark.parametrize("n_out", [3, 7, 12, 30, 70])
def test_dense_kernel_with_long_rows(cuda, n, n_out):
    from hgcalml_b200 import _capi as C
    n_in = 516
    g = torch.Generator(device=cuda).manual_seed(n + n_out)
    x, w = torch.randn((n, n_in), generator=g, device=cuda), torch.randn((n_in, n_out), generator=g, device=cuda)
    y = torch.empty((n, n_out), device=cuda)
    C.check(C.lib.hgc_dense(C.ptr(x), C.ptr(w), None, C.ptr(y), n, n_in, n_out, 0, C.stream_of(x)), "dense")
    # n_in fused multiply-adds, each off by half an ulp of at most the sum of the terms' sizes
    assert ((y.double() - x.double() @ w.double()).abs() <= n_in * 2. ** -24 * (x.double().abs() @ w.double().abs())).all()
    assert C.lib.hgc_dense(C.ptr(x), C.ptr(w), None, C.ptr(y), n, 514, n_out, 0, C.stream_of(x)) == -3
