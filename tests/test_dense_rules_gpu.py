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
