"""A forward-mode tangent on the gradient that enters the activation's backward
reaches the bias gradient (torch's operations carry it; the one-pass kernel
would drop it)."""
import pytest
import torch

from nicr import surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relu", [True, False])
def test_bias_gradient_keeps_the_tangent_of_the_output_gradient(require_gpu, relu):
    fw = torch.autograd.forward_ad
    x = torch.randn((1, 4, 8, 16, 16), device="cuda").bfloat16()
    w = (0.1 * torch.randn((16, 27, 16), device="cuda")).requires_grad_()
    b = torch.zeros(16, device="cuda", requires_grad=True)
    y = surrogate.conv3d_act(x, w, b, relu, False)
    dy, dt = torch.randn_like(y), torch.randn_like(y)
    mask = (y > 0).float() if relu else torch.ones_like(y)
    with fw.dual_level():
        gb, = torch.autograd.grad(y, (b,), fw.make_dual(dy, dt))
        primal, tangent = fw.unpack_dual(gb)
        assert tangent is not None
        for got, ref in ((primal, dy * mask), (tangent, dt * mask)):
            size = ref.double().abs().sum((0, 1, 2, 3))
            assert bool(((got.double() - ref.double().sum((0, 1, 2, 3))).abs() <= 2e-6 * size).all())
