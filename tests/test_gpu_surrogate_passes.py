"""The one-kernel elementwise passes around the surrogate's convolutions against
the torch operations they stand for: the activation's backward with the bias
gradient, the pooling, the upsampled concatenation and the padded input. The
stored values are the same (the pooling's eight summands here have exponents
within FP32's reach, so its sum is exact in any order); the bias gradient's
FP32 sums may differ from FP64 by (terms per thread) x 2^-24 of the sum of
magnitudes, at most 2e-6 at these sizes."""
import numpy as np
import pytest
import torch

from nicr import surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [8, 16, 48, 96, 272, 2048])
@pytest.mark.parametrize("rows", [1, 63, 592 * 4 + 5])
@pytest.mark.parametrize("gy_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("y_dtype", [None, torch.bfloat16, torch.float32])
def test_act_backward(require_gpu, c, rows, gy_dtype, y_dtype):
    g = torch.Generator(device="cuda").manual_seed(c + rows)
    gy = torch.randn((rows, c), generator=g, device="cuda").to(gy_dtype)
    y = None if y_dtype is None else torch.randn((rows, c), generator=g, device="cuda").relu().to(y_dtype)
    with torch.no_grad():   # as the backward without a graph of its own runs
        got, gb = surrogate._act_backward(gy, y)
    ref = gy.float() if y is None else gy.float() * (y > 0)
    assert torch.equal(got, ref.to(torch.bfloat16))
    exact, size = ref.double().sum(0), ref.double().abs().sum(0)
    assert bool(((gb.double() - exact).abs() <= 2e-6 * size + 1e-300).all())


def test_act_backward_passes_nonfinite_values(require_gpu):
    gy = torch.ones((64, 16), device="cuda")
    gy[3, 2], gy[4, 5], gy[5, 6] = float("nan"), float("inf"), float("-inf")
    y = torch.ones((64, 16), device="cuda", dtype=torch.bfloat16)
    y[4, 5] = 0.0        # inf x 0 is NaN, as in the torch product
    y[6, 6] = float("nan")
    with torch.no_grad():
        got, gb = surrogate._act_backward(gy, y)
    ref = gy * (y > 0)
    assert torch.equal(torch.nan_to_num(got.float(), nan=7.0), torch.nan_to_num(ref.to(torch.bfloat16).float(), nan=7.0))
    assert torch.equal(torch.isnan(gb), torch.isnan(ref.sum(0)))


@pytest.mark.parametrize("shape", [(1, 4, 4, 8, 16), (2, 8, 4, 12, 32), (1, 4, 4, 4, 16)])
def test_inference_passes_equal_training_passes(require_gpu, shape):
    """The U-Net's forward without gradients (fused passes) equals the one that records them (torch's)."""
    n, d, h, w, base = shape
    net = surrogate.unet(5, base).cuda()
    x = torch.randn((n, 4 * d, 4 * h, 4 * w, 5), device="cuda")
    with torch.no_grad():
        a = net(x)
    b = net(x)
    assert torch.equal(a, b.detach())
    with torch.no_grad():
        c = net(x.transpose(1, 2).contiguous().transpose(1, 2))   # another stride order: the general path
    assert torch.equal(a, c)


def test_first_layer_needs_no_input_gradient(require_gpu):
    x = torch.randn((1, 4, 8, 16, 16), device="cuda").bfloat16()
    w = torch.randn((16, 27, 16), device="cuda", requires_grad=True)
    b = torch.zeros(16, device="cuda", requires_grad=True)
    y = surrogate.conv3d_act(x, w, b)
    gw, gb = torch.autograd.grad(y.float().square().sum(), (w, b))
    xg = x.clone().requires_grad_()
    y2 = surrogate.conv3d_act(xg, w, b)
    gx2, gw2, gb2 = torch.autograd.grad(y2.float().square().sum(), (xg, w, b))
    assert gx2.shape == x.shape and torch.equal(gb, gb2)
    assert np.allclose(gw.cpu(), gw2.cpu(), rtol=1e-5, atol=1e-5 * float(gw.abs().max()))   # FP32 atomics: order of sums


def test_bias_gradient_is_differentiable(require_gpu):
    """A backward that records a graph keeps torch's operations: the bias
    gradient's derivative along the output gradient is the ReLU's mask."""
    x = torch.randn((1, 4, 8, 16, 16), device="cuda").bfloat16()
    w = (0.1 * torch.randn((16, 27, 16), device="cuda")).requires_grad_()
    b = torch.zeros(16, device="cuda", requires_grad=True)
    y = surrogate.conv3d_act(x, w, b, True, False)
    dy = torch.randn_like(y).requires_grad_()
    gb, = torch.autograd.grad(y, (b,), dy, create_graph=True)
    mask, = torch.autograd.grad(gb.sum(), (dy,))
    assert torch.equal(mask, (y > 0).float())


@pytest.mark.parametrize("y", [None, torch.float32, torch.bfloat16])
def test_act_backward_of_other_layouts(require_gpu, y):
    """Stored activations in another stride order take torch's operations."""
    gy = torch.randn((6, 4, 16), device="cuda")
    act = None if y is None else torch.randn((4, 6, 16), device="cuda").relu().to(y).transpose(0, 1)
    with torch.no_grad():
        got, gb = surrogate._act_backward(gy, act)
    ref = gy if act is None else gy * (act > 0)
    assert torch.equal(got, ref.to(torch.bfloat16))
    assert bool(((gb - ref.sum((0, 1))).abs() <= 2e-6 * ref.abs().sum((0, 1))).all())


def test_forward_mode_stays_refused(require_gpu):
    """The convolutions have no forward-mode rule; the passes around them must not drop the tangent."""
    net = surrogate.unet(5, 16).cuda()
    x = torch.randn((1, 4, 4, 8, 5), device="cuda")
    with torch.no_grad(), torch.autograd.forward_ad.dual_level():
        with pytest.raises((RuntimeError, NotImplementedError)):
            net(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))
