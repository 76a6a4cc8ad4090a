"""The convolutions move 16 bytes at a time: a base that is not 16-byte aligned is
refused before anything is launched (checked here with addresses that nothing
reads, without a GPU), and the Python layer takes a misaligned bias through
separate operations."""
import ctypes

import pytest

import nicr
from nicr import surrogate

OK = 0x10000            # aligned; never read: every call below is refused
OFF = 0x10002
FWD_ACT = ("nicr_conv3d_fwd_act", "nicr_conv3d_fwd_march", "nicr_conv3d_fwd_shift", "nicr_conv3d_fwd_halo")
FWD = ("nicr_conv3d_fwd", "nicr_conv3d_fwd_tma", "nicr_conv3d_fwd_gather", "nicr_conv3d_fwd_mma_sync")
WGRAD = ("nicr_conv3d_wgrad", "nicr_conv3d_wgrad_tma", "nicr_conv3d_wgrad_mma_sync")


@pytest.mark.parametrize("which", ["x", "w", "bias", "y"])
@pytest.mark.parametrize("name", FWD_ACT)
def test_fused_forward_refuses(name, which):
    a = {k: OFF if k == which else OK for k in ("x", "w", "bias", "y")}
    f = getattr(surrogate._lib(), name)
    assert f(a["x"], a["w"], a["bias"], 0, a["y"], 1, 4, 4, 128, 16, 16, None) == 1


@pytest.mark.parametrize("which", ["x", "w"])
@pytest.mark.parametrize("name", FWD)
def test_forward_refuses(name, which):
    a = {k: OFF if k == which else OK for k in ("x", "w")}
    f = getattr(surrogate._lib(), name)
    f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 6 + [ctypes.c_void_p]
    assert f(a["x"], a["w"], OK, 1, 4, 4, 128, 48, 16, None) == 1


@pytest.mark.parametrize("which", ["x", "dy"])
@pytest.mark.parametrize("name", WGRAD)
def test_weight_gradient_refuses(name, which):
    a = {k: OFF if k == which else OK for k in ("x", "dy")}
    f = getattr(nicr.lib(), name)
    f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 6 + [ctypes.c_void_p]
    assert f(a["x"], a["dy"], OK, 1, 4, 4, 128, 16, 16, None) == 1


@pytest.mark.gpu
def test_misaligned_tensors(require_gpu):
    import torch
    x = torch.randn((1, 4, 4, 16, 16), device="cuda").bfloat16()
    w = 0.1 * torch.randn((16, 27, 16), device="cuda")
    b = torch.randn(17, device="cuda")[1:]
    assert b.data_ptr() % 16 != 0
    with torch.no_grad():
        assert torch.equal(surrogate.conv3d_act(x, w, b), surrogate.conv3d_act(x, w, b.clone()))
        flat = torch.zeros(w.numel() + 1, device="cuda", dtype=torch.bfloat16)
        flat[1:] = w.bfloat16().flatten()
        with pytest.raises(RuntimeError):
            surrogate.conv3d_act(x, flat[1:].view(w.shape), b)
        flat = torch.zeros(x.numel() + 1, device="cuda", dtype=torch.bfloat16)
        with pytest.raises(RuntimeError):
            surrogate.conv3d_act(flat[1:].view(x.shape), w, b)
