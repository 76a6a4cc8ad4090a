"""The forward form that stages input lines once (nicr_conv3d_fwd_shift): the
same bits as the form each shape used before (the per-tap TMA form, or the halo
block for Cin x Cout <= 768 with Cout <= 32 on rows of 128 or more), at the
edges of its tiles and rings: one line, one plane, heights that leave lines of
the last group outside, rows shorter than a tile, of exactly one tile and just
beyond, one to four channel boxes, every line count per CTA."""
import pytest
import torch

import conv_ref
from nicr import surrogate

pytestmark = pytest.mark.gpu

# (n, d, h, w, cin, cout)
SHAPES = [(1, 3, 4, 128, 16, 16), (1, 2, 5, 128, 32, 32), (2, 1, 1, 128, 48, 16), (1, 3, 7, 64, 64, 64),
          (1, 4, 9, 64, 96, 32), (1, 2, 6, 32, 80, 48), (1, 3, 16, 16, 16, 64), (1, 2, 24, 8, 32, 48),
          (1, 2, 3, 96, 48, 32), (1, 2, 4, 136, 16, 48), (2, 2, 8, 200, 64, 16), (1, 2, 4, 120, 112, 32),
          (1, 4, 4, 4, 128, 16), (1, 9, 65, 128, 32, 16), (1, 9, 65, 128, 96, 32), (1, 7, 130, 64, 48, 64),
          (1, 4, 75, 256, 16, 32)]


def inputs(shape, seed):
    n, d, h, w, ci, co = shape
    g = torch.Generator().manual_seed(seed)
    return conv_ref.bf16_rounded((n, d, h, w, ci), g).cuda().bfloat16(), conv_ref.bf16_rounded((co, 27, ci), g, 0.2).cuda().bfloat16()


@pytest.mark.parametrize("shape", SHAPES)
def test_same_bits_as_the_former_form(require_gpu, shape):
    x, w = inputs(shape, 1)
    n, d, h, wd, ci, co = shape
    former = "halo" if co <= 32 and ci * co <= 768 and wd >= 128 else "tma"
    a = surrogate.conv3d_raw(x, w, "shift")
    assert surrogate.conv_error() == 0
    b = surrogate.conv3d_raw(x, w, former)
    assert torch.equal(a, b)


@pytest.mark.parametrize("shape", [SHAPES[1], SHAPES[4], SHAPES[8]])
@pytest.mark.parametrize("act", [0, 1, 2, 3])
def test_epilogue(require_gpu, shape, act):
    n, d, h, wd, ci, co = shape
    x, w = inputs(shape, 2)
    b = torch.randn(co, device="cuda")
    y = torch.empty((n, d, h, wd, co), dtype=torch.bfloat16 if act & 2 else torch.float32, device="cuda")
    L = surrogate._lib()
    rc = L.nicr_conv3d_fwd_shift(x.data_ptr(), w.data_ptr(), b.data_ptr(), act, y.data_ptr(), n, d, h, wd, ci, co,
                                 torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    ref = surrogate.conv3d_raw(x, w, "tma") + b
    ref = ref.relu() if act & 1 else ref
    assert torch.equal(y, ref.to(y.dtype))


@pytest.mark.parametrize("shape", [(1, 4, 4, 8, 16, 80), (3, 1, 64, 128, 192, 64)], ids=["Cout 80", "rings too large"])
def test_refuses_what_it_cannot_hold(require_gpu, shape):
    x, w = inputs(shape, 3)
    with pytest.raises(RuntimeError):
        surrogate.conv3d_raw(x, w, "shift")


@pytest.mark.parametrize("shape", [(1, 2, 5, 128, 32, 32), (1, 1, 4, 128, 48, 16), (1, 3, 4, 64, 64, 64)])
@pytest.mark.parametrize("tap", [1, 13, 25])   # planes below, at and above the voxel
def test_infinite_weights_reach_the_same_voxels(require_gpu, shape, tap):
    """An infinite weight times the zero padding is NaN, in planes outside the grid as elsewhere."""
    x, w = inputs(shape, 4)
    w[3, tap, 5] = float("inf")
    n, d, h, wd, ci, co = shape
    a = surrogate.conv3d_raw(x, w, "shift")
    b = surrogate.conv3d_raw(x, w, "halo" if co <= 32 and ci * co <= 768 and wd >= 128 else "tma")
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
