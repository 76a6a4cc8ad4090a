"""The pooling's order of summation. Summands whose exponents differ by more
than FP32's 24 bits make the sum depend on it: the stored averages equal those
of torch's mean and of the order the kernel states, ((((e0 + e4) + (e1 + e5)) +
(e2 + e6)) + (e3 + e7)) / 8 with e[4 z + 2 y + x], each addition rounded to
FP32, and another order gives other values, so the test can tell."""
import numpy as np
import pytest
import torch

from nicr import surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 8, 6, 10, 24), (1, 2, 2, 32, 16), (1, 64, 64, 64, 64)])
def test_average_in_the_stated_order(require_gpu, shape):
    g = torch.Generator(device="cuda").manual_seed(5)
    n, d, h, w, c = shape
    scale = torch.randint(-30, 31, (n, d, h, w, c), generator=g, device="cuda").float().exp2()
    x = (torch.randn((n, d, h, w, c), generator=g, device="cuda") * scale).bfloat16()
    # partners that cancel, so that what an order loses is all that is left
    x[:, 1::2, 0::2, 1::2] = -x[:, 0::2, 0::2, 0::2]
    y = torch.empty((n, d // 2, h // 2, w // 2, c), device="cuda", dtype=torch.bfloat16)
    rc = surrogate._lib().nicr_avgpool2_ndhwc(x.data_ptr(), y.data_ptr(), n, d, h, w, c, surrogate._stream(x))
    assert rc == 0
    f = x.float().cpu().numpy().reshape(n, d // 2, 2, h // 2, 2, w // 2, 2, c)
    e = [f[:, :, k >> 2, :, (k >> 1) & 1, :, k & 1] for k in range(8)]
    order = (((e[0] + e[4]) + (e[1] + e[5])) + (e[2] + e[6])) + (e[3] + e[7])
    other = ((((((e[0] + e[1]) + e[2]) + e[3]) + e[4]) + e[5]) + e[6]) + e[7]
    assert order.dtype == np.float32
    got = y.float().cpu().numpy()

    def stored(v):
        return torch.from_numpy(v * np.float32(0.125)).bfloat16().float().numpy()
    assert np.array_equal(got, stored(order))
    mean = x.float().view(n, d // 2, 2, h // 2, 2, w // 2, 2, c).mean(dim=(2, 4, 6)).to(torch.bfloat16)
    assert torch.equal(y, mean)
    assert not np.array_equal(stored(order), stored(other))
