"""Channel-pair depthwise kernels against the oracle where they can go wrong: odd widths and channel counts, heights that leave
a partial patch or several bands, one to several planes (the march rotates with period 3), several groups per block, rows
that start at any 16-byte remainder, and rows too long for a block (the older kernels take over)."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 1, 1, 1, 1), (1, 2, 2, 3, 5), (2, 3, 3, 4, 7), (1, 5, 4, 9, 33), (2, 4, 5, 13, 107), (1, 3, 2, 30, 54),
    (1, 2, 6, 5, 214), (1, 2, 2, 3, 257), (1, 1, 2, 2, 385), (3, 40, 7, 6, 11),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("skew", [0, 1])
def test_pair_kernels_vs_oracle(shape, dtype, skew):
    from d2conv3d_b200 import _lib, fast_depthwise_conv3d
    gen = torch.Generator().manual_seed(sum(shape))

    def make(*sh):
        flat = torch.zeros(int(np.prod(sh)) + skew, device="cuda", dtype=dtype)
        t = flat[skew:].view(*sh)
        t.copy_(torch.randn(*sh, generator=gen) / 2)
        return t

    C = shape[1]
    x, w, b = make(*shape).requires_grad_(), make(C, 1, 3, 3, 3).requires_grad_(), make(C).requires_grad_()
    gy = make(*shape)
    op = fast_depthwise_conv3d._ops.depthwise_separable_conv3d
    y = op(x, w, b, 1, 1, 1)
    gx, gw, gb = torch.autograd.grad(y, (x, w, b), gy, retain_graph=True)
    only_x, = torch.autograd.grad(y, (x,), gy, retain_graph=True)
    only_w, = torch.autograd.grad(y, (w,), gy)
    d = lambda t: t.detach().double().cpu().numpy()
    wy = orc.depthwise_conv3d_fwd(d(x), d(w), d(b), 1, 1, 1)
    wgx, wgw, wgb = orc.depthwise_conv3d_bwd(d(gy), d(x), d(w), True, 1, 1, 1)
    tol = 1e-5 if dtype == torch.float32 else 2e-3
    for got, want in ((y, wy), (gx, wgx), (only_x, wgx), (gw, wgw), (only_w, wgw), (gb, wgb)):
        assert np.abs(d(got) - want).max() <= tol * max(1.0, np.abs(want).max())
    _lib.device_status()
