"""Layout kernels of the tensor-core tier (input to channels-last, grad_input and grad_weight back) at the edges of their tiles:
volumes off 32 and 64 voxels, channels off 64, enough blocks for the 64-voxel tiles, many taps."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests._util import make_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,tol", [("auto", 1e-4), ("bf16", 2e-2)])
@pytest.mark.parametrize("B,Cin,Cout,dims,G,k", [
    (1, 64, 64, (1, 1, 1), 1, 3), (2, 96, 192, (3, 5, 13), 3, 3), (1, 64, 128, (1, 5, 13), 2, 5), (2, 128, 64, (7, 25, 29), 1, 3),
    (1, 64, 192, (2, 7, 9), 1, 1), (2, 64, 64, (2, 80, 61), 2, 1),
])
def test_layout_kernels(mode, tol, B, Cin, Cout, dims, G, k):
    from d2conv3d_b200 import _lib, dconv_native as dn
    p = make_problem(700 + Cin, B, Cin, Cout, dims, k=k, padding=k // 2, G=G, dtype=np.float32)
    ts = [torch.from_numpy(p[n]).cuda().requires_grad_() for n in ("x", "geo", "mask", "weight", "bias")]
    old = _lib.get_math_mode()
    _lib.set_math_mode(mode)
    try:
        y = dn.deform_conv3d(*ts, 1, k // 2, 1, 1, G)
        y.backward(torch.from_numpy(p["gy"]).cuda())
    finally:
        _lib.set_math_mode(old)
    kw = dict(padding=k // 2, offset_groups=G)
    want = orc.deform_conv3d_fwd(p["x"], p["geo"], p["mask"], p["weight"], p["bias"], **kw)
    wants = orc.deform_conv3d_bwd(p["gy"], p["x"], p["geo"], p["mask"], p["weight"], True, **kw)
    for got, w in [(y.detach(), want), (ts[0].grad, wants[0]), (ts[3].grad, wants[3])]:
        assert np.abs(got.cpu().numpy() - w).max() <= tol * max(np.abs(w).max(), 1e-3)
    _lib.device_status()
