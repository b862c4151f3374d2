"""Exact (CUDA-core) tier against the oracle at the edges of its tiles: 256-voxel tiles that end early, fit or cross a clip,
contraction remainders of the 16-row steps, output tiles of 32 / 64 / 128 channels and one more, sampling from the
channels-last copy with four, two and one thread per voxel sharing, from NCDHW four channels at a time, and row by row."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests._util import make_problem

pytestmark = pytest.mark.gpu

CASES = [
    # (B, Cin, Cout, dims, G, groups, extra)
    (1, 16, 32, (4, 8, 8), 1, 1, {}),                                   # one full tile, sharing by four
    (3, 16, 33, (3, 5, 7), 1, 1, {}),                                   # tiles cross clips, one column past 32
    (1, 32, 64, (2, 5, 26), 4, 1, {}),                                  # 260 voxels, sharing by two
    (2, 48, 68, (2, 6, 11), 4, 1, {}),                                  # 12 channels per group: no sharing
    (1, 160, 136, (2, 4, 9), 2, 1, {}),                                 # two 128-wide output tiles
    (2, 32, 48, (3, 6, 6), 2, 2, dict(stride=(1, 2, 1), padding=(1, 0, 2), dilation=(1, 1, 2))),   # weight groups
    (1, 12, 9, (3, 6, 7), 3, 1, {}),                                    # fewer than 16 channels: NCDHW
    (2, 6, 4, (3, 4, 5), 2, 2, {}),                                     # 3 channels per group: row by row
    (1, 16, 16, (1, 1, 3), 1, 1, dict(k=1, padding=0)),                 # one contraction step
]


@pytest.mark.parametrize("ci", range(len(CASES)))
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("field", [None, "xyz"])
def test_exact_tier_tile_edges(ci, dtype, field):
    import d2conv3d_b200
    from d2conv3d_b200 import _lib, dconv_native
    B, cin, cout, dims, G, groups, extra = CASES[ci]
    cfg = dict(dict(k=3, padding=1), **extra)
    p = make_problem(7100 + ci, B, cin, cout, dims, G=G, groups=groups, dtype=dtype, offset_std=1.5, field_mode=field, **cfg)
    kw = dict(stride=p["stride"], padding=p["padding"], dilation=p["dilation"], groups=groups, offset_groups=G)
    d = lambda a: None if a is None else a.astype(np.float64)
    if field is None:
        want_y = orc.deform_conv3d_fwd(d(p["x"]), d(p["geo"]), d(p["mask"]), d(p["weight"]), d(p["bias"]), **kw)
        want = orc.deform_conv3d_bwd(d(p["gy"]), d(p["x"]), d(p["geo"]), d(p["mask"]), d(p["weight"]), True, **kw)
    else:
        want_y = orc.dyn_dilated_conv3d_fwd(d(p["x"]), d(p["geo"]), d(p["mask"]), d(p["weight"]), d(p["bias"]), field, **kw)
        want = orc.dyn_dilated_conv3d_bwd(d(p["gy"]), d(p["x"]), d(p["geo"]), d(p["mask"]), d(p["weight"]), True, field, **kw)
    ts = [torch.from_numpy(p[n]).cuda().requires_grad_() for n in ("x", "geo", "mask", "weight", "bias")]
    d2conv3d_b200.set_math_mode("fp32")
    try:
        if field is None:
            run = lambda: dconv_native.deform_conv3d(*ts, p["stride"], p["padding"], p["dilation"], groups, G)
        else:
            run = lambda: dconv_native.dyn_dilated_conv3d(*ts, field, p["stride"], p["padding"], p["dilation"], groups, G)
        y = run()
        assert torch.equal(y, run())                     # the forward is reproducible
        y.backward(torch.from_numpy(p["gy"]).cuda())
        _lib.device_status()
    finally:
        d2conv3d_b200.set_math_mode("auto")
    tol = 2e-5 if dtype == np.float32 else 1e-10
    for got, ref, n in zip([y.detach()] + [t.grad for t in ts], [want_y] + list(want), ("y", "x", "geo", "mask", "w", "b")):
        err = np.abs(got.cpu().numpy() - ref).max() / max(np.abs(ref).max(), 1e-30)
        assert err <= tol, (CASES[ci], n, err)
