"""Sampling gradient of the tensor-core tier against the oracle where its lists of contributions can go wrong: volumes that are no
multiple of a brick or of 32 voxels, boxes of input voxels with more cells than a block keeps lists for, samples on voxels (corners
that weigh nothing), more taps than a block takes, several slices per offset group, 32 channels per offset group, all outside."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests._util import make_problem

pytestmark = pytest.mark.gpu

REL = 1e-4        # of each gradient's scale, the bound of the tier's fp32-parity mode

CASES = {
    "one voxel": dict(B=1, Cin=64, Cout=64, dims=(1, 1, 1)),
    "rows shorter than a brick": dict(B=2, Cin=64, Cout=64, dims=(3, 5, 3)),
    "last brick of one column": dict(B=1, Cin=64, Cout=64, dims=(5, 3, 17)),
    "one frame": dict(B=1, Cin=128, Cout=64, dims=(1, 7, 33), G=2),
    "box larger than the lists": dict(B=1, Cin=64, Cout=64, dims=(12, 40, 40), offset_std=25.0),
    "all samples outside": dict(B=1, Cin=64, Cout=64, dims=(3, 6, 7), shift=1000.0),
    "on voxels": dict(B=1, Cin=64, Cout=64, dims=(4, 9, 10), whole=True),
    "more than 27 taps": dict(B=1, Cin=64, Cout=64, dims=(4, 8, 11), k=(3, 3, 5), padding=(1, 1, 2)),
    "four slices a group": dict(B=1, Cin=256, Cout=64, dims=(3, 9, 10)),
    "four slices a group, on voxels": dict(B=1, Cin=256, Cout=64, dims=(3, 9, 10), whole=True),
    "32 channels a group": dict(B=2, Cin=128, Cout=64, dims=(3, 7, 9), G=4),
    "strided": dict(B=1, Cin=64, Cout=64, dims=(5, 12, 13), stride=(1, 2, 2), dilation=(2, 1, 1), padding=(2, 1, 1)),
}
FIELDS = {
    "one slice": dict(B=2, Cin=64, Cout=64, dims=(3, 7, 9)),
    "two slices a group": dict(B=1, Cin=256, Cout=64, dims=(4, 7, 9), G=2),
    "32 channels a group": dict(B=1, Cin=128, Cout=64, dims=(4, 7, 9), G=4),
}


def cu(a):
    return torch.from_numpy(a).cuda().requires_grad_()


def check(ts, want):
    for name, t, w in zip(("x", "geometry", "mask", "weight", "bias"), ts, want):
        scale = max(float(np.abs(w).max()), 1e-30)
        err = float(np.abs(t.grad.cpu().numpy() - w).max())
        assert err <= REL * scale, f"{name}: {err / scale:.2e} of scale"


@pytest.fixture
def dn():
    import d2conv3d_b200
    from d2conv3d_b200 import _lib, dconv_native
    d2conv3d_b200.set_math_mode("auto")
    yield dconv_native
    _lib.device_status()


@pytest.mark.parametrize("name", CASES)
def test_offsets(dn, name):
    cfg = dict(CASES[name])
    shift, whole, g = cfg.pop("shift", 0.0), cfg.pop("whole", False), cfg.get("G", 1)
    cfg.setdefault("padding", 1)
    cfg.setdefault("offset_std", 2.0)
    p = make_problem(910, dtype=np.float32, **cfg)
    if whole:
        p["geo"] = np.rint(p["geo"]).astype(np.float32)
    p["geo"] += np.float32(shift)
    ts = [cu(p[k]) for k in ("x", "geo", "mask", "weight", "bias")]
    dn.deform_conv3d(*ts, p["stride"], p["padding"], p["dilation"], 1, g).backward(torch.from_numpy(p["gy"]).cuda())
    check(ts, orc.deform_conv3d_bwd(p["gy"], p["x"], p["geo"], p["mask"], p["weight"], True, stride=p["stride"],
                                    padding=p["padding"], dilation=p["dilation"], groups=1, offset_groups=g))


@pytest.mark.parametrize("field", ["x", "xyz"])
@pytest.mark.parametrize("name", FIELDS)
def test_field(dn, name, field):
    cfg = FIELDS[name]
    g = cfg.get("G", 1)
    p = make_problem(920, dtype=np.float32, padding=1, field_mode=field, **cfg)
    ts = [cu(p[k]) for k in ("x", "geo", "mask", "weight", "bias")]
    dn.dyn_dilated_conv3d(*ts, field, 1, 1, 1, 1, g).backward(torch.from_numpy(p["gy"]).cuda())
    check(ts, orc.dyn_dilated_conv3d_bwd(p["gy"], p["x"], p["geo"], p["mask"], p["weight"], True, field, padding=1,
                                         offset_groups=g))
