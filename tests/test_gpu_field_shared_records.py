"""Dilation-field forward on the tensor-core tier with several offset groups (one record per tap and voxel, modulation rows
apart): volumes that end inside a tile and off a 16-byte boundary, one to several clips, both arithmetics, 32 channels per
group, with and without a mask."""
import numpy as np
import pytest
import torch


from oracle import oracle as orc
from tests._util import make_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,tol", [("auto", 1e-4), ("bf16", 1e-2)])
@pytest.mark.parametrize("B,Cin,G,dims", [(1, 64, 2, (1, 1, 3)), (2, 128, 2, (3, 5, 7)), (3, 256, 8, (2, 9, 7)), (1, 128, 4, (4, 8, 8)),
                                          (2, 64, 2, (3, 7, 9))])
@pytest.mark.parametrize("masked", [True, False])
def test_groups_share_records(mode, tol, B, Cin, G, dims, masked):
    from d2conv3d_b200 import _lib, dconv_native as dn
    p = make_problem(900 + B, B, Cin, 64, dims, padding=1, G=G, dtype=np.float32, field_mode="xyz")
    mask = p["mask"] if masked else np.ones_like(p["mask"])
    cu = lambda a: torch.from_numpy(a).cuda()
    old = _lib.get_math_mode()
    _lib.set_math_mode(mode)
    try:
        y = dn.dyn_dilated_conv3d(cu(p["x"]), cu(p["geo"]), cu(mask) if masked else None, cu(p["weight"]), cu(p["bias"]), "xyz",
                                  1, 1, 1, 1, G).cpu().numpy()
    finally:
        _lib.set_math_mode(old)
    want = orc.dyn_dilated_conv3d_fwd(p["x"], p["geo"], mask, p["weight"], p["bias"], "xyz", padding=1, offset_groups=G)
    assert np.abs(y - want).max() <= tol * np.abs(want).max()
    _lib.device_status()
