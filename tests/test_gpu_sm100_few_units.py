"""Tensor-core forward where its 24 gather warps have few items of 8 rows, or a number that does not divide among them: calls of one to
a few units (taps x channel slices), tiles of one row to one row more than a tile."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests._util import make_problem

pytestmark = pytest.mark.gpu

REL = {"auto": 1e-4, "bf16": 1e-2}        # of the output's scale, the bounds of the two modes


@pytest.mark.parametrize("mode", REL)
@pytest.mark.parametrize("k", [(1, 1, 1), (1, 1, 2), (1, 1, 3), (1, 2, 2), (1, 1, 5), (1, 2, 3)])
@pytest.mark.parametrize("dims", [(1, 1, 8), (1, 4, 33), (2, 9, 17)])
def test_few_units(mode, k, dims):
    import d2conv3d_b200
    from d2conv3d_b200 import _lib, dconv_native
    dims = tuple(n + kk - 1 for n, kk in zip(dims, k))                  # output of the size given
    p = make_problem(930, 1, 64, 64, dims, k=k, dtype=np.float32, offset_std=1.5)
    d2conv3d_b200.set_math_mode(mode)
    try:
        y = dconv_native.deform_conv3d(*(torch.from_numpy(p[n]).cuda() for n in ("x", "geo", "mask", "weight", "bias")), 1, 0, 1, 1, 1)
    finally:
        d2conv3d_b200.set_math_mode("auto")
    _lib.device_status()
    want = orc.deform_conv3d_fwd(p["x"], p["geo"], p["mask"], p["weight"], p["bias"])
    assert np.abs(y.cpu().numpy() - want).max() <= REL[mode] * np.abs(want).max()
