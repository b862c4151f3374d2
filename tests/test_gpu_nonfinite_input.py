"""One NaN voxel in the input: the outputs whose samples touch it are NaN, and nothing else is -- not the other voxels of its tile,
not the other taps, channels or clips that the same producer thread serves afterwards, and not the other channels' weight
gradient.  Which samples touch it is worked out by the oracle in float64 from an indicator of that voxel.  A sample that has the
voxel for a corner of weight zero may be NaN or not (0 * NaN; the tiers differ in whether they read such a corner)."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests._util import make_problem

pytestmark = pytest.mark.gpu

SHAPES = [
    dict(B=3, Cin=64, Cout=64, dims=(4, 9, 10), G=1),             # ragged last tile, several clips per CTA
    dict(B=2, Cin=256, Cout=64, dims=(3, 7, 9), G=8),             # 32 channels per group (bf16: two groups a unit)
    dict(B=2, Cin=128, Cout=320, dims=(2, 8, 9), G=1),            # two weight stages a unit
    dict(B=2, Cin=128, Cout=64, dims=(3, 6, 8), G=2),             # 64 channels per group
    dict(B=2, Cin=24, Cout=40, dims=(3, 6, 7), G=2),              # CUDA-core tier
]


def cu(a):
    return torch.from_numpy(a).cuda()


def _run(p, x, field, G, keep):
    from d2conv3d_b200 import _lib, dconv_native as dn
    was = _lib.get_keep_samples()
    _lib.set_keep_samples(keep)
    try:
        ts = [cu(a).requires_grad_() for a in (x, p["geo"], p["mask"], p["weight"], p["bias"])]
        y = dn.dyn_dilated_conv3d(*ts, field, 1, 1, 1, 1, G) if field else dn.deform_conv3d(*ts, 1, 1, 1, 1, G)
        with torch.no_grad():
            y_inf = (dn.dyn_dilated_conv3d(*ts, field, 1, 1, 1, 1, G) if field else dn.deform_conv3d(*ts, 1, 1, 1, 1, G))
        grads = torch.autograd.grad(y, ts, cu(p["gy"]))
    finally:
        _lib.set_keep_samples(was)
    _lib.device_status()
    return y.detach(), y_inf, grads


@pytest.mark.parametrize("mode", ["auto", "bf16", "fp32"])
@pytest.mark.parametrize("field", [None, "xyz"])
@pytest.mark.parametrize("keep", [True, False])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_nan_voxel_stays_where_it_is_sampled(mode, field, keep, shape):
    import d2conv3d_b200
    cfg = dict(SHAPES[shape])
    G = cfg["G"]
    p = make_problem(4200 + shape, k=3, padding=1, dtype=np.float32, offset_std=2.0, field_mode=field, **cfg)
    clip, ch = 0, cfg["Cin"] // 2 + 5
    at = tuple(d // 2 for d in cfg["dims"])
    x = p["x"].copy()
    x[(clip, ch) + at] = np.nan

    def reached(corners):
        """Output voxels with a sample of channel ch that gives one of the input voxels `corners` a weight."""
        ind = np.zeros_like(p["x"], dtype=np.float64)
        for c in corners:
            ind[(clip, ch) + c] = 1.0
        kw = dict(padding=1, offset_groups=G, **(dict(mode=field) if field else {}))
        fwd = orc.dyn_dilated_conv3d_fwd if field else orc.deform_conv3d_fwd
        return fwd(ind, p["geo"].astype(np.float64), p["mask"].astype(np.float64), np.ones(p["weight"].shape), None, **kw)[:, :1] > 0

    touched = reached([at])
    # the voxel as an upper corner of weight zero: its lower neighbour then has a weight
    allowed = reached([tuple(np.subtract(at, d)) for d in np.ndindex(2, 2, 2)])
    assert 0 < touched.sum() and allowed.sum() < allowed[clip].size
    d2conv3d_b200.set_math_mode(mode)
    try:
        y0, _, g0 = _run(p, p["x"], field, G, keep)
        y, y_inf, g = _run(p, x, field, G, keep)
    finally:
        d2conv3d_b200.set_math_mode("auto")
    touched, allowed = cu(touched), cu(allowed)
    # the same sums in another order of atomics: fp32 rounding
    near = lambda a, b: bool(((a - b).abs() <= 1e-5 * b.abs().max()).all())  # noqa: E731
    for out in (y, y_inf):
        assert out[touched.expand_as(y)].isnan().all()
        assert near(out[~allowed.expand_as(y)], y0[~allowed.expand_as(y)])
    gx, ggeo, gmask, gw, gb = g
    assert near(gx, g0[0]) and near(gb, g0[4])               # do not depend on x
    others = [c for c in range(cfg["Cin"]) if c != ch]
    assert near(gw[:, others], g0[3][:, others]) and gw[:, ch].isnan().any()
    for a, b in ((ggeo, g0[1]), (gmask, g0[2])):             # per output voxel (and tap)
        assert a[clip].isnan().any() and near(a[clip + 1:], b[clip + 1:])
        assert near(a[~allowed.expand_as(a)], b[~allowed.expand_as(a)])


@pytest.mark.parametrize("mode", ["auto", "bf16"])
@pytest.mark.parametrize("field", ["x", "xy"])
@pytest.mark.parametrize("cin,dims", [(64, (3, 7, 9)), (256, (6, 15, 27))])
def test_corners_that_a_field_cannot_reach(mode, field, cin, dims):
    """An axis without a channel in the field: every sample lies on a voxel along it, and the next one up is no corner of it.  A NaN
    there leaves the gradients of the field and of the modulation alone."""
    import d2conv3d_b200
    p = make_problem(77, B=1, Cin=cin, Cout=64, dims=dims, k=3, padding=1, dtype=np.float32, field_mode=field, G=1)
    at = (0, 5) + tuple(d // 2 for d in dims)
    ind = np.zeros_like(p["x"], dtype=np.float64)
    for d in np.ndindex(2, 2):                              # rows and columns have a channel, frames have none
        ind[(0, 5) + tuple(np.subtract(at[2:], (0,) + d))] = 1.0
    reached = cu(orc.dyn_dilated_conv3d_fwd(ind, p["geo"].astype(np.float64), p["mask"].astype(np.float64), np.ones(p["weight"].shape),
                                            None, field, padding=1, offset_groups=1)[:, :1] > 0)
    assert reached.any() and not reached.all()
    x = p["x"].copy()
    x[at] = np.nan
    d2conv3d_b200.set_math_mode(mode)
    try:
        want, got = (_run(p, a, field, 1, True)[2] for a in (p["x"], x))
    finally:
        d2conv3d_b200.set_math_mode("auto")
    for a, b in ((got[1], want[1]), (got[2], want[2])):
        assert ((a - b).abs() <= 1e-5 * b.abs().max())[~reached.expand_as(a)].all()


@pytest.mark.skipif(os.environ.get("D2C_SM100_PAIR") == "1", reason="already inside")
def test_the_same_with_cta_pairs():
    """The opt-in pair kernel is chosen by an environment variable that the library reads once per process."""
    env = dict(os.environ, D2C_SM100_PAIR="1")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-m", "gpu", os.path.abspath(__file__), "-k", "bf16]"], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
