"""Sampling gradient of the tensor-core tier against the oracle where its lists of contributions can go wrong: volumes that are no
multiple of a brick or of 32 voxels, boxes of input voxels with more cells than a block keeps lists for, samples on voxels (corners
that weigh nothing), more taps than a block takes, several slices per offset group, 32 channels per offset group, all outside."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests._util import make_problem

pytestmark = pytest.mark.gpu

# of each gradient's scale, the bounds of the tier's two modes (bf16: the input is staged in fp16 there)
REL = {"auto": 1e-4, "bf16": 2e-2}

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


def check(ts, want, rel):
    for name, t, w in zip(("x", "geometry", "mask", "weight", "bias"), ts, want):
        scale = max(float(np.abs(w).max()), 1e-30)
        err = float(np.abs(t.grad.cpu().numpy() - w).max())
        assert err <= rel * scale, f"{name}: {err / scale:.2e} of scale"


@pytest.fixture
def dn(mode):
    import d2conv3d_b200
    from d2conv3d_b200 import _lib, dconv_native
    d2conv3d_b200.set_math_mode(mode)
    yield dconv_native
    d2conv3d_b200.set_math_mode("auto")
    _lib.device_status()


@pytest.mark.parametrize("mode", REL)
@pytest.mark.parametrize("name", CASES)
def test_offsets(dn, mode, name):
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
                                    padding=p["padding"], dilation=p["dilation"], groups=1, offset_groups=g), REL[mode])


@pytest.mark.parametrize("mode", REL)
@pytest.mark.parametrize("field", ["x", "xyz"])
@pytest.mark.parametrize("name", FIELDS)
def test_field(dn, mode, name, field):
    cfg = FIELDS[name]
    g = cfg.get("G", 1)
    p = make_problem(920, dtype=np.float32, padding=1, field_mode=field, **cfg)
    ts = [cu(p[k]) for k in ("x", "geo", "mask", "weight", "bias")]
    dn.dyn_dilated_conv3d(*ts, field, 1, 1, 1, 1, g).backward(torch.from_numpy(p["gy"]).cuda())
    check(ts, orc.dyn_dilated_conv3d_bwd(p["gy"], p["x"], p["geo"], p["mask"], p["weight"], True, field, padding=1,
                                         offset_groups=g), REL[mode])


def problem(cin, dims, g, k=(3, 3, 3), stride=(1, 1, 1), b=1, cout=64, seed=1):
    gen = torch.Generator("cuda").manual_seed(seed)
    rand = lambda *n: torch.randn(n, generator=gen, device="cuda")  # noqa: E731
    out = [(d - 1) // s + 1 for d, s in zip(dims, stride)]
    taps = k[0] * k[1] * k[2]
    return [rand(b, cin, *dims), rand(b, 3 * taps * g, *out), torch.sigmoid(rand(b, taps * g, *out)),
            rand(cout, cin, *k) * (taps * cin) ** -0.5, rand(cout)]


def gradients(dn, ts, geo, gy, g, k=(3, 3, 3), stride=(1, 1, 1), field=None):
    ts = [t.clone().requires_grad_() for t in [ts[0], geo] + ts[2:]]
    pad = tuple(n // 2 for n in k)
    y = dn.dyn_dilated_conv3d(*ts, field, stride, pad, 1, 1, g) if field else dn.deform_conv3d(*ts, stride, pad, 1, 1, g)
    return torch.autograd.grad(y, ts, gy)


# lists of contributions or every corner by itself, by what the host knows; "both": the positions decide, where it would be lists, from
# 2048 (32 voxels, tap, slice) on
ROUTES = [
    ("direct", "auto", dict(cin=64, dims=(4, 16, 16), g=1)),                          # three taps a block
    ("lists", "auto", dict(cin=64, dims=(8, 16, 16), g=1)),                           # four
    ("direct", "bf16", dict(cin=64, dims=(8, 16, 16), g=2)),                          # seven, 32 channels a group
    ("direct", "auto", dict(cin=128, dims=(8, 30, 54), g=2, k=(1, 1, 3))),
    ("both", "auto", dict(cin=128, dims=(8, 30, 54), g=2, k=(1, 1, 5))),
    ("direct", "bf16", dict(cin=128, dims=(8, 30, 54), g=2, k=(1, 1, 7))),
    ("both", "bf16", dict(cin=128, dims=(8, 30, 54), g=2, k=(2, 2, 2))),
    ("direct", "auto", dict(cin=64, dims=(16, 60, 60), g=1, stride=(2, 2, 2))),
    ("both", "auto", dict(cin=64, dims=(8, 60, 60), g=1, stride=(1, 2, 2))),
    ("both", "auto", dict(cin=128, dims=(16, 60, 60), g=1, stride=(2, 2, 2))),        # two slices
    ("direct", "auto", dict(cin=64, dims=(8, 60, 60), g=2, stride=(1, 2, 2))),
    ("direct", "auto", dict(cin=64, dims=(8, 30, 54), g=2, k=(1, 3, 5))),
    ("both", "auto", dict(cin=64, dims=(8, 40, 40), g=2)),
    ("direct", "bf16", dict(cin=64, dims=(8, 60, 60), g=2)),                          # 32 channels a group, fp16
    ("lists", "bf16", dict(cin=64, dims=(8, 15, 20), g=1)),                           # 75 x 27
    ("both", "bf16", dict(cin=64, dims=(8, 19, 16), g=1)),                            # 76 x 27
    ("both", "auto", dict(cin=64, dims=(8, 60, 107), g=1)),
]


@pytest.mark.parametrize("route,mode,cfg", ROUTES)
def test_routes(dn, route, mode, cfg):
    from torch.profiler import ProfilerActivity, profile
    cfg = dict(cfg)
    k, stride, g = cfg.get("k", (3, 3, 3)), cfg.get("stride", (1, 1, 1)), cfg["g"]
    ts = problem(**cfg)
    if k == (2, 2, 2):
        ts[1:3] = [t[:, :, 1:, 1:, 1:].contiguous() for t in ts[1:3]]
        pad_out = [d - 1 for d in cfg["dims"]]
    else:
        pad_out = list(ts[1].shape[2:])
    geo = 2 * ts[1]
    gy = torch.randn(1, 64, *pad_out, device="cuda")

    def run():
        if k == (2, 2, 2):
            leaf = [t.clone().requires_grad_() for t in [ts[0], geo] + ts[2:]]
            return torch.autograd.grad(dn.deform_conv3d(*leaf, 1, 0, 1, 1, g), leaf, gy)
        return gradients(dn, ts, geo, gy, g, k, stride)

    run()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        got = run()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    seen = [n for n, kernel in (("lists", "sample_grad_taps_kernel"), ("direct", "sample_grad_direct_kernel")) if kernel in names]
    assert seen == (["lists", "direct"] if route == "both" else [route])
    import d2conv3d_b200
    d2conv3d_b200.set_math_mode("fp32")
    for a, b in zip(got[:3], run()[:3]):
        assert float((a - b).abs().max()) <= REL[mode] * float(b.abs().max())


# positions as the call that asks them may find them: (across, in the plane), share of samples far outside
POSITIONS = {"zero": (0, 0, 0), "whole frames": (0, 2, 0), "ordinary": (2, 2, 0), "scattered": (0.5, 30, 0), "outside": (2, 2, 0.9)}


@pytest.mark.parametrize("mode", REL)
@pytest.mark.parametrize("cin,g,dims", [(64, 1, (8, 60, 107)), (128, 1, (8, 48, 64)), (64, 2, (8, 60, 107)), (256, 4, (7, 9, 13)),
                                        (64, 1, (5, 23, 29))])
@pytest.mark.parametrize("name", POSITIONS)
def test_asked(dn, mode, cin, g, dims, name):
    import d2conv3d_b200
    z, yx, out = POSITIONS[name]
    ts = problem(cin, dims, g)
    geo = ts[1] * torch.tensor([z, yx, yx], device="cuda", dtype=torch.float32).repeat(27 * g)[None, :, None, None, None]
    geo += 1000.0 * (torch.rand_like(geo) < out)
    gy = torch.randn(1, 64, *dims, device="cuda")
    got = gradients(dn, ts, geo, gy, g)
    d2conv3d_b200.set_math_mode("fp32")
    for a, b in zip(got, gradients(dn, ts, geo, gy, g)):
        assert float((a - b).abs().max()) <= REL[mode] * float(b.abs().max())


@pytest.mark.parametrize("mode", REL)
@pytest.mark.parametrize("ones", [True, False])
def test_asked_field(dn, mode, ones):
    """A field of ones puts every sample on a voxel; two slices per group."""
    import d2conv3d_b200
    ts = problem(128, (8, 48, 64), 1)
    geo = torch.ones(1, 3, 8, 48, 64, device="cuda")
    if not ones:
        geo += torch.nn.functional.softplus(ts[1][:, :3])
    gy = torch.randn(1, 64, 8, 48, 64, device="cuda")
    got = gradients(dn, ts, geo, gy, 1, field="xyz")
    d2conv3d_b200.set_math_mode("fp32")
    for a, b in zip(got, gradients(dn, ts, geo, gy, 1, field="xyz")):
        assert float((a - b).abs().max()) <= REL[mode] * float(b.abs().max())


@pytest.mark.parametrize("mode", ["auto"])
def test_asked_chunk_by_chunk(dn, mode):
    """Two clips in chunks of one, offsets zero in one of them: each chunk's positions decide for it; the word is this call's own."""
    import d2conv3d_b200
    ts = problem(64, (8, 60, 107), 1, b=2)
    gy = torch.randn(2, 64, 8, 60, 107, device="cuda")
    was = dn._ops.config.get_max_intermediate_elements()
    for first in (0, 1):
        geo = 2 * ts[1]
        geo[first] = 0
        d2conv3d_b200.set_math_mode(mode)
        dn._ops.config.set_max_intermediate_elements(64 * 27 * 8 * 60 * 107)
        try:
            got = gradients(dn, ts, geo, gy, 1)
        finally:
            dn._ops.config.set_max_intermediate_elements(was)
        d2conv3d_b200.set_math_mode("fp32")
        for a, b in zip(got, gradients(dn, ts, geo, gy, 1)):
            assert float((a - b).abs().max()) <= REL[mode] * float(b.abs().max())


@pytest.mark.parametrize("mode", REL)
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("cin,g,dims", [(64, 1, (3, 7, 9)), (64, 1, (8, 17, 16)), (256, 1, (6, 13, 16)), (128, 4, (8, 17, 16))])
def test_output_gradient_that_is_not_finite(dn, mode, bad, whole, cin, g, dims):
    """One voxel of grad_out: the input voxels that it gives a weight are not finite, nothing else is; a corner of weight zero takes
    nothing (whole: every sample lies on a voxel).  Without and with lists."""
    p = make_problem(930, dtype=np.float32, B=1, Cin=cin, Cout=64, dims=dims, padding=1, offset_std=2.0, G=g)
    if whole:
        p["geo"] = np.rint(p["geo"]).astype(np.float32)
    at = (slice(None), slice(None)) + tuple(d // 2 for d in dims)
    ind = np.zeros(p["gy"].shape, np.float64)
    ind[at] = 1.0
    wide = {n: p[n].astype(np.float64) for n in ("x", "geo", "mask")}
    reached = torch.from_numpy(orc.deform_conv3d_bwd(ind, wide["x"], wide["geo"], wide["mask"], np.ones(p["weight"].shape), True, padding=1,
                                                     offset_groups=g)[0] > 0).cuda()
    assert reached.any() and not reached.all()
    ts = [torch.from_numpy(p[n]).cuda() for n in ("x", "geo", "mask", "weight", "bias")]
    gy = torch.from_numpy(p["gy"]).cuda()
    want = gradients(dn, ts, ts[1], gy, g)
    gy[at] = bad
    got = gradients(dn, ts, ts[1], gy, g)
    assert not got[0][reached].isfinite().any()
    assert float((got[0] - want[0])[~reached].abs().max()) <= 1e-5 * float(want[0].abs().max())
    for a, b in zip(got[1:3], want[1:3]):                     # per output voxel and tap
        a, b = a.clone(), b.clone()
        a[at] = b[at] = 0
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
