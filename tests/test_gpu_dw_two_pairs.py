"""Weight gradient from kept samples with two slice pairs a CTA (at most 256 output channels, enough work for every multiprocessor)
against the kernel that gathers the samples again: an odd number of pairs (the last CTA has one), an odd number of slices (the last
pair has one), accumulators of 64, 192 and 256 columns, a ragged last tile."""
import re

import pytest
import torch

pytestmark = pytest.mark.gpu

BOUND = {"auto": 1e-4, "bf16": 2e-2}        # of the gradient's scale, the bounds of the two modes


@pytest.mark.parametrize("mode", BOUND)
@pytest.mark.parametrize("cin,cout,g,dims", [(192, 64, 1, (4, 60, 70)), (320, 256, 1, (3, 60, 71)), (128, 192, 4, (8, 60, 107)),
                                             (256, 256, 8, (8, 33, 55))])
def test_equals_gather(mode, cin, cout, g, dims):
    from torch.profiler import ProfilerActivity, profile
    import d2conv3d_b200
    from d2conv3d_b200 import _lib, dconv_native
    gen = torch.Generator("cuda").manual_seed(7)
    rand = lambda *s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    ts = [rand(1, cin, *dims), 2 * rand(1, 81 * g, *dims), torch.sigmoid(rand(1, 27 * g, *dims)),
          rand(cout, cin, 3, 3, 3) * (27 * cin) ** -0.5, rand(cout)]
    gy = rand(1, cout, *dims)
    ts[3].requires_grad_()
    res = []
    try:
        d2conv3d_b200.set_math_mode(mode)
        for keep in (True, False):
            d2conv3d_b200.set_keep_samples(keep)
            _lib.profile_read(); _lib.profile_enable(True)
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                res.append(torch.autograd.grad(dconv_native.deform_conv3d(*ts, 1, 1, 1, 1, g), ts[3], gy)[0])
                torch.cuda.synchronize()
            _lib.profile_enable(False)
            assert ("bwd_dw_sm100_saved" if keep else "bwd_dw_sm100") in [n for n, _ in _lib.profile_read()]
            # dw_saved_sm100_kernel<hi/lo mode, two pairs>
            ran = re.findall(r"dw_saved_sm100_kernel<(\d), (\d)>", " ".join(e.key for e in prof.key_averages()))
            assert ran == ([("1" if mode == "auto" else "0", "1")] if keep else [])
    finally:
        d2conv3d_b200.set_math_mode("auto")
        d2conv3d_b200.set_keep_samples(True)
    _lib.device_status()
    assert float((res[0] - res[1]).abs().max()) <= BOUND[mode] * float(res[1].abs().max())
