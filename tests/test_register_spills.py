"""Kernels whose inner loop must hold everything in registers, by ptxas' own report of the last build."""
import re

import pytest

from d2conv3d_b200 import build


def test_narrow_sampling_gradient_does_not_spill():
    """sample_grad_taps_kernel<FieldOut, kF32X, kNarrow = true>: the largest kernel of the backward of layers with 32 channels
    per offset group."""
    found = {name: r for name, r in build.ptxas_report().items() if re.search(r"sample_grad_taps_kernelILb.ELb.ELb1E", name)}
    if not found:
        pytest.skip("the library was not built here")
    assert len(found) == 4
    assert all(stack == stores == loads == 0 for _, stack, stores, loads in found.values()), found


# bytes that a thread loads back from the stack at most: the gathers of the forward's producers and the walk of the lists must stay in
# registers; what ptxas spills there now is a handful of set-up values
@pytest.mark.parametrize("kernel,variants,most", [("fwd_sm100_kernel", 12, 44), ("sample_grad_taps_kernel", 12, 16),
                                                  ("sample_grad_direct_kernel", 14, 16)])
def test_spills_stay_small(kernel, variants, most):
    found = {name: r for name, r in build.ptxas_report().items() if re.search(rf"\d{kernel}I", name)}
    if not found:
        pytest.skip("the library was not built here")
    assert len(found) == variants, sorted(found)
    assert all(loads <= most for _, _, _, loads in found.values()), found
