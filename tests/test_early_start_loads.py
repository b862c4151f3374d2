"""A kernel that starts beside the one that writes its operands must not load them as read-only data: ld.global.nc and __ldg promise
that the words do not change for the kernel's life, and the compiler may move them above the wait.  The forward kernel starts that
way, so everything but the bias, which no kernel of a call writes, is read by ordinary loads after the wait."""
import os
import re

import d2conv3d_b200

CSRC = os.path.join(os.path.dirname(d2conv3d_b200.__file__), "csrc")


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_forward_kernel_reads_staged_operands_by_ordinary_loads():
    kernel = code("deform_sm100_fwd_kernel.cuh")
    assert "wait_for_kernels_before()" in kernel
    assert set(re.findall(r"__ldg\(\s*([\w.]+)", kernel)) == {"p.bias"}
    assert not re.search(r"ldg_nc|global\.nc", kernel)
    assert re.search(r"const volatile int\*>\(p\.nan_flag\)", kernel)
    helpers = set(re.findall(r"ptx::(ldg_\w+)\(", kernel))
    assert helpers
    text = code("sm100_ptx.cuh")
    for h in helpers:
        body = text[text.index(f" {h}("):]
        body = body[:body.index("\n}")]
        assert "asm volatile" in body and "ld.global.v" in body, h
