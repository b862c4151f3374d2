"""What the channel-pair depthwise kernels bulk-copy lies inside the tensor, whatever the alignment of its first and last byte (the
header's own arithmetic, compiled for the host)."""
import os
import shutil
import subprocess

import pytest

from d2conv3d_b200 import build

PROGRAM = r"""
#include <cstdio>
#include "depthwise_pair.cuh"
int main() {
  long bad = 0, n = 0, all = 0;
  const uintptr_t page = 4096;
  for (int size = 2; size <= 4; size += 2)                       // bytes of an element
    for (uintptr_t base = page; base < page + 32; base += size)
      for (uintptr_t end = base + size; end <= base + 96; end += size)
        for (uintptr_t start = base; start < end; start += size)
          for (uintptr_t stop = start + size; stop <= end; stop += size) {
            const d2c::DwpSpan s(start, stop, base, end);
            ++n;
            // whole vectors inside the tensor, in the slot that begins at start's vector
            bad += s.lo % 16 || s.hi % 16 || s.lo > s.hi || s.lo < (start & ~(uintptr_t)15);
            bad += s.hi > s.lo && (s.lo < base || s.hi > end);
            // nothing is left to fetch by elements but what shares a vector with the tensor's first or last byte
            for (uintptr_t e = start; e < stop; e += size)
              if (e < s.lo || e >= s.hi) bad += !(e / 16 * 16 < base || e / 16 * 16 + 16 > end);
            all += s.lo <= start && s.hi >= stop;
          }
  printf("%ld %ld %ld\n", n, all, bad);
}
"""


def test_copied_bytes_lie_inside_the_tensor(tmp_path):
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None:
        pytest.skip("needs nvcc")
    src, exe = tmp_path / "span.cu", tmp_path / "span"
    src.write_text(PROGRAM)
    flags = [f for f in build.NVCC_FLAGS if f != "-O3"]
    subprocess.run([nvcc] + flags + ["-I", os.path.join(build.CSRC), "-o", str(exe), str(src)], check=True, capture_output=True)
    n, all_copied, bad = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and 0 < all_copied < n
