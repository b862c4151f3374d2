"""Builds libd2conv3d.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m d2conv3d_b200.build [--force] [--verbose] [--unit-trace]

The library links only the CUDA runtime (statically); it has no dependency on
torch or Python.  _C.so, built beside it, is the PyTorch front-end (csrc/torch_ops.cpp:
autograd nodes and argument handling over the library's C ABI).  A GPU is not needed
to build either.
"""
import os
import re
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libd2conv3d.so")
TORCH_SRC = os.path.join(CSRC, "torch_ops.cpp")
TORCH_LIB = os.path.join(HERE, "_C.so")
OBJ_DIR = os.path.join(HERE, "build")
TORCH_STAMP = os.path.join(OBJ_DIR, "torch_ops.stamp")

SOURCES = ["d2c_api.cu", "depthwise.cu", "deform_sm100_fwd.cu", "deform_sm100_bwd.cu", "deform_sm100_dw.cu",
           "deform_exact_f32.cu", "deform_exact_f64.cu", "act_norm.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", INCLUDE,
]


def _nvcc():
    return os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def _deps():
    out = [os.path.join(INCLUDE, "d2conv3d.h")]
    for f in os.listdir(CSRC):
        if not f.endswith(".cpp"):
            out.append(os.path.join(CSRC, f))
    return out


def needs_build():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(d) > t for d in _deps())


def _torch_stamp():
    """What the front-end was compiled against; it does not load, or misbehaves, with another one."""
    import torch
    return f"torch {torch.__version__}, python {sys.version_info.major}.{sys.version_info.minor}"


def _torch_needs_build():
    if not os.path.exists(TORCH_LIB) or not os.path.exists(TORCH_STAMP):
        return True
    with open(TORCH_STAMP) as f:
        if f.read() != _torch_stamp():
            return True
    t = os.path.getmtime(TORCH_LIB)
    return any(os.path.getmtime(d) > t for d in (TORCH_SRC, os.path.join(INCLUDE, "d2conv3d.h")))


def build_torch(force=False):
    """The PyTorch front-end _C.so: csrc/torch_ops.cpp against the installed torch, linked to libd2conv3d.so (which it
    finds beside itself)."""
    if not force and not _torch_needs_build():
        return TORCH_LIB
    os.makedirs(OBJ_DIR, exist_ok=True)
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    inc = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], INCLUDE, "/usr/local/cuda/include"]
    lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_C", "-DTORCH_API_INCLUDE_EXTENSION_H",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
           + [a for i in inc for a in ("-isystem", i)]
           + [TORCH_SRC, "-o", TORCH_LIB, "-L", lib_dir, "-lc10", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda",
              "-ltorch_python", "-L", HERE, "-l:libd2conv3d.so", "-L", "/usr/local/cuda/lib64", "-lcudart",
              "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{lib_dir}"])
    p = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if p.returncode != 0:
        sys.stderr.write(p.stdout)
        raise RuntimeError("building the PyTorch front-end failed")
    with open(TORCH_STAMP, "w") as f:
        f.write(_torch_stamp())
    return TORCH_LIB


def build(force=False, verbose=False, unit_trace=False):
    """The kernel library, then the PyTorch front-end.

    unit_trace: compile the forward kernel's per-unit timeline instrumentation in (-DD2C_UNIT_TRACE, see
    csrc/deform_sm100_fwd_kernel.cuh and unit_trace.py); always rebuilds.  Build again without it afterwards: the
    instrumented library is for measurements only."""
    if not force and not unit_trace and not needs_build():
        build_torch()
        return LIB
    os.makedirs(OBJ_DIR, exist_ok=True)
    extra = ["-Xptxas", "-v"] + (["-DD2C_UNIT_TRACE"] if unit_trace else [])
    procs = []
    objs = []
    for src in SOURCES:
        obj = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [_nvcc()] + NVCC_FLAGS + extra + ["-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        with open(os.path.join(OBJ_DIR, src.replace(".cu", ".ptxas")), "w") as f:
            f.write(out)
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {src} ---\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed building libd2conv3d.so")
    cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-cudart", "static", "-Xlinker", "-soname=libd2conv3d.so"]
    subprocess.run(cmd, check=True)
    build_torch(force)
    return LIB


def ptxas_report():
    """{mangled kernel name: (registers, bytes of stack, of spill stores, of spill loads)} of the last build here; kernels of
    sources whose report is missing are absent."""
    out = {}
    for src in SOURCES:
        path = os.path.join(OBJ_DIR, src.replace(".cu", ".ptxas"))
        if not os.path.exists(path):
            continue
        with open(path) as f:
            text = f.read()
        for name, stack, stores, loads, regs in re.findall(
                r"Compiling entry function '(\w+)'.*?(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads"
                r".*?Used (\d+) registers", text, re.S):
            out[name] = (int(regs), int(stack), int(stores), int(loads))
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, unit_trace="--unit-trace" in sys.argv))
