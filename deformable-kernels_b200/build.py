#!/usr/bin/env python3
"""Build libdk_b200.so (the C-ABI library) with nvcc for sm_100a and dk_torch.so (its torch binding) with g++, in-tree.

    python deformable-kernels_b200/build.py [--force] [--verbose]

The library depends on the CUDA runtime only (no torch, no ATen); the binding gets the library's entry points at load
time and needs neither nvcc nor a GPU.  Output: deformable-kernels_b200/lib/ (git-ignored).
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libdk_b200.so")
TORCH_SOURCE = os.path.join(CSRC, "dk_torch.cpp")
TORCH_LIB = os.path.join(LIB_DIR, "dk_torch.so")
SOURCES = ["dk_api.cu", "dk_local.cu", "dk_local_mma.cu", "dk_local_ring.cu", "dk_local_tc.cu", "dk_local_f32.cu", "dk_local_pieces.cu", "dk_deform.cu", "dk_deform_bins.cu", "dk_deform_lines.cu", "dk_deform_mma.cu", "dk_nd.cu", "dk_scale.cu", "dk_global.cu", "dk_static_scratch.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _nvcc():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _deps():
    out = [os.path.join(ROOT, "include", "dk_b200.h")]
    for f in os.listdir(CSRC):
        if f.endswith((".cu", ".cuh", ".h")):
            out.append(os.path.join(CSRC, f))
    return out


def _start_torch_binding(force):
    """The compile of dk_torch.so as a running process (None when it is up to date)."""
    newest = max(os.path.getmtime(p) for p in (TORCH_SOURCE, os.path.join(ROOT, "include", "dk_b200.h")))
    if not force and os.path.exists(TORCH_LIB) and os.path.getmtime(TORCH_LIB) >= newest:
        return None
    import sysconfig
    import torch
    base = os.path.dirname(torch.__file__)
    inc = os.path.join(base, "include")
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    includes = [os.path.join(ROOT, "include"), inc, os.path.join(inc, "torch", "csrc", "api", "include"),
                sysconfig.get_paths()["include"], os.path.join(cuda_home, "include")]
    libs = os.path.join(base, "lib")
    # the system's compiler, not $CXX: torch was linked against the shared libstdc++, and a toolchain that links its own copy
    # into the extension (two sets of iostream facets in one process) crashes in the first formatted error message
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wno-attributes",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
    for d in includes:
        cmd += ["-isystem" if d is not includes[0] else "-I", d]
    cmd += [TORCH_SOURCE, "-o", TORCH_LIB, "-L" + libs, "-Wl,-rpath," + libs, "-ltorch_python", "-ltorch", "-ltorch_cpu",
            "-ltorch_cuda", "-lc10", "-lc10_cuda"]
    return cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish(cmd, p, verbose):
    out, _ = p.communicate()
    if verbose or p.returncode:
        sys.stderr.write(out)
    if p.returncode:
        raise RuntimeError("compile failed: " + " ".join(cmd))


def build(force=False, verbose=False, defines=()):
    os.makedirs(LIB_DIR, exist_ok=True)
    binding = _start_torch_binding(force)
    try:
        return _build_library(force, verbose, defines)
    finally:
        if binding:
            _finish(*binding, verbose)


def _build_library(force, verbose, defines):
    obj_dir = os.path.join(HERE, "build")
    os.makedirs(obj_dir, exist_ok=True)
    newest = max(os.path.getmtime(p) for p in _deps())
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= newest:
        return LIB
    objs, procs = [], []
    for src in SOURCES:
        obj = os.path.join(obj_dir, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [_nvcc()] + NVCC_FLAGS + list(defines) + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for cmd, p in procs:
        _finish(cmd, p, verbose)
    subprocess.check_call([_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs + ["-lcudart"])
    return LIB


if __name__ == "__main__":
    # -DNAME arguments are passed to nvcc (e.g. -DDK_TUNING enables the experiment knobs read from the environment)
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, defines=[a for a in sys.argv[1:] if a.startswith("-D")]))
