"""Builds libgmm_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and the extension module that describes tensors to it.

Run as ``python -m ops_transformer_b200._build`` or through ``__graft_entry__.build()``.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libgmm_b200.so")
DESCRIBE_PATH = os.path.join(PKG_DIR, "_describe.so")
DESCRIBE_SOURCE = os.path.join(CSRC, "describe.cpp")

SOURCES = ["gmm_sm100.cu", "gmm_simt.cu", "gmm_noalloc.cu", "ep_peer.cu", "moe_init_routing.cu", "view_copy.cu", "acl_shim.cpp", "op_api.cpp"]
HEADERS = ["gmm_common.h", "acl_shim.h"]

# -fmad=false: the epilogues reproduce the reference's separately rounded fp32 steps, so the compiler must not
# fuse a multiply and an add.  No fast-math.
NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-fmad=false",
    "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall", "-shared", "-cudart", "static",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def needs_build() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS]
    inc = os.path.join(ROOT, "include")
    for d, _, files in os.walk(inc):
        deps += [os.path.join(d, f) for f in files]
    deps.append(os.path.abspath(__file__))
    return any(os.path.getmtime(d) > t for d in deps)


def described_for() -> str:
    """What the extension module is bound to beside its source: the C++ interface of this torch and the ABI of this Python.  The
    module carries it (``built_for``), so that one left over from another installation is told from a fresh one."""
    import sysconfig

    import torch
    return f"describe.cpp for torch {torch.__version__}, {sysconfig.get_config_var('SOABI')}"


def describe_stale() -> bool:
    if not os.path.exists(DESCRIBE_PATH) or os.path.getmtime(DESCRIBE_PATH) < os.path.getmtime(DESCRIBE_SOURCE):
        return True
    with open(DESCRIBE_PATH, "rb") as f:
        return described_for().encode() + b"\0" not in f.read()


def build_describe(force: bool = False) -> str:
    """The extension module that writes a call's tensors into its description; g++ against torch's headers.  It is written under
    another name and moved into place, so that no process loads half of it."""
    import sysconfig

    import torch
    if not force and not describe_stale():
        return DESCRIBE_PATH
    root = os.path.dirname(torch.__file__)
    part = f"{DESCRIBE_PATH}.{os.getpid()}.part"
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DDESCRIBE_BUILT_FOR="{described_for()}"',
           "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I", sysconfig.get_paths()["include"], "-I", os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"),
           "-o", part, DESCRIBE_SOURCE, "-L", os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("g++ failed building _describe.so")
        os.replace(part, DESCRIBE_PATH)
    finally:
        if os.path.exists(part):
            os.remove(part)
    return DESCRIBE_PATH


def build_library(force: bool = False, verbose: bool = False) -> str:
    build_describe(force)
    if not force and not needs_build():
        return LIB_PATH
    extra = os.environ.get("GMM_B200_NVCC_EXTRA", "").split()  # e.g. -DGMM_DEBUG_KNOBS for kernel experiments
    cmd = [_nvcc()] + NVCC_FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + [
        "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-o", LIB_PATH,
    ] + [os.path.join(CSRC, s) for s in SOURCES]
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    r = subprocess.run(cmd, capture_output=True, text=True, env=env)
    if verbose or r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed building libgmm_b200.so")
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
