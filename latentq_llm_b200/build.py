"""In-tree build of liblatentq.so (nvcc, sm_100a only) and of the extension module _lqhost, the native host path of the short
calls (g++, against the torch and the Python that run this).

    python -m latentq_llm_b200.build [--force] [--verbose]

The shared libraries land next to this file so that they travel with the source
tree; nothing is installed into site-packages and nothing is JIT-cached.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "liblatentq.so")
HOST = os.path.join(PKG, "_lqhost" + sysconfig.get_config_var("EXT_SUFFIX"))       # the suffix names the Python
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC,-fvisibility=hidden", "-shared",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in [*deps, os.path.join(ROOT, "include", "latentq.h"), __file__])


def torch_build() -> str:
    """The torch that this process runs on.  Compiled into _lqhost, whose code holds torch's inline accessors: another torch
    may lay its tensors out differently."""
    import torch
    return f"{torch.__version__} {torch.version.git_version}"


def _host_stale() -> bool:
    if _stale(HOST, [os.path.join(CSRC, "lq_host.cpp")]):
        return True
    with open(HOST, "rb") as f:
        return torch_build().encode() not in f.read()


def build_host(force: bool = False) -> str:
    if not force and not _host_stale():
        return HOST
    import torch
    src, t, nvcc = os.path.join(CSRC, "lq_host.cpp"), os.path.dirname(torch.__file__), shutil.which(NVCC) or NVCC
    inc = [os.path.join(ROOT, "include"), os.path.join(t, "include"), os.path.join(t, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include"), sysconfig.get_paths()["include"]]
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                           f'-DLQ_TORCH_BUILD="{torch_build()}"', *[f"-I{i}" for i in inc], src, "-o", HOST, f"-L{os.path.join(t, 'lib')}", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda",
                           f"-L{PKG}", "-l:liblatentq.so", "-Wl,-rpath,$ORIGIN"])
    return HOST


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale(LIB, [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")]):
        build_host()
        return LIB
    cmd = [NVCC, *NVCC_FLAGS, "--threads", "0"]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB, *sources()]
    subprocess.check_call(cmd)
    build_host(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
