"""In-tree build of libattn_sm100.so (hand-written CUDA for sm_100a only).

``python gpt.c_b200/build.py`` compiles every ``csrc/*.cu`` with nvcc for compute_100a and links
them into ``gpt.c_b200/lib/libattn_sm100.so`` next to the sources, so the library travels with the
tree, and ``csrc/torch_calls.cpp`` into the extension module the Python package calls it through.
nvcc cross-compiles: no GPU is needed to build.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libattn_sm100.so")
CALLS_SRC = os.path.join(CSRC, "torch_calls.cpp")
CALLS = os.path.join(LIB_DIR, "gptc_b200_calls.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v", "--expt-relaxed-constexpr",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def up_to_date() -> bool:
    if not os.path.exists(LIB):
        return False
    deps = sources() + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    deps.append(os.path.join(HERE, "..", "include", "attn_sm100.h"))
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(d) <= t for d in deps)


def build_calls(force: bool = False) -> str:
    """The CPython extension over the library (torch's own headers and libraries; host compiler only)."""
    if not force and os.path.exists(CALLS) and os.path.getmtime(CALLS) >= os.path.getmtime(CALLS_SRC):
        return CALLS
    import torch
    from torch.utils import cpp_extension

    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += ["-isystem" + d for d in cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]]
    cmd += [CALLS_SRC, "-o", CALLS, "-L" + LIB_DIR, "-lattn_sm100", "-Wl,-rpath,$ORIGIN"]
    cmd += ["-L" + d for d in cpp_extension.library_paths("cuda")]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("building the extension module failed:\n" + res.stdout + res.stderr)
    return CALLS


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        build_calls()
        return LIB
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = os.environ.get("NVCC", "nvcc")
    cmd = [nvcc, *NVCC_FLAGS, "-shared", "-o", LIB, *sources()]
    res = subprocess.run(cmd, capture_output=True, text=True)
    log = res.stdout + res.stderr
    with open(os.path.join(LIB_DIR, "build.log"), "w") as f:
        f.write(" ".join(cmd) + "\n" + log)
    if verbose or res.returncode != 0:
        print(log)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed, see gpt.c_b200/lib/build.log")
    build_calls(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
