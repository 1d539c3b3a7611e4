"""In-tree build of libattn_sm100.so (hand-written CUDA for sm_100a only).

``python gpt.c_b200/build.py`` compiles every ``csrc/*.cu`` with nvcc for compute_100a and links
them into ``gpt.c_b200/lib/libattn_sm100.so`` next to the sources, so the library travels with the
tree, and ``csrc/torch_calls.cpp`` into the extension module the Python package calls it through.
nvcc cross-compiles: no GPU is needed to build.

What a file was built from stands beside it (``*.stamp``: a digest of every source and header it can include, of the
compiler flags and, for the extension, of the versions of torch and Python it is tied to), and it is built again when
that differs.
"""
from __future__ import annotations

import glob
import hashlib
import importlib.metadata
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(HERE, "..", "include")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libattn_sm100.so")
CALLS_SRC = os.path.join(CSRC, "torch_calls.cpp")
CALLS = os.path.join(LIB_DIR, "gptc_b200_calls.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v", "--expt-relaxed-constexpr",
]
CXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def digest(files: list[str], *words: str) -> str:
    h = hashlib.sha256("\n".join(words).encode())
    for path in sorted(files):
        with open(path, "rb") as f:
            h.update(f"\n{os.path.basename(path)}\n".encode() + f.read())
    return h.hexdigest()


def headers() -> list[str]:
    return [p for pattern in (os.path.join(CSRC, "*.h"), os.path.join(CSRC, "*.cuh"), os.path.join(INCLUDE, "*.h"))
            for p in glob.glob(pattern)]


def lib_digest() -> str:
    return digest(sources() + headers(), *NVCC_FLAGS)


def calls_digest() -> str:
    return digest([CALLS_SRC, *headers()], *CXX_FLAGS, importlib.metadata.version("torch"), sysconfig.get_config_var("SOABI"))


def is_built_from(path: str, wanted: str) -> bool:
    try:
        with open(path + ".stamp") as f:
            return os.path.exists(path) and f.read() == wanted
    except FileNotFoundError:
        return False


def write_stamp(path: str, wanted: str) -> None:
    with open(path + ".stamp", "w") as f:
        f.write(wanted)


def build_calls(force: bool = False) -> str:
    """The CPython extension over the library (torch's own headers and libraries; host compiler only)."""
    wanted = calls_digest()
    if not force and is_built_from(CALLS, wanted):
        return CALLS
    import torch
    from torch.utils import cpp_extension

    cmd = [os.environ.get("CXX", "g++"), *CXX_FLAGS,
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += ["-isystem" + d for d in cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]]
    cmd += [CALLS_SRC, "-o", CALLS, "-L" + LIB_DIR, "-lattn_sm100", "-Wl,-rpath,$ORIGIN"]
    cmd += ["-L" + d for d in cpp_extension.library_paths("cuda")]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("building the extension module failed:\n" + res.stdout + res.stderr)
    write_stamp(CALLS, wanted)
    return CALLS


def build(force: bool = False, verbose: bool = False) -> str:
    wanted = lib_digest()
    if not force and is_built_from(LIB, wanted):
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
    write_stamp(LIB, wanted)
    build_calls(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
