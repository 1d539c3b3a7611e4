"""B200-native causal self-attention for gpt.c: ctypes access to ``libattn_sm100.so``.

The product is the C-ABI library declared in ``include/attn_sm100.h`` (hand-written sm_100a CUDA).
This package only loads it and offers a thin convenience layer that takes ``torch`` CUDA tensors
for device memory and streams; every call goes through the C ABI with raw pointers, the tensor-level
ones by way of a small extension module (``csrc/torch_calls.cpp``).  There is no
CPU or PyTorch fallback: if the library is missing or the device is not an sm_100 GPU the calls
raise.

The directory name contains a dot, so it cannot be imported with a plain ``import`` statement;
load it with ``importlib`` (see ``load_package`` in ``__graft_entry__.py``) under the module name
``gptc_b200``.
"""
from __future__ import annotations

import ctypes
import os

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "lib", "libattn_sm100.so")
CALLS_PATH = os.path.join(HERE, "lib", "gptc_b200_calls.so")
HEADER_PATH = os.path.join(HERE, "..", "include", "attn_sm100.h")

FLAG_FORCE_GENERIC = 1
FLAG_PREPARE_ONLY = 2
FLAG_CORE_ONLY = 4

# name -> (restype, argtypes); must list every function include/attn_sm100.h declares
_c = ctypes
SIGNATURES = {
    "attn_sm100_version": (_c.c_int, []),
    "attn_sm100_init": (_c.c_int, []),
    "attn_sm100_saved_bytes": (_c.c_size_t, [_c.c_int] * 4),
    "attn_sm100_backward_scratch_bytes": (_c.c_size_t, [_c.c_int] * 4),
    "attn_sm100_forward": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 5 + [_c.c_void_p]),
    "attn_sm100_backward": (_c.c_int, [_c.c_void_p] * 6 + [_c.c_int] * 5 + [_c.c_void_p]),
    "attn_sm100_forward_static": (_c.c_int, [_c.c_void_p] * 3 + [_c.c_int] * 4 + [_c.c_void_p]),
    "attn_sm100_static_status": (_c.c_int, [_c.POINTER(_c.c_int), _c.c_int]),
    "attn_sm100_selftest_wait_limit": (_c.c_int, [_c.c_uint, _c.c_void_p]),
    "attn_sm100_device_status": (_c.c_int, [_c.POINTER(_c.c_int), _c.c_int]),
    "attn_sm100_strerror": (_c.c_char_p, [_c.c_int]),
    "linear_sm100_forward": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 3 + [_c.c_void_p]),
    "linear_sm100_backward_scratch_bytes": (_c.c_size_t, [_c.c_int] * 3),
    "linear_sm100_backward": (_c.c_int, [_c.c_void_p] * 7 + [_c.c_int] * 3 + [_c.c_void_p]),
    "linear_sm100_backward_plan": (_c.c_int, [_c.c_int] * 6 + [_c.POINTER(_c.c_int)]),
    "layernorm_sm100_forward": (_c.c_int, [_c.c_void_p] * 3 + [_c.c_float] + [_c.c_void_p] * 3 + [_c.c_int] * 2 + [_c.c_void_p]),
    "layernorm_sm100_backward": (_c.c_int, [_c.c_void_p] * 8 + [_c.c_int] * 2 + [_c.c_void_p]),
    "tensor_sm100_fill": (_c.c_int, [_c.c_void_p, _c.c_size_t, _c.c_float, _c.c_void_p]),
    "tensor_sm100_arange": (_c.c_int, [_c.c_void_p, _c.c_size_t, _c.c_int, _c.c_int, _c.c_void_p]),
    "tensor_sm100_copy": (_c.c_int, [_c.c_void_p, _c.c_void_p, _c.c_size_t, _c.c_void_p]),
    "tensor_sm100_axpy": (_c.c_int, [_c.c_size_t, _c.c_float, _c.c_void_p, _c.c_void_p, _c.c_void_p]),
    "tensor_sm100_gelu_forward": (_c.c_int, [_c.c_void_p, _c.c_void_p, _c.c_size_t, _c.c_void_p]),
    "tensor_sm100_gelu_backward": (_c.c_int, [_c.c_void_p, _c.c_void_p, _c.c_void_p, _c.c_size_t, _c.c_void_p]),
    "xent_sm100_forward": (_c.c_int, [_c.c_void_p] * 4 + [_c.c_int] * 2 + [_c.c_void_p]),
    "xent_sm100_selftest_wait_limit": (_c.c_int, [_c.c_void_p] * 4 + [_c.c_int] * 3 + [_c.c_uint, _c.c_void_p]),
    "xent_sm100_backward": (_c.c_int, [_c.c_void_p] * 4 + [_c.c_int] * 2 + [_c.c_void_p]),
    "adamw_sm100_step": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] + [_c.c_float] * 5 + [_c.c_int, _c.c_void_p]),
}

_lib = None
_calls_module = None
_entry_classes = {}  # name of an entry point -> the class of its function in lib()


class AttnError(RuntimeError):
    def __init__(self, code: int, where: str):
        self.code = code
        msg = lib().attn_sm100_strerror(code).decode()
        super().__init__(f"{where} failed with status {code}: {msg}")


def lib() -> ctypes.CDLL:
    """Load libattn_sm100.so (once).  Raises if it has not been built."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise FileNotFoundError(
                f"{LIB_PATH} is missing: build it with `python gpt.c_b200/build.py`; there is no fallback path")
        handle = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in SIGNATURES.items():
            fn = getattr(handle, name)
            fn.restype = res
            fn.argtypes = args
            _entry_classes[name] = fn.__class__ = _entry_class(handle._FuncPtr)
        _lib = handle
        _shorten_calls()
    return _lib


def _entry_class(plain):
    """A class for one function of the library: a ctypes function like any other, which the extension module may give a
    shorter way from a call's arguments to the C ABI.  That way knows the signature above, so a function that is given
    another one becomes an ordinary ctypes function."""

    class Entry(plain):
        _flags_ = plain._flags_
        _restype_ = plain._restype_

        def __setattr__(self, name, value):
            if name in ("restype", "argtypes", "errcheck"):
                self.__class__ = plain
            plain.__setattr__(self, name, value)

        def __delattr__(self, name):
            if name in ("restype", "argtypes", "errcheck"):
                self.__class__ = plain
            plain.__delattr__(self, name)

    return Entry


def _shorten_calls():
    if _calls_module is not None:
        _calls_module.shorten_calls(_entry_classes)


def _calls():
    """The extension module over the C ABI (once).  Raises if it has not been built."""
    global _calls_module
    if _calls_module is None:
        import importlib.util

        import torch  # noqa: F401  (its libraries have to be loaded first)

        lib()
        if not os.path.exists(CALLS_PATH):
            raise FileNotFoundError(
                f"{CALLS_PATH} is missing: build it with `python gpt.c_b200/build.py`; there is no fallback path")
        spec = importlib.util.spec_from_file_location("gptc_b200_calls", CALLS_PATH)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        mod.set_error(AttnError)
        _calls_module = mod
        _shorten_calls()
    return _calls_module


def _raw(stream):
    return None if stream is None else stream.cuda_stream


def _check(code: int, where: str) -> None:
    if code != 0:
        raise AttnError(code, where)


def init() -> None:
    _check(lib().attn_sm100_init(), "attn_sm100_init")


def device_status(clear: bool = True) -> int:
    """Synchronise the current device and return its kernel status word (0 = fine)."""
    st = ctypes.c_int(0)
    rc = lib().attn_sm100_device_status(ctypes.byref(st), 1 if clear else 0)
    if rc not in (0, -6):
        raise AttnError(rc, "attn_sm100_device_status")
    return st.value


def static_status(clear: bool = True) -> int:
    """The same for the status word of attn_sm100_forward_static (a separate word inside the library)."""
    st = ctypes.c_int(0)
    rc = lib().attn_sm100_static_status(ctypes.byref(st), 1 if clear else 0)
    if rc not in (0, -6):
        raise AttnError(rc, "attn_sm100_static_status")
    return st.value


def saved_bytes(B: int, T: int, H: int, D: int) -> int:
    return lib().attn_sm100_saved_bytes(B, T, H, D)


def backward_scratch_bytes(B: int, T: int, H: int, D: int) -> int:
    return lib().attn_sm100_backward_scratch_bytes(B, T, H, D)


class Saved:
    """What forward leaves behind for backward (all device buffers, owned by torch)."""

    def __init__(self, saved, out, lse, shape, flags):
        self.saved, self.out, self.lse, self.shape, self.flags = saved, out, lse, shape, flags


def forward_into(qkv, out, out_copy, lse, saved, n_heads: int, flags: int = 0, stream=None) -> None:
    """Raw call: every buffer is supplied by the caller (torch CUDA tensors or None)."""
    _calls().forward_into(qkv, out, out_copy, lse, saved, n_heads, flags, _raw(stream))


def backward_into(saved, out, lse, dout, dqkv, scratch, n_heads: int, flags: int = 0, stream=None) -> None:
    _calls().backward_into(saved, out, lse, dout, dqkv, scratch, n_heads, flags, _raw(stream))


def forward(qkv, n_heads: int, flags: int = 0, keep_copy: bool = False):
    """qkv [B, T, 3C] fp32 CUDA tensor -> (out [B, T, C], Saved)."""
    out, out_copy, lse, saved, shape = _calls().forward(qkv, n_heads, flags, keep_copy)
    return out, Saved(saved, out if out_copy is None else out_copy, lse, shape, flags)


def backward(ctx: Saved, dout):
    """dout [B, T, C] -> dqkv [B, T, 3C] = [dq | dk | dv]."""
    return _calls().backward(ctx.saved, ctx.out, ctx.lse, dout, ctx.shape, ctx.flags)


# ---------------------------------------------------------------------------------------------
# Linear either side of the attention layer (include/linear_sm100.h); mirrors the reference's
# linear_forward_cuda_kernel / linear_backward_cuda_kernel (kernels/src/cuda/Linear.cu:37-92).
# ---------------------------------------------------------------------------------------------
def linear_forward(x, w, bias=None, planes=None, stream=None):
    """y[..., N] = x[..., K] @ w[N, K].T + bias.  `planes`: optional uint8 CUDA tensor of
    saved_bytes(...) bytes that receives y as bf16 hi/lo planes for the attention kernels."""
    return _calls().linear_forward(x, w, bias, planes, _raw(stream))


def linear_backward(dy, x, w, dw, db=None, stream=None, want_dx=True):
    """Returns dx = dy @ w (None when want_dx is false); accumulates dy.T @ x into dw (skipped when dw is
    None) and the column sums of dy into db."""
    return _calls().linear_backward(dy, x, w, dw, db, _raw(stream), want_dx)


# ---------------------------------------------------------------------------------------------
# LayerNorm (include/layernorm_sm100.h); mirrors layer_norm_{forward,backward}_cuda_kernel
# (kernels/src/cuda/LayerNorm.cu:115-165).
# ---------------------------------------------------------------------------------------------
def layernorm_forward(x, w, b=None, eps: float = 1e-5, stream=None):
    """Returns (y, mean, rstd) for x [..., C]."""
    return _calls().layernorm_forward(x, w, b, eps, _raw(stream))


def layernorm_backward(dy, x, mean, rstd, w, dw, db, dx, stream=None) -> None:
    """Accumulates into dw, db (may be None) and dx, like the reference."""
    _calls().layernorm_backward(dy, x, mean, rstd, w, dw, db, dx, _raw(stream))
