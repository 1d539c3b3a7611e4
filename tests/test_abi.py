"""CPU tests of the C-ABI boundary: the library loads, exports every declared symbol, and rejects
bad arguments before touching the GPU."""
import ctypes
import os
import re

import pytest

INCLUDE = os.path.join(os.path.dirname(__file__), "..", "include")
HEADERS = ["attn_sm100.h", "linear_sm100.h", "layernorm_sm100.h", "tensor_sm100.h", "xent_sm100.h", "adamw_sm100.h"]


def declared_functions():
    names = set()
    for header in HEADERS:
        text = open(os.path.join(INCLUDE, header)).read()
        text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
        names |= set(re.findall(r"\b((?:attn|linear|layernorm|tensor|xent|adamw)_sm100_\w+)\s*\(", text))
    return sorted(names)


def test_header_declares_something():
    names = declared_functions()
    assert "attn_sm100_forward" in names and "attn_sm100_backward" in names


def test_library_exports_every_declared_symbol(pkg):
    handle = pkg.lib()
    for name in declared_functions():
        assert hasattr(handle, name), f"{name} declared under include/ but not exported"
    assert set(pkg.SIGNATURES) == set(declared_functions())


def test_version_and_strerror(pkg):
    L = pkg.lib()
    assert L.attn_sm100_version() >= 100
    assert L.attn_sm100_strerror(0) == b"success"
    for code in (-1, -2, -3, -4, -5, -6):
        assert len(L.attn_sm100_strerror(code)) > 8
    assert L.attn_sm100_strerror(-99) == b"unknown error"


def test_size_queries(pkg):
    # two bf16 planes of B*T*3C elements, each padded to 256 bytes
    assert pkg.saved_bytes(8, 1024, 12, 64) == 2 * 8 * 1024 * 3 * 768 * 2
    assert pkg.saved_bytes(1, 1, 1, 3) == 2 * 256
    # dO planes, delta, and 256 bytes for the backward kernel's item counter
    assert pkg.backward_scratch_bytes(8, 1024, 12, 64) == 2 * 8 * 1024 * 768 * 2 + 8 * 12 * 1024 * 4 + 256
    for bad in [(0, 1, 1, 1), (1, -1, 1, 1), (1, 1, 0, 1), (1, 1, 1, 0), (4096, 4096, 64, 64)]:
        assert pkg.saved_bytes(*bad) == 0
        assert pkg.backward_scratch_bytes(*bad) == 0


def test_linear_scratch_is_only_asked_for_where_it_is_used(pkg):
    size = pkg.lib().linear_sm100_backward_scratch_bytes
    assert size(8192, 50257, 768) == 0 and size(4096, 8193, 64) == 0  # read as they are, every fourth row at a time
    assert size(8192, 768, 768) == 0
    # a padded copy: too few rows, a dy that stays in L2, rows on 16-byte boundaries
    for M, N, pitch in ((4095, 50257, 50272), (1024, 50257, 50272), (4096, 8191, 8192), (8192, 100, 128), (8192, 50260, 50272)):
        assert size(M, N, 768) == M * pitch * 4


def test_argument_errors_are_reported_before_any_cuda_call(pkg):
    L = pkg.lib()
    one = ctypes.c_void_p(16)
    # NULL pointers
    assert L.attn_sm100_forward(None, one, None, one, one, 1, 1, 1, 64, 0, None) == -1
    assert L.attn_sm100_backward(one, one, one, None, one, one, 1, 1, 1, 64, 0, None) == -1
    # shapes
    assert L.attn_sm100_forward(one, one, None, one, one, 0, 1, 1, 64, 0, None) == -2
    assert L.attn_sm100_backward(one, one, one, one, one, one, 1, 1, 1, -3, 0, None) == -2
    # alignment
    odd = ctypes.c_void_p(20)
    assert L.attn_sm100_forward(odd, one, None, one, one, 1, 1, 1, 64, 0, None) == -4
    # shapes no kernel takes
    assert L.attn_sm100_forward(one, one, None, one, one, 1, 1, 1, 300, 0, None) == -3
    assert L.attn_sm100_forward(one, one, None, one, one, 1, 9000, 1, 32, 0, None) == -3
    assert L.attn_sm100_device_status(None, 0) == -1


def test_missing_library_raises(pkg, monkeypatch):
    monkeypatch.setattr(pkg, "_lib", None)
    monkeypatch.setattr(pkg, "LIB_PATH", "/nonexistent/libattn_sm100.so")
    with pytest.raises(FileNotFoundError):
        pkg.lib()


def test_no_cpu_fallback_without_gpu(pkg):
    """Without a CUDA device init must fail loudly instead of computing anything on the host."""
    import torch

    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    assert pkg.lib().attn_sm100_init() != 0
    with pytest.raises(pkg.AttnError):
        pkg.init()


@pytest.fixture
def fresh(pkg, monkeypatch):
    """The library loaded anew, as in a program that has made no tensor-level call yet (the module is loaded again by one)."""
    monkeypatch.setattr(pkg, "_lib", None)
    monkeypatch.setattr(pkg, "_calls_module", None)
    monkeypatch.setattr(pkg, "_entry_classes", {}, raising=False)
    return pkg


def test_functions_are_the_same_objects_before_and_after_the_extension_is_loaded(fresh):
    """What lib() gives does not depend on what has been called before, and is a ctypes function in both cases."""
    names = sorted(fresh.SIGNATURES)
    before = [getattr(fresh.lib(), n) for n in names]
    classes = [type(f) for f in before]
    address = [ctypes.cast(f, ctypes.c_void_p).value for f in before]
    assert before[names.index("tensor_sm100_axpy")](5, 1.0, None, None, None) == -1
    fresh._calls()
    for name, fn, cls, at in zip(names, before, classes, address):
        assert getattr(fresh.lib(), name) is fn and type(fn) is cls and isinstance(fn, ctypes._CFuncPtr)
        assert ctypes.cast(fn, ctypes.c_void_p).value == at and at
        assert fn.argtypes == fresh.SIGNATURES[name][1] and fn.restype is fresh.SIGNATURES[name][0]
    assert before[names.index("tensor_sm100_axpy")](5, 1.0, None, None, None) == -1


@pytest.mark.parametrize("loaded_before", [False, True])
def test_a_changed_signature_acts_on_every_call(fresh, loaded_before):
    if loaded_before:
        fresh._calls()
    fn = fresh.lib().tensor_sm100_fill
    assert fn(None, 2, 0.5, None) == -1
    fn.errcheck = lambda result, func, args: result - 100
    fresh._calls()
    assert fn(None, 2, 0.5, None) == -101  # a call whose arguments are plain numbers
    del fn.errcheck
    fn.restype = ctypes.c_uint
    assert fn(None, 2, 0.5, None) == 2 ** 32 - 1
    fn.argtypes = [ctypes.c_void_p] * 4
    with pytest.raises(ctypes.ArgumentError):
        fn(None, 2, 0.5, None)


def test_extension_answers_like_ctypes(pkg):
    """The entry points the extension puts in front of the ctypes functions: the same results for numbers, None, ctypes
    objects and wrong arguments (all rejected or done before the GPU is touched), the same attributes."""
    plain_lib = ctypes.CDLL(pkg.LIB_PATH)
    for name, (res, args) in pkg.SIGNATURES.items():
        getattr(plain_lib, name).restype, getattr(plain_lib, name).argtypes = res, args
    pkg._calls()
    fast = pkg.lib()
    calls = [("tensor_sm100_axpy", (0, 1.0, None, None, None)), ("tensor_sm100_axpy", (5, 1.0, None, None, 0)),
             ("tensor_sm100_axpy", (5, 1, None, None, None)), ("tensor_sm100_copy", (ctypes.c_void_p(0), None, ctypes.c_size_t(3), None)),
             ("tensor_sm100_fill", (None, 2, 0.5, None)), ("tensor_sm100_arange", (None, 2, -1, -1, None)),
             ("tensor_sm100_gelu_forward", (None, None, 1, None)), ("tensor_sm100_gelu_backward", (None, None, None, 1, None)),
             ("xent_sm100_forward", (None, None, None, None, 1, 1, None)), ("xent_sm100_backward", (1, 1, 1, 1, -1, 2, None)),
             ("attn_sm100_saved_bytes", (8, 1024, 12, 64)), ("attn_sm100_saved_bytes", (2 ** 32 + 1, 1, 1, 3)),
             ("attn_sm100_backward_scratch_bytes", (1, -1, 1, 1)), ("attn_sm100_backward_scratch_bytes", (True, 7, 2, 64))]
    for name, args in calls:
        assert getattr(fast, name)(*args) == getattr(plain_lib, name)(*args), (name, args)
    for args in ((1,), ("a", 1.0, None, None, None), (1, "a", None, None, None), (1.5, 1.0, None, None, None), (1, 1.0, 2.5, None, None)):
        with pytest.raises((TypeError, ctypes.ArgumentError)) as ours:
            fast.tensor_sm100_axpy(*args)
        with pytest.raises((TypeError, ctypes.ArgumentError)) as plain:
            plain_lib.tensor_sm100_axpy(*args)
        assert ours.type is plain.type
    assert fast.tensor_sm100_axpy.argtypes == pkg.SIGNATURES["tensor_sm100_axpy"][1]
