"""Failure detection on the device without a fault: a bounded wait that runs out.

Every tcgen05 kernel of the library waits on its barriers through one helper with a time limit;
when the limit passes the kernel records which wait gave up and returns normally.  The reference
has no counterpart (it checks cudaGetLastError after each launch, kernels/src/cuda/Attention.cu:119);
this test drives the helper through attn_sm100_selftest_wait_limit, whose kernel waits on a barrier
nothing completes, and checks that the status is reported, can be cleared, and that the context
keeps working afterwards.
"""
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_wait_limit_reports_status_and_context_survives(pkg, oracle):
    pkg.init()
    assert pkg.device_status() == 0
    L = pkg.lib()
    stream = torch.cuda.current_stream().cuda_stream

    t0 = time.perf_counter()
    assert L.attn_sm100_selftest_wait_limit(2000, stream) == 0  # 2 ms
    code = pkg.device_status(clear=False)
    elapsed = time.perf_counter() - t0
    assert code == 1900, code
    assert elapsed < 1.0, f"the wait took {elapsed:.3f} s for a 2 ms limit"
    # the word is sticky until cleared ...
    assert pkg.device_status(clear=True) == 1900
    # ... and clean afterwards
    assert pkg.device_status() == 0

    # the context is still usable: a forward pass right after matches the oracle
    B, T, H, D = 1, 160, 2, 64
    g = torch.Generator(device="cpu").manual_seed(5)
    x = torch.randn(B, T, 3 * H * D, generator=g)
    out, _ = pkg.forward(x.cuda(), H)
    ref = oracle.forward(x.numpy(), H)
    assert np.abs(out.cpu().numpy() - ref).max() < 2e-3
    assert pkg.device_status() == 0


def test_wait_limit_argument_range(pkg):
    L = pkg.lib()
    assert L.attn_sm100_selftest_wait_limit(0, None) == -2
    assert L.attn_sm100_selftest_wait_limit(100001, None) == -2


def test_cross_entropy_rows_that_never_arrive(pkg):
    """Several rows per CTA, of which the later ones are never fetched: the kernel ends, says so, and the rows before are right."""
    L = pkg.lib()
    rows, C, loaded = 400, 50257, 170  # up to three rows per CTA of 148; 22 CTAs get two of theirs, the others one
    x = torch.randn(rows, C, generator=torch.Generator().manual_seed(9)).cuda()
    targets, y = torch.zeros(rows, device="cuda"), torch.full((rows, C), 7.0, device="cuda")
    loss = torch.zeros(1, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    args = (x.data_ptr(), targets.data_ptr(), y.data_ptr(), loss.data_ptr(), rows, C)
    assert pkg.device_status() == 0
    t0 = time.perf_counter()
    assert L.xent_sm100_selftest_wait_limit(*args, loaded, 2000, stream) == 0
    assert pkg.device_status(clear=True) == 1252
    assert time.perf_counter() - t0 < 1.0
    want = torch.log_softmax(x.double(), -1)
    assert (y[:loaded] - want[:loaded]).abs().max().item() <= 2e-6 * want.abs().max().item()
    assert bool((y[loaded:] == 7.0).all())
    # the context is still usable
    assert L.xent_sm100_forward(*args, stream) == 0
    assert pkg.device_status() == 0
    assert (y - want).abs().max().item() <= 2e-6 * want.abs().max().item()


def test_cross_entropy_wait_limit_argument_range(pkg):
    L = pkg.lib()
    p = torch.zeros(8, device="cuda").data_ptr()
    for rows, C, loaded, limit in ((0, 30000, 0, 1), (1, 29999, 0, 1), (1, 53249, 0, 1), (1, 30000, 2, 1), (1, 30000, -1, 1),
                                   (1, 30000, 0, 0), (1, 30000, 0, 100001)):
        assert L.xent_sm100_selftest_wait_limit(p, p, p, p, rows, C, loaded, limit, None) == -2
