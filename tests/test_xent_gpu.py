"""Parity of the cross-entropy kernels (include/xent_sm100.h) against the float64 numpy restatement of the
reference in oracle/ops_oracle.py, pinned to the reference's own CPU kernel by tests/test_ops_oracle.py
(kernels/src/cpu/CrossEntropyLoss.c; kernels/src/cuda/CrossEntropyLoss.cu:8-129 has the same arithmetic but
accumulates the loss into its output, which is what the CUDA kernels here do too):
log-softmax, mean negative log-likelihood accumulated into the loss, and the backward that works on what
dout already holds.  Tolerance: fp32 with fast exponentials, 2e-6 absolute on log-softmax values of order
10, 1e-7 + 1e-5 relative on the gradient.  On the loss 1e-6 relative for its terms, and what adding them up one by one
rounds: the kernel's blocks add into one float in no fixed order, each addition is off by at most half a unit in the last
place of the sum, and such errors, spread evenly, have a standard deviation of sqrt(rows / 12) units; six of them are
allowed (7e-5 at 2048 rows and a loss of 10.5, where one in some dozen runs was more than 1.2e-5 off).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import ops_oracle as ops  # noqa: E402

pytestmark = pytest.mark.gpu


def stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("rows,C", [(64, 50257), (1000, 1003), (7, 5), (2048, 512), (1, 1)])
def test_cross_entropy_forward_backward_vs_cpu(pkg, rows, C):
    L = pkg.lib()
    rng = np.random.default_rng(rows + C)
    logits = (rng.standard_normal((rows, C)) * 3.0).astype(np.float32)
    targets = rng.integers(0, C, size=rows).astype(np.float32)
    g = rng.standard_normal(rows).astype(np.float32)

    logsm_ref, loss_ref = ops.xent_forward(logits, targets)

    lt, tt, gt = (torch.from_numpy(a).cuda() for a in (logits, targets, g))
    logsm = torch.empty_like(lt)
    loss = torch.full((1,), 0.25, device="cuda")  # accumulates on top of what is there
    assert L.xent_sm100_forward(lt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), loss.data_ptr(), rows, C, stream()) == 0
    assert np.abs(logsm.cpu().numpy() - logsm_ref).max() <= 2e-6 * max(1.0, np.abs(logsm_ref).max())
    unit = float(np.spacing(np.float32(loss_ref + 0.25)))
    assert abs(loss.item() - 0.25 - loss_ref) <= 1e-6 * max(1.0, abs(loss_ref)) + 2e-6 + 6 * np.sqrt(rows / 12) * unit

    # backward from a zero-filled dout (what the layer does) ...
    dout = torch.zeros_like(lt)
    assert L.xent_sm100_backward(gt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), dout.data_ptr(), rows, C, stream()) == 0
    d_ref = ops.xent_backward(g, targets, logsm_ref)
    assert np.abs(dout.cpu().numpy() - d_ref).max() <= 1e-7 + 1e-5 * np.abs(d_ref).max()

    # ... and from a dout that already holds something: the reference's formula on its contents
    d0 = (rng.standard_normal((rows, C)) * 0.01).astype(np.float32)
    dout = torch.from_numpy(d0.copy()).cuda()
    assert L.xent_sm100_backward(gt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), dout.data_ptr(), rows, C, stream()) == 0
    d_ref2 = ops.xent_backward(g, targets, logsm_ref, d0)
    assert np.abs(dout.cpu().numpy() - d_ref2).max() <= 1e-6 + 1e-5 * np.abs(d_ref2).max()
    torch.cuda.synchronize()


@pytest.mark.parametrize("rows,C", [(5, 50257), (9, 12000), (3, 9)])
def test_cross_entropy_masked_classes(pkg, rows, C):
    """Logits of -inf: probability 0, whatever their place in the row."""
    L = pkg.lib()
    logits = np.random.default_rng(C).standard_normal((rows, C)).astype(np.float32)
    logits[:, : C * 8 // 9] = -np.inf
    logits[0], logits[0, 0] = -np.inf, 1.0  # one class left
    targets = np.full(rows, C - 1, np.float32)
    targets[0] = 0
    lt, tt = torch.from_numpy(logits).cuda(), torch.from_numpy(targets).cuda()
    logsm, loss = torch.empty_like(lt), torch.zeros(1, device="cuda")
    assert L.xent_sm100_forward(lt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), loss.data_ptr(), rows, C, stream()) == 0
    got, (ref, loss_ref) = logsm.cpu().numpy(), ops.xent_forward(logits, targets)
    masked = np.isneginf(logits)
    assert np.isneginf(got[masked]).all()
    assert np.abs(got[~masked] - ref[~masked]).max() <= 2e-6 * max(1.0, np.abs(ref[~masked]).max())
    assert abs(loss.item() - loss_ref) <= 1e-5 * max(1.0, abs(loss_ref))


@pytest.mark.parametrize("rows,C,offsets", [
    (1, 30000, (0, 0)), (3, 29999, (1, 2)),              # the shortest rows that are kept in shared memory, the longest that are not
    (400, 50257, (0, 0)), (300, 50257, (3, 3)),          # several rows per CTA, up to three loose values either side of the words
    (297, 31001, (1, 2)), (149, 32768, (2, 1)),          # logits and log-probabilities on different addresses modulo 16
    (150, 53248, (0, 0)), (150, 53247, (1, 1)), (2, 53249, (0, 0)),  # every place of the ring full; a row too long for it
])
def test_cross_entropy_rows_in_shared_memory(pkg, rows, C, offsets):
    """Rows on any 4-byte boundary, with values that are -inf, against the oracle; nothing is written outside."""
    L = pkg.lib()
    rng = np.random.default_rng(rows * 7 + C)
    logits = (rng.standard_normal((rows, C)) * 3.0).astype(np.float32)
    logits[rows // 2, : C // 2] = -np.inf  # masked classes, whole pieces of them
    targets = rng.integers(C // 2, C, size=rows).astype(np.float32)
    targets[0], targets[-1] = C - 1, C - 2
    g = rng.standard_normal(rows).astype(np.float32)
    with np.errstate(invalid="ignore"):
        logsm_ref, loss_ref = ops.xent_forward(logits, targets)

    def place(a, off):  # a copy that starts `off` floats past a 16-byte boundary, in a buffer of sevens
        buf = torch.full((a.size + 16,), 7.0, device="cuda")
        v = buf[4 + off:4 + off + a.size].view(a.shape)
        v.copy_(torch.from_numpy(a))
        return buf, v

    def outside(buf, off, n):
        return bool((buf[:4 + off] == 7.0).all()) and bool((buf[4 + off + n:] == 7.0).all())

    _, lt = place(logits, offsets[0])
    sbuf, logsm = place(np.zeros_like(logits), offsets[1])
    tt, gt = torch.from_numpy(targets).cuda(), torch.from_numpy(g).cuda()
    loss = torch.zeros(1, device="cuda")
    assert L.xent_sm100_forward(lt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), loss.data_ptr(), rows, C, stream()) == 0
    got = logsm.cpu().numpy()
    masked = np.isneginf(logits)
    assert np.isneginf(got[masked]).all()
    assert np.abs(got[~masked] - logsm_ref[~masked]).max() <= 2e-6 * np.abs(logsm_ref[~masked]).max()
    unit = float(np.spacing(np.float32(loss_ref)))
    assert abs(loss.item() - loss_ref) <= 1e-6 * abs(loss_ref) + 2e-6 + 6 * np.sqrt(rows / 12) * unit
    assert outside(sbuf, offsets[1], logits.size)
    d0 = (rng.standard_normal((rows, C)) * 0.01).astype(np.float32)
    dbuf, dout = place(d0, offsets[0])
    assert L.xent_sm100_backward(gt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), dout.data_ptr(), rows, C, stream()) == 0
    d_ref = ops.xent_backward(g, targets, np.where(masked, -np.inf, logsm_ref), d0)
    assert np.abs(dout.cpu().numpy() - d_ref).max() <= 1e-6 + 1e-5 * np.abs(d_ref).max()
    assert outside(dbuf, offsets[0], logits.size)
    assert pkg.device_status() == 0


@pytest.mark.parametrize("rows,C,offsets", [
    (148, 53248, (0, 0)), (149, 53248, (0, 0)), (296, 30000, (0, 0)), (297, 53248, (0, 0)),  # one row per SM, up to two, more
    (299, 32768, (2, 1)),
])
def test_cross_entropy_rows_on_even_addresses(pkg, rows, C, offsets):
    """Either side of where up to two rows per SM, all on the same address modulo 16, are taken at once."""
    test_cross_entropy_rows_in_shared_memory(pkg, rows, C, offsets)


def test_cross_entropy_keeps_rows_apart(pkg):
    """A NaN or an infinity stays in its own row; a row of -inf has no probabilities."""
    L = pkg.lib()
    rows, C = 310, 30003
    logits = np.random.default_rng(5).standard_normal((rows, C)).astype(np.float32)
    bad = {3: (0, np.nan), 4: (C - 1, np.nan), 160: (7777, np.inf), 200: (slice(None), -np.inf)}
    for row, (col, value) in bad.items():
        logits[row, col] = value
    lt, tt = torch.from_numpy(logits).cuda(), torch.zeros(rows, device="cuda")
    logsm, loss = torch.empty_like(lt), torch.zeros(1, device="cuda")
    assert L.xent_sm100_forward(lt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), loss.data_ptr(), rows, C, stream()) == 0
    got = logsm.cpu().numpy()
    rest = np.setdiff1d(np.arange(rows), list(bad))
    for row in bad:  # an infinite logit: log(inf) below it everywhere, inf - inf at its place
        assert not np.isfinite(got[row]).any()
    ref, _ = ops.xent_forward(logits[rest], np.zeros(len(rest), np.float32))
    assert np.abs(got[rest] - ref).max() <= 2e-6 * np.abs(ref).max()


@pytest.mark.parametrize("rows,C", [(7, 9), (5, 1000), (5, 1024), (5, 12000), (3, 29999), (4, 50257)])
def test_cross_entropy_passes_nan_on(pkg, rows, C):
    """One NaN makes its row and the loss NaN, also where a thread sees no other value, or only -inf beside it."""
    L = pkg.lib()
    logits = np.random.default_rng(C).standard_normal((rows, C)).astype(np.float32)
    for row, col in enumerate((0, C - 1, C // 2)[:rows - 1]):
        logits[row, col] = np.nan
    logits[1, : C - 2] = -np.inf
    lt, tt = torch.from_numpy(logits).cuda(), torch.full((rows,), C - 2.0, device="cuda")
    logsm, loss = torch.empty_like(lt), torch.zeros(1, device="cuda")
    assert L.xent_sm100_forward(lt.data_ptr(), tt.data_ptr(), logsm.data_ptr(), loss.data_ptr(), rows, C, stream()) == 0
    got = logsm.cpu().numpy()
    bad = np.isnan(logits).any(1)
    assert np.isnan(got[bad]).all() and np.isfinite(got[~bad]).all() and np.isnan(loss.item())
    assert pkg.device_status() == 0


def test_cross_entropy_argument_errors(pkg):
    L = pkg.lib()
    assert L.xent_sm100_forward(None, None, None, None, 1, 1, None) == -1
    t = torch.zeros(8, device="cuda")
    p = t.data_ptr()
    assert L.xent_sm100_forward(p, p, p, p, 0, 4, None) == -2
    assert L.xent_sm100_backward(p, p, p, p, 4, 0, None) == -2
