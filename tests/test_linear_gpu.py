"""Parity of the tcgen05 Linear kernels (include/linear_sm100.h) against the float64 numpy restatement of the
reference's Linear (kernels/src/cpu/Linear.c:4-31 forward, :33-88 backward) in oracle/ops_oracle.py, pinned to
the reference's own CPU kernel by tests/test_ops_oracle.py: y = x W^T + b, dx = dy W, dW += dy^T x,
db += colsum(dy).

Tolerance: the kernels use TF32 inputs (the upper 19 bits of each fp32 operand: truncation, relative
error below 2^-10 per operand) with fp32 accumulation, the precision class of the reference's CUDA
path (cuBLAS TF32 tensor-op math).  Every product is therefore within 2^-9 of the exact one, which
gives the element-wise bound |err| <= 2^-9 * (|a| @ |b|) plus the fp32 accumulation error; the fused
bf16 planes must reproduce y itself to 2^-16 relative.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import ops_oracle as ops  # noqa: E402
from test_linear_plan import EVEN, FIXED, LONG, SMS, TEAMS, plan  # noqa: E402

pytestmark = pytest.mark.gpu

SHAPES = [
    # (M, N, K)                      what
    (8 * 128, 2304, 768),          # QKV projection, config 1
    (2 * 1024, 768, 768),          # c_proj
    (300, 2304, 768),              # ragged M (tail tile)
    (256, 96, 64),                 # N, K below one tile
    (1000, 3072, 768),             # MLP up-projection shape
    (260, 50257, 768),             # vocabulary projection: rows of y not 16-byte aligned, plain stores
    (130, 1001, 64),               # the same path with a ragged last tile in every direction
    (70, 95, 64),                  # 31 of 32 columns in the last block: the padded copy of dy reads its last word alone
    (70, 94, 32),                  # rows of dy start 0 or 2 floats past a 16-byte boundary
    (9, 16415, 32),                # long contraction for dx (513 steps): cut into pieces that add into a zeroed dx
    (260, 16392, 768),             # weight above 48 MB with 16-byte-aligned rows of y: row-fastest tile order, copy-engine stores
]


def within(got, ref, a, b):
    """a [M, L], b [L, N]: got must be within the TF32 truncation bound of ref = a @ b."""
    a64, b64 = np.abs(a.astype(np.float64)), np.abs(b.astype(np.float64))
    lim = 2.0 ** -9 * (a64 @ b64) + 2.0 ** -20 * a.shape[1] * a64.max() * b64.max()
    excess = np.abs(got.astype(np.float64) - ref) - lim
    assert excess.max() <= 0, f"max error {np.abs(got - ref).max():.3e}, exceeds the bound by {excess.max():.3e}"


def inputs(M, N, K, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((M, K), dtype=np.float32)
    w = (rng.standard_normal((N, K), dtype=np.float32) * 0.05).astype(np.float32)
    b = rng.standard_normal(N, dtype=np.float32)
    dy = rng.standard_normal((M, N), dtype=np.float32)
    return x, w, b, dy


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_linear_forward_vs_cpu(pkg, M, N, K):
    x, w, b, _ = inputs(M, N, K, 11)
    ref = ops.linear_forward(x, w, b)
    y = pkg.linear_forward(torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), torch.from_numpy(b).cuda())
    assert pkg.device_status() == 0
    within(y.cpu().numpy(), ref, x, w.T)
    # without bias
    y0 = pkg.linear_forward(torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), None)
    within(y0.cpu().numpy(), ref - b, x, w.T)


def test_linear_forward_planes_feed_attention(pkg, oracle):
    """The fused bf16 planes equal the split of y, and attention run from them (core only) matches
    attention run from y itself."""
    B, T, H, D = 2, 256, 4, 64
    C = H * D
    x, w, b, _ = inputs(B * T, 3 * C, C, 5)
    xt, wt, bt = (torch.from_numpy(a).cuda() for a in (x, w, b))
    planes = torch.empty(pkg.saved_bytes(B, T, H, D), device="cuda", dtype=torch.uint8)
    y = pkg.linear_forward(xt.view(B, T, C), wt, bt, planes=planes)
    assert pkg.device_status() == 0
    n = B * T * 3 * C
    plane_bytes = pkg.saved_bytes(B, T, H, D) // 2
    hi = planes[: 2 * n].view(torch.bfloat16).float()
    lo = planes[plane_bytes: plane_bytes + 2 * n].view(torch.bfloat16).float()
    yy = y.reshape(-1)
    assert torch.equal(hi, yy.bfloat16().float())
    assert ((hi + lo) - yy).abs().max().item() <= 2.0 ** -16 * yy.abs().max().item()
    # attention from the planes (split pass skipped) == attention from y
    out_a = torch.empty(B, T, C, device="cuda")
    lse_a = torch.empty(B, H, T, device="cuda")
    pkg.forward_into(y, out_a, None, lse_a, planes, H, pkg.FLAG_CORE_ONLY)
    out_b, _ = pkg.forward(y, H)
    assert pkg.device_status() == 0
    assert torch.equal(out_a, out_b)
    ref = oracle.forward(y.cpu().numpy(), H)
    assert np.abs(out_a.cpu().numpy() - ref).max() < 2e-3


@pytest.mark.parametrize("M,N,K", [s for s in SHAPES if s[2] % 32 == 0])
def test_linear_backward_vs_cpu(pkg, M, N, K):
    x, w, b, dy = inputs(M, N, K, 23)
    rng = np.random.default_rng(99)
    dw0 = rng.standard_normal((N, K), dtype=np.float32)
    db0 = rng.standard_normal(N, dtype=np.float32)
    dx_ref, dw_ref, db_ref = ops.linear_backward(dy, x, w, dw0, db0)
    dw = torch.from_numpy(dw0.copy()).cuda()
    db = torch.from_numpy(db0.copy()).cuda()
    dx = pkg.linear_backward(torch.from_numpy(dy).cuda(), torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), dw, db)
    assert pkg.device_status() == 0
    within(dx.cpu().numpy(), dx_ref, dy, w)
    within(dw.cpu().numpy(), dw_ref, dy.T, x)
    assert np.abs(db.cpu().numpy() - db_ref).max() <= 1e-5 * np.sqrt(M) * 8


@pytest.mark.parametrize("M,N,K", [
    (1, 96, 64), (16, 128, 32), (17, 260, 96),   # one tile of 16 or 32 activation rows, one CTA or two
    (48, 1001, 128), (129, 384, 512), (250, 130, 1024), (348, 768, 3072),  # clusters of 6 and 8 CTAs, unaligned columns
    (2600, 3000, 512), (6000, 1104, 256), (8192, 1152, 384), (3000, 520, 1600),  # tiles of 256, 192 and 128 columns, several per CTA
])
def test_linear_tile_shapes(pkg, M, N, K):
    """Forward with bias and planes, dx, dW and db where the choice of kernel, tile shape and split changes."""
    x, w, b, dy = inputs(M, N, K, 47)
    xt, wt, bt, dyt = (torch.from_numpy(a).cuda() for a in (x, w, b, dy))
    planes = torch.zeros(2 * ((M * N * 2 + 255) // 256 * 256), dtype=torch.uint8, device="cuda") if N % 8 == 0 else None
    y = pkg.linear_forward(xt, wt, bt, planes=planes)
    within(y.cpu().numpy(), ops.linear_forward(x, w, b), x, w.T)
    if planes is not None:
        hi, lo = (p[: M * N * 2].view(torch.bfloat16).view(M, N) for p in planes.chunk(2))
        assert torch.equal(hi, y.bfloat16()) and torch.equal(lo, (y - hi.float()).bfloat16())
    dw, db = torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda")
    dx = pkg.linear_backward(dyt, xt, wt, dw, db)
    assert pkg.device_status() == 0
    dx_ref, dw_ref, db_ref = ops.linear_backward(dy, x, w, np.zeros_like(w), np.zeros_like(b))
    within(dx.cpu().numpy(), dx_ref, dy, w)
    within(dw.cpu().numpy(), dw_ref, dy.T, x)
    assert np.abs(db.cpu().numpy() - db_ref).max() <= 1e-5 * np.sqrt(M) * 8


@pytest.mark.parametrize("M,N,K", [(1024, 257, 256), (1025, 1001, 96), (1026, 513, 384), (1027, 94, 512), (1300, 9999, 64), (1111, 16387, 32),
                                   (4096, 8193, 256), (4097, 8195, 96), (4099, 8318, 384), (4101, 8190, 320), (4098, 8197, 640),
                                   (9999, 3357, 128), (4111, 16387, 32)])
def test_linear_backward_from_every_fourth_row(pkg, M, N, K):
    """Rows of dy that start on 4- or 8-byte boundaries: from a padded copy, and from 4096 rows and 2^25 values on without
    one; there dW has rows that only the shifted views reach and tiles of each width, whole and not, dx a contraction that
    is cut into pieces (the last one)."""
    x, w, _, dy = inputs(M, N, K, 53)
    xt, wt, dyt = (torch.from_numpy(a).cuda() for a in (x, w, dy))
    dw0 = np.random.default_rng(3).standard_normal((N, K), dtype=np.float32)
    pad = torch.full((N + 16, K), 7.0, device="cuda")  # rows either side of dW stay as they are
    dw = pad[8:8 + N]
    dw.copy_(torch.from_numpy(dw0))
    db = torch.full((N + 8,), 0.5, device="cuda")
    dx = torch.empty_like(xt)
    need = pkg.lib().linear_sm100_backward_scratch_bytes(M, N, K)
    assert (need == 0) == (M >= 4096)
    scratch = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert pkg.lib().linear_sm100_backward(dyt.data_ptr(), xt.data_ptr(), wt.data_ptr(), dx.data_ptr(), dw.data_ptr(),
                                           db[3:].data_ptr(), scratch.data_ptr() if need else None, M, N, K,
                                           torch.cuda.current_stream().cuda_stream) == 0
    assert pkg.device_status() == 0
    dx_ref, dw_ref, db_ref = ops.linear_backward(dy, x, w, dw0, np.full(N, 0.5, np.float32))
    assert np.abs(db.cpu().numpy()[3:3 + N] - db_ref).max() <= 1e-5 * np.sqrt(M) * 8
    assert bool((db[:3] == 0.5).all()) and bool((db[3 + N:] == 0.5).all())
    within(dx.cpu().numpy(), dx_ref, dy, w)
    within(dw.cpu().numpy(), dw_ref, dy.T, x)
    assert bool((pad[:8] == 7.0).all()) and bool((pad[8 + N:] == 7.0).all())


@pytest.mark.parametrize("N", [8193, 8194, 8195, 16387])  # the last one: contraction in pieces
def test_linear_input_gradient_keeps_rows_apart(pkg, N):
    """Values of dy that are not finite stay in their own row of dx and their own column's row of dW, where dy's rows start
    on 4- or 8-byte boundaries and every fourth one is read through a view that starts up to three values early."""
    M, K = 4102, 96
    x, w, _, dy = inputs(M, N, K, 61)
    bad = {3: (N - 1, np.inf), 4: (N - 2, np.nan), 517: (N - 3, -np.inf), 1025: (N - 1, np.nan), M - 1: (N - 1, np.inf)}
    for row, (col, value) in bad.items():
        dy[row, col] = value
    rest = np.setdiff1d(np.arange(M), list(bad))
    dw = torch.zeros(N, K, device="cuda")
    dx = pkg.linear_backward(*(torch.from_numpy(a).cuda() for a in (dy, x, w)), dw).cpu().numpy()
    assert pkg.device_status() == 0
    assert not np.isfinite(dx[list(bad)]).any()
    within(dx[rest], dy[rest].astype(np.float64) @ w.astype(np.float64), dy[rest], w)
    dw = dw.cpu().numpy()
    assert not np.isfinite(dw[-3:]).any()
    within(dw[:-3], dy[:, :-3].T.astype(np.float64) @ x.astype(np.float64), dy[:, :-3].T, x)


def test_linear_backward_parts_can_be_skipped(pkg):
    M, N, K = 512, 768, 768
    x, w, b, dy = inputs(M, N, K, 31)
    dyt, xt, wt = (torch.from_numpy(a).cuda() for a in (dy, x, w))
    dw_full = torch.zeros(N, K, device="cuda")
    dx_full = pkg.linear_backward(dyt, xt, wt, dw_full, None)
    # dx only
    dx_only = pkg.linear_backward(dyt, xt, wt, None, None)
    assert torch.equal(dx_only, dx_full)
    # dW only (accumulates on top of what is there)
    dw_only = torch.zeros(N, K, device="cuda")
    assert pkg.linear_backward(dyt, xt, wt, dw_only, None, want_dx=False) is None
    assert pkg.device_status() == 0
    within(dw_only.cpu().numpy(), dy.astype(np.float64).T @ x.astype(np.float64), dy.T, x)


@pytest.mark.parametrize("M,N,K", [(16, 96, 64), (37, 768, 768), (300, 2304, 768), (2048, 768, 768), (9, 16415, 32)])
@pytest.mark.parametrize("want_dx,want_dw,want_db", [(True, True, True), (True, True, False), (True, False, True), (False, True, True)])
def test_linear_backward_kernels_beside_each_other(pkg, M, N, K, want_dx, want_dw, want_db):
    """dx, dW and db read the same tensors, none of them before what wrote dy, x and w nor after what reads the results:
    back to back, with every input written by the kernel before and every result read by the kernel behind.  Small and
    large tiles, clusters, pieces that add into zeros, a padded copy."""
    L = pkg.lib()
    rounds = 12
    x, w, _, dy = inputs(M, N, K, 41)
    st = torch.cuda.current_stream().cuda_stream
    src = [torch.from_numpy(dy).cuda() * (i + 1) for i in range(rounds)]
    xs = [torch.from_numpy(x).cuda() * 2.0 ** -i for i in range(rounds)]
    wt = torch.from_numpy(w).cuda()

    def copy(dst, source):
        assert L.tensor_sm100_copy(dst.data_ptr(), source.data_ptr(), source.numel(), st) == 0

    def once(i, g, xi):
        copy(xi, xs[i])
        copy(g, src[i])
        dw = torch.zeros(N, K, device="cuda") if want_dw else None
        db = torch.zeros(N, device="cuda") if want_db else None
        dx = pkg.linear_backward(g, xi, wt, dw, db, want_dx=want_dx)
        out = [torch.empty_like(t) if t is not None else None for t in (dx, dw, db)]
        for o, t in zip(out, (dx, dw, db)):
            if t is not None:
                copy(o, t)
                t.fill_(float("nan"))
        return out

    got, alone = [], []
    g, xi = torch.empty_like(src[0]), torch.empty_like(xs[0])
    for i in range(rounds):
        got.append(once(i, g, xi))
    torch.cuda.synchronize()
    for i in range(rounds):
        alone.append(once(i, g, xi))
        torch.cuda.synchronize()
    assert pkg.device_status() == 0
    for a, b in zip(got, alone):
        for u, v in zip(a, b):
            # the order of additions in memory is free: up to 32 pieces, each within an ulp of the sum so far
            assert (u is None and v is None) or (u - v).abs().max().item() <= 2.0 ** -19 * v.abs().max().item()


@pytest.mark.parametrize("M,N,K", [(900, 5120, 1280), (257, 4096, 512), (3000, 12001, 512)])
def test_linear_input_gradient_in_two_pieces(pkg, M, N, K):
    """A contraction in two pieces that add into zeros: within the bound, and the same in every call."""
    x, w, _, dy = inputs(M, N, K, 43)
    g, xt, wt = (torch.from_numpy(t).cuda() for t in (dy, x, w))
    first = pkg.linear_backward(g, xt, wt, None, None)
    assert pkg.device_status() == 0
    within(first.cpu().numpy(), dy.astype(np.float64) @ w.astype(np.float64), dy, w)
    for _ in range(5):
        assert torch.equal(pkg.linear_backward(g, xt, wt, None, None), first)


@pytest.mark.parametrize("M,N,K", [
    (1500, 1600, 1600),                    # seven column tiles, of 7 and 8 blocks of 32
    (1203, 160, 736), (2373, 384, 1152),   # more tiles of dW than of dx per CTA, one tile row; ranges that end inside tiles
    (200, 2500, 3200),                     # tiles of dW only 7 blocks deep, more than CTAs: not cut
    (4500, 3072, 768), (4500, 768, 3072),  # dy and x larger than L2: teams of three CTAs beside, of six below each other
    (640, 33, 32), (1025, 129, 4288),      # one column of a tile in use; long rows
])
@pytest.mark.parametrize("with_db", [True, False])
def test_linear_backward_in_one_launch(pkg, M, N, K, with_db):
    """dx, dW and db of one launch, in which every CTA takes tiles of dx and a range of dW; db starts on any address."""
    x, w, _, dy = inputs(M, N, K, 59)
    rng = np.random.default_rng(7)
    dw0, db0 = rng.standard_normal((N, K), dtype=np.float32), rng.standard_normal(N, dtype=np.float32)
    xt, wt, dyt, dw = (torch.from_numpy(a).cuda() for a in (x, w, dy, dw0.copy()))
    db = torch.full((N + 12,), 0.5, device="cuda")
    at = 4 if N % 32 == 0 else 3
    db[at:at + N] = torch.from_numpy(db0).cuda()
    dx = torch.full((M + 2, K), 3.0, device="cuda")
    need = pkg.lib().linear_sm100_backward_scratch_bytes(M, N, K)
    scratch = torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")
    assert pkg.lib().linear_sm100_backward(dyt.data_ptr(), xt.data_ptr(), wt.data_ptr(), dx[1:].data_ptr(), dw.data_ptr(),
                                           db[at:].data_ptr() if with_db else None, scratch.data_ptr() if need else None, M, N, K,
                                           torch.cuda.current_stream().cuda_stream) == 0
    assert pkg.device_status() == 0
    dx_ref, dw_ref, db_ref = ops.linear_backward(dy, x, w, dw0, db0)
    within(dx[1:-1].cpu().numpy(), dx_ref, dy, w)
    within(dw.cpu().numpy(), dw_ref, dy.T, x)
    assert bool((dx[0] == 3.0).all()) and bool((dx[-1] == 3.0).all())
    # fp32 sums of M values, 8 at a time, then 8 such sums, then pieces: at most 2^-20 of the sum of magnitudes
    err = np.abs(db[at:at + N].cpu().numpy() - (db_ref if with_db else db0))
    assert (err <= 2.0 ** -20 * (np.abs(dy).sum(0) + np.abs(db0))).all()
    assert bool((db[:at] == 0.5).all()) and bool((db[at + N:] == 0.5).all())


@pytest.mark.parametrize("M,N,K,team,down", TEAMS)
@pytest.mark.parametrize("with_db", [True, False])
def test_linear_backward_in_one_launch_by_teams(pkg, M, N, K, team, down, with_db):
    """The same at sizes of which tests/test_linear_plan.py says that they run that way, by teams of every kind."""
    assert torch.cuda.get_device_properties(0).multi_processor_count == SMS
    p = plan(pkg, M, N, K)
    assert (p["together"], p["views"], p["team"], p["down"]) == (1, 1, team, down)
    test_linear_backward_in_one_launch(pkg, M, N, K, with_db)


@pytest.mark.parametrize("M,N,K", [(1000, 33555, 64), (1025, 32801, 96), (3001, 16387, 320), (2050, 16386, 1536)])
def test_linear_backward_from_every_fourth_row_of_fewer(pkg, M, N, K):
    """Below 4096 rows, with a contraction of dx that is cut into pieces: views of dy, or a copy where K is large beside M (the
    last one)."""
    x, w, _, dy = inputs(M, N, K, 71)
    dw0 = np.random.default_rng(3).standard_normal((N, K), dtype=np.float32)
    xt, wt, dyt, dw = (torch.from_numpy(a).cuda() for a in (x, w, dy, dw0))
    db = torch.zeros(N, device="cuda")
    dx = pkg.linear_backward(dyt, xt, wt, dw, db)
    assert pkg.device_status() == 0
    dx_ref, dw_ref, db_ref = ops.linear_backward(dy, x, w, dw0, np.zeros(N, np.float32))
    within(dx.cpu().numpy(), dx_ref, dy, w)
    within(dw.cpu().numpy(), dw_ref, dy.T, x)
    assert np.abs(db.cpu().numpy() - db_ref).max() <= 1e-5 * np.sqrt(M) * 8


@pytest.mark.parametrize("M,N,K", [(4096, 8195, 64), (1000, 33555, 64), (5001, 16386, 160)])
def test_linear_backward_from_every_fourth_row_in_part(pkg, M, N, K):
    """dx without dW, which needs no x; dW that lies over w, so that the products follow each other."""
    L = pkg.lib()
    x, w, _, dy = inputs(M, N, K, 79)
    xt, wt, dyt = (torch.from_numpy(a).cuda() for a in (x, w, dy))
    st = torch.cuda.current_stream().cuda_stream
    need = L.linear_sm100_backward_scratch_bytes(M, N, K)
    scratch = torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")
    sp = scratch.data_ptr() if need else None
    dx = torch.full((M + 2, K), 3.0, device="cuda")
    db = torch.zeros(N, device="cuda")
    assert L.linear_sm100_backward(dyt.data_ptr(), None, wt.data_ptr(), dx[1:].data_ptr(), None, db.data_ptr(), sp, M, N, K, st) == 0
    assert pkg.device_status() == 0
    dx_ref, dw_ref, db_ref = ops.linear_backward(dy, x, w, w, np.zeros(N, np.float32))
    within(dx[1:-1].cpu().numpy(), dx_ref, dy, w)
    assert bool((dx[0] == 3.0).all()) and bool((dx[-1] == 3.0).all())
    assert np.abs(db.cpu().numpy() - db_ref).max() <= 1e-5 * np.sqrt(M) * 8
    dx.fill_(3.0), db.zero_()
    assert L.linear_sm100_backward(dyt.data_ptr(), xt.data_ptr(), wt.data_ptr(), dx[1:].data_ptr(), wt.data_ptr(), db.data_ptr(), sp,
                                   M, N, K, st) == 0
    assert pkg.device_status() == 0
    within(dx[1:-1].cpu().numpy(), dx_ref, dy, w)
    within(wt.cpu().numpy(), dw_ref, dy.T, x)
    assert np.abs(db.cpu().numpy() - db_ref).max() <= 1e-5 * np.sqrt(M) * 8


@pytest.mark.parametrize("M,N,K", LONG)
def test_linear_weight_gradient_in_several_sums(pkg, M, N, K):
    assert torch.cuda.get_device_properties(0).multi_processor_count == SMS
    p = plan(pkg, M, N, K)
    assert p["dw_sum"] <= 160 < p["dw_of_a_cta"]
    test_linear_backward_in_one_launch(pkg, M, N, K, True)


@pytest.mark.parametrize("M,N,K,blocks", EVEN)
def test_linear_weight_gradient_in_pieces_of_one_size(pkg, M, N, K, blocks):
    assert plan(pkg, M, N, K)["dw_of_a_cta"] == blocks
    test_linear_backward_in_one_launch(pkg, M, N, K, True)


@pytest.mark.parametrize("M,N,K", FIXED)
def test_linear_input_gradient_in_turn(pkg, M, N, K):
    """From views of dy, in pieces that one CTA takes in turn, or below 4096 rows in pieces apart that are added up behind the launch:
    the same bits in every call, with and without dW, on either alignment of dx; nothing outside it is written."""
    L = pkg.lib()
    p = plan(pkg, M, N, K)
    assert p["views"] == 4 and p["dx_pieces"] > 2 and p["dx_fixed_order"]
    x, w, _, dy = inputs(M, N, K, 83)
    xt, wt, dyt = (torch.from_numpy(a).cuda() for a in (x, w, dy))
    need = L.linear_sm100_backward_scratch_bytes(M, N, K)
    scratch = torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")
    dw, db = torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda")

    def dx(with_dw, off):
        buf = torch.full((M * K + 32,), float("nan"), device="cuda")
        out = buf[16 + off:16 + off + M * K].view(M, K)
        assert L.linear_sm100_backward(dyt.data_ptr(), xt.data_ptr(), wt.data_ptr(), out.data_ptr(), dw.data_ptr() if with_dw else None,
                                       db.data_ptr() if with_dw else None, scratch.data_ptr() if need else None, M, N, K,
                                       torch.cuda.current_stream().cuda_stream) == 0
        assert bool(buf[:16 + off].isnan().all()) and bool(buf[16 + off + M * K:].isnan().all())
        return out

    first = dx(True, 0)
    assert pkg.device_status() == 0
    dx_ref, dw_ref, db_ref = ops.linear_backward(dy, x, w, np.zeros((N, K), np.float32), np.zeros(N, np.float32))
    within(first.cpu().numpy(), dx_ref, dy, w)
    within(dw.cpu().numpy(), dw_ref, dy.T, x)
    assert np.abs(db.cpu().numpy() - db_ref).max() <= 1e-5 * np.sqrt(M) * 8
    for with_dw, off in ((True, 0), (False, 0), (True, 4), (False, 4), (False, 0)):
        assert torch.equal(dx(with_dw, off), first)


@pytest.mark.parametrize("M,N,K", [(1411, 4800, 1600), (2305, 2312, 1568), (8001, 760, 3072)])
def test_linear_tiles_of_256_rows(pkg, M, N, K):
    """Forward with bias and planes and dx alone, where tiles of 256 rows by 256 or 192 columns are taken: the last ones with
    fewer rows and columns, one with rows in its lower half only."""
    x, w, b, _ = inputs(M, N, K, 73)
    xt, wt, bt = (torch.from_numpy(a).cuda() for a in (x, w, b))
    planes = torch.zeros(2 * ((M * N * 2 + 255) // 256 * 256), dtype=torch.uint8, device="cuda")
    y = pkg.linear_forward(xt, wt, bt, planes=planes)
    within(y.cpu().numpy(), ops.linear_forward(x, w, b), x, w.T)
    hi, lo = (p[: M * N * 2].view(torch.bfloat16).view(M, N) for p in planes.chunk(2))
    assert torch.equal(hi, y.bfloat16()) and torch.equal(lo, (y - hi.float()).bfloat16())
    # x as the gradient of a [M, K] result
    w2 = np.ascontiguousarray(w.T[:, : N // 32 * 32])
    dx = pkg.linear_backward(xt, torch.empty(M, w2.shape[1], device="cuda"), torch.from_numpy(w2).cuda(), None, None)
    assert pkg.device_status() == 0
    within(dx.cpu().numpy(), x.astype(np.float64) @ w2.astype(np.float64), x, w2)


def test_linear_backward_results_over_operands(pkg):
    """Where dW lies over w, dx comes from w as it was; where db lies over dy, dW comes from dy as it was."""
    M, N, K = 1024, 512, 512
    x, w, _, dy = inputs(M, N, K, 67)
    xt, wt, dyt = (torch.from_numpy(a).cuda() for a in (x, w, dy))
    dx = pkg.linear_backward(dyt, xt, wt, wt, dyt[0])
    assert pkg.device_status() == 0
    dx_ref, dw_ref, _ = ops.linear_backward(dy, x, w, w, np.zeros(N, np.float32))
    within(dx.cpu().numpy(), dx_ref, dy, w)
    within(wt.cpu().numpy(), dw_ref, dy.T, x)


def test_linear_argument_errors(pkg):
    L = pkg.lib()
    assert L.linear_sm100_forward(None, None, None, None, None, 1, 4, 4, None) == -1
    t = torch.zeros(64, device="cuda")
    p = t.data_ptr()
    assert L.linear_sm100_forward(p, p, None, p, None, 0, 4, 4, None) == -2
    assert L.linear_sm100_forward(p, p, None, p, None, 4, 4, 6, None) == -3
    assert L.linear_sm100_forward(p, p, None, p, p, 4, 12, 8, None) == -3  # planes need N % 8 == 0
    assert L.linear_sm100_backward(p, p, p, p, p, None, None, 4, 32, 48, None) == -3  # K % 32
    assert L.linear_sm100_backward(p, p, p, p, p, None, None, 4, 50, 32, None) == -1  # scratch needed, none given
    assert L.linear_sm100_backward_scratch_bytes(260, 50257, 768) == 260 * 50272 * 4
    assert L.linear_sm100_backward_scratch_bytes(260, 2304, 768) == 0
