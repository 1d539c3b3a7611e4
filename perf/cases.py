"""What the speed of this library is judged by: the calls that programs built on gpt.c make, over the range of
sizes they make them at.

A case is a dict of plain values, ``kind`` first:

  attention  the causal self-attention layer alone, forward or forward and backward (pkg.forward, pkg.backward)
  block      a whole pre-LayerNorm transformer block out of the library's entry points, in the order of gpt.c's
             block: LayerNorm, QKV projection that also writes the attention kernels' bf16 planes, attention,
             output projection, residual, LayerNorm, MLP with GELU, residual; backward the same way round
  head       the vocabulary projection, and in training the cross-entropy over it and both backward passes
  adamw      the optimizer step over every parameter of a model

``prepare`` makes what a program holds before the call, ``run`` makes the call(s) and returns everything they
produce.  ``listed`` are the named sizes, ``draw`` gives further ones of the same ranges.
"""
import ctypes
import importlib.util
import os
import sys

import torch

VOCAB = 50257  # classes of the GPT-2 tokenizer: rows of logits start on 4-byte boundaries only


def package():
    """The package directory has a dot in its name, so it is loaded by path (from the working folder)."""
    if "gptc_b200" not in sys.modules:
        here = os.path.join(os.getcwd(), "gpt.c_b200")
        spec = importlib.util.spec_from_file_location("gptc_b200", os.path.join(here, "__init__.py"),
                                                      submodule_search_locations=[here])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["gptc_b200"] = mod
        spec.loader.exec_module(mod)
        mod.init()
    return sys.modules["gptc_b200"]


def listed():
    return [
        # the smallest training call: a unit test, a toy model, the last short batch of a file
        {"name": "attention_toy_train", "kind": "attention", "B": 1, "T": 40, "H": 2, "D": 64, "backward": True},
        # block size 128, batch 8, 12 heads: the training command of gpt.c's README
        {"name": "attention_t128_train", "kind": "attention", "B": 8, "T": 128, "H": 12, "D": 64, "backward": True},
        # the full GPT-2 124M block size: the workload bench.py times by default
        {"name": "attention_t1024_train", "kind": "attention", "B": 8, "T": 1024, "H": 12, "D": 64, "backward": True},
        # prefill, or evaluation of a validation set: forward only, GPT-2 medium shape
        {"name": "attention_medium_prefill", "kind": "attention", "B": 32, "T": 1024, "H": 16, "D": 64, "backward": False},
        # GPT-2 XL shape, the largest attention call of the benchmark
        {"name": "attention_xl_train", "kind": "attention", "B": 64, "T": 1024, "H": 25, "D": 64, "backward": True},
        # a model whose head size is not 64 (the same width cut into 6 heads): the fp32 kernels
        {"name": "attention_d128_train", "kind": "attention", "B": 4, "T": 1024, "H": 6, "D": 128, "backward": True},
        # generation without a key/value cache: every new token runs the whole prompt of a single sequence again
        {"name": "block_generate", "kind": "block", "B": 1, "T": 37, "H": 12, "backward": False},
        # one of the 12 blocks of a GPT-2 124M training step at full block size
        {"name": "block_124m_train", "kind": "block", "B": 8, "T": 1024, "H": 12, "backward": True},
        # a block of GPT-2 XL width over ragged rows: a batch that memory limits, a sequence that is no power of two
        {"name": "block_xl_ragged_train", "kind": "block", "B": 3, "T": 500, "H": 25, "backward": True},
        # logits of one sequence during generation
        {"name": "head_generate", "kind": "head", "rows": 37, "C": 768, "V": VOCAB, "backward": False},
        # vocabulary projection and loss of a GPT-2 124M training step, both directions
        {"name": "head_124m_train", "kind": "head", "rows": 8192, "C": 768, "V": VOCAB, "backward": True},
        # the optimizer step of GPT-2 124M: 148 tensors
        {"name": "adamw_124m", "kind": "adamw", "layers": 12, "C": 768, "V": VOCAB, "block": 1024},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention_other", "block", "block", "head", "adamw"])
    backward = rng.random() < 0.7
    if kind == "attention":
        c = {"kind": "attention", "B": _log(rng, 1, 64), "T": _log(rng, 8, 4096), "H": rng.randint(1, 25), "D": 64, "backward": backward}
        while c["B"] * c["T"] * c["H"] > 64 * 1024 * 25 or c["B"] * c["H"] * c["T"] ** 2 > 64 * 25 * 1024 ** 2:
            c["B"] = (c["B"] + 1) // 2 if c["B"] > 1 else 1
            c["T"] -= c["T"] // 8 if c["B"] == 1 else 0
        return c
    if kind == "attention_other":  # any other head size up to 128
        c = {"kind": "attention", "B": _log(rng, 1, 8), "T": _log(rng, 8, 2048), "H": rng.randint(1, 16),
             "D": rng.choice([3, 16, 20, 32, 40, 48, 80, 96, 100, 128]), "backward": backward}
        while c["B"] * c["H"] * c["T"] ** 2 * c["D"] > 4 * 6 * 1024 ** 2 * 128:
            c["T"] -= c["T"] // 8
        return c
    if kind == "block":
        c = {"kind": "block", "B": _log(rng, 1, 16), "T": _log(rng, 8, 1024), "H": rng.choice([6, 8, 12, 16, 20, 25]), "backward": backward}
        while c["B"] * c["T"] * c["H"] ** 2 > 8192 * 12 ** 2:
            c["B"], c["T"] = max(1, c["B"] - 1), c["T"] - (c["T"] // 8 if c["B"] == 1 else 0)
        return c
    if kind == "head":
        return {"kind": "head", "rows": _log(rng, 1, 6000), "C": 64 * rng.choice([6, 8, 12]),
                "V": rng.choice([VOCAB, VOCAB, 50304, _log(rng, 60, 40000)]), "backward": backward}
    return {"kind": "adamw", "layers": rng.randint(1, 12), "C": 64 * rng.randint(2, 12), "V": _log(rng, 60, VOCAB),
            "block": rng.choice([128, 256, 1024])}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, shape, std=1.0):
    t = torch.empty(shape, device="cuda", dtype=torch.float32)
    return t.normal_(0.0, std, generator=g)


def _zeros(*shape):
    return torch.zeros(shape, device="cuda", dtype=torch.float32)


def _block_shapes(C):
    """The block's parameters: name -> shape."""
    return {"ln1_w": (C,), "ln1_b": (C,), "qkv_w": (3 * C, C), "qkv_b": (3 * C,), "proj_w": (C, C), "proj_b": (C,),
            "ln2_w": (C,), "ln2_b": (C,), "fc_w": (4 * C, C), "fc_b": (4 * C,), "out_w": (C, 4 * C), "out_b": (C,)}


def prepare(case, seed):
    pkg = package()
    g = _generator(seed)
    s = dict(case, pkg=pkg, lib=pkg.lib())
    if case["kind"] == "attention":
        B, T, C = case["B"], case["T"], case["H"] * case["D"]
        s["qkv"] = _normal(g, (B, T, 3 * C))
        if case["backward"]:
            s["dout"] = _normal(g, (B, T, C))
    elif case["kind"] == "block":
        B, T, C = case["B"], case["T"], 64 * case["H"]
        s["x"] = _normal(g, (B, T, C))
        # weights N(0, 0.02), the LayerNorm gains around one, as a model in training has them
        s["p"] = {n: _normal(g, sh, 0.02) for n, sh in _block_shapes(C).items()}
        s["p"]["ln1_w"] += 1.0
        s["p"]["ln2_w"] += 1.0
        if case["backward"]:
            s["dy"] = _normal(g, (B, T, C))
            s["d"] = {n: _zeros(*sh) for n, sh in _block_shapes(C).items()}
    elif case["kind"] == "head":
        rows, C, V = case["rows"], case["C"], case["V"]
        s["x"] = _normal(g, (rows, C))
        s["w"] = _normal(g, (V, C), 0.02)
        if case["backward"]:
            # targets are class indices held as floats, the loss gradient is one per row: gpt.c's convention
            s["targets"] = torch.randint(0, V, (rows,), device="cuda", generator=g).float()
            s["ones"] = torch.ones(rows, device="cuda", dtype=torch.float32)
            s["dw"] = _zeros(V, C)
    else:
        C = case["C"]
        shapes = [(case["V"], C), (case["block"], C)]
        shapes += [sh for _ in range(case["layers"]) for sh in _block_shapes(C).values()] + [(C,), (C,)]
        lengths = [sh[0] * (sh[1] if len(sh) > 1 else 1) for sh in shapes]
        starts, total = [], 0
        for n in lengths:  # every tensor starts on a 256-byte boundary of its flat buffer
            starts.append(total)
            total += (n + 63) // 64 * 64
        s["p"], s["g"], s["m"], s["v"] = _normal(g, total, 0.02), _normal(g, total, 1e-3), _normal(g, total, 1e-3), _normal(g, total, 1e-3)
        s["v"].square_()
        s["lists"] = [(ctypes.c_void_p * len(lengths))(*[s[k].data_ptr() + 4 * at for at in starts]) for k in "pgmv"]
        s["lengths"] = (ctypes.c_int * len(lengths))(*lengths)
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _ok(code):
    if code != 0:
        raise RuntimeError("status %d" % code)


def _attention(s):
    pkg = s["pkg"]
    out, ctx = pkg.forward(s["qkv"], s["H"])
    if not s["backward"]:
        return {"out": out, "lse": ctx.lse}
    return {"out": out, "lse": ctx.lse, "dqkv": pkg.backward(ctx, s["dout"])}


def _block(s):
    pkg, lib, p, x, H = s["pkg"], s["lib"], s["p"], s["x"], s["H"]
    B, T, C = x.shape
    n = x.numel()
    stream = torch.cuda.current_stream().cuda_stream
    h1, mean1, rstd1 = pkg.layernorm_forward(x, p["ln1_w"], p["ln1_b"])
    planes = torch.empty(pkg.saved_bytes(B, T, H, 64), device=x.device, dtype=torch.uint8)
    qkv = pkg.linear_forward(h1, p["qkv_w"], p["qkv_b"], planes=planes)
    a = torch.empty_like(x)
    lse = torch.empty((B, H, T), device=x.device, dtype=torch.float32)
    pkg.forward_into(qkv, a, None, lse, planes, H, flags=pkg.FLAG_CORE_ONLY)
    r = pkg.linear_forward(a, p["proj_w"], p["proj_b"])
    _ok(lib.tensor_sm100_axpy(n, 1.0, x.data_ptr(), r.data_ptr(), stream))
    h2, mean2, rstd2 = pkg.layernorm_forward(r, p["ln2_w"], p["ln2_b"])
    f = pkg.linear_forward(h2, p["fc_w"], p["fc_b"])
    u = torch.empty_like(f)
    _ok(lib.tensor_sm100_gelu_forward(f.data_ptr(), u.data_ptr(), f.numel(), stream))
    y = pkg.linear_forward(u, p["out_w"], p["out_b"])
    _ok(lib.tensor_sm100_axpy(n, 1.0, r.data_ptr(), y.data_ptr(), stream))
    if not s["backward"]:
        return {"y": y}
    d, dy = s["d"], s["dy"]
    du = pkg.linear_backward(dy, u, p["out_w"], d["out_w"], d["out_b"])
    df = torch.empty_like(f)
    _ok(lib.tensor_sm100_gelu_backward(du.data_ptr(), f.data_ptr(), df.data_ptr(), f.numel(), stream))
    dh2 = pkg.linear_backward(df, h2, p["fc_w"], d["fc_w"], d["fc_b"])
    dr = torch.empty_like(x)  # the residual's gradient, onto which LayerNorm adds
    _ok(lib.tensor_sm100_copy(dr.data_ptr(), dy.data_ptr(), n, stream))
    pkg.layernorm_backward(dh2, r, mean2, rstd2, p["ln2_w"], d["ln2_w"], d["ln2_b"], dr)
    da = pkg.linear_backward(dr, a, p["proj_w"], d["proj_w"], d["proj_b"])
    dqkv = pkg.backward(pkg.Saved(planes, a, lse, (B, T, H, 64), 0), da)
    dh1 = pkg.linear_backward(dqkv, h1, p["qkv_w"], d["qkv_w"], d["qkv_b"])
    pkg.layernorm_backward(dh1, x, mean1, rstd1, p["ln1_w"], d["ln1_w"], d["ln1_b"], dr)
    return {"y": y, "dx": dr, "d": d}


def _head(s):
    pkg, lib, x, w = s["pkg"], s["lib"], s["x"], s["w"]
    rows, V = s["rows"], s["V"]
    stream = torch.cuda.current_stream().cuda_stream
    logits = pkg.linear_forward(x, w)
    if not s["backward"]:
        return {"logits": logits}
    logsm = torch.empty_like(logits)
    loss = torch.empty(1, device=x.device, dtype=torch.float32)
    _ok(lib.tensor_sm100_fill(loss.data_ptr(), 1, 0.0, stream))  # the loss is accumulated
    _ok(lib.xent_sm100_forward(logits.data_ptr(), s["targets"].data_ptr(), logsm.data_ptr(), loss.data_ptr(), rows, V, stream))
    dlogits = torch.empty_like(logits)
    _ok(lib.tensor_sm100_fill(dlogits.data_ptr(), rows * V, 0.0, stream))  # and so is the logits' gradient
    _ok(lib.xent_sm100_backward(s["ones"].data_ptr(), s["targets"].data_ptr(), logsm.data_ptr(), dlogits.data_ptr(), rows, V, stream))
    dx = pkg.linear_backward(dlogits, x, w, s["dw"])
    return {"loss": loss, "logsm": logsm, "dlogits": dlogits, "dx": dx, "dw": s["dw"]}


def _adamw(s):
    p, g, m, v = s["lists"]
    _ok(s["lib"].adamw_sm100_step(p, g, m, v, s["lengths"], len(s["lengths"]), 3e-4, 0.9, 0.999, 0.01, 1e-8, 10,
                                  torch.cuda.current_stream().cuda_stream))
    return {"p": s["p"], "m": s["m"], "v": s["v"]}


def run(state):
    return {"attention": _attention, "block": _block, "head": _head, "adamw": _adamw}[state["kind"]](state)


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without, and how close two right results are
# ---------------------------------------------------------------------------------------------
def _attention_flops(B, T, H, D, backward):
    """Causal: half of every T x T product counts; two products forward, four backward."""
    return (6 if backward else 2) * B * H * T * T * D


def work(case):
    kind = case["kind"]
    if kind == "adamw":
        C = case["C"]
        n = (case["V"] + case["block"] + 2 + case["layers"] * (12 * C + 13)) * C
        return {"bytes": 28 * n, "flops": 16 * n}  # p, m, v read and written, g read
    back = case["backward"]
    if kind == "attention":
        B, T, H, D = case["B"], case["T"], case["H"], case["D"]
        C = H * D
        words = B * T * 4 * C + B * H * T + (B * T * 4 * C if back else 0)  # qkv, out, lse; dout, dqkv
        return {"bytes": 4 * words, "flops": _attention_flops(B, T, H, D, back)}
    if kind == "block":
        B, T, H = case["B"], case["T"], case["H"]
        C = 64 * H
        rows, params = B * T, (12 * C + 13) * C
        words = 2 * rows * C + params + (2 * rows * C + 2 * params if back else 0)  # x, y; dy, dx; gradients are added to
        return {"bytes": 4 * words, "flops": (3 if back else 1) * 24 * rows * C * C + _attention_flops(B, T, H, 64, back)}
    rows, C, V = case["rows"], case["C"], case["V"]
    words = rows * C + V * C + rows * V  # x, w; logits, or their log-softmax
    if back:
        words += rows * V + rows * C + 2 * V * C  # dlogits, dx, dw added to
    return {"bytes": 4 * words, "flops": (6 if back else 2) * rows * C * V}


def tolerance(case):
    kind = case["kind"]
    if kind == "adamw":
        return {"rel": 1e-6, "max": 1e-4}  # a dozen fp32 operations per element, no sums
    if kind == "attention":
        # head size 64: operands of 16 significant bits, fp32 sums; other sizes fp32 (the backward reads q, k, v with 16 bits)
        return {"rel": 1e-4, "max": 4e-3} if case["D"] == 64 else {"rel": 1e-5, "max": 1e-3}
    # TF32 products (10 bits after the leading one), fp32 sums; a block chains up to a dozen of them
    return {"rel": 3e-3, "max": 0.1} if kind == "block" else {"rel": 1e-3, "max": 0.05}
