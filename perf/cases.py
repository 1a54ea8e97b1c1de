"""What a user of this framework has it do, as measurable cases.

Every case is one pass through the public entry points (``attn_fwd``, ``attn_bwd``, ``gemm`` / ``make_gemm``,
``quantize_mx``).  Sizes are those of the repository's benchmark and tests, plus the two calls a serving loop makes per
generated token: attention of one query row over a cache of keys, and the MLP products of one small batch of rows.
"""

import math

import torch

import warpy_kernels as wk

FP8 = torch.float8_e4m3fn
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _attn(name, op, dtype, B, Hq, Hkv, Nq, Nk, d, causal, layout="bhnd", used=False):
    """``op``: "fwd", "bwd" (the gradients alone) or "train" (forward, then backward)."""
    return {"name": name, "kind": "attn", "op": op, "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hkv, "Nq": Nq, "Nk": Nk,
            "d": d, "causal": causal, "layout": layout, "used": used}


def _gemm(name, dtype, M, N, K, act="", trans="", prepared=False, quantise=False):
    return {"name": name, "kind": "gemm", "dtype": dtype, "M": M, "N": N, "K": K, "act": act, "trans": trans,
            "prepared": prepared, "quantise": quantise}


def listed():
    return [
        # a short cross attention of a small model: one call is over before the host has made the next one
        _attn("fwd_fp8_short", "fwd", "fp8", 1, 2, 1, 300, 777, 64, False),
        # prompt processing / the forward of training: the benchmark's headline shape
        _attn("fwd_fp8_prefill", "fwd", "fp8", 4, 32, 32, 4096, 4096, 128, True),
        # a long prompt with grouped heads: the largest call
        _attn("fwd_fp8_long", "fwd", "fp8", 1, 64, 8, 32768, 32768, 128, True),
        # one generated token for 16 sequences of different lengths, keys and values in a [B, N, H, d] cache
        _attn("fwd_fp8_decode", "fwd", "fp8", 16, 64, 8, 1, 8192, 128, False, layout="bnhd", used=True),
        # gradients of the headline shape
        _attn("bwd_fp8", "bwd", "fp8", 4, 32, 32, 4096, 4096, 128, True),
        # gradients of a small batch with a ragged length and grouped heads
        _attn("bwd_fp8_ragged", "bwd", "fp8", 2, 4, 2, 1000, 1000, 128, True),
        # a training step's attention in bf16, tensors as a projection leaves them ([B, N, H, d])
        _attn("train_bf16", "train", "bf16", 2, 32, 8, 2048, 2048, 128, True, layout="bnhd"),
        # a square bf16 product of ordinary size
        _gemm("gemm_bf16", "bf16", 2048, 2048, 2048),
        # the up projection of an MLP over a prompt, both operands MXFP8
        _gemm("gemm_mx", "mx", 8192, 14336, 4096),
        # the same layer's down projection for a small batch of rows (one generated token each): bf16 activations are
        # quantised, the weights' launch was prepared when the model was loaded
        _gemm("gemm_mx_decode", "mx", 128, 4096, 14336, prepared=True, quantise=True),
        # a whole MLP in MXFP8: quantise, up projection with GELU and MXFP8 output, down projection of those codes
        {"name": "mlp_mx", "kind": "mlp", "M": 4096, "N": 14336, "K": 4096},
        # quantising the activations of a prompt
        {"name": "quantise", "kind": "quantise", "dtype": "bf16", "M": 8192, "K": 14336},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(rng, lo, hi, step):
    """A multiple of ``step``, spread over the logarithm of the range."""
    return max(1, round(_log(rng, lo, hi) / step)) * step


def _draw_attn(rng):
    op = rng.choice(["fwd", "fwd", "decode", "bwd", "train"])
    dtype = rng.choice(["fp8", "fp8", "bf16"])
    Hkv, group = rng.choice([1, 2, 4, 8]), rng.choice([1, 1, 2, 4, 8])
    d, layout = rng.choice([64, 128, 128]), rng.choice(["bhnd", "bnhd"])
    if op == "decode":
        Hkv = rng.choice([1, 2, 4, 8])
        Nk = _log(rng, 256, 16384)
        B = _log(rng, 1, max(1.5, min(64, 3e8 / (2 * Hkv * Nk * d))))
        return _attn("", "fwd", dtype, B, Hkv * group, Hkv, rng.choice([1, 1, 1, 2, 4]), Nk, d, False, layout, True)
    Nq = _log(rng, 64, 16384)
    Nk = Nq if rng.random() < 0.7 else _log(rng, max(64, Nq / 4), min(16384, Nq * 4))
    per_head = (4 if op == "fwd" else 14) * Nq * Nk * d
    most = (4e12 if op == "fwd" else 2e12) / (Hkv * group * per_head)
    B = _log(rng, 1, max(1.2, min(8, most)))
    while B * Hkv * group * per_head > 6e12 and Hkv > 1:
        Hkv //= 2
    return _attn("", op, dtype, B, Hkv * group, Hkv, Nq, Nk, d, rng.random() < 0.6, layout)


def _draw_gemm(rng):
    dtype = rng.choice(["bf16", "bf16", "fp16", "mx", "mx", "mx"])
    M = _steps(rng, 128, 8192, 128)
    N, K = _steps(rng, 512, 14336, 128), _steps(rng, 512, 14336, 128 if dtype == "mx" else 64)
    act = rng.choice(["", "", "gelu", "dgelu"])
    trans = rng.choice(["", "", "b", "a"]) if dtype != "mx" else ""
    serving = dtype == "mx" and M <= 1024
    return _gemm("", dtype, M, N, K, act, trans, prepared=serving and rng.random() < 0.7,
                 quantise=serving and rng.random() < 0.5)


def draw(rng):
    what = rng.choice(["attn", "attn", "attn", "gemm", "gemm", "mlp", "quantise"])
    if what == "attn":
        case = _draw_attn(rng)
    elif what == "gemm":
        case = _draw_gemm(rng)
    elif what == "mlp":
        case = {"kind": "mlp", "M": _steps(rng, 128, 4096, 128), "N": _steps(rng, 1024, 14336, 128),
                "K": _steps(rng, 1024, 4096, 128)}
    else:
        case = {"kind": "quantise", "dtype": rng.choice(["bf16", "fp32"]), "M": _log(rng, 1, 8192),
                "K": _steps(rng, 224, 14336, 32)}
    case.pop("name", None)
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------
def _heads(gen, B, H, N, d, layout):
    """``[B, H, N, d]`` normal values, stored in that order or as ``[B, N, H, d]``."""
    if layout == "bnhd":
        return torch.randn(B, N, H, d, device="cuda", generator=gen, dtype=torch.bfloat16).transpose(1, 2)
    return torch.randn(B, H, N, d, device="cuda", generator=gen, dtype=torch.bfloat16)


def _to_fp8(x, Hkv):
    """e4m3 codes (in the memory layout of ``x``) and the ``[B, Hkv]`` scale amax / 448 of each batch item and group."""
    B, H = x.shape[:2]
    scale = (x.abs().amax(dim=(2, 3)).view(B, Hkv, H // Hkv).amax(2).float() / 448.0).clamp_min(1e-12)
    return (x / scale.repeat_interleave(H // Hkv, 1).to(x.dtype)[:, :, None, None]).to(FP8), scale


def _prepare_attn(c, gen):
    B, Hq, Hkv, Nq, Nk, d, lay = c["B"], c["Hq"], c["Hkv"], c["Nq"], c["Nk"], c["d"], c["layout"]
    q, k, v = _heads(gen, B, Hq, Nq, d, lay), _heads(gen, B, Hkv, Nk, d, lay), _heads(gen, B, Hkv, Nk, d, lay)
    scales = ()
    if c["dtype"] == "fp8":
        (q, sq), (k, sk), (v, sv) = _to_fp8(q, Hkv), _to_fp8(k, Hkv), _to_fp8(v, Hkv)
        scales = (sq, sk, sv)
    s = {"q": q, "k": k, "v": v, "scales": scales}
    if c["used"]:  # lengths from half of the cache to all of it
        s["used"] = torch.randint(max(1, Nk // 2), Nk + 1, (B,), device="cuda", generator=gen, dtype=torch.int32)
    if c["op"] != "fwd":
        s["dout"] = _heads(gen, B, Hq, Nq, d, lay)
    if c["op"] == "bwd":
        s["saved"] = wk.attn_fwd(q, k, v, *scales, causal=c["causal"])
    return s


def _mx(gen, rows, K):
    return wk.quantize_mx(torch.randn(rows, K, device="cuda", generator=gen, dtype=torch.bfloat16))


def _prepare_gemm(c, gen):
    M, N, K = c["M"], c["N"], c["K"]
    s = {"options": {}}
    if c["dtype"] == "mx":
        s["a"], sa = _mx(gen, M, K)
        s["b"], sb = _mx(gen, N, K)
        s["options"].update(a_scale_mx=sa, b_scale_mx=sb)
        if c["quantise"]:
            s["x"] = torch.randn(M, K, device="cuda", generator=gen, dtype=torch.bfloat16)
    else:
        dt = DTYPES[c["dtype"]]
        s["a"] = torch.randn(*((K, M) if c["trans"] == "a" else (M, K)), device="cuda", generator=gen, dtype=dt)
        s["b"] = torch.randn(*((K, N) if c["trans"] == "b" else (N, K)), device="cuda", generator=gen, dtype=dt)
        if c["trans"]:
            s["options"][c["trans"] + "_trans"] = True
    if c["act"]:
        s["options"]["act"] = c["act"]
    if c["act"] == "gelu":
        s["options"]["store_pre"] = True
    if c["act"] == "dgelu":
        out_dtype = torch.float16 if c["dtype"] == "fp16" else torch.bfloat16
        s["options"]["pre"] = torch.randn(M, N, device="cuda", generator=gen, dtype=out_dtype)
    if c["prepared"]:
        s["launch"], *s["results"] = wk.make_gemm(s["a"], s["b"], **s["options"])
    return s


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "attn":
        s = _prepare_attn(case, gen)
    elif case["kind"] == "gemm":
        s = _prepare_gemm(case, gen)
    elif case["kind"] == "mlp":
        M, N, K = case["M"], case["N"], case["K"]
        s = {"x": torch.randn(M, K, device="cuda", generator=gen, dtype=torch.bfloat16)}
        s["up"], s["up_scale"] = _mx(gen, N, K)
        s["down"], s["down_scale"] = _mx(gen, K, N)
        # weights of unit gain, so that the activations stay of order one
        s["alpha"] = torch.full((1,), 1.0 / math.sqrt(K), device="cuda")
        s["beta"] = torch.full((1,), 1.0 / math.sqrt(N), device="cuda")
    else:
        s = {"x": torch.randn(case["M"], case["K"], device="cuda", generator=gen).to(DTYPES[case["dtype"]])}
    s["case"] = case
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------
def _run_attn(c, s):
    q, k, v, scales, causal = s["q"], s["k"], s["v"], s["scales"], c["causal"]
    if c["used"]:
        return wk.attn_fwd(q, k, v, *scales, causal=causal, seqused_k=s["used"], return_lse=False)[0]
    if c["op"] == "fwd":
        return wk.attn_fwd(q, k, v, *scales, causal=causal)
    saved = s["saved"] if c["op"] == "bwd" else wk.attn_fwd(q, k, v, *scales, causal=causal)
    # attn_bwd takes the three descales between dout and causal; bf16 inputs have none
    grads = wk.attn_bwd(q, k, v, *saved, s["dout"], *scales, causal=causal)
    return grads if c["op"] == "bwd" else (saved, grads)


def run(state):
    c, s = state["case"], state
    if c["kind"] == "attn":
        return _run_attn(c, s)
    if c["kind"] == "quantise":
        return wk.quantize_mx(s["x"])
    if c["kind"] == "mlp":
        x8, xs = wk.quantize_mx(s["x"])
        h, _, h8, hs = wk.gemm(x8, s["up"], a_scale_mx=xs, b_scale_mx=s["up_scale"], scale_b=s["alpha"], act="gelu",
                               out_mx=True)
        return h, wk.gemm(h8, s["down"], a_scale_mx=hs, b_scale_mx=s["down_scale"], scale_b=s["beta"])
    if c["quantise"]:  # new activations into the buffers that the product reads
        wk.quantize_mx(s["x"], q=s["a"], s=s["options"]["a_scale_mx"])
    if c["prepared"]:
        s["launch"]()
        return s["results"]
    return wk.gemm(s["a"], s["b"], **s["options"])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _work_attn(c):
    B, Hq, Hkv, Nq, Nk, d = (c[x] for x in ("B", "Hq", "Hkv", "Nq", "Nk", "d"))
    size = 1 if c["dtype"] == "fp8" else 2
    keys = 0.75 * Nk if c["used"] else Nk  # the mean of the lengths
    pairs = Nq * keys
    if c["causal"]:  # the mask is aligned to the last key: row i sees keys up to i + Nk - Nq
        lo, hi = max(0, Nk - Nq + 1), Nk
        pairs = (lo + hi) * (hi - lo + 1) / 2
    rows, kv = B * Hq * Nq * d, 2 * B * Hkv * keys * d
    lse = 0 if c["used"] else 8 * B * Hq * Nq
    fwd = {"bytes": rows * (size + 2) + kv * size + lse, "flops": 4 * B * Hq * pairs * d}
    # q, k, v, out, dout and lse in; dq, dk, dv out
    bwd = {"bytes": rows * (size + 6) + kv * (size + 2) + lse / 2, "flops": 10 * B * Hq * pairs * d}
    parts = {"fwd": [fwd], "bwd": [bwd], "train": [fwd, bwd]}[c["op"]]
    return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}


def work(case):
    if case["kind"] == "attn":
        return _work_attn(case)
    if case["kind"] == "quantise":
        return {"bytes": case["M"] * case["K"] * ((2 if case["dtype"] == "bf16" else 4) + 1 + 1 / 32), "flops": 0}
    M, N, K = case["M"], case["N"], case["K"]
    code = 1 + 1 / 32  # an e4m3 value and its share of a scale
    if case["kind"] == "mlp":  # x and both weights in, the hidden activations (bf16 and MXFP8) and the result out
        return {"bytes": 2 * M * K + 2 * N * K * code + M * N * (2 + code) + 2 * M * K, "flops": 4 * M * N * K}
    size = code if case["dtype"] == "mx" else 2
    outs = {"": 1, "gelu": 2, "dgelu": 2}[case["act"]]  # the pre-activations are a second output, or an input
    acts = 2 if case["quantise"] else size
    return {"bytes": M * K * acts + N * K * size + 2 * M * N * outs, "flops": 2 * M * N * K}


def tolerance(case):
    if case["kind"] == "quantise":
        return "exact"
    if case["kind"] == "attn" and case["dtype"] == "fp8":
        # probabilities (and in the backward dO and dS) are rounded to e4m3: 2.5 % per value, root mean square, and
        # which way a value falls depends on the scale an implementation gives it
        return {"rel": 0.03}
    if case["kind"] == "mlp":
        # bf16 outputs; a hidden value near a rounding boundary may fall on either side and move its block's scale
        return {"rel": 1e-2, "max": 0.4, "differ": 1e-3}
    return {"rel": 1e-2}
