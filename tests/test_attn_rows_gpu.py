"""GPU: the attention forward for few query rows and small problems (packed query heads, keys split over warps and the
CTAs of a cluster), FP8 and BF16: packed rows around multiples of 16, keys around multiples of a step, caches with
lengths of their own down to 0, causal rows without a key, late peaks."""

import pytest
import torch

from oracle import reference_math as R
from tests.helpers import fwd_errors

pytestmark = pytest.mark.gpu

# (B, Hq, Hkv, Nq, Nk, d, causal)
SHAPES = [
    (1, 1, 1, 1, 1, 128, False), (1, 1, 1, 1, 33, 64, False), (3, 8, 1, 1, 500, 128, False),
    (2, 16, 4, 1, 2049, 128, False), (1, 64, 8, 2, 4097, 128, True), (2, 4, 4, 3, 31, 64, True),
    (1, 8, 2, 8, 1000, 128, True), (5, 2, 1, 16, 130, 64, False), (1, 4, 2, 33, 64, 128, True),
    (1, 2, 1, 300, 777, 64, False), (1, 2, 1, 200, 90, 128, True), (40, 32, 8, 1, 700, 128, False),
    # FP8 from 1024 keys on: products with the packed rows on the N side, 8 or 16 of them
    (1, 1, 1, 1, 1024, 128, False), (2, 8, 1, 1, 1153, 64, False), (3, 9, 3, 3, 1500, 128, True),
    (1, 32, 2, 2, 3333, 64, True), (20, 16, 2, 1, 1280, 128, False), (1, 2, 1, 8, 1031, 128, True),
    # more than 32 packed rows, ragged, with keys enough to be worth dividing
    (1, 4, 2, 33, 1500, 128, True), (1, 2, 1, 100, 1900, 64, True), (1, 1, 1, 49, 3100, 128, False),
]

# calls within the same limits whose CTAs would crowd the GPU: 128-row tiles with P in two terms, for any number of keys
CROWDED = [(8, 8, 8, 128, 128, 128), (4, 8, 8, 180, 180, 64), (36, 4, 4, 37, 574, 64), (14, 2, 2, 47, 720, 128),
           (40, 32, 32, 17, 707, 128), (30, 16, 16, 32, 1100, 64)]


def _inputs(cuda, shape, fp8, seed=0):
    # not centred over the sequence as randn_qkv does it: with one key that leaves V = 0, and 0 / 0 for a cosine
    B, Hq, Hkv, Nq, Nk, d = shape[:6]
    g = torch.Generator(device=cuda).manual_seed(seed)
    q, k, v = (torch.randn(B, h, n, d, device=cuda, generator=g) for h, n in ((Hq, Nq), (Hkv, Nk), (Hkv, Nk)))
    if not fp8:
        q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
        return (q, k, v), (q.float(), k.float(), v.float())
    q8 = R.quantize_qkv(q, k, v)
    return q8, R.dequantize_qkv(*q8)


def _check(errs):
    # P carries 8 bits for BF16 inputs; for FP8 11 (f16) below 1024 keys and 7 (two e4m3 terms) in the decode kernel and on
    # the 128-row tiles.  Its rounding errors average out over the keys and the output's own rounding to bf16 is of the same
    # size: the gates of the bf16 forward hold for both
    assert errs["out"] <= 1e-2 and errs["lse"] <= 1e-2 and errs["max_abs"] <= 2e-2 and errs["cos"] >= 0.999, errs


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("shape", SHAPES)
def test_matches_the_oracle(cuda, shape, fp8):
    from warpy_kernels import attn_fwd

    B, Hq, Hkv, Nq, Nk, d, causal = shape
    args, deq = _inputs(cuda, shape, fp8)
    out, lse, pmax = attn_fwd(*args, causal=causal)
    out_ref, lse_ref = R.attention_reference(*deq, causal)
    _check(fwd_errors(out, lse, out_ref, lse_ref, Nq, Nk, causal))
    rep = Hq // Hkv
    s = (deq[0] @ deq[1].repeat_interleave(rep, 1).transpose(-1, -2)) / d**0.5
    if causal:
        s = s.masked_fill(torch.arange(Nk, device=cuda) > torch.arange(Nq, device=cuda)[:, None] + Nk - Nq, float("-inf"))
    seen = torch.isfinite(lse)
    want = torch.softmax(s, -1).amax(-1)
    assert torch.allclose(pmax[seen], want[seen], rtol=2e-3, atol=1e-6) and bool((pmax[~seen] == 0).all())
    again = attn_fwd(*args, causal=causal)
    assert all(torch.equal(x, y) for x, y in zip(again, (out, lse, pmax)))


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("Nk,fill", [(600, 400.0), (1700, float("nan"))])
def test_cache_lengths(cuda, fp8, causal, Nk, fill):
    """A [B, N, H, d] cache whose items attend to lengths of their own, the rest of it filled with what must not count."""
    from warpy_kernels import attn_fwd

    shape = (5, 16, 4, 2, Nk, 128)
    args, deq = _inputs(cuda, shape, fp8, seed=4)
    used = [Nk, 1, 0, 257, 64]
    k, v = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in args[1:3])
    for b, n in enumerate(used):
        k[b, :, n:] = torch.full_like(k[b, :, n:].float(), fill).to(k.dtype)
        v[b, :, n:] = torch.full_like(v[b, :, n:].float(), -fill).to(v.dtype)
    lengths = torch.tensor(used, dtype=torch.int32, device=cuda)
    out, lse, pmax = attn_fwd(args[0], k, v, *args[3:], causal=causal, seqused_k=lengths)
    only = attn_fwd(args[0], k, v, *args[3:], causal=causal, seqused_k=lengths, return_lse=False)
    assert torch.equal(only[0], out) and only[1] is None
    for b, n in enumerate(used):
        if n == 0:
            assert bool((out[b] == 0).all()) and bool(torch.isinf(lse[b]).all()) and bool((pmax[b] == 0).all())
            continue
        out_ref, lse_ref = R.attention_reference(deq[0][b : b + 1], deq[1][b : b + 1, :, :n], deq[2][b : b + 1, :, :n], causal)
        _check(fwd_errors(out[b : b + 1], lse[b : b + 1], out_ref, lse_ref, 2, n, causal))


@pytest.mark.parametrize("fp8", [True, False])
def test_late_peaks(cuda, fp8):
    """Scores hundreds of nats above the first ones: the row reference of a warp moves (BF16), or is the maximum of each
    split's first tile, which both peaks are in (FP8)."""
    from tests.test_attn_fwd_range_gpu import late_peak_qkv
    from warpy_kernels import attn_fwd

    q, k, v = late_peak_qkv(1, 8, 1, 1, 3000, 128, [(100, 90.0), (2000, 300.0)], device=cuda)
    args = R.quantize_qkv(q, k, v) if fp8 else (q.bfloat16(), k.bfloat16(), v.bfloat16())
    deq = R.dequantize_qkv(*args) if fp8 else tuple(x.float() for x in args)
    out, lse, pmax = attn_fwd(*args)
    out_ref, lse_ref = R.attention_reference(*deq, False)
    errs = fwd_errors(out, lse, out_ref, lse_ref, 1, 3000, False)
    assert errs["out"] <= 1e-2 and errs["lse"] <= 5e-2, errs  # lse near 400: fp32 logits in base 2
    assert pmax.min().item() > 0.99


@pytest.mark.parametrize("layout", ["bhnd", "bnhd"])
@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", CROWDED)
def test_crowded_problems(cuda, shape, causal, fp8, layout):
    """The line between the kernels for few rows and the 128-row tiles costs no precision: the same gates on this side,
    with lengths per sequence and without."""
    from warpy_kernels import attn_fwd

    B, Hq, Hkv, Nq, Nk, d = shape
    args, deq = _inputs(cuda, shape, fp8, seed=9)
    if layout == "bnhd":
        args = (*(x.transpose(1, 2).contiguous().transpose(1, 2) for x in args[:3]), *args[3:])
    used = [Nk if b % 3 else (Nk * (b + 1)) // B for b in range(B)]
    for lengths in (None, torch.tensor(used, dtype=torch.int32, device=cuda)):
        out, lse, pmax = attn_fwd(*args, causal=causal, seqused_k=lengths)
        for b in range(0, B, max(1, B // 4)):
            n = Nk if lengths is None else used[b]
            out_ref, lse_ref = R.attention_reference(deq[0][b : b + 1], deq[1][b : b + 1, :, :n], deq[2][b : b + 1, :, :n], causal)
            _check(fwd_errors(out[b : b + 1], lse[b : b + 1], out_ref, lse_ref, Nq, n, causal))
        again = attn_fwd(*args, causal=causal, seqused_k=lengths)
        assert all(torch.equal(x, y) for x, y in zip(again, (out, lse, pmax)))


def test_a_tuned_entry_leaves_few_rows_alone(cuda, tmp_path, monkeypatch):
    """The tuner chooses between the kernels with 128-row tiles, under a key that rounds lengths up to 1024: its entry,
    here also for each of them in turn, changes nothing for a token per sequence or a small problem of the same bucket,
    but does apply to the calls it is for."""
    from warpy_kernels import attn_fwd
    from warpy_kernels.attn import autotune_attn_fwd, make_attn_fwd
    from warpy_kernels_b200 import utils
    from warpy_kernels_b200.attn import fwd_api

    few = [_inputs(cuda, shape, True)[0] for shape in ((4, 8, 2, 1, 3000, 128), (1, 8, 2, 2, 700, 128), (1, 4, 1, 60, 900, 128))]
    large = _inputs(cuda, (3, 16, 4, 900, 1000, 128), True)[0]
    monkeypatch.setattr(utils, "TUNE_CACHE_PATH", str(tmp_path / "none.json"))
    want = [attn_fwd(*args) for args in few]
    monkeypatch.setattr(utils, "TUNE_CACHE_PATH", str(tmp_path / "tune.json"))
    best, _ = autotune_attn_fwd(*large[:3], iters=2, verbose=False, q_descale=large[3], k_descale=large[4], v_descale=large[5])
    entries = utils._entries()
    assert entries == {utils.tune_key("fwd", 128, False, 900, 1000, 4): best}
    for ctas in (best["ctas_per_sm"], 1, 2):
        for nk in (1000, 3000):
            utils.tune_store(utils.tune_key("fwd", 128, False, 1, nk, 4), {"ctas_per_sm": ctas})
        assert fwd_api._tuned_ctas_per_sm(*large[:2], False) == ctas
        for args, (out, lse, pmax) in zip(few, want):
            for x, y in zip(attn_fwd(*args), (out, lse, pmax)):
                assert torch.equal(x, y)
            launch, prepared, _, _ = make_attn_fwd(*args)
            launch()
            assert torch.equal(prepared, out)


# (B, Hq, Hkv, Nq, d, causal): 8 and up to 16 packed rows, one and two groups of them, both head dimensions
SECOND_PASS = [(1, 8, 1, 1, 128, False), (1, 8, 1, 2, 128, True), (1, 8, 1, 1, 64, False), (1, 6, 1, 5, 64, True)]


@pytest.mark.parametrize("used", [3000, 2900])
@pytest.mark.parametrize("shape", SECOND_PASS)
def test_decode_second_pass(cuda, shape, used):
    """Peaks 120 nats above the rest in tiles of 128 keys that are not the first of their split (eight splits of three tiles): each
    of these splits goes through its keys a second time, with the maximum it then knows.  The peaks weigh the same, so a
    split that gets its second pass wrong shows.  One length ends inside a tile with a peak, before keys and values that
    must not count."""
    from tests.test_attn_fwd_range_gpu import late_peak_qkv
    from warpy_kernels import attn_fwd

    B, Hq, Hkv, Nq, d, causal = shape
    q, k, v = late_peak_qkv(B, Hq, Hkv, Nq, 3000, d, [(300, 120.0), (2200, 120.0), (2850, 120.0)], device=cuda)
    args = R.quantize_qkv(q, k, v)
    deq = R.dequantize_qkv(*args)
    nan = torch.full_like(args[1][:, :, used:].float(), float("nan")).to(args[1].dtype)
    args[1][:, :, used:], args[2][:, :, used:] = nan, nan
    lengths = torch.full((B,), used, dtype=torch.int32, device=cuda)
    out, lse, pmax = attn_fwd(*args, causal=causal, seqused_k=lengths)
    out_ref, lse_ref = R.attention_reference(deq[0], deq[1][:, :, :used], deq[2][:, :, :used], causal)
    errs = fwd_errors(out, lse, out_ref, lse_ref, Nq, used, causal)
    assert errs["out"] <= 1e-2 and errs["lse"] <= 5e-2, errs  # lse near 170: fp32 logits in base 2
    assert torch.allclose(pmax, torch.full_like(pmax, 1 / 3), rtol=2e-2)
    again = attn_fwd(*args, causal=causal, seqused_k=lengths)
    assert all(torch.equal(x, y) for x, y in zip(again, (out, lse, pmax)))
