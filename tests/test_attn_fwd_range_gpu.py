"""GPU: attention forward on rows whose late keys lie far above the first ones.

The tensor-core kernels fix one reference exponent per query row from the row's first 64 keys and can represent
scores up to 2^100 (69 nats) above it; the reference has no such limit because its reference moves with every key
tile (``warpy_kernels/attn/fwd_base.py:337-360``).  Query blocks that leave the range are recomputed by the
library in fp32 when the call is given its flag workspace, as the Python wrappers always do.  These
tests put peaks of 120 to 400 nats behind the first tile and apply the usual gates against the oracle, then check
the raw C-ABI behaviour without a workspace: the status word says ``WK_ERR_RANGE`` (nothing faults).

Small problems would go to the kernels for few query rows, which hold scores of any range; ``ctas_per_sm`` keeps a call
on the kernels these tests are about.
"""

import ctypes
import math

import pytest
import torch

from oracle import reference_math as R
from tests.helpers import fwd_errors

pytestmark = pytest.mark.gpu

WK_ERR_RANGE = 110


def late_peak_qkv(B, Hq, Hkv, Nq, Nk, d, peaks, seed=0, device="cuda"):
    """Near-uniform logits except for keys ``peaks = [(index, gap_nats), ...]`` that rise ``gap_nats`` above the rest
    (the recipe of the reference's long-tail case, ``tests/fixtures.py:81-88``, with the peak moved off key 0)."""
    g = torch.Generator(device=device).manual_seed(seed)
    q = 1.0 + 0.1 * torch.randn(B, Hq, Nq, d, device=device, generator=g)
    k = 0.01 * torch.randn(B, Hkv, Nk, d, device=device, generator=g)
    for index, gap in peaks:
        k[:, :, index, :] = gap / math.sqrt(d)
    v = torch.randn(B, Hkv, Nk, d, device=device, generator=g)
    return q, k, v


def gates(errs):
    assert errs["out"] <= 6e-2 and errs["cos"] >= 0.999 and errs["max_abs"] <= 2e-2, errs
    assert errs["lse"] <= 5e-2, errs


CASES = [
    # (B, Hq, Hkv, Nq, Nk, peaks, causal, ctas_per_sm)
    (1, 2, 1, 384, 640, [(300, 120.0)], False, 2),
    (1, 2, 1, 384, 640, [(300, 120.0)], True, 2),
    (2, 4, 2, 300, 777, [(100, 90.0), (500, 250.0)], True, 2),      # two rising peaks, ragged, GQA
    (1, 2, 2, 256, 2304, [(1500, 400.0)], False, None),             # persistent kernel (from 2048 keys on)
    (1, 4, 1, 640, 2176, [(70, 80.0), (2100, 160.0)], True, 1),     # persistent kernel, causal
]


@pytest.mark.parametrize("case", CASES)
def test_fp8_late_peaks_match_oracle(cuda, case):
    from warpy_kernels import attn_fwd
    from warpy_kernels_b200.attn import fwd_api

    B, Hq, Hkv, Nq, Nk, peaks, causal, ctas = case
    q, k, v = late_peak_qkv(B, Hq, Hkv, Nq, Nk, 128, peaks, device=cuda)
    q8, k8, v8, sq, sk, sv = R.quantize_qkv(q, k, v)
    out, lse, pmax = attn_fwd(q8, k8, v8, sq, sk, sv, causal=causal, ctas_per_sm=ctas)
    qd, kd, vd = R.dequantize_qkv(q8.cpu(), k8.cpu(), v8.cpu(), sq.cpu(), sk.cpu(), sv.cpu())
    out_ref, lse_ref = R.attention_reference(qd, kd, vd, causal)
    gates(fwd_errors(out, lse, out_ref, lse_ref, Nq, Nk, causal))
    # rows that see a peak put nearly all their weight on it
    assert pmax.max().item() > 0.99
    # the flag scratch is handed back all zero, so the next call on the stream starts clean
    assert int(fwd_api._block_flags(cuda, 16).count_nonzero()) == 0
    again = attn_fwd(q8, k8, v8, sq, sk, sv, causal=causal, ctas_per_sm=ctas)
    assert torch.equal(again[0], out) and torch.equal(again[1], lse)


@pytest.mark.parametrize("causal", [False, True])
def test_bf16_late_peaks_match_oracle(cuda, causal):
    from warpy_kernels import attn_fwd

    q, k, v = late_peak_qkv(1, 4, 2, 300, 700, 128, [(200, 100.0), (650, 300.0)], seed=2, device=cuda)
    qb, kb, vb = q.bfloat16(), k.bfloat16(), v.bfloat16()
    out, lse, _ = attn_fwd(qb, kb, vb, causal=causal, ctas_per_sm=2)
    out_ref, lse_ref = R.attention_reference(qb.float().cpu(), kb.float().cpu(), vb.float().cpu(), causal)
    errs = fwd_errors(out, lse, out_ref, lse_ref, 300, 700, causal)
    assert errs["out"] <= 1e-2 and errs["lse"] <= 1e-2, errs  # the reference's bf16 gates (tests/attn/test_fwd.py)


def test_rows_inside_the_range_are_not_recomputed(cuda):
    """A 60-nat peak stays inside the range: the tensor-core result is kept and passes the gates."""
    from warpy_kernels import attn_fwd

    q, k, v = late_peak_qkv(1, 2, 1, 256, 512, 128, [(300, 60.0)], device=cuda)
    q8, k8, v8, sq, sk, sv = R.quantize_qkv(q, k, v)
    out, lse, _ = attn_fwd(q8, k8, v8, sq, sk, sv, causal=False, ctas_per_sm=2)
    qd, kd, vd = R.dequantize_qkv(q8.cpu(), k8.cpu(), v8.cpu(), sq.cpu(), sk.cpu(), sv.cpu())
    out_ref, lse_ref = R.attention_reference(qd, kd, vd, False)
    gates(fwd_errors(out, lse, out_ref, lse_ref, 256, 512, False))


def test_without_workspace_the_status_word_reports_the_range(cuda):
    """Raw C ABI, ``workspace = NULL``: no recomputation, ``wk_status()`` returns ``WK_ERR_RANGE`` once and clears it."""
    from warpy_kernels_b200 import _lib
    from warpy_kernels_b200.attn.fwd_api import _FwdArgs

    lib = _lib.lib()
    B, H, Nq, Nk, d = 1, 1, 128, 256, 128
    q, k, v = late_peak_qkv(B, H, H, Nq, Nk, d, [(200, 150.0)], device=cuda)
    q8, k8, v8, sq, sk, sv = R.quantize_qkv(q, k, v)
    out = torch.empty(B, H, Nq, d, dtype=torch.bfloat16, device=cuda)
    lse = torch.empty(B, H, Nq, dtype=torch.float32, device=cuda)
    pmax = torch.empty_like(lse)
    a = _FwdArgs()
    a.q, a.k, a.v, a.out, a.lse, a.pmax = (t.data_ptr() for t in (q8, k8, v8, out, lse, pmax))
    a.q_descale, a.k_descale, a.v_descale = sq.data_ptr(), sk.data_ptr(), sv.data_ptr()
    a.q_strides = (ctypes.c_int64 * 3)(*q8.stride()[:3])
    a.k_strides = (ctypes.c_int64 * 3)(*k8.stride()[:3])
    a.v_strides = (ctypes.c_int64 * 3)(*v8.stride()[:3])
    a.out_strides = (ctypes.c_int64 * 3)(*out.stride()[:3])
    a.lse_strides = (ctypes.c_int64 * 2)(H * Nq, Nq)
    a.B, a.Hq, a.Hkv, a.Nq, a.Nk, a.d = B, H, H, Nq, Nk, d
    a.causal, a.write_lse, a.lse_natural, a.seqused_k = 0, 1, 0, None
    a.softmax_scale, a.ctas_per_sm = 1.0 / math.sqrt(d), 0
    a.workspace, a.workspace_bytes = None, 0
    assert lib.wk_attn_fwd_fp8(ctypes.byref(a), _lib.stream_ptr(cuda)) == 0
    assert lib.wk_status() == WK_ERR_RANGE
    assert lib.wk_status() == 0
    # the same call with the workspace: recomputed, clean status, right answer
    ws = torch.zeros(lib.wk_attn_fwd_workspace_bytes(B, H, Nq), dtype=torch.uint8, device=cuda)
    a.workspace, a.workspace_bytes, a.ctas_per_sm = ws.data_ptr(), ws.numel(), 2
    assert lib.wk_attn_fwd_fp8(ctypes.byref(a), _lib.stream_ptr(cuda)) == 0
    assert lib.wk_status() == 0 and int(ws.count_nonzero()) == 0
    qd, kd, vd = R.dequantize_qkv(q8.cpu(), k8.cpu(), v8.cpu(), sq.cpu(), sk.cpu(), sv.cpu())
    out_ref, lse_ref = R.attention_reference(qd, kd, vd, False)
    gates(fwd_errors(out, lse, out_ref, lse_ref, Nq, Nk, False))
    # a workspace that is too small is rejected before anything is launched
    a.workspace_bytes = 0
    assert lib.wk_attn_fwd_fp8(ctypes.byref(a), _lib.stream_ptr(cuda)) == -1


@pytest.mark.parametrize("bf16,ctas", [(False, 1), (False, 2), (True, 2)])
def test_head_dim_64_late_peaks_match_oracle(cuda, bf16, ctas):
    """Head dimension 64 takes the same path."""
    from warpy_kernels import attn_fwd

    q, k, v = late_peak_qkv(1, 4, 2, 300, 700, 64, [(200, 100.0), (650, 300.0)], seed=3, device=cuda)
    if bf16:
        qx, kx, vx = q.bfloat16(), k.bfloat16(), v.bfloat16()
        out, lse, _ = attn_fwd(qx, kx, vx, causal=True, ctas_per_sm=ctas)
        out_ref, lse_ref = R.attention_reference(qx.float().cpu(), kx.float().cpu(), vx.float().cpu(), True)
        errs = fwd_errors(out, lse, out_ref, lse_ref, 300, 700, True)
        assert errs["out"] <= 1e-2 and errs["lse"] <= 1e-2, errs
    else:
        q8, k8, v8, sq, sk, sv = R.quantize_qkv(q, k, v)
        out, lse, _ = attn_fwd(q8, k8, v8, sq, sk, sv, causal=True, ctas_per_sm=ctas)
        qd, kd, vd = R.dequantize_qkv(q8.cpu(), k8.cpu(), v8.cpu(), sq.cpu(), sk.cpu(), sv.cpu())
        out_ref, lse_ref = R.attention_reference(qd, kd, vd, True)
        gates(fwd_errors(out, lse, out_ref, lse_ref, 300, 700, True))
    assert out.shape == q.shape


# (B, Hq, Hkv, Nq, Nk, d): more marked blocks than SMs (a CTA of the persistent kernel recomputes several); a ragged last
# block whose rows partly lie in range; keys that end inside a group of 4 and of 32
RECOMPUTED = [(2, 8, 2, 1300, 1301, 128), (3, 4, 1, 1155, 1099, 64)]


@pytest.mark.parametrize("bf16,ctas", [(False, 1), (False, 2), (True, 2)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", RECOMPUTED)
def test_recomputed_rows(cuda, shape, causal, bf16, ctas):
    """Rows beyond the range are as exact as fp32 and a bf16 output allow; sequences of different lengths, one of them
    without a peak; natural lse; pmax."""
    from warpy_kernels import attn_fwd
    from warpy_kernels_b200.attn import fwd_api

    B, Hq, Hkv, Nq, Nk, d = shape
    q, k, v = late_peak_qkv(B, Hq, Hkv, Nq, Nk, d, [(700, 120.0), (901, 260.0)], seed=5, device=cuda)
    args = (q.bfloat16(), k.bfloat16(), v.bfloat16()) if bf16 else R.quantize_qkv(q, k, v)
    deq = tuple(x.float() for x in args) if bf16 else R.dequantize_qkv(*args)
    used = [Nk, 650, 903][:B]
    out, lse, pmax = attn_fwd(*args, causal=causal, ctas_per_sm=ctas, lse_natural=True,
                              seqused_k=torch.tensor(used, dtype=torch.int32, device=cuda))
    assert int(fwd_api._block_flags(cuda, 16).count_nonzero()) == 0
    for b, n in enumerate(used):
        s = deq[0][b] @ deq[1][b, :, :n].repeat_interleave(Hq // Hkv, 0).transpose(-1, -2) / math.sqrt(d)
        if causal:
            s = s.masked_fill(torch.arange(n, device=cuda) > torch.arange(Nq, device=cuda)[:, None] + n - Nq, float("-inf"))
        far = s.amax(-1) - s[..., :64].amax(-1) > 75.0  # 69 nats, and what fp32 logits near 260 may be off
        assert bool(far.any()) == (n > 700)
        if n <= 700:
            continue
        want = torch.softmax(s.double(), -1) @ deq[2][b, :, :n].repeat_interleave(Hq // Hkv, 0).double()
        # the output's own rounding to bf16 (2^-9) twice over
        assert R.rel_l2(out[b][far].double(), want[far]) < 2**-8
        assert torch.allclose(lse[b][far].double(), torch.logsumexp(s[far].double(), -1), rtol=1e-5)
        assert torch.allclose(pmax[b][far].double(), torch.softmax(s[far].double(), -1).amax(-1), rtol=2e-3)


@pytest.mark.parametrize("shape", [(1, 2, 1, 300, 900, 128), (2, 4, 2, 200, 700, 64)])
def test_first_scores_overflow_to_minus_infinity(cuda, shape):
    """The first 100 keys' scores are -inf in fp32, so the row reference is too and every row is computed again: those keys
    have no weight and the others theirs."""
    from warpy_kernels import attn_fwd

    B, Hq, Hkv, Nq, Nk, d = shape
    q, k, v = late_peak_qkv(B, Hq, Hkv, Nq, Nk, d, [], seed=11, device=cuda)
    k[:, :, 100:] = 0.0
    q, k = q * 1e20, k.clone()
    k[:, :, :100] = -1e20  # q . k about -1e42
    out, lse, pmax = attn_fwd(q.bfloat16(), k.bfloat16(), v.bfloat16(), ctas_per_sm=2)
    want = v.bfloat16().double()[:, :, 100:].mean(2).repeat_interleave(Hq // Hkv, 1)[:, :, None].expand(out.shape)
    assert R.rel_l2(out.double(), want) < 2**-8
    assert torch.allclose(lse, torch.full_like(lse, math.log2(Nk - 100)), rtol=1e-5)
    assert torch.allclose(pmax, torch.full_like(pmax, 1 / (Nk - 100)), rtol=1e-4)
