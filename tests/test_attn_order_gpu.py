"""GPU: the order in which the blocks of a causal problem are handed out (longest first over bands of heads).  A head
computed alone gives what it gives in the batch."""

import pytest
import torch

from oracle import reference_math as R
from tests.helpers import randn_qkv

pytestmark = pytest.mark.gpu


def _heads(t, b, h, n=1):
    return t[b : b + 1, h : h + n].contiguous()


# (B, Hq, Hkv, Nq, Nk, d): one band; as many heads as blocks do not divide; more blocks than are banded; rows without keys;
# heads too large for one band
BF16_SHAPES = [(2, 6, 3, 700, 700, 128), (1, 5, 5, 130, 900, 64), (3, 8, 4, 900, 300, 64), (2, 16, 8, 4200, 4200, 64),
               (1, 14, 7, 9000, 9000, 128)]


@pytest.mark.parametrize("shape", BF16_SHAPES)
def test_bf16_backward_order(cuda, shape):
    from warpy_kernels import attn_bwd, attn_fwd

    B, Hq, Hkv, Nq = shape[:4]
    group = Hq // Hkv
    q, k, v = [t.bfloat16() for t in randn_qkv(*shape, device=cuda)]
    dout = torch.randn(q.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(7)).bfloat16()
    saved = attn_fwd(q, k, v, causal=True)
    dq, dk, dv = attn_bwd(q, k, v, *saved, dout, causal=True)
    for b, hkv in {(0, 0), (B - 1, Hkv - 1), (B // 2, Hkv // 2)}:
        hq = hkv * group
        one = attn_bwd(_heads(q, b, hq, group), _heads(k, b, hkv), _heads(v, b, hkv),
                       *(_heads(t, b, hq, group) for t in saved), _heads(dout, b, hq, group), causal=True)
        assert torch.equal(one[0], _heads(dq, b, hq, group))
        assert torch.equal(one[1], _heads(dk, b, hkv)) and torch.equal(one[2], _heads(dv, b, hkv))


# one band with a remainder; rows without keys; heads too large for one band (the persistent FP8 kernel from 2048 keys on)
FWD_SHAPES = [(2, 6, 3, 2100, 2100, 128), (3, 8, 4, 4500, 2300, 64), (1, 14, 7, 9000, 9000, 128)]


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("shape", FWD_SHAPES)
def test_forward_order(cuda, shape, fp8):
    from warpy_kernels import attn_fwd

    B, Hq, Hkv = shape[:3]
    group = Hq // Hkv
    q, k, v = randn_qkv(*shape, device=cuda)
    if fp8:
        q, k, v, *scales = R.quantize_qkv(q, k, v)
    else:
        (q, k, v), scales = [t.bfloat16() for t in (q, k, v)], []
    got = attn_fwd(q, k, v, *scales, causal=True)
    for b, hkv in {(0, 0), (B - 1, Hkv - 1), (B // 2, Hkv // 2)}:
        one = attn_fwd(_heads(q, b, hkv * group, group), _heads(k, b, hkv), _heads(v, b, hkv),
                       *(s[b : b + 1, hkv : hkv + 1].contiguous() for s in scales), causal=True)
        want = [_heads(t, b, hkv * group, group) for t in got]
        if fp8:
            # which of the persistent kernel's groups takes a tile depends on the blocks its CTA had before, and with it
            # the order of the fp32 sums: a few ulp of fp32 in lse and pmax, a rounding of bf16 (2^-8 at most) in out
            assert R.rel_l2(one[0], want[0]) < 2**-8
            assert all(torch.allclose(x, w, rtol=2**-20, atol=2**-20) for x, w in zip(one[1:], want[1:]))
        else:
            assert all(torch.equal(x, w) for x, w in zip(one, want))


# enough blocks that no block is divided over a cluster in the batch; in the head alone it is, so the fp32 sums are in
# another order and the bf16 results (2^-9 apart at most where they round differently) agree to less than 2^-8
@pytest.mark.parametrize("shape", [(2, 6, 3, 2100, 2100, 128), (3, 16, 8, 1500, 1000, 64)])
def test_fp8_backward_order(cuda, shape):
    from warpy_kernels import attn_bwd, attn_fwd

    B, Hq, Hkv = shape[:3]
    group = Hq // Hkv
    q, k, v, *scales = R.quantize_qkv(*randn_qkv(*shape, device=cuda))
    dout = torch.randn(q.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(7)).bfloat16()
    saved = attn_fwd(q, k, v, *scales, causal=True)
    grads = attn_bwd(q, k, v, *saved, dout, *scales, causal=True)
    for b, hkv in {(0, 0), (B - 1, Hkv - 1), (B // 2, Hkv // 2)}:
        hq = hkv * group
        one = attn_bwd(_heads(q, b, hq, group), _heads(k, b, hkv), _heads(v, b, hkv),
                       *(_heads(t, b, hq, group) for t in saved), _heads(dout, b, hq, group),
                       *(s[b : b + 1, hkv : hkv + 1].contiguous() for s in scales), causal=True)
        want = (_heads(grads[0], b, hq, group), _heads(grads[1], b, hkv), _heads(grads[2], b, hkv))
        assert all(R.rel_l2(x, w) < 2**-8 for x, w in zip(one, want))


# no more query blocks than SMs: below 2048 keys, with a two-term launch beside the main one, and from 2048 keys on
@pytest.mark.parametrize("shape,causal", [((1, 16, 16, 1100, 1100, 128), True), ((2, 8, 2, 1024, 1300, 64), False),
                                          ((1, 9, 9, 2048, 2304, 128), True)])
def test_few_blocks_repeat_to_the_bit(cuda, shape, causal):
    """With a kernel of another stream on most SMs, so that many CTAs have to wait for one: a block must not go to a
    running CTA then, whose sums would be in another order."""
    from warpy_kernels import attn_fwd

    q, k, v = randn_qkv(*shape, device=cuda)
    q8, k8, v8, *scales = R.quantize_qkv(q, k, v)
    busy = R.quantize_qkv(*randn_qkv(1, 1, 1, 100 * 128, 16384, 128, device=cuda))  # 100 query blocks
    side = torch.cuda.Stream()
    want = attn_fwd(q8, k8, v8, *scales, causal=causal)
    attn_fwd(*busy)
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(side):
            attn_fwd(*busy)
        got = [attn_fwd(q8, k8, v8, *scales, causal=causal) for _ in range(4)]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for one in got for a, b in zip(one, want))
