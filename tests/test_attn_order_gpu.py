"""GPU: the order in which the blocks of a causal problem are handed out (longest first over bands of heads).  Every head
computed alone gives the same bits as in the batch."""

import pytest
import torch

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
