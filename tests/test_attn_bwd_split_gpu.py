"""GPU: the FP8 backward of problems with fewer key or query blocks than SMs: a block's tiles divided among the CTAs of a
cluster (1 to 8 of them, uneven shares, CTAs without a tile), the dQ kernel beside the dK/dV kernel."""

import pytest
import torch

from oracle import reference_math as R
from tests.helpers import randn_qkv
from tests.test_attn_bwd_gpu import _oracle_grads, check_grads

pytestmark = pytest.mark.gpu

# (B, Hq, Hkv, Nq, Nk, d): few key blocks with many query tiles and the reverse; ragged; grouped heads; one block only
SHAPES = [(1, 1, 1, 64, 64, 128), (1, 1, 1, 2000, 130, 128), (1, 1, 1, 130, 2000, 64), (1, 8, 1, 513, 513, 128),
          (1, 16, 2, 300, 100, 64), (2, 4, 2, 1000, 1000, 128), (1, 2, 1, 1152, 1152, 128), (3, 3, 1, 700, 640, 64)]


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_few_blocks(cuda, shape, causal):
    from warpy_kernels import attn_bwd, attn_fwd

    q, k, v = randn_qkv(*shape, device=cuda)
    q8, k8, v8, sq, sk, sv = R.quantize_qkv(q, k, v)
    dout = torch.randn(q.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(7)).bfloat16()
    out, lse, pmax = attn_fwd(q8, k8, v8, sq, sk, sv, causal=causal)
    got = attn_bwd(q8, k8, v8, out, lse, pmax, dout, sq, sk, sv, causal=causal)
    check_grads(got, _oracle_grads(q8, k8, v8, sq, sk, sv, dout, causal))
    for _ in range(2):  # the parts are added up in a fixed order
        again = attn_bwd(q8, k8, v8, out, lse, pmax, dout, sq, sk, sv, causal=causal)
        assert all(torch.equal(x, y) for x, y in zip(again, got))
