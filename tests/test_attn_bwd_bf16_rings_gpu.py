"""GPU: the BF16 backward where its rings and buffer pairs begin and end: one to seven tiles of keys (dQ: K ring of three,
V ring of two, two sets of dS) and of queries (dK/dV: two stages, two groups), remainders of every kind."""

import pytest
import torch

from tests.helpers import randn_qkv
from tests.test_attn_bwd_gpu import _bf16_case

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 1, 127, 129, 64), (1, 2, 2, 128, 256, 128), (1, 2, 1, 300, 384, 128),
          (2, 1, 1, 513, 385, 64), (1, 3, 1, 640, 641, 128), (1, 1, 1, 130, 896, 128), (1, 2, 1, 900, 65, 128)]


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_tile_counts(cuda, shape, causal):
    q, k, v = randn_qkv(*shape, device=cuda)
    dout = torch.randn(q.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(7))
    _bf16_case(cuda, q, k, v, dout, causal)
