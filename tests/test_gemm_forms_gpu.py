"""GPU: the forms of the GEMM kernel that small problems take: 128-column tiles and K split over the CTAs of a cluster.

Shapes on both sides of each choice: the fewest K blocks a range may have, ranges of unequal length, one 128-column tile
over the edge of the last 256-column one, half of a pair outside M.  The sum over K is taken in another order than the
oracle's, so the bound is the bf16 rounding of the output (2^-9 relative) plus fp32 sums."""

import pytest
import torch

from oracle import reference_math as R

pytestmark = pytest.mark.gpu

FP8 = torch.float8_e4m3fn
# (M, N, K blocks): narrow, narrow with 2 and 4 ranges, pairs with 2 ranges; 17 and 35 blocks do not divide evenly
SHAPES = [(128, 128, 1), (128, 128, 16), (128, 640, 17), (128, 4096, 35), (256, 1024, 64), (640, 2048, 33),
          (2048, 640, 82), (2176, 640, 83)]


@pytest.mark.parametrize("kind", ["bf16", "fp8"])
@pytest.mark.parametrize("shape", SHAPES)
def test_split_and_narrow_forms(cuda, kind, shape):
    from warpy_kernels import gemm, quantize_mx

    m, n, kb = shape
    k = kb * (128 if kind == "fp8" else 64)
    g = torch.Generator(device=cuda).manual_seed(0)
    a = torch.randn(m, k, device=cuda, generator=g).bfloat16()
    b = torch.randn(n, k, device=cuda, generator=g).bfloat16()
    kw, ref = {}, {}
    if kind == "fp8":
        (a, sa), (b, sb) = quantize_mx(a), quantize_mx(b)
        kw = {"a_scale_mx": sa, "b_scale_mx": sb}
    out = gemm(a, b, **kw)
    want = R.gemm_reference(a, b, **kw)
    assert R.rel_l2(out, want) <= 3e-3  # 2^-9 relative rounding of the output, root mean square below 2^-9
    for pair in (True, False):  # every form adds up K in the same order
        assert torch.equal(gemm(a, b, cta_pair=pair, **kw), out)
    # the fused epilogue behind the exchange: column scales, GELU with its input kept, MXFP8 copy
    cols = torch.rand(n, device=cuda, generator=g) + 0.5
    post, pre, q, s = gemm(a, b, scale_b=cols, act="gelu", store_pre=True, out_mx=True, **kw)
    x = want * cols
    assert R.rel_l2(pre, x) <= 3e-3
    assert R.rel_l2(post, torch.nn.functional.gelu(x)) <= 4e-3  # the same, on values that GELU shrinks
    assert R.rel_l2(R.mx_dequant(q, s), post.float()) <= 4e-2
