"""GPU: the entry points' compiled host side (``_host``) against the prepared launches, which are set up in Python:
same kernels, so the same bits; and the calls it must leave to the Python code (copies, errors)."""

import pytest
import torch

from oracle import reference_math as R
from tests.helpers import randn_qkv

pytestmark = pytest.mark.gpu

FP8 = torch.float8_e4m3fn


def _qkv(cuda, fp8, layout, d):
    q, k, v = randn_qkv(2, 4, 2, 130, 200, d, seed=3, device=cuda)
    if fp8:
        q, k, v, *scales = R.quantize_qkv(q, k, v)
    else:
        q, k, v, scales = q.bfloat16(), k.bfloat16(), v.bfloat16(), ()
    if layout == "bnhd":
        q, k, v = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in (q, k, v))
    return q, k, v, tuple(scales)


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("layout,d", [("bhnd", 128), ("bnhd", 64)])
def test_attention_matches_prepared_launches(cuda, fp8, layout, d):
    from warpy_kernels import attn_bwd, attn_fwd
    from warpy_kernels.attn import make_attn_bwd, make_attn_fwd
    from warpy_kernels_b200 import _lib

    q, k, v, scales = _qkv(cuda, fp8, layout, d)
    used = torch.tensor([200, 77], dtype=torch.int32, device=cuda)
    for options in ({}, {"lse_natural": True, "softmax_scale": 0.07}, {"seqused_k": used}, {"return_lse": False}):
        got = attn_fwd(q, k, v, *scales, causal=True, **options)
        assert _lib.host().attn_fwd(q, k, v, *(scales or (None,) * 3), True, **options) is not None
        launch, *want = make_attn_fwd(q, k, v, *scales, causal=True, **options)
        launch()
        for x, y in zip(got, want):
            assert (x is None and y is None) or (torch.equal(x, y) and x.stride() == y.stride())
    out, lse, pmax = attn_fwd(q, k, v, *scales, causal=True)
    dout = torch.randn_like(out, memory_format=torch.preserve_format)
    got = attn_bwd(q, k, v, out, lse, pmax, dout, *scales, causal=True)
    launch, finish = make_attn_bwd(q, k, v, out, lse, pmax, dout, *scales, causal=True)
    launch()
    assert all(torch.equal(x, y) for x, y in zip(got, finish()))


@pytest.mark.parametrize("kind", ["bf16", "fp16", "fp8"])
@pytest.mark.parametrize("options", [{}, {"act": "gelu", "store_pre": True}, {"act": "gelu"}, {"act": "dgelu"},
                                     {"accum": True}, {"out_mx": True}, {"scales": True}, {"group_m": 2, "bn": 256}])
def test_gemm_matches_prepared_launches(cuda, kind, options):
    from warpy_kernels import gemm, make_gemm

    g = torch.Generator(device=cuda).manual_seed(0)
    m, n, k = 128, 512, 256
    dt = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp8": FP8}[kind]
    odt = torch.float16 if kind == "fp16" else torch.bfloat16
    a = torch.randn(m, k, device=cuda, generator=g).to(dt)
    b = torch.randn(n, k, device=cuda, generator=g).to(dt)
    c = torch.randn(m, n, device=cuda, generator=g).to(odt)
    kw = dict(options)
    if kw.pop("scales", False):
        kw.update(scale_a=torch.rand(m, device=cuda, generator=g), scale_b=torch.rand(n, device=cuda, generator=g))
        if kind == "fp8":
            kw["a_scale_mx"] = torch.randint(120, 130, (m, k // 32), device=cuda, generator=g, dtype=torch.uint8)
    if kw.get("act") == "dgelu":
        kw["pre"] = c
    got = gemm(a, b, c.clone() if kw.get("accum") else None, **kw)
    launch, *want = make_gemm(a, b, c.clone() if kw.get("accum") else None, **kw)
    launch()
    got = got if isinstance(got, tuple) else (got,)
    assert len(got) == len(want)
    for x, y in zip(got, want):
        assert (x is None and y is None) or torch.equal(x.view(torch.uint8), y.view(torch.uint8))


def test_what_is_left_to_python(cuda):
    from warpy_kernels import attn_fwd, gemm, quantize_mx
    from warpy_kernels_b200 import _lib

    host = _lib.host()
    q, k, v, scales = _qkv(cuda, True, "bhnd", 128)
    base = attn_fwd(q, k, v, *scales)
    wide = torch.zeros(2, 4, 130, 136, device=cuda, dtype=torch.uint8).view(FP8)  # a row stride TMA cannot take
    wide[..., :128] = q
    assert host.attn_fwd(wide[..., :128], k, v, *scales) is None
    assert torch.equal(attn_fwd(wide[..., :128], k, v, *scales)[0], base[0])
    assert torch.equal(attn_fwd(q, k, v, *(s.double() for s in scales))[0], base[0])
    with pytest.raises(ValueError):
        attn_fwd(q, k[:, :, :, :64], v, *scales)
    with pytest.raises(NotImplementedError):
        attn_fwd(q.half(), k.half(), v.half())
    with pytest.raises(TypeError):
        attn_fwd(q, k, v, *scales, no_such_option=1)
    with pytest.raises(ValueError):
        attn_fwd(q, k, v, *scales, softmax_scale=-1.0)
    a = torch.zeros(128, 64, device=cuda, dtype=torch.bfloat16)
    with pytest.raises(ValueError):
        gemm(a, a[:, :32])
    with pytest.raises(ValueError):
        quantize_mx(a[:, :40])


def test_arguments_without_a_value_are_left_to_python(cuda):
    """An option whose truth value raises, and a whole number beyond a C long: the error of the Python code, not a default."""
    from warpy_kernels import attn_bwd, attn_fwd, gemm

    q, k, v, scales = _qkv(cuda, True, "bhnd", 128)
    saved = attn_fwd(q, k, v, *scales)
    two = torch.tensor([1, 0], device=cuda)
    for option in ("causal", "return_lse", "lse_natural"):
        with pytest.raises(RuntimeError, match="ambiguous"):
            attn_fwd(q, k, v, *scales, **{option: two})
    with pytest.raises(RuntimeError, match="ambiguous"):
        attn_bwd(q, k, v, *saved, torch.ones_like(saved[0]), *scales, causal=two)
    with pytest.raises(ValueError, match="ctas_per_sm"):
        attn_fwd(q, k, v, *scales, ctas_per_sm=2**70)
    a = torch.zeros(128, 64, device=cuda, dtype=torch.bfloat16)
    for option in ("out_mx", "store_pre", "a_trans", "b_trans", "accum", "cta_pair"):
        with pytest.raises(RuntimeError, match="ambiguous"):
            gemm(a, a, **{option: two})
