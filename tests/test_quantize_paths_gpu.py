"""GPU: the quantiser's load and store widths: rows that start on 16-byte but not 32-byte boundaries, row strides, block
counts that are no multiple of the four whose scale bytes leave together, and the last, partly filled CTA.  Bit-exact."""

import numpy as np
import pytest
import torch

from oracle import c_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols,offset,stride", [(1, 32, 0, 32), (5, 32, 8, 40), (33, 96, 0, 96), (7, 160, 8, 168),
                                                     (129, 480, 0, 512), (513, 32, 0, 32), (300, 1056, 0, 1056)])
def test_bit_exact_whatever_the_alignment(cuda, dtype, rows, cols, offset, stride):
    from warpy_kernels import quantize_mx

    g = torch.Generator(device=cuda).manual_seed(0)
    flat = torch.randn(offset + rows * stride, device=cuda, generator=g).to(dtype)
    x = torch.as_strided(flat, (rows, cols), (stride, 1), offset)
    q, s = quantize_mx(x)
    host = x.cpu().contiguous()
    host = host.view(torch.int16).numpy().view(np.uint16) if dtype == torch.bfloat16 else host.numpy()
    want_q, want_s = c_oracle.quantize_mx(host)
    assert np.array_equal(s.cpu().numpy(), want_s)
    assert np.array_equal(q.view(torch.uint8).cpu().numpy(), want_q)
