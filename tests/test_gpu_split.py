"""Split-precision products whose sizes fill no tile, k-step or vector: from 2^25
terms in all on, any n and any k from 96 on run on the tensor cores, smaller ones
in FP32 (test_gpu_split_routes.py checks the route as well). B is split from the
columns of the row-major matrix, A from its rows, mostly inside the product."""
import numpy as np
import pytest

from qflex_gb300 import BF16X3, FP16X3, TF32X3, Context

pytestmark = pytest.mark.gpu

# Of sum |a| |b| per element. Operands carry 22 bits or more (2^-22 per
# product), a chunk of two k-steps 24 truncating additions in BF16x3, 12 in the
# others (2^-23 each), the chunks k / 16 FP32 additions (2^-24 each), two parts
# (sqrt 2): below 6e-6 for k <= 400, 2e-5 for k <= 4100.
CASES = [(64, 64, 96, 6e-6), (65, 67, 97, 6e-6), (129, 130, 111, 6e-6), (1000, 200, 100, 6e-6),
         (100, 1025, 129, 6e-6), (300, 2051, 255, 6e-6), (257, 1100, 333, 6e-6), (70, 1500, 4100, 2e-5),
         (3001, 690, 1100, 2e-5), (128, 4096, 2048, 2e-5)]


@pytest.mark.parametrize("precision", [FP16X3, TF32X3, BF16X3], ids=["fp16x3", "tf32x3", "bf16x3"])
@pytest.mark.parametrize("m,n,k,tol", CASES)
@pytest.mark.parametrize("batch,extra", [(1, 0), (2, 1)])
def test_any_size(built_lib, precision, m, n, k, tol, batch, extra):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    stride = m * k + k * n + m * n + extra
    buf = torch.randn((batch, stride), dtype=torch.complex64, device="cuda", generator=gen)
    # Columns of B of very different size: each has its own scale.
    B = buf[:, m * k:m * k + k * n].view(batch, k, n)
    B *= torch.exp2(torch.arange(n, device="cuda") % 41 - 20.0)
    keep = buf.clone()
    torch.cuda.synchronize()
    ctx = Context(0, precision)
    at = buf.data_ptr()
    ctx.multiply(at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, batch, stride)
    ctx.synchronize()
    assert torch.equal(buf[:, :m * k + k * n], keep[:, :m * k + k * n])
    assert torch.equal(buf[:, m * k + k * n + m * n:], keep[:, m * k + k * n + m * n:])
    for row in buf:
        A, B = (x.to(torch.complex128) for x in (row[:m * k].view(m, k), row[m * k:m * k + k * n].view(k, n)))
        C = row[m * k + k * n:m * k + k * n + m * n].view(m, n)
        assert float(((C - A @ B).abs() / (A.abs() @ B.abs())).max()) < tol
