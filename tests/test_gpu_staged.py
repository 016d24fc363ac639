"""The FP32 products that run one tile per block, at odd sizes, partial tiles
and strides that leave rows on 8-byte boundaries."""
import pytest

from qflex_gb300 import FP32, Context

pytestmark = pytest.mark.gpu

# (m, n, k, batch, elements between entries beyond their own): tiles of 128 x 64
# in rounds that persistent blocks fill badly or on rows of 8 bytes, tiles of
# 256 x 16 on rows of 8 bytes.
STAGED = [(1478, 310, 331, 7, 0), (1850, 257, 256, 6, 1), (1729, 1021, 151, 2, 1), (1634, 41, 387, 4, 0),
          (129, 1217, 501, 3, 1), (30001, 11, 161, 1, 0), (74497, 16, 41, 1, 0), (15001, 9, 153, 6, 1),
          (40001, 13, 29, 4, 0)]


@pytest.mark.parametrize("m,n,k,batch,extra", STAGED)
def test_one_tile_per_block(built_lib, m, n, k, batch, extra):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    buf = torch.randn((batch, m * k + k * n + m * n + extra), dtype=torch.complex64, device="cuda", generator=gen)
    keep = buf.clone()
    torch.cuda.synchronize()
    ctx = Context(0, FP32)
    at = buf.data_ptr()
    ctx.multiply(at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, batch, buf.shape[1])
    ctx.synchronize()
    out = slice(m * k + k * n, m * k + k * n + m * n)
    assert torch.equal(buf[:, :out.start], keep[:, :out.start]) and torch.equal(buf[:, out.stop:], keep[:, out.stop:])
    # 2 k rounded additions of each part: 2 k 2^-24 of the sum of magnitudes,
    # times sqrt 2 for the two parts.
    tol = 2 * k * 2.0 ** -24 * 2 ** 0.5
    for row in buf:
        A, B, C = row[:m * k].view(m, k).cdouble(), row[m * k:out.start].view(k, n).cdouble(), row[out].view(m, n)
        assert float(((C - A @ B).abs() / (A.abs() @ B.abs())).max()) < tol
