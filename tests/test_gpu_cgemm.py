"""The tiled complex64 products on the FP32 pipes at the edges of every tile
shape (columns 8, 16, 32, 64; rows 16, 128, 256; k-steps of 8 and 16), odd
sizes, batches and strides that leave outputs on 8-byte boundaries."""
import numpy as np
import pytest

from qflex_gb300 import FP32, Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (256, 8, 8), (255, 7, 9), (600, 5, 3), (256, 16, 16), (257, 15, 33), (128, 32, 16), (129, 31, 17), (16, 256, 16),
    (17, 300, 40), (32, 64, 7), (128, 64, 8), (130, 65, 8), (129, 63, 100), (1000, 200, 1), (2, 2, 31),
    (70000, 16, 16), (40000, 8, 64), (5000, 64, 64)])
@pytest.mark.parametrize("batch,extra", [(1, 0), (3, 1)])
def test_tiled_product(built_lib, m, n, k, batch, extra):
    import torch
    g = np.random.default_rng(m + n + k)
    stride = m * k + k * n + m * n + extra
    buf = (g.standard_normal((batch, stride)) + 1j * g.standard_normal((batch, stride))).astype(np.complex64)
    d = torch.from_numpy(buf).cuda()
    torch.cuda.synchronize()
    ctx = Context(0, FP32)
    at = d.data_ptr()
    ctx.multiply(at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, batch, stride)
    ctx.synchronize()
    out = d.cpu().numpy()
    # 2 k rounded additions of each part: 2 k 2^-24 of the sum of magnitudes,
    # times sqrt 2 for the two parts.
    tol = 2 * k * 2.0 ** -24 * 2 ** 0.5
    for row, got in zip(buf, out):
        A, B = row[:m * k].reshape(m, k).astype(complex), row[m * k:m * k + k * n].reshape(k, n).astype(complex)
        C = got[m * k + k * n:m * k + k * n + m * n].reshape(m, n)
        assert np.max(np.abs(C - A @ B) / (np.abs(A) @ np.abs(B))) < tol
        assert np.array_equal(got[:m * k + k * n], row[:m * k + k * n])
        assert np.array_equal(got[m * k + k * n + m * n:], row[m * k + k * n + m * n:])


def test_product_without_terms_is_zero(built_lib):
    import torch
    C = torch.full((300, 20), 7, dtype=torch.complex64, device="cuda")
    ctx = Context(0, FP32)
    torch.cuda.synchronize()
    ctx.multiply(C.data_ptr() + 8, C.data_ptr() + 16, C.data_ptr(), 300, 20, 0)
    ctx.synchronize()
    assert not C.any()


@pytest.mark.parametrize("m,n,k", [
    (16, 16, 32), (33, 31, 17), (64, 8, 191), (65, 7, 192), (16, 16, 192), (31, 33, 257), (130, 9, 1000), (64, 64, 4096),
    (2, 3, 700), (1000, 24, 300), (512, 130, 511)])
@pytest.mark.parametrize("batch,extra", [(1, 0), (3, 1)])
def test_few_tiles(built_lib, m, n, k, batch, extra):
    """Small tiles, and k in runs (from 192 terms on) summed afterwards."""
    test_tiled_product(built_lib, m, n, k, batch, extra)


@pytest.mark.parametrize("m,n,k", [
    (10000, 16, 33), (9999, 9, 16), (16001, 12, 100), (5000, 32, 40), (6001, 17, 15), (3000, 200, 128), (2999, 193, 131),
    (64, 3000, 20), (33, 2999, 131), (1586, 161, 513), (1001, 300, 700)])
@pytest.mark.parametrize("batch,extra", [(1, 0), (2, 1)])
def test_one_wave(built_lib, m, n, k, batch, extra):
    """Tiles for products that the SMs hold at once, and of 64 rows."""
    test_tiled_product(built_lib, m, n, k, batch, extra)
