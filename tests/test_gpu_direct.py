"""Split-precision products at the edges of tiles and blocks of the kernel that
splits A itself, and on rows whose magnitude changes from one block of 32 values
to the next. Sizes that no contraction has run in FP32 here below 2^25 terms in
all or 96 a sum; test_gpu_split_routes.py has such edges above that line."""
import numpy as np
import pytest

from qflex_gb300 import BF16X3, FP16X3, TF32X3, Context

pytestmark = pytest.mark.gpu

# Error of an element against FP64, relative to sum |a| |b|: operands carried
# to 22 bits (2 * 2^-23 each), twelve truncating additions per chunk of two
# k-steps (2^-23 each), the chunks' FP32 additions (k / 32 * 2^-24), real and
# imaginary part together (sqrt 2): below 4e-6 for k <= 256.
TOL = 4e-6


def _rows(kind, g, m, k):
    block = np.arange(k) // 32
    scale = {"gauss": np.zeros(k), "grow": 13.0 * block, "shrink": -13.0 * block,
             "zeros": np.where(block == 0, -np.inf, 0.0), "tiny": np.full(k, -118.0),
             "jump": np.where(block % 2 == 0, 0.0, 3.0)}[kind]
    return (g.standard_normal((m, k)) + 1j * g.standard_normal((m, k))) * np.exp2(scale)


@pytest.mark.parametrize("kind", ["gauss", "grow", "shrink", "zeros", "tiny", "jump"])
@pytest.mark.parametrize("m,n,k,batch,extra", [
    (64, 64, 16, 1, 0), (128, 128, 32, 1, 0), (129, 64, 64, 2, 0), (300, 128, 64, 1, 1), (192, 256, 128, 3, 1),
    (1024, 1024, 32, 1, 0), (20000, 64, 16, 1, 0)])
def test_direct_product(built_lib, kind, m, n, k, batch, extra, precision=FP16X3, tol=TOL):
    import torch
    g = np.random.default_rng(m + n + k)
    stride = m * k + k * n + m * n + extra  # an odd stride leaves rows on 8-byte boundaries
    buf = np.zeros((batch, stride), np.complex64)
    scale_b = 2.0 ** 40 if kind == "tiny" else 1.0
    with np.errstate(under="ignore"):
        for row in buf:
            row[:m * k] = _rows(kind, g, m, k).reshape(-1)
            row[m * k:m * k + k * n] = (g.standard_normal(k * n) + 1j * g.standard_normal(k * n)) * scale_b
    d = torch.from_numpy(buf).cuda()
    torch.cuda.synchronize()
    ctx = Context(0, precision)
    at = d.data_ptr()
    ctx.multiply(at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, batch, stride)
    ctx.synchronize()
    out = d.cpu().numpy()
    for row, got in zip(buf, out):
        A, B = row[:m * k].reshape(m, k).astype(complex), row[m * k:m * k + k * n].reshape(k, n).astype(complex)
        C = got[m * k + k * n:m * k + k * n + m * n].reshape(m, n)
        assert np.isfinite(C).all()
        assert np.max(np.abs(C - A @ B) / (np.abs(A) @ np.abs(B) + 1e-300)) < tol
        assert np.array_equal(got[:m * k + k * n], row[:m * k + k * n])
        assert np.array_equal(got[m * k + k * n + m * n:], row[m * k + k * n + m * n:])


@pytest.mark.parametrize("kind", ["gauss", "grow", "tiny"])
@pytest.mark.parametrize("m,n,k,batch,extra", [
    (256, 16, 96, 1, 0), (300, 17, 100, 2, 0), (257, 31, 129, 1, 1), (1000, 32, 256, 1, 0), (384, 33, 128, 3, 1),
    (257, 50, 97, 1, 0), (20000, 63, 112, 1, 0), (300, 64, 96, 2, 0)])
def test_narrow_tiles(built_lib, kind, m, n, k, batch, extra):
    """Tiles of 32 and 64 columns, also of products that FP32 kernels ran."""
    test_direct_product(built_lib, kind, m, n, k, batch, extra)


@pytest.mark.parametrize("kind", ["gauss", "jump", "tiny"])
@pytest.mark.parametrize("m,n,k,batch,extra", [
    (129, 128, 160, 1, 0), (256, 129, 256, 1, 0), (257, 640, 161, 1, 1), (640, 1100, 192, 2, 0), (383, 1500, 130, 1, 0),
    (20000, 256, 256, 1, 0), (128, 1100, 192, 1, 0)])
def test_pairs(built_lib, kind, m, n, k, batch, extra):
    """Tiles of two CTAs, also with an empty second half, and of one beside them."""
    test_direct_product(built_lib, kind, m, n, k, batch, extra)


# 3xTF32: chunks of 16 values, so k / 16 FP32 additions: below 6e-6 for k <= 400.
@pytest.mark.parametrize("m,n,k,batch,extra", [
    (64, 64, 16, 1, 0), (128, 128, 32, 1, 0), (129, 64, 64, 2, 0), (300, 130, 97, 1, 1), (257, 640, 111, 1, 1),
    (640, 1100, 160, 2, 0), (383, 1500, 400, 1, 0), (20000, 256, 64, 1, 0), (128, 1100, 192, 1, 0)])
def test_tf32(built_lib, m, n, k, batch, extra):
    test_direct_product(built_lib, "gauss", m, n, k, batch, extra, TF32X3, 6e-6)


# BF16x3: 24 truncating additions per chunk of two k-steps of 16.
@pytest.mark.parametrize("m,n,k,batch,extra", [
    (129, 64, 65, 1, 0), (256, 128, 128, 1, 0), (300, 130, 97, 1, 1), (257, 640, 111, 1, 1), (640, 1100, 160, 2, 0),
    (383, 1500, 400, 1, 0), (20000, 256, 80, 1, 0)])
def test_bf16(built_lib, m, n, k, batch, extra):
    test_direct_product(built_lib, "gauss", m, n, k, batch, extra, BF16X3, 6e-6)
