"""Split-precision multiplies that run on the tensor cores, each checked to do
so: its result differs in some bit from that of the FP32 kernels, which take
the smaller products of a split-precision context (below 96 terms a sum or 2^25
in all, unless n and k are powers of two)."""
import pytest

from qflex_gb300 import BF16X3, FP16X3, FP32, TF32X3, Context

pytestmark = pytest.mark.gpu


def _multiply(precision, buf, m, n, k):
    import torch
    out = buf.clone()
    torch.cuda.synchronize()
    ctx = Context(0, precision)
    at = out.data_ptr()
    ctx.multiply(at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, out.shape[0], out.shape[1])
    ctx.synchronize()
    return out


def check(precision, A, B, extra, tol):
    """C = A B of (batch, m, k) and (batch, k, n), entries `extra` elements
    further apart than they need, against complex128: every element within
    `tol` of its sum |a| |b|, nothing else written, and not the FP32 kernels."""
    import torch
    batch, m, k = A.shape
    n = B.shape[2]
    buf = torch.zeros((batch, m * k + k * n + m * n + extra), dtype=torch.complex64, device="cuda")
    buf[:, :m * k] = A.reshape(batch, -1)
    buf[:, m * k:m * k + k * n] = B.reshape(batch, -1)
    got = _multiply(precision, buf, m, n, k)
    C = slice(m * k + k * n, m * k + k * n + m * n)
    assert torch.equal(got[:, :m * k + k * n], buf[:, :m * k + k * n])
    assert torch.equal(got[:, C.stop:], buf[:, C.stop:])
    assert not torch.equal(got[:, C], _multiply(FP32, buf, m, n, k)[:, C])
    for a, b, c in zip(A.to(torch.complex128), B.to(torch.complex128), got[:, C].view(batch, m, n)):
        assert float(((c - a @ b).abs() / (a.abs() @ b.abs())).max()) < tol


def randn(shape, seed):
    import torch
    return torch.randn(shape, dtype=torch.complex64, device="cuda",
                       generator=torch.Generator(device="cuda").manual_seed(seed))


# Of sum |a| |b| per element, k <= 320: operands carried to 22 bits of the
# largest component of their 32 values (2 * 2^-23 each, a block's largest
# component up to four times its mean magnitude), twelve truncating additions
# per chunk of two k-steps (2^-23 each), the chunks' FP32 additions (k / 32 *
# 2^-24), real and imaginary part together (sqrt 2): below 6e-6.
@pytest.mark.parametrize("m,n,k,batch", [(640, 512, 320, 1), (129, 4096, 256, 1), (40000, 128, 160, 2),
                                         (70000, 32, 256, 1), (20000, 64, 192, 2)])
def test_block_exponents(built_lib, m, n, k, batch):
    """Every row's blocks of 32 values have scales of their own, far apart, in
    more blocks than the ring of exponents has places: a sum takes each at the
    scale of its block, in pairs of CTAs and alone."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    scale = torch.randint(-30, 31, (batch, m, (k + 31) // 32), device="cuda", generator=gen)
    A = randn((batch, m, k), k) * torch.exp2(scale.repeat_interleave(32, -1)[..., :k])
    check(FP16X3, A, randn((batch, k, n), n), 0, 6e-6)


@pytest.mark.parametrize("precision,m,n,k", [
    (FP16X3, 300, 640, 200), (FP16X3, 20000, 256, 256), (FP16X3, 100, 1000, 400), (FP16X3, 60000, 32, 128),
    (TF32X3, 300, 640, 200), (TF32X3, 20000, 256, 256), (TF32X3, 100, 1000, 400), (BF16X3, 300, 640, 200),
    (BF16X3, 20000, 256, 256)])
def test_abandoned_products(built_lib, precision, m, n, k):
    """Products whose pipeline waits run out at once (limit 1 ns), in pairs and
    alone, end with the error and with every copy landed: the products after
    them, in the same context and at the default limit, are right."""
    import torch

    from qflex_gb300 import QflexGb300Error
    A, B = randn((1, m, k), k)[0], randn((1, k, n), n)[0]
    C = torch.zeros((m, n), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    ctx = Context(0, precision)
    want = A.to(torch.complex128) @ B.to(torch.complex128)
    bound = A.abs().double() @ B.abs().double()
    for _ in range(3):
        ctx.set_option("tc_wait_ns", 1)
        for _ in range(4):
            ctx.multiply(A.data_ptr(), B.data_ptr(), C.data_ptr(), m, n, k)
            with pytest.raises(QflexGb300Error, match="pipeline wait expired"):
                ctx.synchronize()
        ctx.set_option("tc_wait_ns", 0)
        ctx.multiply(A.data_ptr(), B.data_ptr(), C.data_ptr(), m, n, k)
        ctx.synchronize()
        # Bound as for test_block_exponents, k <= 400 (3xTF32: chunks of 16 terms).
        assert float(((C - want).abs() / bound).max()) < 8e-6
