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


def _parts(A, B):
    """Real and imaginary part of A B by products of real matrices in 64 bits:
    where they have infinities and NaN."""
    a, b = A.cdouble(), B.cdouble()
    return a.real @ b.real - a.imag @ b.imag, a.real @ b.imag + a.imag @ b.real


@pytest.mark.parametrize("precision,m,n,k,batch,options", [
    (FP32, 300, 70, 161, 3, {}), (FP32, 40, 30, 700, 2, {}), (FP32, 70000, 16, 19, 1, {}), (FP32, 20, 600, 9, 1, {}),
    (FP16X3, 640, 500, 161, 1, {}), (FP16X3, 3001, 70, 200, 2, {}), (FP16X3, 40000, 17, 100, 1, {}),
    (FP16X3, 100, 2051, 255, 2, {}), (FP16X3, 640, 500, 161, 1, {"tc_chunk": 1}),
    (TF32X3, 640, 500, 161, 1, {}), (TF32X3, 100, 2051, 255, 2, {}), (BF16X3, 640, 500, 161, 1, {}),
    (BF16X3, 100, 2051, 255, 2, {})])
@pytest.mark.parametrize("case", ["inf_a", "inf_b", "nan_a", "nan_b", "largest", "none"])
def test_infinities_and_nan(built_lib, precision, m, n, k, batch, options, case):
    """Sizes that only a multiply has: infinities stay infinities and reach no
    other element, also next to values that round to infinity in fewer bits."""
    import torch
    A, B = randn((batch, m, k), k), randn((batch, k, n), n)
    if case == "inf_a":
        A[-1, m - 1, k - 1] = complex(float("inf"), 1)
    elif case == "inf_b":
        B[0, 3, n - 2] = complex(2, -float("inf"))
        B[0, 5, n - 2] = complex(-1, -float("inf"))
    elif case == "nan_a":
        A[0, 5, 7] = complex(0, float("nan"))
    elif case == "nan_b":
        B[-1, k - 1, 0] = complex(float("nan"), 0)
    elif case == "largest":
        A[0, 2, 1] = 3.4028234e38
        B *= 2.0 ** -40
    buf = torch.zeros((batch, m * k + k * n + m * n), dtype=torch.complex64, device="cuda")
    buf[:, :m * k] = A.reshape(batch, -1)
    buf[:, m * k:m * k + k * n] = B.reshape(batch, -1)
    torch.cuda.synchronize()
    ctx = Context(0, precision)
    for name, value in options.items():
        ctx.set_option(name, value)
    at = buf.data_ptr()
    for again in range(2):  # a product without them afterwards is not run twice
        ctx.multiply(at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, batch, buf.shape[1])
        ctx.synchronize()
    for a, b, row in zip(A, B, buf):
        c = row[m * k + k * n:].view(m, n)
        for got, want in zip((c.real, c.imag), _parts(a, b)):
            assert torch.equal(got.isnan(), want.isnan())
            assert torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
        good = c.isfinite()
        # 2 k additions of each part at 2^-24, and as for test_block_exponents.
        tol = 2 * k * 2.0 ** -24 * 2 ** 0.5 + 6e-6
        want, bound = (x.nan_to_num(0, 0, 0) for x in (a.to(torch.complex128) @ b.to(torch.complex128),
                                                      a.abs().double() @ b.abs().double()))
        assert float((torch.where(good, c.to(torch.complex128) - want, 0).abs() / (bound + 1e-300))[good].max()) < tol


EDGES = [(300, 1000, 113, 1, 1), (129, 4097, 97, 1, 0), (40000, 130, 97, 1, 1), (4097, 257, 111, 2, 1),
         (128, 1024, 300, 1, 1), (64, 5467, 96, 1, 0), (383, 1500, 130, 1, 0), (640, 1100, 192, 2, 0),
         (257, 640, 257, 1, 1), (8193, 129, 161, 1, 0), (3001, 690, 319, 1, 0)]
# Few columns: 3xFP16, tiles of 32 and 64, with rows on 16 and on 8 bytes.
NARROW = [(65537, 17, 100, 1, 0), (40001, 31, 129, 2, 1), (262144, 16, 96, 1, 0), (20000, 32, 256, 1, 1),
          (70001, 50, 97, 1, 1), (20001, 63, 112, 1, 0), (30000, 64, 97, 2, 1), (16385, 33, 128, 1, 0),
          (100000, 48, 96, 1, 0)]


@pytest.mark.parametrize("precision,m,n,k,batch,extra",
                         [(p, *e) for p in (FP16X3, TF32X3, BF16X3) for e in EDGES] + [(FP16X3, *e) for e in NARROW])
def test_edges(built_lib, precision, m, n, k, batch, extra):
    """Partial tiles, k-steps and blocks, one row into a pair's second half, odd
    sizes and strides, and columns of B of very different size."""
    import torch
    B = randn((batch, k, n), n) * torch.exp2(torch.arange(n, device="cuda") % 41 - 20.0)
    check(precision, randn((batch, m, k), k), B, extra, 8e-6)  # as for test_block_exponents; 3xTF32 chunks of 16


@pytest.mark.parametrize("precision,m,n,k", [
    (p, m, n, k) for p in (FP16X3, TF32X3, BF16X3) for m, n, k in [(1000, 500, 200), (129, 4096, 256)]] + [
    (FP16X3, 60000, 31, 128), (FP16X3, 20000, 60, 97), (FP16X3, 100, 2000, 255)])
def test_wide_ranges(built_lib, precision, m, n, k):
    """Components from 1 down to 2^-60 side by side in a row of A and in a column
    of B. 3xTF32 and BF16x3 keep the bits of each; 3xFP16 counts them from the
    largest of 32 values of A's row (of the row, where A's planes are made
    before the product: m <= 128 with n > 1024) and of B's column."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    A, B = (randn((1, *s), s[0]) * torch.exp2(-torch.randint(0, 61, s, device="cuda", generator=gen))
            for s in ((m, k), (k, n)))
    if precision != FP16X3:
        check(precision, A, B, 0, 8e-6)
        return
    buf = torch.cat([A.reshape(1, -1), B.reshape(1, -1), torch.zeros((1, m * n), dtype=torch.complex64, device="cuda")], 1)
    C = _multiply(precision, buf, m, n, k)[0, m * k + k * n:].view(m, n).cdouble()
    assert not torch.equal(C, _multiply(FP32, buf, m, n, k)[0, m * k + k * n:].view(m, n).cdouble())
    a, b = A[0].cdouble(), B[0].cdouble()

    def largest(x, dim):
        return torch.maximum(x.real.abs(), x.imag.abs()).amax(dim, keepdim=True)
    if m <= 128 and n > 1024:
        top_a = largest(a, 1).expand(m, k)
    else:
        pad = torch.nn.functional.pad(torch.view_as_real(a), (0, 0, 0, -k % 32)).abs().amax(-1)
        top_a = pad.view(m, -1, 32).amax(-1).repeat_interleave(32, -1)[:, :k]
    top_b = largest(b, 0).expand(k, n)
    # A value within 2^-22 of the largest component, each part of a complex one.
    bound = 2.0 ** -22 * 2 ** 0.5 * (top_a @ b.abs() + a.abs() @ top_b) + 8e-6 * (a.abs() @ b.abs())
    assert float(((C - a @ b).abs() / bound).max()) < 1


@pytest.mark.parametrize("precision,m,n,k", [(FP16X3, 640, 500, 161), (BF16X3, 100, 2051, 255), (FP16X3, 65537, 17, 100),
                                             (FP32, 64, 64, 600)])
@pytest.mark.parametrize("how", ["legacy stream", "graph"])
def test_streams(built_lib, precision, m, n, k, how):
    """The legacy stream, and a caller's graph replayed on new operands, with an
    infinity in some of them."""
    import torch
    buf = torch.zeros((1, m * k + k * n + m * n), dtype=torch.complex64, device="cuda")
    at = buf.data_ptr()
    args = (at, at + 8 * m * k, at + 8 * (m * k + k * n), m, n, k, 1, buf.shape[1])
    ctx = Context(0, precision)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    if how == "graph":
        ctx.set_stream(side.cuda_stream)
        with torch.cuda.stream(side):
            ctx.multiply(*args)  # takes the context's buffers
            ctx.synchronize()
            graph.capture_begin()
            ctx.multiply(*args)
            graph.capture_end()
    else:
        ctx.set_stream(0)
    for seed in range(4):
        x = randn((1, m * k + k * n), seed)
        if seed in (1, 2):
            x[0, 3 * k + 5] = complex(float("inf"), 1)
        buf[:, :m * k + k * n] = x
        torch.cuda.synchronize()
        graph.replay() if how == "graph" else ctx.multiply(*args)
        torch.cuda.synchronize()
        ctx.synchronize()
        a, b = x[0, :m * k].view(m, k), x[0, m * k:].view(k, n)
        c = buf[0, m * k + k * n:].view(m, n)
        rows = torch.arange(m, device="cuda") != (3 if seed in (1, 2) else -1)
        want, bound = a[rows].cdouble() @ b.cdouble(), a[rows].abs().double() @ b.abs().double()
        assert float(((c[rows] - want).abs() / bound).max()) < 2 * k * 2.0 ** -24 * 2 ** 0.5 + 6e-6
        for got, part in zip((c.real, c.imag), _parts(a, b)):
            assert torch.equal(got.isnan(), part.isnan()) and torch.equal(got.isposinf(), part.isposinf())


@pytest.mark.parametrize("precision,m,n,k,batch,extra", [
    (TF32X3, 32769, 1024, 32, 1, 1), (TF32X3, 4100, 8192, 32, 1, 0), (TF32X3, 2100, 16384, 32, 2, 1),
    (TF32X3, 16385, 256, 32, 4, 1), (TF32X3, 3000, 4096, 64, 2, 0), (BF16X3, 32769, 1024, 64, 1, 1),
    (BF16X3, 4100, 8192, 64, 1, 0), (BF16X3, 2100, 16384, 64, 2, 1)])
def test_short_sums(built_lib, precision, m, n, k, batch, extra):
    """Products of 32 and 64 terms: real and imaginary parts in MMAs of their own
    where a tile's store bounds it, and pairs for many tiles."""
    check(precision, randn((batch, m, k), m), randn((batch, k, n), n), extra, 8e-6)
