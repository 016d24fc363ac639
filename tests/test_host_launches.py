"""What the library's host code launches, on a CUDA runtime without a GPU."""
from tests.fake_cuda import fake_lib, run_fake  # noqa: F401  (fixtures)


def test_every_kernel_runs_on_every_device(run_fake):  # noqa: F811
    """One process, contexts on two devices: whatever runs on the first runs on
    the second. Limits of dynamic shared memory belong to a device."""
    run_fake('''
fake.fake_devices(2)
products = [(70000, 8, 16), (70000, 16, 16), (70000, 32, 16), (32, 70000, 16), (64, 70000, 16), (70000, 64, 16),
            (70000, 64, 8), (64, 8, 600), (64, 64, 600), (5000, 12, 100), (3000, 200, 128)]
splits = [(128, 128, 32), (4096, 64, 256), (4096, 256, 16), (4096, 256, 256), (65536, 32, 128), (512, 9000, 4096),
          (100, 2048, 64)]
circuit, grid, ordering = rqc.random_circuit(3, 3, 8, seed=1), rqc.grid_text(3, 3), rqc.row_sweep_ordering(3, 3)
seen = []
for device in (0, 1):
    for precision in (FP32, TF32X3, FP16X3, BF16X3):
        ctx = Context(device, precision)
        for m, n, k in products if precision == FP32 else splits:
            ctx.multiply(A, B, C, m, n, k)
            ctx.multiply(A, B, C, m, n, k, 3, 1 << 30)
        ctx.evaluate(circuit, ordering, grid, "0" * 9, "1" * 9, 1 << 40)
        if precision not in (FP32, TF32X3):
            ctx.set_option("exact_gates", 0)
            ctx.evaluate(circuit, ordering, grid, "0" * 9, "1" * 9, 1 << 40)
        if precision != FP32:
            for variant in range(1, 5):
                ctx.set_option("tc_variant", variant)
                ctx.multiply(A, B, C, 4096, 256, 256)
    seen.append(kernels())
assert seen[0] == seen[1] and len(set(seen[0])) > 20, (len(seen[0]), len(seen[1]))
''')


def test_multiply_without_room_for_planes(run_fake):  # noqa: F811
    """A multiply of sizes that no contraction has takes its planes' memory
    when it can be had; otherwise fewer entries at a time, and FP32 when those
    of one entry find no room. Free memory that comes in no large enough piece
    is no error, and neither is what follows."""
    run_fake('''
m, n, k, batch = 1000, 700, 1100, 6
entry = 4 * (2 * n * 1104 + 2 * n)  # planes, scales and largest components of B
for limit in (fake.fake_largest_block, fake.fake_memory):
    for room, piece in ((1 << 40, 6), (6 * entry, 6), (3 * entry, 3), (entry, 1), (entry - (1 << 16), 0), (1 << 20, 0)):
        ctx = Context(0, FP16X3)
        ctx.multiply(A, B, C, 4, 4, 4)  # the context's FP32 scratch and control block exist
        ctx.multiply(A, B, C, 64, 64, 16)
        log()
        limit(room)
        ctx.multiply(A, B, C, m, n, k, batch, 1 << 30)
        names = kernels()
        direct = [x for x in names if x.startswith("cgemm_direct_kernel")]
        fp32 = [x for x in names if x.startswith("cgemm_kernel")]
        # One FP32 launch: the product, or what runs only if sums were not finite.
        assert (len(direct), len(fp32)) == (-(-batch // piece) if piece else 0, 1), (room, names)
        ctx.multiply(A, B, C, 70000, 64, 5)
        ctx.synchronize()
        limit(1 << 40)
        # Sizes of contractions have no other way.
        limit(1 << 16)
        try:
            ctx.multiply(A, B, C, 4096, 4096, 4096)
            raise SystemExit("no error")
        except QflexGb300Error as e:
            assert e.code == 2 and "out of memory" in str(e), str(e)
        limit(1 << 40)
        ctx.multiply(A, B, C, 4096, 4096, 4096)
        assert kernels()[-1].startswith("cgemm_direct_kernel")
        ctx.close()
''')


def test_one_kernel_or_separate_kernels(run_fake):  # noqa: F811
    """Which form a small program takes depends on the strings of a call and on
    its gate chains: separate kernels where one SM would be the slower (each of
    these was measured in both forms)."""
    run_fake('''
from qflex_gb300 import FP16X3, FP32
for (rows, cols, depth), precision, strings, one in [
        ((4, 5, 16), FP32, 1, True), ((4, 5, 16), FP16X3, 1, True), ((4, 5, 16), FP32, 152, True),
        ((4, 5, 16), FP32, 4096, False), ((4, 5, 16), FP16X3, 1024, False), ((2, 3, 32), FP32, 1, False),
        ((2, 3, 32), FP16X3, 1, False), ((2, 3, 32), FP16X3, 32, False), ((2, 3, 32), FP16X3, 152, True),
        ((2, 3, 32), FP32, 4096, True), ((3, 3, 21), FP16X3, 1, False), ((3, 3, 21), FP16X3, 304, True),
        ((3, 3, 12), FP16X3, 152, True), ((3, 3, 12), FP16X3, 4096, False), ((5, 5, 8), FP32, 4096, True)]:
    net = (rqc.random_circuit(rows, cols, depth, seed=depth), rqc.row_sweep_ordering(rows, cols), rqc.grid_text(rows, cols))
    ctx = Context(0, precision)
    log()
    ctx.evaluate_many(*net, "0" * (rows * cols), ["0" * (rows * cols)] * strings, 1 << 40)
    assert (ctx.stats()["launches"] == 1) == one, (rows, cols, depth, precision, strings)
    # Passes of one string at a time are calls of one string.
    if strings > 1:
        ctx.set_option("max_batch", 1)
        ctx.evaluate_many(*net, "0" * (rows * cols), ["0" * (rows * cols)] * 3, 1 << 40)
        single = ctx.stats()["launches"] == 3
        ctx.set_option("max_batch", 0)
        ctx.evaluate_many(*net, "0" * (rows * cols), ["0" * (rows * cols)], 1 << 40)
        assert (ctx.stats()["launches"] == 1) == single
''')


def test_launch_count(run_fake):  # noqa: F811
    """stats()["launches"] is the number of kernels an evaluation launches, also
    where FP32 products sum k in runs, added up by a second kernel."""
    run_fake('''
runs = 0
nets = [(4, 4, 16), (4, 5, 16), (4, 4, 24), (5, 5, 16)]
nets = [(rqc.random_circuit(r, c, d, seed=3), rqc.row_sweep_ordering(r, c), rqc.grid_text(r, c), r * c) for r, c, d in nets]
nets.append((rqc.random_circuit(6, 6, 24, seed=0), rqc.ordering_6x6(cut_values=(1,)), rqc.grid_text(6, 6), 36))
nets.append((rqc.random_circuit(7, 7, 32, seed=0), rqc.ordering_7x7((0,), (1,)), rqc.grid_text(7, 7), 49))
# Patches that share four bonds of dimension 4 and keep others: (4, 64, 256).
merge = [f"expand a {q}" for q in range(5)] + [f"expand b {q}" for q in (5, 6, 7)] + ["merge a b"]
nets.append((rqc.random_circuit(4, 4, 16, seed=3), "\\n".join(merge + [f"expand b {q}" for q in range(8, 16)]) + "\\n",
             rqc.grid_text(4, 4), 16))
fake.fake_memory(1 << 45)
for circuit, ordering, grid, qubits in nets:
    for precision in (FP32, TF32X3, FP16X3, BF16X3, FP64):
        for strings in (1, 2):
            ctx = Context(0, precision)
            ctx.set_profiling(True)  # operation by operation
            log()
            ctx.evaluate_many(circuit, ordering, grid, "0" * qubits, ["0" * qubits] * strings, float(1 << 50))
            names = kernels()
            runs += sum(x.startswith("split_finish_kernel") for x in names)
            assert len(names) == ctx.stats()["launches"], (qubits, precision, strings, len(names), ctx.stats())
            ctx.close()
assert runs > 4, runs
''')


def test_buffers_across_streams(run_fake):  # noqa: F811
    """A product that uses the context's buffers (planes, runs of k) on another
    stream than the one before it waits for that one; products that use none run
    side by side, and a captured product waits for nothing outside its graph."""
    run_fake('''
def steps():
    return [(w[0], x.split("stream=")[1].split()[0]) for x in log() for w in [x.split()]
            if w[0] in ("launch", "wait", "record")]
for precision, size in ((FP32, (64, 64, 600)), (FP32, (1, 4, 9000)), (FP16X3, (4096, 256, 256)), (BF16X3, (640, 700, 200))):
    ctx = Context(0, precision)
    ctx.multiply(A, B, C, *size)
    assert not [s for s in steps() if s[0] != "launch"]  # the context's own stream
    ctx.set_stream(0x10)
    last = None
    for stream in ("0x10", "0x20", "0x20", "0x10"):
        ctx.set_stream(int(stream, 16))
        ctx.multiply(A, B, C, *size)
        got = steps()
        assert {s for _, s in got} == {stream} and got[-1][0] == "record", got
        assert [w for w, _ in got].count("wait") == (last not in (None, stream)), (precision, size, got)
        assert last in (None, stream) or got[0][0] == "wait", got
        last = stream
    ctx.set_stream(0x30)
    plain = Context(0, FP32)
    for stream in (0x10, 0x20):
        plain.set_stream(stream)
        plain.multiply(A, B, C, 70000, 64, 16)
        assert [w for w, _ in steps()] == ["launch"]
    # 0x30 is being captured.
    fake.fake_capturing(0x30, 1)
    ctx.multiply(A, B, C, *size)
    assert all(w == "launch" for w, _ in steps())
    fake.fake_capturing(0x30, 0)
''')


def test_fp32_tiles_per_block(run_fake):  # noqa: F811
    """Which FP32 products run one tile per block: those measured slower in
    persistent blocks (rounds of tiles that fill half the chip, rows on 8
    bytes), and none of the sizes that contractions have beside them."""
    from tests.test_gpu_staged import STAGED
    run_fake(f"staged = {STAGED!r}" + '''
persistent = [(2048, 2048, 2048, 1), (32768, 64, 64, 16), (1024, 1024, 1024, 4), (157583, 13, 9, 7), (40000, 40, 10, 1),
              (65536, 16, 512, 1), (10143, 11, 585, 4), (5000, 200, 300, 1), (1048576, 16, 16, 1), (300, 30, 700, 1)]
ctx = Context(0, FP32)
for product in staged + persistent:
    ctx.multiply(A, B, C, *product[:4], 1 << 30)
    name = kernels()[0]
    assert name.startswith("cgemm_staged_kernel" if product in staged else "cgemm_kernel"), (product, name)
''')


def test_small_permutations_move_short_runs(run_fake):  # noqa: F811
    """Runs of at most four elements up to 2^17, where longer ones leave too few
    threads; the schedules on either side of the line are right."""
    run_fake('''
import numpy as np
ctx = Context(0, FP32)
for dims, order in [((25, 5, 24, 4), (0, 2, 3, 1)), ((16, 24, 26), (1, 2, 0)), ((3, 3, 2, 5, 2, 5, 4, 4), (7, 5, 2, 0, 4, 1, 6, 3)),
                    ((8, 16, 1023), (2, 1, 0)), ((131071,), (0,)), ((1025, 128), (1, 0)), ((7, 18725), (1, 0)),
                    ((13, 9, 16, 71), (3, 1, 0, 2)), ((71, 13, 9, 16), (1, 3, 0, 2))]:
    ctx.permute(A, B, dims, order)
    name = kernels()[0]
    run = int(name.split("<")[1].split(",")[0])
    size = int(np.prod(dims))
    assert name.startswith("permute_runs_kernel") and (run <= 4 if size <= 1 << 17 else run in (1, 8, 16)), (dims, name)
    x = np.arange(size).astype(np.complex64)
    assert np.array_equal(_lib.check_permute(x, dims, order), x.reshape(dims).transpose(order).reshape(-1)), dims
''')


def test_products_of_a_split_precision(run_fake):  # noqa: F811
    """Which products of a split-precision context run on the tensor cores, and
    in which tiles."""
    from tests.test_gpu_split_routes import EDGES, NARROW
    run_fake(f"edges, narrow = {EDGES!r}, {NARROW!r}" + '''
kinds = {FP16X3: 1, TF32X3: 0, BF16X3: 2}
for precision, kind in kinds.items():
    ctx = Context(0, precision)
    def direct(m, n, k, batch=1, extra=0):
        ctx.multiply(A, B, C, m, n, k, batch, 1 << 30)
        return [x for x in kernels() if x.startswith(("cgemm_direct", "cgemm_tf32", "cgemm_fp16", "cgemm_bf16"))]
    for e in edges:
        m, n = e[:2]
        name, = direct(*e)
        if precision == BF16X3 and m <= 128 or m <= 128 and n > 1024:
            assert not name.startswith("cgemm_direct"), (e, name)
        else:
            columns = 128 if n > 64 or kind != 1 else 64 if n > 32 else 32
            assert name.startswith(f"cgemm_direct_kernel<{kind}, {columns},"), (e, name)
            assert name.endswith("true>") == (m > 128 and e[2] > {1: 128, 0: 64, 2: 0}[kind] and columns == 128), (e, name)
    for e in narrow:
        names = direct(*e)
        if precision == FP16X3:
            assert len(names) == 1 and names[0].startswith(f"cgemm_direct_kernel<1, {32 if e[1] <= 32 else 64}, false>"), (e, names)
        else:
            assert bool(names) == (e[1] == 64), (e, names)
    # Below 2^25 terms in all, or 96 a sum, FP32 kernels.
    for m, n, k in [(64, 5461, 96), (40000, 130, 95), (257, 640, 161), (300, 130, 97), (262144, 15, 96), (255, 50, 4000)]:
        assert not direct(m, n, k), (precision, m, n, k)
    assert direct(64, 64, 16) and direct(128, 128, 32)  # sizes of contractions
''')


def test_kernels_of_an_evaluation(run_fake):  # noqa: F811
    """The 3xFP16 products of one 7x7 slice: at the default choices they split A
    themselves and no permutation writes planes; in chunks of one k-step, or at
    another kernel choice, permutations write planes and the product loads them."""
    run_fake('''
net = (rqc.random_circuit(7, 7, 32, seed=0), rqc.ordering_7x7((0,), (1,)), rqc.grid_text(7, 7), "0" * 49, ["0" * 49])
for option, kernel in ((None, "cgemm_direct_kernel<1,"), (("tc_chunk", 1), "cgemm_fp16x3_kernel"),
                       (("tc_variant", 1), "cgemm_fp16x3_pair_kernel"), (("tc_variant", 2), "cgemm_fp16x3_deep_kernel"),
                       (("tc_variant", 3), "cgemm_fp16x3_wide_kernel"), (("tc_variant", 4), "cgemm_fp16x3_narrow_kernel")):
    ctx = Context(0, FP16X3)
    if option:
        ctx.set_option(*option)
    log()
    ctx.evaluate_many(*net, float(1 << 50))
    names = kernels()
    writing = [x for x in names if x.startswith("permute_kernel<float2, true>")]
    assert [x for x in names if x.startswith(kernel)], (option, set(names))
    assert bool(writing) == (option is not None), (option, len(writing))
    assert option is None or not [x for x in names if x.startswith("cgemm_direct")], option
''')


def test_products_of_few_terms(run_fake):  # noqa: F811
    """Which kernel 3xTF32 and BF16x3 products of 16 to 64 terms take (each line
    measured on both sides)."""
    run_fake('''
for precision, (m, n, k, batch), want in [
        (TF32X3, (16384, 4096, 32, 1), "cgemm_tf32x3_separate_kernel"), (TF32X3, (32769, 1024, 32, 1), "cgemm_tf32x3_separate_kernel"),
        (TF32X3, (65536, 512, 32, 1), "cgemm_direct_kernel<0, 128, true>"), (TF32X3, (16384, 256, 32, 4), "cgemm_direct_kernel<0, 128, true>"),
        (TF32X3, (16384, 8192, 64, 1), "cgemm_direct_kernel<0, 128, true>"), (TF32X3, (16384, 8192, 16, 1), "cgemm_direct_kernel<0, 128, false>"),
        (TF32X3, (512, 512, 64, 1), "cgemm_direct_kernel<0, 128, false>"), (TF32X3, (65536, 64, 64, 4), "cgemm_direct_kernel<0, 128, false>"),
        (TF32X3, (512, 512, 128, 1), "cgemm_direct_kernel<0, 128, true>"), (BF16X3, (16384, 4096, 64, 1), "cgemm_bf16x3_separate_kernel"),
        (BF16X3, (65536, 512, 64, 1), "cgemm_direct_kernel<2, 128, true>"), (BF16X3, (16384, 4096, 32, 1), "cgemm_direct_kernel<2, 128, true>"),
        (BF16X3, (16384, 4096, 128, 1), "cgemm_direct_kernel<2, 128, true>"), (BF16X3, (2048, 2048, 64, 1), "cgemm_direct_kernel<2, 128, true>")]:
    ctx = Context(0, precision)
    ctx.multiply(A, B, C, m, n, k, batch, 1 << 31)
    names = kernels()
    assert names[-1].startswith(want), (precision, m, n, k, batch, names)
    ctx.close()
''')
