"""Products of vectors in contractions that run as one kernel."""
import pytest

from qflex_gb300 import FP16X3, FP32, Context, rqc

pytestmark = pytest.mark.gpu


def _two_patches(rows, cols, first, merge, late):
    """Rows 0 .. first - 1 into patch a, the others into b, merged at the end
    or (late) before the last rows."""
    sites = [[i * cols + j for j in range(cols)] for i in range(rows)]
    into = merge.split()[-1]
    lines = [f"expand a {q}" for row in sites[:first] for q in row]
    rest = sites[first:]
    b = rest[:1] if late else rest
    lines += [f"expand b {q}" for row in b for q in row] + [merge]
    return "\n".join(lines + [f"expand {into} {q}" for row in rest[len(b):] for q in row]) + "\n"


@pytest.mark.parametrize("precision", [FP32, FP16X3], ids=["fp32", "fp16x3"])
@pytest.mark.parametrize("rows,cols,first,merge,late,shape", [
    (3, 3, 1, "merge a b", False, (64, 1, 16)), (3, 3, 2, "merge a b", False, (1, 1, 64)),
    (3, 3, 1, "merge a b", True, (1, 64, 64)), (3, 3, 1, "merge b a", True, (64, 1, 64)),
    (4, 3, 2, "merge a b", True, (1, 64, 64)), (4, 4, 3, "merge a b", False, (1, 1, 256))])
def test_vector_products_sum_as_separate_kernels_do(built_lib, precision, rows, cols, first, merge, late, shape):
    """Bit for bit the amplitudes of the same program run operation by
    operation, whose vector products sum by lanes (the other products of these
    programs have fewer than 192 terms and sum them in one order)."""
    circuit, grid = rqc.random_circuit(rows, cols, 16, seed=16), rqc.grid_text(rows, cols)
    ordering = _two_patches(rows, cols, first, merge, late)
    initial, *finals = rqc.random_bitstrings(rows * cols, 9, 3)
    one, ops = Context(0, precision), Context(0, precision)
    ops.set_profiling(True)
    got = one.evaluate_many(circuit, ordering, grid, initial, finals, 1 << 40)
    want = ops.evaluate_many(circuit, ordering, grid, initial, finals, 1 << 40)
    assert one.stats()["launches"] == 1 < ops.stats()["launches"]
    shapes = [tuple(s[:3]) for s in one.shapes()]
    assert shape in shapes and all(k < 192 for m, n, k in shapes if m > 1 and n > 1)
    assert got == want
