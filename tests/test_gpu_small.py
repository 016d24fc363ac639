"""Contractions that run as one kernel (tensors in shared memory) against the
same programs run operation by operation (profiling on)."""
import numpy as np
import pytest

from qflex_gb300 import BF16X3, FP16X3, FP32, Context, rqc
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu

# Both add the same products in FP32; only vector products and the order of a
# warp's partial sums differ, a few roundings of 2^-24 in sums of up to 1024.
TOL = 2e-6


def _cases():
    for I, J, depth in [(2, 3, 8), (3, 3, 12), (4, 4, 16), (4, 5, 16), (3, 5, 10), (5, 5, 11)]:
        yield I, J, depth, rqc.row_sweep_ordering(I, J)
    lines = rqc.row_sweep_ordering(4, 4).splitlines()
    # A bond cut summed over all its values, and two open output qubits.
    yield 4, 4, 16, "\n".join(["cut () 5 6"] + lines) + "\n"
    yield 4, 4, 16, "\n".join(lines[:8] + ["cut () 14", "cut () 15"] + ["merge a b"] +
                              [ln.replace(" a ", " b ") for ln in lines[8:]]) + "\n"


@pytest.mark.parametrize("precision", [FP32, FP16X3, BF16X3], ids=["fp32", "fp16x3", "bf16x3"])
@pytest.mark.parametrize("case", list(_cases()), ids=lambda c: f"{c[0]}x{c[1]}_d{c[2]}_{c[3][:3]}_{len(c[3])}")
def test_one_kernel_matches_operations(built_lib, case, precision):
    I, J, depth, ordering = case
    circuit, grid = rqc.random_circuit(I, J, depth, seed=depth), rqc.grid_text(I, J)
    initial, *finals = rqc.random_bitstrings(I * J, 6, 3)
    if "cut () 14" in ordering:
        finals = [f[:14] + "xx" for f in finals]
    one, ops = Context(0, precision), Context(0, precision)
    ops.set_profiling(True)
    for strings in (finals, finals[:1]):
        got = one.evaluate_many(circuit, ordering, grid, initial, strings, 1 << 40)
        want = ops.evaluate_many(circuit, ordering, grid, initial, strings, 1 << 40)
        assert [s for s, _ in got] == [s for s, _ in want]
        assert rel_err([a for _, a in got], [a for _, a in want]) < TOL
        assert one.stats()["launches"] < ops.stats()["launches"] or one.stats()["n_ops"] > 200
    # Limited passes give the same amplitudes.
    one.set_option("max_batch", 2)
    again = one.evaluate_many(circuit, ordering, grid, initial, finals, 1 << 40)
    assert np.array_equal([a for _, a in again], [a for _, a in one.evaluate_many(
        circuit, ordering, grid, initial, finals, 1 << 40)])
