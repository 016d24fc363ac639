"""3xFP16 evaluations whose products load both operands' planes (chunks of one
k-step, or a kernel choice other than 0): permutations write A's planes for the
product that follows."""
import numpy as np
import pytest

from qflex_gb300 import FP16X3, Context, rqc
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


def _cases():
    circuit, ordering, grid, initial, finals = rqc.workload("c2")
    yield circuit, ordering, grid, initial, finals[:2]
    yield (rqc.random_circuit(7, 7, 32, seed=0), rqc.ordering_7x7((0,), (1,)), rqc.grid_text(7, 7), "",
           rqc.random_bitstrings(49, 2, 5))


@pytest.fixture(scope="module")
def cases(built_lib):
    """The networks and their amplitudes by the complex128 oracle."""
    from oracle import qflex_oracle as qo
    out = []
    for circuit, ordering, grid, initial, finals in _cases():
        inp = [qo.Input(qo.Circuit.loads(circuit), qo.load_ordering(ordering), qo.Grid.loads(grid), initial, f) for f in finals]
        out.append((circuit, ordering, grid, initial, finals,
                    [qo.evaluate_circuit(i, np.complex128, float(1 << 40))[0][1] for i in inp]))
    return out


@pytest.mark.parametrize("option", [("tc_chunk", 1), ("tc_variant", 1), ("tc_variant", 2), ("tc_variant", 3),
                                    ("tc_variant", 4)], ids=lambda o: f"{o[0]}_{o[1]}")
def test_permutations_write_planes(cases, option):
    """Planes written by permutations (scaled per 32 values of a row) against
    planes split from permuted operands (scaled per row), and both against the
    complex128 oracle; fewer kernels are launched where permutations write them."""
    for circuit, ordering, grid, initial, finals, want in cases:
        got = []
        for fuse in (1, 0):
            ctx = Context(0, FP16X3)
            ctx.set_option(*option)
            ctx.set_option("fuse_splits", fuse)
            ctx.set_profiling(True)  # every launch counts, none in a graph
            got.append([x for _, x in ctx.evaluate_many(circuit, ordering, grid, initial, finals, 1 << 40)])
            got.append(ctx.stats()["launches"])
        written, few, split, many = got
        assert few < many
        assert rel_err(written, want) < 1e-5 and rel_err(split, want) < 1e-5
