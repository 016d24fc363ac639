"""The run schedule of permutations with dimensions that are not powers of
two, on host buffers, over random ranks, dimensions and orders."""
import random

import numpy as np
import pytest

from qflex_gb300._lib import check_permute


@pytest.mark.parametrize("seed", range(30))
def test_runs_match_transpose(built_lib, seed):
    rng = random.Random(seed)
    for _ in range(25):
        rank = rng.randint(1, 7)
        while True:
            top = rng.choice([3, 7, 20, 60, 300])
            dims = [rng.randint(1, top) for _ in range(rank)]
            if np.prod(dims) <= 1 << 16:
                break
        dims[rng.randrange(rank)] = rng.choice([3, 5, 15, 17, 31, 33])  # not all powers of two
        order = list(range(rank))
        if rng.random() < 0.8:
            rng.shuffle(order)
        a = np.arange(np.prod(dims)).astype(np.complex64)
        assert np.array_equal(check_permute(a, dims, order), a.reshape(dims).transpose(order).reshape(-1)), (dims, order)
