"""Products that read A through a permutation: their copies and block reads,
run on host buffers, against numpy's transpose of the same array."""
import random

import numpy as np
import pytest

from qflex_gb300._lib import check_gather


def _source(size):
    return (np.arange(size) + 1j * np.arange(size)).astype(np.complex64)


@pytest.mark.parametrize("seed", range(40))
def test_gather_matches_transpose(built_lib, seed):
    """Index orders of tensors with index dimensions 2..32: accepted exactly
    when the source's three lowest digits belong to the operand's seven lowest
    row digits or five lowest value digits, and then equal to the transpose."""
    rng = random.Random(seed)
    accepted = 0
    for _ in range(40):
        lg = [rng.randint(1, 5) for _ in range(rng.randint(2, 7))]
        if not 11 <= sum(lg) <= 17:
            continue
        order = list(range(len(lg)))
        rng.shuffle(order)
        if rng.random() < 0.3:
            order.sort()
        kl = rng.randint(4, sum(lg) - 7)
        # Digits of the operand, least significant first, as source digits.
        start = [sum(lg[i + 1:]) for i in range(len(lg))]
        digits = [start[i] + b for i in reversed(order) for b in range(lg[i])]
        block = set(digits[:min(kl, 5)]) | set(digits[kl:kl + 7])
        src = _source(1 << sum(lg))
        got = check_gather(src, [1 << x for x in lg], order, 1 << (sum(lg) - kl))
        assert (got is not None) == ({0, 1, 2} <= block)
        if got is not None:
            accepted += 1
            want = src.reshape([1 << x for x in lg]).transpose(order).reshape(got.shape)
            assert np.array_equal(got, want)
    assert accepted


def test_gather_refuses_what_no_block_holds(built_lib):
    src = _source(1 << 12)
    assert check_gather(src, [64, 64], [1, 0], 64) is None           # fewer than 128 rows
    assert check_gather(src, [512, 8], [1, 0], 512) is None          # rows of 8 values
    assert check_gather(src, [16, 16, 16], [0, 1, 2], 256) is not None


@pytest.mark.parametrize("n", [8, 16, 32, 64, 256])
@pytest.mark.parametrize("seed", range(8))
def test_tile_gather_matches_transpose(built_lib, seed, n):
    """The same for the tiled CUDA-core products, whose tile depends on the
    product's columns, rows and terms."""
    rng = random.Random(1000 * n + seed)
    accepted = 0
    for _ in range(60):
        lg = [rng.randint(1, 5) for _ in range(rng.randint(2, 7))]
        if not 8 <= sum(lg) <= 17:
            continue
        order = list(range(len(lg)))
        rng.shuffle(order)
        if rng.random() < 0.3:
            order.sort()
        src = _source(1 << sum(lg))
        kl = rng.randint(2, sum(lg) - 3)
        got = check_gather(src, [1 << x for x in lg], order, 1 << (sum(lg) - kl), n)
        if got is not None:
            accepted += 1
            want = src.reshape([1 << x for x in lg]).transpose(order).reshape(got.shape)
            assert np.array_equal(got, want)
    assert accepted
