"""Launch counts of the calls that queue several products: a wide-digit product
of up to 2^12 points is two launches, a longer one four, whoever queues it."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bb():
    import bigint_b200

    bigint_b200.init(0)
    return bigint_b200


def rand_limbs(rng, n):
    a = rng.integers(0, 2**64, n, dtype=np.uint64)
    a[-1] |= np.uint64(1 << 63)
    return a


def tree_launches(bb, leaves):
    bb.product_tree(np.full(leaves, 3, dtype=np.uint64))
    return bb.last_launch_count()


def test_tree_levels(bb):
    """A tree of twice the leaves has one more level, of width w = leaves."""
    for leaves in (256, 1024, 2048):  # 2 w limbs are 2^9, 2^11, 2^12 points
        assert tree_launches(bb, 2 * leaves) - tree_launches(bb, leaves) == 2, leaves
    for leaves in (4096, 8192):
        assert tree_launches(bb, 2 * leaves) - tree_launches(bb, leaves) == 4, leaves


def test_tree_level_in_pieces(bb):
    """A level of more than 2^14 transform products takes its launches again for
    each 2^14: from 129 limbs the levels of 2^23 leaves have 2^15, 2^14, ... products."""
    small, large = (tree_launches(bb, n) for n in (1 << 21, 1 << 23))
    # two more levels, of 2^21 and 2^22 limbs; the level of 128 limbs has 2^13 and
    # 2^15 products, on the wide-digit transform from 193 limbs of product on
    assert large - small == 2 * 4 + 2


@pytest.mark.parametrize("n,one", [(300, 2), (2048, 2), (2049, 4), (20000, 4)])
def test_products_of_a_list(bb, n, one):
    rng = np.random.default_rng([SEED, n])
    a, b = rand_limbs(rng, n), rand_limbs(rng, n)
    bb.ntt_mul(a, b)
    assert bb.last_launch_count() == one
    outs = [np.zeros(2 * n, dtype=np.uint64) for _ in range(3)]
    bb.mul_many([(a, b)] * 3, outs)
    assert bb.last_launch_count() == 3 * one


def test_power(bb):
    """x^2 is one product; x^3 a square and a product."""
    rng = np.random.default_rng(SEED + 9)
    x = rand_limbs(rng, 400)
    bb.fast_pow(x, 2)
    assert bb.last_launch_count() == 2
    bb.fast_pow(x, 3)
    assert bb.last_launch_count() == 4


def test_blocks_beyond_one_transform(bb):
    """Two blocks of one operand against one of the other: three spectra of two
    launches, and two sums of three, the second with the merge."""
    rng = np.random.default_rng(SEED + 10)
    a, b = rand_limbs(rng, 512), rand_limbs(rng, 256)
    bb.set_block_limbs(256)
    try:
        bb.mul(a, b)
        assert bb.last_launch_count() == 3 * 2 + 2 * 3 + 1
    finally:
        bb.set_block_limbs(0)


def test_kernel_times_are_of_one_kind(bb):
    """Times of products with other kernels are not averaged in."""
    rng = np.random.default_rng(SEED + 11)
    short, long = rand_limbs(rng, 500), rand_limbs(rng, 5000)
    bb.set_kernel_timing(True)
    try:
        for _ in range(3):
            bb.ntt_mul(long, long[:4000])
        for _ in range(2):
            bb.ntt_mul(short, short[:400])
        times, n = bb.kernel_times()
        assert n == 2 and [k for k, _ in times] == ["k_wide_short", "none", "none", "k_wide_carry"]
    finally:
        bb.set_kernel_timing(False)
