"""Products under tuned transform splits (set_split, set_batch_split): splits that
only one of the two transforms is built for, and every column and row length of
the wide-digit kernels."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu

M61 = (1 << 61) - 1


@pytest.fixture(scope="module")
def bb():
    import bigint_b200

    bigint_b200.init(0)
    return bigint_b200


@contextlib.contextmanager
def split(bb, log_points, column, batch=False):
    set_ = bb.set_batch_split if batch else bb.set_split
    set_(log_points, column)
    try:
        yield
    finally:
        set_(log_points, 0)


def rand_limbs(rng, n):
    a = rng.integers(0, 2**64, n, dtype=np.uint64)
    a[-1] |= np.uint64(1 << 63)
    return a


def mod61(x):
    return int.from_bytes(np.ascontiguousarray(x).tobytes(), "little") % M61


def run_plan(bb, pairs, flags=0):
    """Results and launch count of a plan of the products (a is b: a square)."""
    import torch

    dev = [(torch.from_numpy(a.view(np.int64)).cuda(), torch.from_numpy(b.view(np.int64)).cuda()) for a, b in pairs]
    out = [torch.full((a.size + b.size,), -1, dtype=torch.int64, device="cuda") for a, b in pairs]
    prods = [(x.data_ptr(), x.numel(), (x if a is b else y).data_ptr(), y.numel(), o.data_ptr())
             for (a, b), (x, y), o in zip(pairs, dev, out)]
    torch.cuda.synchronize()
    plan = bb.BatchPlan(prods, flags=flags)
    plan.run(0)
    bb.device_status(0)
    launches = plan.launches
    plan.close()
    return [o.cpu().numpy().view(np.uint64) for o in out], launches


# a column of 2^8 of 2^23 32-bit digits: 2^15-point rows of three primes, which
# are not built there, and 2^14-point rows of wide digits, which are
def test_split_of_the_wide_transform_alone(bb):
    rng = np.random.default_rng([SEED, 81])
    a, b = rand_limbs(rng, 1 << 21), rand_limbs(rng, 1 << 21)
    with split(bb, 23, 8):
        assert mod61(bb.ntt_mul(a, b)) == mod61(a) * mod61(b) % M61
    with split(bb, 23, 8, batch=True):
        (got,), _ = run_plan(bb, [(a, b)])
        assert mod61(got) == mod61(a) * mod61(b) % M61


def test_batch_split_beyond_the_mixed_launches(bb, port):
    """Several short lengths share their launches, whatever split one has."""
    rng = np.random.default_rng([SEED, 82])
    pairs = [(rand_limbs(rng, n), rand_limbs(rng, m)) for n, m in ((900, 1000), (2000, 1900), (1000, 3000))]
    _, launches = run_plan(bb, pairs)
    with split(bb, 13, 2, batch=True):
        got, n = run_plan(bb, pairs)
    assert n == launches == 4
    for (a, b), c in zip(pairs, got):
        want = port.mul(a, b)
        assert np.array_equal(c[: want.size], want) and not c[want.size :].any()


# every column and row length of the wide-digit kernels, the lazy primes
# (2^13 points and more): columns of all lengths over rows of 2^8 points and
# less, rows of all lengths over the shortest columns, the longest of each
@pytest.mark.parametrize("col,row", [(5, 8), (6, 7), (7, 6), (8, 5), (9, 5), (10, 5), (11, 5), (5, 9), (5, 10), (5, 11),
                                     (5, 12), (5, 13), (5, 14), (8, 14), (11, 11), (9, 13)])
@pytest.mark.parametrize("batch", [False, True])
def test_wide_splits(bb, port, col, row, batch):
    rng = np.random.default_rng([SEED, col, row])
    n = 1 << (col + row)  # limbs of the product: the longest of this many points
    a, b = rand_limbs(rng, n - n // 3), rand_limbs(rng, n // 3)  # more and less than half the points
    c = np.full(n // 2, 0xFFFFFFFFFFFFFFFF, dtype=np.uint64)
    with split(bb, col + row + 1, col, batch):
        assert (bb.get_batch_split if batch else bb.get_split)(col + row + 1) == col
        got = run_plan(bb, [(a, b), (c, c)])[0] if batch else [bb.ntt_mul(a, b), bb.ntt_mul(c)]
    for (x, y), z in zip([(a, b), (c, c)], got):
        assert port.mod_m61(z) == port.mod_m61(x) * port.mod_m61(y) % M61


# six and seven primes on columns of every length: the lazy sets at 2^16 points,
# the strict ones at 2^21 and 2^19, and 2^24 and 2^23, the longest
@pytest.mark.parametrize("quarters,col,log_n", [(q, col, ln) for q, ls in ((5, (16, 21)), (6, (16, 19))) for ln in ls
                                                for col in range(max(5, ln - 14), min(12, ln - 4))]
                         + [(5, 10, 24), (6, 10, 23)])
def test_long_digit_splits(bb, port, quarters, col, log_n):
    rng = np.random.default_rng([SEED, quarters, col, log_n])
    n = quarters << (log_n - 2)  # limbs of the product: the longest in 80 or 96 bits
    a, b = rand_limbs(rng, n - n // 2 + 7), rand_limbs(rng, n // 2 - 7)
    with split(bb, log_n + 1, col):
        got = bb.ntt_mul(a, b), bb.ntt_mul(a[: n // 2])
    assert port.mod_m61(got[0]) == port.mod_m61(a) * port.mod_m61(b) % M61
    assert port.mod_m61(got[1]) == port.mod_m61(a[: n // 2]) ** 2 % M61


# classes of 80- and 96-bit digits (2^16 points of a class together), squares among
# them, on short transforms and on longer ones
@pytest.mark.parametrize("quarters,log_n,count", [(5, 12, 20), (6, 12, 20), (6, 13, 10), (5, 16, 2), (6, 16, 2)])
def test_long_digit_classes(bb, port, quarters, log_n, count):
    rng = np.random.default_rng([SEED, quarters, log_n])
    n = quarters << (log_n - 2)
    pairs = []
    for k in range(count):
        a = rand_limbs(rng, n // 2 - k)
        pairs += [(a, a), (a, rand_limbs(rng, n // 2 - 2 * k))]
    got, launches = run_plan(bb, pairs)
    assert launches == 2 * (2 if log_n <= 12 else 4)  # one class of squares, one of products
    for (a, b), c in zip(pairs, got):
        want = port.mul(a, b)
        assert np.array_equal(c[: want.size], want) and not c[want.size :].any()
