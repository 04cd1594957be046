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
