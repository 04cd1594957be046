"""BGPU_INDEPENDENT on the products that make use of it: at most 129 limbs forced
onto the transform, whose forward pass starts under the previous product's carry
scan when the two have the same layout."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import SEED, rand_limbs

pytestmark = pytest.mark.gpu


def run(bb, port, steps):
    """Queue the steps back to back on one stream and check every result.  A step
    is (a, b): limb arrays, or the number of an earlier step for its result; b
    None squares."""
    torch = pytest.importorskip("torch")
    host, dev, queue = [], [], []

    def operand(x):
        if isinstance(x, int):
            return host[x], dev[x]
        return x, torch.from_numpy(x.view(np.int64)).cuda()

    for a, b in steps:
        ha, da = operand(a)
        hb, db = (ha, da) if b is None else operand(b)
        want = port.mul(ha, hb)
        host.append(np.concatenate([want, np.zeros(ha.size + hb.size - want.size, dtype=np.uint64)]))
        dev.append(torch.full((ha.size + hb.size,), -1, dtype=torch.int64, device="cuda"))
        queue.append((da, db, dev[-1]))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(2):
        for da, db, out in queue:
            bb.mul_device(da.data_ptr(), da.numel(), db.data_ptr(), db.numel(), out.data_ptr(),
                          stream=stream.cuda_stream, method=bb.BGPU_METHOD_NTT | bb.BGPU_INDEPENDENT)
        bb.device_status(stream.cuda_stream)
    for k, out in enumerate(dev):
        assert np.array_equal(out.cpu().numpy().view(np.uint64), host[k]), k


def ones(n):
    return np.full(n, 0xFFFFFFFFFFFFFFFF, dtype=np.uint64)


@pytest.mark.parametrize("na,nb", [(1, 1), (8, 9), (40, 24), (64, 65), (128, 1)])
def test_equal_lengths(bb, port, na, nb):
    rng = np.random.default_rng([SEED, na, nb])
    run(bb, port, [(ones(na), ones(nb)) if k % 5 == 0 else (rand_limbs(rng, na), rand_limbs(rng, nb))
                   for k in range(60)])


def test_unequal_lengths_and_squares(bb, port):
    rng = np.random.default_rng(SEED + 51)
    sizes = [(64, 64), (64, 64), (30, 30), (64, 64), (64, None), (64, None), (60, 60), (4, 100), (129 - 64, 64),
             (20, None), (20, 20)]
    run(bb, port, [(rand_limbs(rng, a), None if b is None else rand_limbs(rng, b)) for a, b in sizes * 5])


def test_operand_is_the_previous_result(bb, port):
    rng = np.random.default_rng(SEED + 52)
    steps = []
    for k in range(0, 40, 4):  # 32, 64 and 96 limbs; the same layout as before, and another
        steps += [(rand_limbs(rng, 16), rand_limbs(rng, 16)), (k, ones(32)), (ones(32), k + 1), (k + 1, None)]
    run(bb, port, steps)


def test_wide_digit_products_between(bb, port):
    """The scratch memory and its last user change hands between the two transforms."""
    rng = np.random.default_rng(SEED + 53)
    steps = []
    for k in range(20):
        steps.append((rand_limbs(rng, 60), rand_limbs(rng, 60)))
        if k % 3:
            steps.append((ones(65 + 700 * k), rand_limbs(rng, 65 + k)))
    run(bb, port, steps)
