"""Wide-digit products (64-, 80- and 96-bit digits) at the edges of their
dispatch: lengths around the longest product of each transform, operands longer than half the transform, long runs of
propagating carries, unaligned buffers, 28-bit Digits, both prime sets."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu

ONES = np.uint64(0xFFFFFFFFFFFFFFFF)
M61 = (1 << 61) - 1


def rand_limbs(rng, n):
    a = rng.integers(0, 2**64, n, dtype=np.uint64)
    a[-1] |= np.uint64(1 << 63)
    return a


def mod61(x):
    return int.from_bytes(np.ascontiguousarray(x).tobytes(), "little") % M61


@pytest.fixture(scope="module")
def bb():
    import bigint_b200

    bigint_b200.init(0)
    return bigint_b200


# total limbs around 2^k + 1 (the longest product of a 2^k-point transform) and
# around the shortest transform; the long operand of the second pair fills more
# than half of the points
@pytest.mark.parametrize("log_n", [9, 10, 11, 13, 14, 16, 18])
@pytest.mark.parametrize("extra", [0, 1, 2])
def test_length_edges(bb, port, log_n, extra):
    rng = np.random.default_rng([SEED, log_n, extra])
    total = (1 << log_n) + extra
    for na in (total // 2, total - 5, total - total // 3):
        a, b = rand_limbs(rng, na), rand_limbs(rng, total - na)
        assert np.array_equal(bb.ntt_mul(a, b), port.mul(a, b)), (na, total - na)
    a = rand_limbs(rng, total // 2)
    assert np.array_equal(bb.ntt_mul(a), port.mul(a, a))


# the same around the longest products of 2^k 80-bit digits (5/4 2^k limbs) and
# 96-bit digits (6/4 2^k limbs), with the digits' odd half words and last partial digit
@pytest.mark.parametrize("quarters", [5, 6])
@pytest.mark.parametrize("log_n", [15, 16, 17, 18, 19])
def test_digit_width_edges(bb, port, quarters, log_n):
    rng = np.random.default_rng([SEED, quarters, log_n])
    for extra in (-1, 0, 1):
        total = (quarters << (log_n - 2)) + extra
        for na in (total // 2, total - 5, total - total // 3):
            a, b = rand_limbs(rng, na), rand_limbs(rng, total - na)
            assert np.array_equal(bb.ntt_mul(a, b), port.mul(a, b)), (na, total - na)
        a = rand_limbs(rng, total // 2)
        assert np.array_equal(bb.ntt_mul(a), port.mul(a, a))


@pytest.mark.parametrize("n", [600, 750, 1500, 70000, 80000])
def test_propagating_carries(bb, port, n):
    """Products whose chunks all propagate a carry or stop it only at the ends."""
    ones = np.full(n, ONES)
    one = np.array([1], dtype=np.uint64)
    assert np.array_equal(bb.ntt_mul(ones, one), ones)
    assert np.array_equal(bb.ntt_mul(ones), port.mul(ones, ones))
    a = np.full(n, ONES)
    a[0] = 1  # (B^n - B + 1)(B^(n/2) + 1): runs of ones met by a carry
    b = np.zeros(n // 2 + 1, dtype=np.uint64)
    b[0] = b[-1] = 1
    assert np.array_equal(bb.ntt_mul(a, b), port.mul(a, b))


def test_unaligned_device_buffers(bb, port):
    import torch

    rng = np.random.default_rng(SEED + 3)
    a, b = rand_limbs(rng, 3001), rand_limbs(rng, 1777)
    ta = torch.zeros(3002, dtype=torch.int64, device="cuda")
    tb = torch.zeros(1778, dtype=torch.int64, device="cuda")
    out = torch.full((3001 + 1777 + 2,), -1, dtype=torch.int64, device="cuda")
    ta[1:] = torch.from_numpy(a.view(np.int64))
    tb[1:] = torch.from_numpy(b.view(np.int64))
    st = torch.cuda.current_stream().cuda_stream
    bb.mul_device(ta.data_ptr() + 8, a.size, tb.data_ptr() + 8, b.size, out.data_ptr() + 8, st)
    bb.device_status(st)
    got = out.cpu().numpy().view(np.uint64)
    want = port.mul(a, b)
    assert np.array_equal(got[1 : 1 + want.size], want)
    assert got[0] == ONES and got[-1] == ONES  # nothing written outside the product


@pytest.mark.parametrize("na,nb", [(2500, 2300), (40000, 37450), (150000, 20000), (131073, 131071),
                                   (2900, 2900), (3500, 3500), (330000, 310000), (400000, 380000)])
def test_digits28(bb, port, na, nb):
    rng = np.random.default_rng([SEED, na])
    a = rng.integers(0, 1 << 28, na).astype(np.uint32)
    b = rng.integers(0, 1 << 28, nb).astype(np.uint32)
    a[-1] |= 1 << 27
    b[-1] |= 1
    assert np.array_equal(bb.mul_digits(a, b), port.mul_digits(a, b))
    full = np.full(na, (1 << 28) - 1, dtype=np.uint32)
    assert np.array_equal(bb.mul_digits(full, b), port.mul_digits(full, b))


@pytest.mark.parametrize("log_n", [22, 23, 24])
def test_large_residue(bb, log_n):
    """The longest lazy transform and the shorter strict ones, modulo 2^61 - 1."""
    rng = np.random.default_rng([SEED, log_n, 61])
    total = 1 << log_n
    for na in (total // 2, total - total // 4 + 3):
        a, b = rand_limbs(rng, na), np.full(total - na, ONES)
        c = bb.ntt_mul(a, b)
        assert mod61(c) == mod61(a) * mod61(b) % M61, (na, total - na)


@pytest.mark.parametrize("quarters,log_n", [(5, 20), (5, 21), (6, 19), (6, 22)])
def test_large_width_residue(bb, quarters, log_n):
    """80- and 96-bit digits on the longest lazy and on strict transforms."""
    rng = np.random.default_rng([SEED, quarters, log_n])
    total = quarters << (log_n - 2)
    for na in (total // 2, total - total // 4 + 3):
        a, b = rand_limbs(rng, na), np.full(total - na, ONES)
        c = bb.ntt_mul(a, b)
        assert mod61(c) == mod61(a) * mod61(b) % M61, (na, total - na)


def _run_batch(bb, port, sizes, squares=(), flags=0):
    import torch

    rng = np.random.default_rng([SEED, len(sizes)])
    host = [(rand_limbs(rng, na), rand_limbs(rng, nb)) for na, nb in sizes]
    dev = [tuple(torch.from_numpy(x.view(np.int64)).cuda() for x in p) for p in host]
    outs = [torch.full((2 * na if i in squares else na + nb,), -1, dtype=torch.int64, device="cuda")
            for i, (na, nb) in enumerate(sizes)]
    prods = []
    for i, (a, b) in enumerate(dev):
        b = a if i in squares else b
        prods.append((a.data_ptr(), a.numel(), b.data_ptr(), b.numel(), outs[i].data_ptr()))
    plan = bb.BatchPlan(prods, flags=flags)
    for _ in range(2):
        plan.run(0)
        bb.device_status(0)
    plan.close()
    for i, (a, b) in enumerate(host):
        want = port.mul(a, a if i in squares else b)
        got = outs[i].cpu().numpy().view(np.uint64)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any(), (i, sizes[i])


# one length on its own; long classes beside the mixed-length launches, a class
# holding products much shorter than its longest (their carry blocks end
# early), operands over half the points, squares; every class on branches
@pytest.mark.parametrize("sizes,squares", [
    ([(700, 600), (1100, 90), (1023, 2)], ()),
    ([(4097, 4097), (8000, 9), (5000, 7000), (300, 400), (1000, 900), (60, 70)], (2,)),
    ([(5000, 5240), (6000, 6288), (6100, 6100), (4097, 4097)] * 4, (1, 6)),  # 80- and 96-bit digits, the longest ones
    ([(16384, 16385), (16385, 16385), (40000, 30), (33000, 700)], (1,)),
])
@pytest.mark.parametrize("per_class", [False, True])
def test_batch_classes(bb, port, sizes, squares, per_class):
    _run_batch(bb, port, sizes * 3, [s + k * len(sizes) for s in squares for k in range(3)],
               bb.BGPU_BATCH_PER_CLASS if per_class else 0)


# levels of equally spaced products: fewer than a group, more than 128, and (the
# longest) several groups of launches a level
@pytest.mark.parametrize("n", [1300, 20_000, 77_777, 2_500_000])
def test_decimal_levels(bb, n):
    rng = np.random.default_rng([SEED, n])
    a = rng.integers(0, 1 << 28, n).astype(np.uint32)
    a[-1] |= 1
    text = bb.to_decimal(a)
    back, neg = bb.from_decimal(text)
    assert not neg and np.array_equal(back, a)
    p = (1 << 61) - 1  # the text itself, modulo a prime
    want = 0
    for d in a[::-1].tolist():
        want = ((want << 28) + d) % p
    got = 0
    for i in range(0, len(text), 18):
        piece = text[i : i + 18]
        got = (got * 10 ** len(piece) + int(piece)) % p
    assert got == want


# text that is not digits alone, in and out of the blocks of 64 characters
@pytest.mark.parametrize("text,value", [
    ("0" * 200 + "7" * 300, int("7" * 300)),
    ("-" + "0" * 63 + "9" * 64, -int("9" * 64)),
    ("x" * 70 + "-" + "12,345." * 40 + "6", -int("12345" * 40 + "6")),
    ("1" + "0" * 127 + "-" + "5" * 129, int("1" + "0" * 127 + "5" * 129)),
    ("0" * 64, 0),
    ("3" * 63 + ":" + "4" * 64 + "/", int("3" * 63 + "4" * 64)),
])
def test_decimal_text_blocks(bb, text, value):
    digits, neg = bb.from_decimal(text)
    got = sum(int(d) << (28 * k) for k, d in enumerate(digits))
    assert (-got if neg else got) == value
