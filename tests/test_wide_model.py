"""CPU model of the wide-digit products: the prime sets' bounds and the
single-precision CRT of the carry pass (bigint_b200/csrc/wide_kernels.cu)."""
from __future__ import annotations

import math
import os
import random
import re

import numpy as np
import pytest

from conftest import ROOT

ARITH = open(os.path.join(ROOT, "bigint_b200", "csrc", "arith.cuh")).read()
MAX_LOG = {2: 22, 3: 25, 4: 20, 5: 24, 6: 18, 7: 23}
BITS = {2: 64, 3: 64, 4: 80, 5: 80, 6: 96, 7: 96}
SETS = sorted(BITS)


def prime_sets():
    rows = re.findall(r"\{(\d), \{([\du, ]+)\},\s+\{([\du, ]+)\}, \w+, \d+\}", ARITH)
    nums = [[int(x) for x in re.findall(r"\d+", r)] for _, r, _ in rows]
    gens = [[int(x) for x in re.findall(r"\d+", r)] for _, _, r in rows]
    return nums, gens


def factors(n):
    f, i = set(), 2
    while i * i <= n:
        while n % i == 0:
            f.add(i)
            n //= i
        i += 1
    return f | ({n} if n > 1 else set())


@pytest.mark.parametrize("ps", SETS)
def test_wide_prime_set(ps):
    nums, gens = prime_sets()
    assert len(nums) == 8 and [len(x) for x in nums] == [3, 3, 5, 5, 6, 6, 7, 7]
    m = 1
    for p, g in zip(nums[ps], gens[ps]):
        assert all(p % d for d in range(2, math.isqrt(p) + 1))
        assert (p - 1) % (1 << MAX_LOG[ps]) == 0
        assert all(pow(g, (p - 1) // f, p) != 1 for f in factors(p - 1))
        assert p < (1 << 30 if ps % 2 == 0 else 1 << 31)
        m *= p
    worst = (1 << (MAX_LOG[ps] - 1)) * ((1 << BITS[ps]) - 1) ** 2
    assert worst < m
    # the fraction x / M leaves 0.05 on either side of the floor
    assert worst / m < 0.9
    assert sum(sorted(nums[ps])[-4:]) < 1 << 32 or ps % 2  # four products of a column below 2^64


@pytest.mark.parametrize("ps", SETS)
def test_single_precision_crt(ps):
    """q = floor(sum y_i / p_i) from the top bits of y_i in float32, at random
    coefficients and at the ends of the range."""
    nums, _ = prime_sets()
    p = nums[ps]
    m = math.prod(p)
    inv = np.array([256.0 / x for x in p], dtype=np.float32)
    bias = np.float32(0.05 - 8388608.0 * float(np.sum(inv.astype(np.float64))))
    top = (1 << (MAX_LOG[ps] - 1)) * ((1 << BITS[ps]) - 1) ** 2
    rng = random.Random(7)
    xs = [0, 1, 2, top, top - 1] + [rng.randrange(top + 1) for _ in range(3000)]
    xs += [min(top, q * (m // len(p)) + d) for q in range(len(p)) for d in (0, 1)]
    for x in xs:
        y = [x * pow(m // pi, -1, pi) % pi for pi in p]
        f = bias
        for yi, k in zip(y, inv):
            t = np.float32(8388608.0 + (yi >> 8))  # exact: 2^23 + a 23-bit integer
            f = np.float32(np.float64(t) * np.float64(k) + np.float64(f))  # fused
        q = int(f)
        assert 0 <= q < len(p)
        assert sum(yi * (m // pi) for yi, pi in zip(y, p)) - q * m == x
