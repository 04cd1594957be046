"""The carry scans' block flags against what earlier products leave in the
shared scratch memory."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# Runs in a process of its own, where the n-th product of the engine has scan
# epoch n.  An FFT product with operand 1 leaves its other operand's 8-bit
# digits as 64-bit words in the scratch, at the offset where the scan of the
# next product (2^14 points) would find its flags if these lay behind its
# residues: each digit is that product's flag word "inclusive, no carry".  That
# product is a run of ones through every chunk with a carry entering at the
# bottom, so each block waits for the flag of the one below.
PROGRAM = """
import numpy as np
import bigint_b200 as bb
bb.init(0)
ONES = (1 << 64) - 1
third = np.full(16000, ONES // 3, dtype=np.uint64)
third[:3] = ONES
b = np.ones(3, dtype=np.uint64)
want = int.from_bytes(third.tobytes(), "little") * ((1 << 128) + (1 << 64) + 1)
for k in range(1, 8):
    digits = np.ones(32000, dtype=np.uint8)
    digits[16384:16448] = (2 * k) << 4 | 8
    _, st = bb.fft_mul(digits.view(np.uint64), np.ones(1, dtype=np.uint64), digit_bits=8, stats=True)
    assert (st.fft_bits, st.log2_points, st.fell_back) == (8, 15, 0)
    got, st = bb.ntt_mul(third, b, stats=True)
    assert st.log2_points == 15
    assert int.from_bytes(got.tobytes(), "little") == want, k
"""


def test_stale_words_are_no_flags():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
