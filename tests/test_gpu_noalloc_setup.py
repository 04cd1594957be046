"""The no-allocation entry point's first call in a process, on a stream that does
not wait for the legacy default stream its tables are copied on."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes as C
import numpy as np
import torch
import bigint_b200 as bb
f = bb.lib.bgpu_mul_u64_device_noalloc
f.argtypes = [C.c_void_p, C.c_size_t, C.c_void_p, C.c_size_t, C.c_void_p, C.c_void_p]
rng = np.random.default_rng(5)
a = rng.integers(0, 2**64, 4000, dtype=np.uint64)
b = rng.integers(0, 2**64, 3001, dtype=np.uint64)
da, db = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
out = torch.empty(7001, dtype=torch.int64, device="cuda")
s = torch.cuda.Stream()
torch.cuda.synchronize()
assert f(da.data_ptr(), a.size, db.data_ptr(), b.size, out.data_ptr(), s.cuda_stream) == 0
got = int.from_bytes(out.cpu().numpy().tobytes(), "little")
assert got == int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
"""


def test_first_call_on_its_own_stream():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=180)
    assert r.returncode == 0, r.stdout + r.stderr
