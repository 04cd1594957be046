"""What a batch takes before its kernels run: building a plan, and the one-shot
call, which queues its launches without a graph."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

from conftest import SEED, rand_limbs

pytestmark = pytest.mark.gpu


def make(torch, rng, n, lo, hi, squares=()):
    bits = np.exp2(rng.uniform(lo, hi, (n, 2))).astype(np.int64)
    host, dev, prods = [], [], []
    for i, (x, y) in enumerate(bits // 64 + 1):
        a, b = rand_limbs(rng, int(x)), rand_limbs(rng, int(y))
        b = a if i in squares else b
        da = torch.from_numpy(a.view(np.int64)).cuda()
        db = da if i in squares else torch.from_numpy(b.view(np.int64)).cuda()
        out = torch.full((a.size + b.size,), -1, dtype=torch.int64, device="cuda")
        host.append((a, b))
        dev.append((da, db, out))
        prods.append((da.data_ptr(), a.size, db.data_ptr(), b.size, out.data_ptr()))
    torch.cuda.synchronize()
    return host, dev, prods


def check(port, host, dev):
    for i, ((a, b), (_, _, out)) in enumerate(zip(host, dev)):
        want = port.mul(a, b)
        got = out.cpu().numpy().view(np.uint64)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any(), i


# small products alone; mixed-length launches; long classes on branches with small products beside them
@pytest.mark.parametrize("lo,hi", [(6, 12), (10, 17), (8, 20)])
def test_one_shot(bb, port, lo, hi):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng([SEED, lo, hi])
    host, dev, prods = make(torch, rng, 40, lo, hi, squares=(3, 17))
    s = torch.cuda.Stream()
    for stream in (0, s.cuda_stream):
        for _, _, out in dev:
            out.fill_(-1)
        torch.cuda.synchronize()
        bb.mul_batch_device(prods, stream=stream)
        check(port, host, dev)


def test_one_shot_descriptors_arrive_first(bb, port):
    """The launches of a one-shot call wait for its descriptors: hundreds of
    KB from pageable memory, other ones each time, on a stream that does not wait for
    the legacy default stream."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(SEED + 73)
    n, count = 3, 16384
    a = rng.integers(0, 2**64, (count, n), dtype=np.uint64)
    b = rng.integers(0, 2**64, (count, n), dtype=np.uint64)
    da, db = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    out = torch.zeros((count, 2 * n), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    for turn in range(4):  # product i against operand i + turn
        bb.mul_batch_device([(da.data_ptr() + 8 * n * i, n, db.data_ptr() + 8 * n * ((i + turn) % count), n,
                              out.data_ptr() + 16 * n * i) for i in range(count)], stream=s.cuda_stream)
        got = out.cpu().numpy().view(np.uint64)
        for i in range(0, count, 501):
            want = port.mul(a[i], b[(i + turn) % count])
            assert np.array_equal(got[i, : want.size], want) and not got[i, want.size :].any(), (turn, i)


def test_one_shot_from_threads_while_plans_are_built(bb, port):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(SEED + 71)
    work = [make(torch, rng, 24, 8, 19) for _ in range(3)]
    errors = []

    def go(k):
        try:
            s = torch.cuda.Stream()
            for _ in range(6):
                if k == 2:
                    plan = bb.BatchPlan(work[k][2])
                    plan.run(s.cuda_stream)
                    bb.device_status(s.cuda_stream)
                    plan.close()
                else:
                    bb.mul_batch_device(work[k][2], stream=s.cuda_stream)
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=go, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for host, dev, _ in work:
        check(port, host, dev)


def test_builds_make_no_streams(bb):
    """The branches' streams and events are the engine's: a one-shot call makes no
    stream, and a plan none but those its graph takes, one a branch.  The driver
    numbers streams as they are made."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(SEED + 72)
    _, _, prods = make(torch, rng, 64, 10, 18)
    cu = C.CDLL("libcuda.so.1")

    def next_id():
        s, n = C.c_void_p(), C.c_ulonglong()
        assert cu.cuStreamCreate(C.byref(s), 1) == 0  # CU_STREAM_NON_BLOCKING
        assert cu.cuStreamGetId(s, C.byref(n)) == 0 and cu.cuStreamDestroy_v2(s) == 0
        return n.value

    bb.BatchPlan(prods).close()  # the engine's streams, where this is the first plan
    first = next_id()
    bb.mul_batch_device(prods)
    assert next_id() - first == 1
    first = next_id()
    plans = [bb.BatchPlan(prods) for _ in range(10)]
    made = next_id() - first - 1
    for p in plans:
        p.close()
    assert made <= 10 * 6, made
