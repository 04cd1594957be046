"""Performance cases: the work programs give this library, through its public
entry points.

Each case is a dict of plain values.  `listed()` holds a fixed set, `draw(rng)`
one more of the same ranges; `prepare` makes what a program holds before the
call, `run` makes one call, `work` counts what the call cannot do without, and
`exact` computes the same outputs with Python integers.
"""
import math
import sys

import numpy as np
import torch

import bigint_b200 as bb

# Case kinds
#   mul       product of two device-resident limb arrays (bits of each)
#   square    square of one device-resident limb array
#   batch     one run of a batch plan of independent products of uneven length
#   tree      pairwise product tree over device-resident 64-bit leaves
#   digits    product of two host-resident BigInts in 28-bit Digits (mul_digits)
#   inverse   BigFloat reciprocal of a host-resident number (Newton steps)
#   decimal   a BigInt printed as decimal text and read back


def listed():
    return [
        # A few hundred bits to a few thousand: RSA-sized operands, the lower
        # levels of any recursion; the cost is the call and one launch.
        {"name": "small", "kind": "mul", "abits": 4096, "bbits": 3008},
        # A product just above the schoolbook range: launches and the gaps
        # between them.
        {"name": "medium", "kind": "mul", "abits": 65536, "bbits": 50048},
        # The plain 2^20-bit product.
        {"name": "mul_2p20", "kind": "mul", "abits": 1 << 20, "bbits": 1 << 20},
        # The headline product, 2^24-bit operands.
        {"name": "mul_2p24", "kind": "mul", "abits": 1 << 24, "bbits": 1 << 24},
        # Lengths as a computation leaves them: unequal, no power of two.
        {"name": "ragged", "kind": "mul", "abits": 9_000_001, "bbits": 31_234_567},
        # BigInt operator* on host-resident 28-bit Digits: the call a program
        # linked against the drop-in makes, transfers included.
        {"name": "digits_2p20", "kind": "digits", "adigits": 40_000, "bdigits": 37_450},
        # A large square, the step of fast_pow and of square-root iterations.
        {"name": "square_2p27", "kind": "square", "abits": 150_000_000, "bbits": 0},
        # The largest product one transform holds.
        {"name": "mul_2p30", "kind": "mul", "abits": 1 << 30, "bbits": 1 << 30},
        # Independent products of uneven length in one batch plan.
        {"name": "batch_4096", "kind": "batch", "count": 4096, "lo": 10, "hi": 22, "sizes": 5},
        # Binary splitting: 2^20 leaves in [2^32, 2^64) to one 2^26-bit product.
        {"name": "tree_2p20", "kind": "tree", "leaves": 1 << 20},
        # BigFloat reciprocal at 20000 28-bit digits (about 170 000 decimals).
        {"name": "reciprocal", "kind": "inverse", "digits": 20_000, "precision": 20_000},
        # A number of about a million decimal digits printed and read back.
        {"name": "decimal", "kind": "decimal", "digits": 120_000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mul", "mul", "mul", "mul", "square", "batch", "tree", "digits", "inverse", "decimal"])
    if kind == "mul":
        return {"kind": kind, "abits": _log_uniform(rng, 2048, 1 << 30), "bbits": _log_uniform(rng, 2048, 1 << 30)}
    if kind == "square":
        return {"kind": kind, "abits": _log_uniform(rng, 2048, 1 << 29), "bbits": 0}
    if kind == "batch":
        return {"kind": kind, "count": _log_uniform(rng, 64, 4096), "lo": 10, "hi": rng.randint(14, 22),
                "sizes": rng.randint(0, 1 << 30)}
    if kind == "tree":
        return {"kind": kind, "leaves": _log_uniform(rng, 1 << 10, 1 << 20)}
    if kind == "digits":
        return {"kind": kind, "adigits": _log_uniform(rng, 500, 2_000_000), "bdigits": _log_uniform(rng, 500, 2_000_000)}
    if kind == "inverse":
        n = _log_uniform(rng, 200, 40_000)
        return {"kind": kind, "digits": n, "precision": n}
    return {"kind": kind, "digits": _log_uniform(rng, 500, 120_000)}


def _limbs_of(bits):
    return (bits + 63) // 64


def _random_limbs(gen, n, bits=None):
    """n uniform random limbs on the GPU (int64 bit patterns); with `bits`, a
    number of exactly that many bits."""
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda", generator=gen)
    if bits is not None:
        top = (bits - 1) % 64  # bit of the top limb that is the highest one set
        mask = (1 << (top + 1)) - 1 if top < 63 else -1
        high = 1 << top if top < 63 else -(1 << 63)
        x[-1] = (x[-1] & mask) | high
    return x


def _random_digits(gen, n):
    """n uniform random 28-bit digits with a nonzero top digit, on the host."""
    d = torch.randint(0, 1 << 28, (n,), dtype=torch.int64, device="cuda", generator=gen)
    d[-1] |= 1 << 27
    return d.cpu().numpy().astype(np.uint32)


def _batch_sizes(case):
    """Operand lengths in bits, log-uniform in [2^lo, 2^hi], fixed by the case."""
    r = np.random.default_rng(case["sizes"])
    return np.exp2(r.uniform(case["lo"], case["hi"], (case["count"], 2))).astype(np.int64)


def prepare(case, seed):
    bb.init(0)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("mul", "square"):
        a = _random_limbs(gen, _limbs_of(case["abits"]), case["abits"])
        b = a if kind == "square" else _random_limbs(gen, _limbs_of(case["bbits"]), case["bbits"])
        st.update(a=a, b=b, out=torch.empty(a.numel() + b.numel(), dtype=torch.int64, device="cuda"))
    elif kind == "batch":
        bits = _batch_sizes(case)
        limbs = (bits + 63) // 64
        place = (limbs + 31) // 32 * 32  # each array on a 256-byte boundary, as an allocator gives it
        at = np.concatenate([[0], np.cumsum(place.reshape(-1))])
        osize = (limbs.sum(axis=1) + 31) // 32 * 32
        oat = np.concatenate([[0], np.cumsum(osize)])
        x = _random_limbs(gen, int(at[-1]))
        out = torch.zeros(int(oat[-1]), dtype=torch.int64, device="cuda")
        px, po = x.data_ptr(), out.data_ptr()
        prods = []
        for i in range(case["count"]):
            prods.append((px + 8 * int(at[2 * i]), int(limbs[i, 0]), px + 8 * int(at[2 * i + 1]), int(limbs[i, 1]),
                          po + 8 * int(oat[i])))
        st.update(x=x, out=out, plan=bb.BatchPlan(prods))
    elif kind == "tree":
        n = case["leaves"]
        leaves = _random_limbs(gen, n)
        leaves |= 1 << 32  # at least 2^32
        width = 1 << max(0, (n - 1).bit_length())
        st.update(leaves=leaves, out=torch.empty(width, dtype=torch.int64, device="cuda"))
    elif kind == "digits":
        st.update(a=_random_digits(gen, case["adigits"]), b=_random_digits(gen, case["bdigits"]))
    elif kind == "inverse":
        st.update(a=_random_digits(gen, case["digits"]), precision=case["precision"])
    else:
        st.update(a=_random_digits(gen, case["digits"]))
    return st


def _padded(x, n):
    """x with zeros up to n elements: how many digits a result has depends on
    its value."""
    out = np.zeros(max(n, x.size), x.dtype)
    out[: x.size] = x
    return out


def _padded_text(text, ndigits):
    return _padded(np.frombuffer(text.encode(), dtype=np.uint8), int(ndigits * 28 * math.log10(2)) + 2)


def run(st):
    kind = st["kind"]
    if kind in ("mul", "square"):
        a, b, out = st["a"], st["b"], st["out"]
        bb.mul_device(a.data_ptr(), a.numel(), b.data_ptr(), b.numel(), out.data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
        return out
    if kind == "batch":
        st["plan"].run(torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if kind == "tree":
        bb.product_tree_device(st["leaves"].data_ptr(), st["leaves"].numel(), st["out"].data_ptr(), st["out"].numel(),
                               torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if kind == "digits":
        digits, point = bb.mul_digits(st["a"], st["b"], 0, 0)
        return digits, point
    if kind == "inverse":
        digits, point, neg = bb.reciprocal_digits(st["a"], st["a"].size, False, st["precision"])
        return _padded(digits, 2 * st["precision"] + 16), point, neg
    text = bb.to_decimal(st["a"])
    digits, neg = bb.from_decimal(text)
    return _padded_text(text, st["a"].size), digits, neg


def _mul_work(na, nb, square=False):
    """A product of na and nb 64-bit limbs: operands in, product out; the
    operations of three length-n transforms at 5 n log2 n, n = na + nb (two for
    a square), or of the schoolbook method where that is less."""
    n = na + nb
    transform = (2 if square else 3) * 5.0 * n * max(1.0, math.log2(n))
    return 8 * ((na if square else n) + n), min(transform, 2.0 * na * nb)


def work(case):
    kind = case["kind"]
    if kind in ("mul", "square"):
        na = _limbs_of(case["abits"])
        nbytes, flops = _mul_work(na, na if kind == "square" else _limbs_of(case["bbits"]), kind == "square")
    elif kind == "batch":
        nbytes = flops = 0
        for na, nb in ((_batch_sizes(case) + 63) // 64).tolist():
            by, fl = _mul_work(na, nb)
            nbytes, flops = nbytes + by, flops + fl
    elif kind == "tree":
        n, nbytes, flops, size = case["leaves"], 16 * case["leaves"], 0, 1
        while size < n:
            flops += _mul_work(size, size)[1] * (n / (2 * size))
            size *= 2
    elif kind == "digits":
        na, nb = case["adigits"], case["bdigits"]
        nbytes, flops = 8 * (na + nb), _mul_work((na * 7 + 15) // 16, (nb * 7 + 15) // 16)[1]
    elif kind == "inverse":
        n = (case["precision"] * 7 + 15) // 16
        nbytes = 4 * (case["digits"] + case["precision"])
        flops = 4 * _mul_work(n, n)[1]  # two products a step over halving precisions
    else:
        n = (case["digits"] * 7 + 15) // 16
        text = int(case["digits"] * 28 * math.log10(2)) + 1
        nbytes, flops = 2 * (4 * case["digits"] + text), 0
        size = n
        while size >= 2:  # one product a level each way
            flops += 3 * _mul_work(size / 2, size / 2)[1] * (n / size)
            size /= 2
    return {"bytes": int(nbytes), "flops": int(flops)}


# ---- the outputs from Python integers ---------------------------------------------


def _int_of_limbs(x):
    return int.from_bytes(x.cpu().numpy().tobytes(), "little")


def _limbs_of_int(v, n):
    return torch.from_numpy(np.frombuffer(v.to_bytes(8 * n, "little"), dtype=np.int64).copy())


def _int_of_digits(d):
    """Value of 28-bit digits: pairs of digits are 7 bytes."""
    d = np.concatenate([d, np.zeros(d.size % 2, np.uint32)]).astype(np.uint64)
    pairs = d[0::2] | (d[1::2] << np.uint64(28))
    return int.from_bytes(np.ascontiguousarray(pairs.view(np.uint8).reshape(-1, 8)[:, :7]).tobytes(), "little")


def _digits_of_int(v):
    n = (v.bit_length() + 55) // 56
    b = np.zeros((n, 8), np.uint8)
    b[:, :7] = np.frombuffer(v.to_bytes(7 * n, "little"), dtype=np.uint8).reshape(n, 7)
    pairs = b.reshape(-1).view(np.uint64)
    d = np.empty(2 * n, np.uint32)
    d[0::2] = pairs & np.uint64((1 << 28) - 1)
    d[1::2] = pairs >> np.uint64(28)
    return d[: len(d) - (1 if d[-1] == 0 else 0)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mul", "square"):
        if max(case["abits"], case["bbits"]) > 1 << 22 or case["abits"] + case["bbits"] > 1 << 23:
            return None
        st = prepare(case, seed)
        a, b = _int_of_limbs(st["a"]), _int_of_limbs(st["b"])
        return _limbs_of_int(a * b, st["out"].numel())
    if kind == "tree":
        if case["leaves"] > 1 << 15:
            return None
        st = prepare(case, seed)
        v = [x % (1 << 64) for x in st["leaves"].tolist()]
        while len(v) > 1:
            v = [v[i] * v[i + 1] if i + 1 < len(v) else v[i] for i in range(0, len(v), 2)]
        return _limbs_of_int(v[0], st["out"].numel())
    if kind == "digits":
        if max(case["adigits"], case["bdigits"]) > 150_000:
            return None
        st = prepare(case, seed)
        d = _digits_of_int(_int_of_digits(st["a"]) * _int_of_digits(st["b"]))
        return d, 0
    if kind == "decimal":
        if case["digits"] > 4_000:
            return None
        if hasattr(sys, "set_int_max_str_digits"):
            sys.set_int_max_str_digits(0)
        st = prepare(case, seed)
        text = str(_int_of_digits(st["a"]))
        return _padded_text(text, st["a"].size), st["a"], False
    # a batch is thousands of products and the reciprocal's digits are those of
    # its own truncated iteration: neither has a value here
    return None
