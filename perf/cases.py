"""The calls that users of this package make, as measurable cases.

One pass of a case is one call (or the fixed sequence of calls) through the
public entry points: the Python mirror of the C ABI, and cbl_batch_noalloc by
ctypes, which is how a program binds it. Positions are taken from the seed, a
few percent below the case's size, so that another seed is another position
of the same cost.

192-bit results are whole numbers and are returned as their bytes. Mode-0
(double-double) results are returned as the pair of floats that the library
hands out, with an exact value beside them (exact()).
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import clbellard_gb300 as C

# The seven series (numer, sign, den0, den1) of the formula, for exact().
SERIES = [(32, 1, 4, 1), (1, 1, 4, 3), (256, 0, 10, 1), (64, 1, 10, 3), (4, 1, 10, 5), (4, 1, 10, 7), (1, 0, 10, 9)]
TAIL_DD = 10                       # tail terms k = d .. d+9 of the double-double mode


def listed():
    return [
        # One early position asked for interactively: latency of one whole call.
        {"name": "position_1e3", "kind": "compute", "position": 1000, "precision": 1},
        # Position 1e6, mode 2: the usual first try of a new user.
        {"name": "position_1e6", "kind": "compute", "position": 10 ** 6, "precision": 2},
        # An arbitrary (not 5-aligned) hex position, as spot checks P against P-8 use.
        {"name": "hexpos_1e8", "kind": "hexpos", "position": 10 ** 8 + 3, "precision": 1},
        # A prepared position run again and read back: moduli up to 4e9, all below 2^32.
        {"name": "prepared_1e9", "kind": "prepared", "position": 10 ** 9, "precision": 1},
        # The headline workload: hex position 1e10 through the one-call entry point.
        {"name": "position_1e10", "kind": "compute", "position": 10 ** 10, "precision": 1},
        # A sweep of uneven positions in one call (a table of digits).
        {"name": "batch_512", "kind": "batch", "positions": 512, "low": 10 ** 3, "high": 10 ** 8, "precision": 1},
        # The allocation-free call of a program that owns its device memory.
        {"name": "noalloc_64", "kind": "noalloc", "positions": 64, "low": 10 ** 3, "high": 10 ** 7, "precision": 1},
        # Work mode: one balanced job of position 1e11 (moduli up to 4e11).
        {"name": "job_1e11", "kind": "job", "position": 10 ** 11, "series": 2, "at": 0.5, "terms": 1 << 28,
         "precision": 1},
        # Work mode far out: a job of position 1e13, whose moduli pass 2^44.
        {"name": "job_1e13", "kind": "job", "position": 10 ** 13, "series": 5, "at": 0.8, "terms": 1 << 27,
         "precision": 1},
        # The 106-bit mode on a whole position, kernel by kernel as the reference's host drives it.
        {"name": "dd_1e7", "kind": "dd", "position": 10 ** 7, "precision": 0},
        # The 106-bit mode's work-mode job at position 1e10 (two-word moduli), an odd number of terms.
        {"name": "dd_job_1e10", "kind": "dd_job", "position": 10 ** 10, "series": 3, "at": 0.6,
         "terms": (1 << 25) - 39, "precision": 0},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["compute", "compute", "hexpos", "prepared", "batch", "noalloc", "job", "job", "dd", "dd_job"])
    if kind in ("compute", "hexpos", "prepared"):
        return {"kind": kind, "position": _log(rng, 10 ** 3, 10 ** 10), "precision": rng.choice([1, 2])}
    if kind == "batch":
        return {"kind": kind, "positions": _log(rng, 2, 1024), "low": 10 ** 3, "high": _log(rng, 10 ** 4, 10 ** 8),
                "precision": 1}
    if kind == "noalloc":
        return {"kind": kind, "positions": rng.randint(1, 64), "low": 10 ** 3, "high": _log(rng, 10 ** 4, 10 ** 7),
                "precision": 1}
    if kind == "job":
        return {"kind": kind, "position": _log(rng, 10 ** 10, 10 ** 14), "series": rng.randrange(7),
                "at": round(rng.uniform(0.0, 0.9), 3), "terms": _log(rng, 1 << 16, 1 << 29), "precision": 1}
    if kind == "dd":
        return {"kind": kind, "position": _log(rng, 10 ** 4, 5 * 10 ** 7), "precision": 0}
    return {"kind": kind, "position": _log(rng, 10 ** 9, 10 ** 11), "series": rng.randrange(7),
            "at": round(rng.uniform(0.0, 0.9), 3), "terms": _log(rng, 1 << 14, 1 << 26), "precision": 0}


# ------------------------------------------------------------------ inputs --
def _near(rng, position):
    """A position up to 2 % below the given one."""
    return position - rng.randrange(0, max(1, position // 50))


def _d_of(position):
    """Series length d of a reference position: d is odd and about 2/5 of it."""
    d = ((position - 1) * 2 - 3) // 5
    return d if d % 2 else d - 1


def _job_range(case, rng, d):
    k0 = min(int(case["at"] * d) + rng.randrange(0, 1 << 12), d - 2)
    return k0, min(k0 + case["terms"], d)


def _inputs(case, seed):
    rng = random.Random(seed)
    if case["kind"] in ("batch", "noalloc"):
        return {"positions": [max(5, _log(rng, case["low"], case["high"])) for _ in range(case["positions"])]}
    position = _near(rng, case["position"])
    d = _d_of(position)
    inp = {"position": position, "d": d}
    if case["kind"] in ("job", "dd_job"):
        inp["k0"], inp["k1"] = _job_range(case, rng, d)
    return inp


def prepare(case, seed):
    state = dict(_inputs(case, seed), kind=case["kind"], series=case.get("series"))
    if case["kind"] == "noalloc":
        fn = C.load().cbl_batch_noalloc
        fn.argtypes = [ctypes.POINTER(ctypes.c_uint64), ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
        fn.restype = ctypes.c_int
        n = len(state["positions"])
        state["fn"] = fn
        state["array"] = (ctypes.c_uint64 * n)(*state["positions"])
        state["out"] = torch.empty((n, 3), dtype=torch.int64, device="cuda")
        return state
    state["ctx"] = C.Context(0, case["precision"])
    if case["kind"] == "prepared":
        state["ctx"].prepare([state["position"]])
    return state


# -------------------------------------------------------------------- a pass --
def _bytes(values):
    """192-bit integers as rows of 24 bytes, most significant first."""
    return np.frombuffer(b"".join(v.to_bytes(24, "big") for v in values), dtype=np.uint8).reshape(-1, 24)


def run(state):
    kind = state["kind"]
    if kind == "noalloc":
        rc = state["fn"](state["array"], len(state["positions"]), state["out"].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError("cbl_batch_noalloc: %d" % rc)
        return state["out"]
    ctx = state["ctx"]
    if kind == "compute":
        return np.frombuffer(bytes.fromhex(ctx.compute(state["position"])), dtype=np.uint8)
    if kind == "hexpos":
        return np.frombuffer(bytes.fromhex(ctx.compute_hexpos(state["position"])), dtype=np.uint8)
    if kind == "prepared":
        ctx.run_prepared()
        return _bytes(ctx.read_results())
    if kind == "batch":
        return _bytes(ctx.batch(state["positions"]))
    if kind == "job":
        return np.frombuffer(bytes.fromhex(ctx.run_job_range(state["position"], state["series"], state["k0"],
                                                             state["k1"])), dtype=np.uint8)
    d = state["d"]
    if kind == "dd":
        ctx.Set0ans()
        for f in range(7):
            ctx.Set0mem()
            ctx.BatchCalc(0, d, f, d)
            ctx.AddAns(f)
        hi, lo = ctx.read_ans()
    else:
        ctx.Set0mem()
        ctx.BatchCalc(state["k0"], state["k1"], state["series"], d)
        ctx.AddAns(state["series"])
        hi, lo = ctx.read_partial()
    return {"hi": hi, "lo": lo}


# ---------------------------------------------------------- necessary work --
def _term_products(d, f, k0, k1):
    """32x32-bit products of the terms k in [k0, k1): one modular squaring per
    bit of the exponent 10(d-k) (1 + 1 products below 2^32, 3 + 3 above), and
    six 32-bit digits of the fraction (one product per word of the modulus)."""
    _, _, den0, den1 = SERIES[f]
    total, n = 0.0, k1 - k0
    bins = min(n, 256)
    for i in range(bins):
        k = k0 + (2 * i + 1) * n // (2 * bins)
        squarings = max(1, (10 * (d - k)).bit_length())
        wide = den0 * k + den1 >= 1 << 32
        total += squarings * (6 if wide else 2) + 6 * (2 if wide else 1)
    return total * n / max(1, bins)


def work(case):
    if case["kind"] in ("batch", "noalloc"):
        lo, hi, n = math.log(case["low"]), math.log(max(case["high"], case["low"] + 1)), case["positions"]
        positions = [int(math.exp(lo + (hi - lo) * (2 * i + 1) / (2 * n))) for i in range(n)]
        products = sum(_term_products(_d_of(p), 2, 0, _d_of(p)) * 7 for p in positions)
        return {"bytes": (8 + 24) * n, "flops": 2.0 * products}
    d = _d_of(case["position"])
    if case["kind"] in ("job", "dd_job"):
        k0 = min(int(case["at"] * d), d - 2)
        products = _term_products(d, case["series"], k0, min(k0 + case["terms"], d))
    else:
        products = sum(_term_products(d, f, 0, d) for f in range(7))
    return {"bytes": 24 if case["precision"] else 16, "flops": 2.0 * products}


# ------------------------------------------------------------- exact values --
def _mulmod(a, b, m):
    """a b mod m for a, b < m < 2^40 in 64-bit integers."""
    return ((a * (b >> 20)) % m * (1 << 20) + a * (b & 0xFFFFF)) % m


def _pow2mod(e, m):
    """2^e mod m, elementwise, m < 2^40, from the exponent's top bit down."""
    small = int(m.max()) < 1 << 31
    r = torch.ones_like(m) % m
    for i in range(int(e.max()).bit_length() - 1, -1, -1):
        r = (r * r) % m if small else _mulmod(r, r, m)
        r = (r << ((e >> i) & 1)) % m
    return r


FRACTION_BITS = 8 * 22


def _fraction_sum(f, d, k0, k1, device):
    """sum over k in [k0, k1), k < d, of the signed frac(2^(10(d-k)) / m), in
    units of 2^-176, from eight 22-bit digits of each fraction."""
    _, sign, den0, den1 = SERIES[f]
    total = 0
    for a in range(k0, k1, 1 << 24):
        k = torch.arange(a, min(k1, a + (1 << 24)), dtype=torch.int64, device=device)
        m = den0 * k + den1
        r = _pow2mod(10 * (d - k), m)
        s = 1 - 2 * ((k + sign) & 1)
        for j in range(1, 9):
            r = r << 22
            total += int((s * (r // m)).sum()) << (FRACTION_BITS - 22 * j)
            r = r % m
    return total


def _tail_sum(f, d):
    _, sign, den0, den1 = SERIES[f]
    total = 0
    for i in range(TAIL_DD):
        k = d + i
        t = (1 << (FRACTION_BITS - 10 * i)) // (den0 * k + den1)
        total += -t if (k + sign) & 1 else t
    return total


def _as_pair(x):
    """x / 2^176 mod 1 as the nearest double and the rest."""
    x %= 1 << FRACTION_BITS
    hi = x / (1 << FRACTION_BITS)                            # correctly rounded
    n, q = hi.as_integer_ratio()
    rest = x * q - (n << FRACTION_BITS)
    return {"hi": hi, "lo": rest / (q << FRACTION_BITS)}


def exact(case, seed):
    if case["kind"] not in ("dd", "dd_job"):
        return None                                          # whole numbers
    inp = _inputs(case, seed)
    d = inp["d"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    total = 0
    if case["kind"] == "dd":
        for f in range(7):
            s = _fraction_sum(f, d, 0, d, device) + _tail_sum(f, d)
            total += SERIES[f][0] * s
    else:
        f = case["series"]
        s = _fraction_sum(f, d, inp["k0"], inp["k1"], device)
        if inp["k1"] == d:
            s += _tail_sum(f, d)
        total = SERIES[f][0] * s
    return _as_pair(total)
