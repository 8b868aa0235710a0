"""The measured cases: what a user of the GPU worker has it do.

Every case goes through the C-ABI (include/mps_gpu.h) the way a host program
does: a context (or a server) opened once, items as Factor= lines describe
them, and result buffers that the caller owns.  The context is the handle
that such a program keeps for all of its items, so one per process is shared
by the cases; an item is new work on every call.

Sizes are those of workloads.py (c1 .. c5), of the tests and of the host
program (whose chunks are 2^24 to 2^32 integers), from the smallest call the
library has a path for (2^19 integers) to a configuration in full.  A case
fixes an item; the seed of prepare() moves the start of its prime range (as
the next shard of a run does) or, where the range itself is the point, its c.
"""
from __future__ import annotations

import ctypes
import math
import os
import random
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "mass-prime-siever_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import mps_b200 as mps  # noqa: E402

BASES = (2, 3, 5, 6, 7, 10, 12)
MODS = (1, 2, 6, 12)


def listed() -> list[dict]:
    return [
        # the smallest call: one small range, in the loop of a caller that cannot allocate
        dict(name="noalloc 2^19 at 1e9", kind="noalloc", b=10, c=111, P0=10**9, width=2**19, N0=0, N1=10**7, mod=6, res=4),
        # one small ragged chunk: what a feeder thread of the reference hands over
        dict(name="chunk 2^20 at 1e9", kind="chunk", b=7, c=-3, P0=10**9, width=2**20 + 77, N0=0, N1=10**6, mod=1, res=0),
        # GpuSiever::filter: host-sieved primes, flags back
        dict(name="filter 250k primes", kind="filter", b=10, c=111, P0=10**9, primes=250_001, N0=0, N1=10**7, mod=6, res=4),
        # GpuSiever::sieve_filter on the self-test item, the host program's smallest chunk
        dict(name="sieve_filter 2^24 at 1e10", kind="sieve_filter", b=2, c=-25, P0=10**10, width=2**24, N0=3_600_000,
             N1=5_000_000, mod=2, res=1),
        # the small configuration in full: small primes, thousands of relations and orders
        dict(name="c1 in full", kind="item", b=2, c=-25, P0=10**6, width=99 * 10**6, N0=0, N1=100_000, mod=2, res=1,
             vary="c"),
        # an ordinary chunk of the host program in the middle of a run
        dict(name="chunk 2^28 at 1e12", kind="chunk", b=10, c=111, P0=10**12, width=2**28, N0=0, N1=10**7, mod=6, res=4),
        # the plain GPU configuration, a fifth of its range
        dict(name="c2, 2e9 wide", kind="item", b=10, c=111, P0=10**12, width=2 * 10**9, N0=0, N1=10**7, mod=6, res=4),
        # the residue-class configuration in full: the largest case
        dict(name="c3 in full", kind="item", b=2, c=-25, P0=95 * 10**12, width=2 * 10**10, N0=3_600_000, N1=5_000_000,
             mod=2, res=1),
        # every exponent of the widest N range: the largest baby-step tables, no class to split on
        dict(name="widest N, 5e8 wide", kind="item", b=3, c=2, P0=10**11, width=5 * 10**8, N0=0, N1=10**7, mod=1, res=0),
        # the mixed batch: 64 items, the first 10^8 of each range
        dict(name="c4 batch, 64 items", kind="batch", items=64, items_seed=20261203, lo_digits=9, hi_digits=14,
             lo_width=10**8, hi_width=10**8),
        # many small items over the whole range of the library, 2^49 (integer arithmetic) and beyond included
        dict(name="batch, 48 small items to 1e17", kind="batch", items=48, items_seed=7, lo_digits=9, hi_digits=17,
             lo_width=10**6, hi_width=2 * 10**7),
        # a burst of requests at the server
        dict(name="serve 16 items", kind="serve", items=16, items_seed=20261208, lo_digits=9, hi_digits=14,
             lo_width=10**7, hi_width=10**8),
    ]


# ------------------------------------------------------------------ items --

def _expected(K: float, P0: float, width: float) -> float:
    """Relations an item is expected to have: the sum of K/p over its primes (p > K)."""
    return K * math.log(math.log(P0 + width) / math.log(P0))


def _in_class(n0: int, n1: int, mod: int) -> float:
    return max(1.0, (n1 - n0) / mod)


def _coprime_c(rng: random.Random, b: int) -> int:
    while True:
        c = rng.randint(-999, 999)
        if c != 0 and math.gcd(b, abs(c)) == 1:
            return c


def _draw_spec(rng: random.Random, lo_digits: float, hi_digits: float, lo_width: float, hi_width: float) -> dict:
    """One item with the distributions of the mixed batch (workloads.draw_item)."""
    b = rng.choice(BASES)
    N0 = rng.randint(0, 10**6)
    mod = rng.choice(MODS)
    return dict(b=b, c=_coprime_c(rng, b), P0=int(10 ** rng.uniform(lo_digits, hi_digits)),
                width=int(math.exp(rng.uniform(math.log(lo_width), math.log(hi_width)))), N0=N0,
                N1=N0 + int(10 ** rng.uniform(4, 7)), mod=mod, res=rng.randrange(mod))


def _specs(case: dict) -> list[dict]:
    """The items of a case as the case gives them (before the seed moves them)."""
    if "items" not in case:
        return [case]
    rng = random.Random(case["items_seed"])
    return [_draw_spec(rng, case["lo_digits"], case["hi_digits"], case["lo_width"], case["hi_width"])
            for _ in range(case["items"])]


def _width(case: dict, spec: dict) -> int:
    if case["kind"] == "filter":
        return int(case["primes"] * math.log(spec["P0"]) * 1.1) + 1000
    return spec["width"]


def _moved(case: dict, spec: dict, rng: random.Random) -> tuple:
    """(b, c, P0, P1, N0, N1, mod, res) of a spec for one seed."""
    c, P0, width = spec["c"], spec["P0"], _width(case, spec)
    if case.get("vary") == "c":
        c = _coprime_c(rng, spec["b"])
    else:
        P0 += rng.randrange(P0 // 64)
    return (spec["b"], c, P0, P0 + width, spec["N0"], spec["N1"], spec["mod"], spec["res"])


def draw(rng: random.Random) -> dict:
    """One more case: a way in, and an item (or a set of them) of the ranges above.

    Redrawn until the ranges are wide enough for ten relations or more, which
    is what a run sieves for, and no dearer than the largest listed case."""
    top = max(work(c)["flops"] for c in listed())
    kind = rng.choice(("noalloc", "chunk", "filter", "sieve_filter", "item", "item", "batch", "serve"))
    while True:
        if kind == "batch":
            case = dict(kind=kind, items=rng.randint(4, 64), items_seed=rng.randrange(1 << 30), lo_digits=9,
                        hi_digits=rng.choice((14, 17)), lo_width=10**6, hi_width=int(10 ** rng.uniform(6.5, 8)))
        elif kind == "serve":
            case = dict(kind=kind, items=rng.randint(4, 24), items_seed=rng.randrange(1 << 30), lo_digits=9, hi_digits=14,
                        lo_width=10**7, hi_width=int(10 ** rng.uniform(7.2, 8.2)))
        else:
            lo, hi = {"noalloc": (2**14, 2**19), "chunk": (2**18, 2**28), "sieve_filter": (2**20, 2**28),
                      "item": (10**8, 10**10), "filter": (1, 2)}[kind]
            case = dict(kind=kind, **_draw_spec(rng, 9, 11 if kind == "filter" else 14, lo, hi))
            if kind == "filter":
                case["primes"] = int(math.exp(rng.uniform(math.log(1000), math.log(10**6))))
                del case["width"]
            if kind == "sieve_filter":
                case["P0"] |= 1
        relations = sum(_expected(_in_class(s["N0"], s["N1"], s["mod"]), s["P0"], _width(case, s)) for s in _specs(case))
        if relations >= 10 and work(case)["flops"] <= top:
            return case


# -------------------------------------------------------------- the handle --

_handles: dict = {}


def _siever() -> mps.Siever:
    if "siever" not in _handles:
        _handles["siever"] = mps.Siever(0)
    return _handles["siever"]


def _server() -> mps.Server:
    if "server" not in _handles:
        _handles["server"] = mps.Server(0)
    return _handles["server"]


def _noalloc():
    if "noalloc" not in _handles:
        fn = mps.load_library().mps_chunk_relations_noalloc
        fn.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.POINTER(mps.Item), ctypes.POINTER(mps.Relation),
                       ctypes.c_size_t, ctypes.POINTER(ctypes.c_size_t)]
        fn.restype = ctypes.c_int
        _handles["noalloc"] = fn
    return _handles["noalloc"]


# ------------------------------------------------------------------ passes --

def _primes(lo: int, count: int) -> np.ndarray:
    """The first `count` primes >= lo (host-sieved, as the reference's feeder threads do)."""
    width = int(count * math.log(lo) * 1.1) + 1000
    root = math.isqrt(lo + width) + 1
    small = np.ones(root + 1, dtype=bool)
    small[:2] = False
    for q in range(2, math.isqrt(root) + 1):
        if small[q]:
            small[q * q::q] = False
    keep = np.ones(width, dtype=bool)
    for q in np.flatnonzero(small).tolist():
        keep[(-lo) % q::q] = False
    found = np.flatnonzero(keep)[:count].astype(np.uint64) + np.uint64(lo)
    if found.size < count:
        raise ValueError("the range holds too few primes")
    return found


class State:
    """One prepared call: the handle, the item(s) and the caller's own buffers."""

    def __init__(self, case: dict, seed: int):
        rng = random.Random(seed * 1_000_003 + 17)
        self.kind = case["kind"]
        specs = _specs(case)
        moved = [_moved(case, s, rng) for s in specs]
        self.items = [mps.make_item(*m) for m in moved]
        self.item = self.items[0]
        self.lo, self.hi = moved[0][2], moved[0][3]
        expected = 0.0
        for s in specs:
            K = _in_class(s["N0"], s["N1"], s["mod"])
            small = min(s["P0"] + _width(case, s), K + 1) / 6 if K > s["P0"] else 0.0   # the primes below K
            expected += small + _expected(K, s["P0"], _width(case, s))
        self.cap = 256 + 4 * int(expected)
        self.out = np.zeros((self.cap, 3), dtype=np.int64)              # p, M, q
        self.rel = self.out.ctypes.data_as(ctypes.POINTER(mps.Relation))
        self.n = ctypes.c_size_t()
        self.lib = mps.load_library()
        if self.kind == "serve":
            self.handle = _server()
            self.counts = np.zeros(len(self.items), dtype=np.int64)
        elif self.kind == "noalloc":
            self.fn = _noalloc()
        else:
            self.handle = _siever()
        if self.kind == "batch":
            self.array = (mps.Item * len(self.items))(*self.items)
            self.which = np.zeros(self.cap, dtype=np.int32)             # the item of each relation
        if self.kind == "filter":
            self.primes = _primes(self.lo, case["primes"])
            self.flags = np.zeros(self.primes.size, dtype=np.uint8)
        if self.kind == "sieve_filter":
            self.flagged = np.zeros(self.cap, dtype=np.int64)

    def check(self, rc: int):
        if rc != mps.MPS_OK:
            raise mps.MpsError(rc, self.kind)


def prepare(case: dict, seed: int) -> State:
    return State(case, seed)


def run(s: State):
    n = ctypes.byref(s.n)
    if s.kind == "noalloc":
        s.check(s.fn(s.lo, s.hi, ctypes.byref(s.item), s.rel, s.cap, n))
    elif s.kind == "chunk":
        s.check(s.lib.mps_chunk_relations(s.handle.ctx, s.lo, s.hi, ctypes.byref(s.item), s.rel, s.cap, n))
    elif s.kind == "item":
        s.check(s.lib.mps_item_relations(s.handle.ctx, ctypes.byref(s.item), s.rel, s.cap, n))
    elif s.kind == "sieve_filter":
        out = s.flagged.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))
        s.check(s.lib.mps_sieve_filter(s.handle.ctx, s.lo, s.hi, ctypes.byref(s.item), out, s.cap, n))
        return {"flagged": s.flagged, "count": s.n.value}
    elif s.kind == "filter":
        s.check(s.lib.mps_filter(s.handle.ctx, s.primes.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), s.primes.size,
                                 ctypes.byref(s.item), s.flags.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8))))
        return {"flags": s.flags}
    elif s.kind == "batch":
        which = s.which.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32))
        s.check(s.lib.mps_batch_relations(s.handle.ctx, s.array, len(s.items), s.rel, which, s.cap, n))
        return {"relations": s.out, "item": s.which, "count": s.n.value}
    else:                                                               # serve: all at once, each result as it is done
        tickets = [s.handle.submit(it) for it in s.items]
        at = 0
        for k, t in enumerate(tickets):
            if not s.handle.wait(t)["done"]:
                raise RuntimeError("the server did not finish an item")
            dst = ctypes.cast(s.out[at:].ctypes.data, ctypes.POINTER(mps.Relation))
            s.check(s.lib.mps_serve_result(s.handle.sv, t, dst, s.cap - at, n))
            s.counts[k] = s.n.value
            at += s.n.value
            s.handle.release(t)
        return {"relations": s.out, "counts": s.counts}
    return {"relations": s.out, "count": s.n.value}


def work(case: dict) -> dict:
    """What a pass cannot do without.  Bytes: the items (and primes) in, the
    relations (or flags) out.  Operations: a mark per sieving prime and odd
    multiple (2.2 an odd number), one modular exponentiation a prime (log2 p
    products of six operations each) and, for the quarter of the primes that
    the quadratic and power-residue conditions leave, 2 sqrt(K) products of
    baby and giant steps over the K exponents of the class."""
    flops = byts = 0.0
    for s in _specs(case):
        width, P0 = _width(case, s), s["P0"]
        K = _in_class(s["N0"], s["N1"], s["mod"])
        primes = width / math.log(P0 + width)
        byts += ctypes.sizeof(mps.Item) + 24 * _expected(K, P0, width)
        if case["kind"] == "filter":
            byts += 9 * case["primes"]
        else:
            flops += 2.2 * width / 2
        flops += primes * 6 * (math.log2(P0 + width) + 0.25 * 2 * math.sqrt(K))
    return {"bytes": byts, "flops": flops}
