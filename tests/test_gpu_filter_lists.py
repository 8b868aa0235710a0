"""filter on the lists a caller may hand over: repeats, and numbers on both
sides of 2^49 in one list."""
from __future__ import annotations

import time

import pytest

from oracle.oracle import make_item as oracle_item

pytestmark = pytest.mark.gpu


def test_one_prime_many_times(siever, mps_lib, oracle):
    """100,000 places of one prime with a relation: a pass over the list, not one per place."""
    spec = (2, -25, 10**6, 10**6 + 200_000, 0, 60_000, 2, 1)
    it = mps_lib.make_item(*spec)
    hit = oracle.relations(spec[2], spec[3], oracle_item(*spec))[0][0]
    siever.filter([hit], it)
    t0 = time.perf_counter()
    assert siever.filter([hit] * 100_000, it) == [1] * 100_000
    assert time.perf_counter() - t0 < 1.0


def test_arithmetic_by_chunk(mps_lib, oracle):
    """A list of two chunks, below and above 2^49: each runs as it does alone (with
    four chains the two arithmetics' solves end after different step counts)."""
    low = oracle.primes(10**9, 10**9 + 200_000, 1 << 16)[:4096]
    high = oracle.primes(2**49, 2**49 + 20_000, 1 << 16)
    it = mps_lib.make_item(3, 2, 10**9, 2**50, 0, 10**7, 1, 0)
    with mps_lib.Siever(0, chunk_odds=4096, chains=4) as s:
        flags, steps = [], 0
        for part in (low, high):
            flags += s.filter(part, it)
            steps += s.stats()["bsgs_steps"]
        assert s.filter(low + high, it) == flags
        assert s.stats()["bsgs_steps"] == steps
        # in one chunk: the same flags
        mixed = low[:2000] + high + low[2000:3000]
        assert s.filter(mixed, it) == flags[:2000] + flags[4096:] + flags[2000:3000]


@pytest.mark.parametrize("P0,counts", [(10**9, (1, 2, 31, 1000, 16383, 16384)), (2**49, (1, 33, 8191, 8192))])
@pytest.mark.parametrize("mod,res", [(1, 0), (6, 4), (1001, 7), (2**20 - 3, 5)])
def test_short_and_long_lists(mps_lib, oracle, P0, counts, mod, res):
    """Lists on both sides of the length from which the primes are split: the oracle's
    flags, with only the kernels that a list needs (a short one: no split's)."""
    primes = oracle.primes(P0, P0 + 24 * 16_384 + 100_000, 1 << 16)
    spec = (3, 2, P0, primes[-1] + 1, 0, 10**7, mod, res)
    hits = {r[0] for r in oracle.relations(P0, primes[max(counts)] + 1, oracle_item(*spec))}
    it = mps_lib.make_item(*spec)
    with mps_lib.Siever(0) as s:
        for n in counts:
            assert s.filter(primes[:n], it) == [int(p in hits) for p in primes[:n]]
            split = n in (16384, 8192) and 10**7 // mod >= 1536
            assert s.stats()["kernel_launches"] == (6 if split else 4)
