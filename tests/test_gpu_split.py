"""The split by primes l | p - 1 and the lane solve: exponent counts on both
sides of every limit, class moduli that hold split primes themselves, bases
that are l-th powers, and primes beyond 2^49 (integer arithmetic) with planted
solutions.  Relations are compared with the oracle's, exactly, on the sieved
path, on the given-primes path and with the split off (an explicit modulus)."""
from __future__ import annotations

import random

import pytest

from oracle.oracle import make_item as oracle_item

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def unsplit(mps_lib):
    with mps_lib.Siever(0, class_modulus=720720) as s:
        yield s


@pytest.mark.parametrize("K", [1, 2, 17, 64, 65, 511, 513, 1023, 1025, 4095, 4097, 65_537, 1_600_003])
def test_exponent_counts(siever, unsplit, mps_lib, oracle, K):
    for b, c, mod, res in ((2, -25, 1, 0), (10, 111, 6, 4)):
        spec = (b, c, 1000, 1_500_000, 12_345, 12_345 + K * mod, mod, res)
        it = mps_lib.make_item(*spec)
        want = oracle.relations(spec[2], spec[3], oracle_item(*spec))
        assert siever.item_relations(it) == want
        assert unsplit.item_relations(it) == want
        primes = oracle.primes(spec[2], spec[3], 1 << 18)
        assert [p for p, f in zip(primes, siever.filter(primes, it)) if f] == [r[0] for r in want]


@pytest.mark.parametrize("mod,res", [(23, 5), (29 * 31, 400), (4 * 101, 6), (4253, 17), (5 * 7 * 11 * 13 * 17, 3)])
@pytest.mark.parametrize("b", [3, 2**23, 3**5, -7])
def test_class_moduli_and_power_bases(siever, mps_lib, oracle, mod, res, b):
    spec = (b, 7, 10**6, 10**6 + 1_500_000, 0, 3_000_000, mod, res)
    assert siever.item_relations(mps_lib.make_item(*spec)) == oracle.relations(spec[2], spec[3], oracle_item(*spec))


@pytest.mark.parametrize("bits", [33, 40, 48, 49, 50, 57, 61])
def test_planted_solutions(siever, mps_lib, oracle, bits):
    """b^n + c == 0 (mod p) for a chosen n: the first, the last, and others in between."""
    rng = random.Random(bits)
    lo = (1 << bits) - 30_000 if bits != 49 else 1 << 49
    for p in rng.sample(oracle.primes(lo, lo + 30_000, 1 << 12), 12):
        b = rng.choice([2, 3, 10, 12, 1_000_003])
        N0, K, mod = rng.randrange(10**6), rng.choice([50, 3_000, 200_000, 1_600_000]), rng.choice([1, 2, 6])
        N1 = N0 + K * mod
        n = rng.choice([N0, N1 - 1, rng.randrange(N0, N1)])
        spec = (b, p - pow(b, n, p), p, p + 1, N0, N1, mod, n % mod)
        want = oracle.relations(p, p + 1, oracle_item(*spec))
        assert len(want) == 1
        it = mps_lib.make_item(*spec)
        assert siever.item_relations(it) == want
        assert siever.filter([p], it) == [1]
