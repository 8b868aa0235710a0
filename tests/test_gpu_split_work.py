"""The split by primes l | p - 1 does its work: relations alone would not show a
split that no longer happens, so the baby and giant steps left are compared,
on every path, with those of the power-residue split alone."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

# b, c, P0, width, N0, N1, mod, res: both arithmetics; widths below and above 148 segments of the sieve
ITEMS = [(3, 2, 10**9, 1 << 21, 0, 10**7, 1, 0), (10, 111, 10**12, 1 << 25, 0, 10**7, 6, 4),
         (3, 2, 2**49, 1 << 22, 0, 2_000_000, 1, 0)]


@pytest.mark.parametrize("b,c,P0,width,N0,N1,mod,res", ITEMS)
def test_steps_left_by_the_split(mps_lib, b, c, P0, width, N0, N1, mod, res):
    it = mps_lib.make_item(b, c, P0, P0 + width, N0, N1, mod, res)
    steps, entries, relations = {}, {}, {}
    for name, tuning in (("split", {}), ("unsplit", {"class_modulus": 144})):
        with mps_lib.Siever(0, chains=2, **tuning) as s:
            relations[name] = s.chunk_relations(P0, P0 + width, it)
            steps[name, "chunk"], entries[name] = s.stats()["bsgs_steps"], s.stats()["entries"]
            assert s.item_relations(it) == relations[name]
            steps[name, "wave"] = s.stats()["bsgs_steps"]
    assert relations["split"] == relations["unsplit"] and entries["split"] == entries["unsplit"]
    for path in ("chunk", "wave"):
        assert steps["split", path] < 0.55 * steps["unsplit", path]
    # of two l of one size class the sieve keeps either one
    assert abs(steps["split", "chunk"] - steps["split", "wave"]) < 0.01 * steps["split", "chunk"]


@pytest.mark.parametrize("b,c,P0,width,N0,N1,mod,res", ITEMS)
def test_given_primes_are_split_as_sieved_ones(mps_lib, oracle, b, c, P0, width, N0, N1, mod, res):
    width = min(width, 1 << 22)
    primes = oracle.primes(P0, P0 + width, 1 << 19)
    it = mps_lib.make_item(b, c, P0, P0 + width, N0, N1, mod, res)
    with mps_lib.Siever(0) as s:
        want = s.chunk_relations(P0, P0 + width, it)
        sieved = s.stats()
        flags = s.filter(primes, it)
        given = s.stats()
    assert [p for p, f in zip(primes, flags) if f] == [r[0] for r in want]
    assert given["entries"] == sieved["entries"]
    assert abs(given["bsgs_steps"] - sieved["bsgs_steps"]) < 0.01 * sieved["bsgs_steps"]


def test_no_split_of_a_given_prime_is_lost(mps_lib, oracle):
    """filter in a context whose buffers fit the list, all of whose primes are entries
    (b = 2, c = -4: n = 2 solves every prime, N0 = 3 leaves it out): as many steps as
    in a context with larger buffers."""
    lo = 10**9
    primes = oracle.primes(lo, lo + (1 << 21), 1 << 18)
    it = mps_lib.make_item(2, -4, lo, lo + (1 << 21), 3, 5_000_003, 1, 0)
    with mps_lib.Siever(0) as s:
        s.filter(primes, it)
        fitted = s.stats()
        s.chunk_relations(lo, lo + 1000, it)                  # (a chunk's buffers are larger)
        s.filter(primes, it)
        large = s.stats()
    assert fitted["entries"] == len(primes)
    assert fitted["bsgs_steps"] == large["bsgs_steps"]


def test_full_event_lists_lose_no_relation(mps_lib):
    """70,000 primes p == 1 (mod 5 7 11 13 17 19): six small l each, eight times what the
    list holds.  Flags and relations as without the split."""
    step = 2 * 5 * 7 * 11 * 13 * 17 * 19
    with mps_lib.Siever(0, class_modulus=144) as s:
        cand = [1 + step * k for k in range(1000, 900_000)]
        primes = [p for p, f in zip(cand, s.is_prime(cand)) if f][:70_000]
        assert len(primes) == 70_000
        it = mps_lib.make_item(3, 2, primes[0], primes[-1] + 1, 0, 10**7, 1, 0)
        want = s.filter(primes, it)
    assert 0 < sum(want) < 70_000
    with mps_lib.Siever(0) as s:
        for _ in range(2):
            assert s.filter(primes, it) == want
