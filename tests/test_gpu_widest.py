"""The widest N range (10^7) with every exponent a candidate: solutions planted at
the last exponent, the first, and around 2^23, where no single-precision quotient
is exact by its error bound.  Moduli whose power-residue split leaves period 1, 2
and 3."""
from __future__ import annotations

import random

import pytest

from oracle.oracle import make_item as oracle_item

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mod", [1, 2, 3])
@pytest.mark.parametrize("bits", [32, 45, 52])
def test_planted_at_the_ends(siever, mps_lib, oracle, mod, bits):
    rng = random.Random(bits * 10 + mod)
    lo = 1 << bits
    for p in rng.sample(oracle.primes(lo, lo + 20_000, 1 << 12), 8):
        for b in (3, 10, 2**4 * 3**4):
            for n in (10**7 - 1, 10**7 - 2, 2**23, 2**23 + 1, 0):
                spec = (b, p - pow(b, n, p), p, p + 1, 0, 10**7, mod, n % mod)
                want = oracle.relations(p, p + 1, oracle_item(*spec))
                assert siever.item_relations(mps_lib.make_item(*spec)) == want and len(want) == 1
