"""filter on primes in any order: ascending lists (with repeats) and shuffled
ones take different ways to their flags, which must be the oracle's."""
from __future__ import annotations

import random

import pytest

from oracle.oracle import make_item as oracle_item

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["ascending", "repeated", "shuffled", "descending", "one"])
def test_filter_flags_in_any_order(siever, mps_lib, oracle, order):
    spec = (2, -25, 10**6, 10**6 + 200_000, 0, 60_000, 2, 1)
    primes = oracle.primes(spec[2], spec[3], 1 << 16)
    want = {r[0] for r in oracle.relations(spec[2], spec[3], oracle_item(*spec))}
    if order == "repeated":
        primes = sorted(primes + primes[::3])
    elif order == "shuffled":
        random.Random(5).shuffle(primes)
    elif order == "descending":
        primes = primes[::-1]
    elif order == "one":
        primes = [min(want)]
    assert want and siever.filter(primes, mps_lib.make_item(*spec)) == [int(p in want) for p in primes]
