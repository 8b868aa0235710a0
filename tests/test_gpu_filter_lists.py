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
