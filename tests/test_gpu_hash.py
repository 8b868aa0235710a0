"""The fingerprint tables on both sides of 2^30, where the hash's multiplier changes:
every kind and chain count that uses them gives the oracle's relations."""
from __future__ import annotations

import pytest

from oracle.oracle import make_item as oracle_item

pytestmark = pytest.mark.gpu

SPAN = 60_000


@pytest.mark.parametrize("table_kind", [0, 3])
@pytest.mark.parametrize("chains", [1, 2, 4])
def test_relations_around_the_change(mps_lib, oracle, table_kind, chains):
    with mps_lib.Siever(0, table_kind=table_kind, chains=chains) as s:
        for lo in (10**6, 2**30 - SPAN, 2**30 - SPAN // 2, 2**30):
            spec = (7, -2, lo, lo + SPAN, 3, 2_000_003, 1, 0)
            want = oracle.relations(lo, lo + SPAN, oracle_item(*spec))
            it = mps_lib.make_item(*spec)
            assert len(want) > 1 and s.item_relations(it) == want and s.chunk_relations(lo, lo + SPAN, it) == want
            primes = oracle.primes(lo, lo + SPAN, 1 << 14)
            assert [p for p, f in zip(primes, s.filter(primes, it)) if f] == [r[0] for r in want]
