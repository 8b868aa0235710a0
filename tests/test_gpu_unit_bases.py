"""Items with |b| <= 1 (b^n takes one or two values), and primes for which the
candidates' step B = b^L is 1 or -1: relations equal the oracle's, and no
baby-step giant-step solve is spent on them."""
from __future__ import annotations

import pytest

from oracle.oracle import make_item as oracle_item

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [1, -1, 0])
@pytest.mark.parametrize("mod,res", [(1, 0), (2, 1), (6, 4)])
@pytest.mark.parametrize("P0", [900, 10**9, (1 << 49) - 50_000])
def test_unit_bases(siever, mps_lib, oracle, b, mod, res, P0):
    width = 100_000
    in_range = [p for p in oracle.primes(P0, P0 + width, 1 << 16) if p >= 1000]
    # c = -1 and 1: solved by every prime or none; c = a prime of the range +-1: by that prime alone
    for c in (-1, 1, in_range[3] - 1, in_range[7] + 1, in_range[11]):
        spec = (b, c, P0, P0 + width, 5, 5 + 6 * 200_000, mod, res)
        it = mps_lib.make_item(*spec)
        want = oracle.relations(spec[2], spec[3], oracle_item(*spec))
        assert siever.item_relations(it) == want
        assert siever.stats()["bsgs_steps"] == 0
        assert siever.chunk_relations(P0, P0 + width, it) == want
        assert siever.stats()["bsgs_steps"] == 0
        assert siever.filter(in_range, it) == [int(p in {r[0] for r in want}) for p in in_range]


@pytest.mark.parametrize("p,b", [(2147483647, 2), (2147483647, 2**31 - 2), (4278255361, 4278255360), (65537, 2)])
def test_step_of_order_one_and_two(siever, mps_lib, oracle, p, b):
    for c in (-1, 1, 3, -8, p - 4):
        for mod, res in ((1, 0), (31, 3), (16, 7)):
            spec = (b, c, p, p + 1, 0, 9_000_000, mod, res)
            want = oracle.relations(p, p + 1, oracle_item(*spec))
            assert siever.item_relations(mps_lib.make_item(*spec)) == want
