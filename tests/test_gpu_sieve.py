"""The sieve's segment sizes: a range shorter than 148 segments is cut into
smaller ones, so the ranges here lie on both sides of each switch, ragged."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

SEGS = 148


@pytest.mark.parametrize("words", [256, 512, 1024, 2048])
@pytest.mark.parametrize("extra", [-1, 0, 31])
def test_survivors_on_both_sides_of_a_segment_size(siever, oracle, words, extra):
    n_odds = SEGS * words * 32 + extra
    lo = 10**10 + 4321
    hi = lo + 2 * n_odds
    assert siever.survivors(lo, hi, cap=1 << 20) == oracle.survivors(lo, hi, 1 << 21)
