"""What the tuner times is what the class then runs: the untuned configuration it
compares with, and the sieve's segment sizes on a full wave."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

WIDEST = (3, 2, 10**11, 10**11 + 10**9, 0, 10**7, 1, 0)


def test_default_is_what_an_untuned_class_runs(mps_lib):
    """10^7 exponents run four chains untuned: the default reported is theirs, not that
    of two chains (7% slower)."""
    it = mps_lib.make_item(*WIDEST)
    ns = {}
    for name, tuning in (("untuned", {}), ("four", {"chains": 4}), ("two", {"chains": 2})):
        with mps_lib.Siever(0, **tuning) as s:
            ns[name] = min(s.autotune([it])[0]["default_ns_per_prime"] for _ in range(3))
    assert abs(ns["untuned"] - ns["four"]) < abs(ns["untuned"] - ns["two"])


def test_sieve_is_timed_on_a_full_wave(mps_lib):
    """The default segment's time in the report is that of chunk_odds odd numbers, as a
    chunk of that many shows it."""
    lo, odds = WIDEST[2], 1 << 26
    it = mps_lib.make_item(*WIDEST)
    with mps_lib.Siever(0, chunk_odds=odds) as s:
        report = s.autotune([it])[0]
        s.tune_clear()
        chunk = []
        for _ in range(4):
            s.chunk_relations(lo | 1, (lo | 1) + 2 * odds, it)
            chunk.append(s.stats()["sieve_ms"])
    assert 0.8 * min(chunk) < report["sieve_default_ms"] < 1.25 * min(chunk)
    assert report["sieve_best_ms"] <= report["sieve_default_ms"]
