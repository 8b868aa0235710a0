"""Waves of fewer segments than the GPU has SMs: item, batch and served calls cut them
into smaller ones, of 256, 512, 1024 or 2048 words; every size gives the oracle's
relations, for one run and for many, ragged ones."""
from __future__ import annotations

import pytest

from oracle.oracle import make_item as oracle_item

pytestmark = pytest.mark.gpu

SEGS = 148


def spec_of(lo, n_odds, k=0):
    return (7, -3 + 6 * k, lo, lo + 2 * n_odds - 1, 10, 400_000 + 1000 * k, 1, 0)


@pytest.mark.parametrize("words", [256, 512, 1024, 2048])
@pytest.mark.parametrize("segs", [SEGS // 2 + 1, SEGS - 1, SEGS])
def test_item_of_few_segments(siever, mps_lib, words, segs):
    for extra in (-7, 0, 5):
        spec = spec_of(10**10 + 4321, segs * words * 32 + extra)
        it = mps_lib.make_item(*spec)
        want = siever.chunk_relations(spec[2], spec[3], it)      # (the chunk path's sizes are tested with the oracle)
        assert want and siever.item_relations(it) == want


@pytest.mark.parametrize("n_odds", [1, 2, 4097, 8191, 8192, 8193, 70_000])
def test_smallest_items(siever, mps_lib, oracle, n_odds):
    for lo in (2, 3, 10**6, 10**12 + 1, 2**49 - 40_000):
        spec = spec_of(lo, n_odds)
        want = oracle.relations(spec[2], spec[3], oracle_item(*spec))
        assert siever.item_relations(mps_lib.make_item(*spec)) == want


def test_batch_and_server_of_ragged_runs(siever, mps_lib, oracle):
    specs = [spec_of(10**9 + 10**7 * k, 100 + 977 * k * k, k) for k in range(24)]
    items = [mps_lib.make_item(*s) for s in specs]
    want = [oracle.relations(s[2], s[3], oracle_item(*s)) for s in specs]
    got = siever.batch_relations(items)
    assert [[r[1:] for r in got if r[0] == k] for k in range(len(specs))] == want
    with mps_lib.Server(0) as sv:
        tickets = [sv.submit(it) for it in items]
        for t, w in zip(tickets, want):
            assert sv.wait(t)["done"] and sv.result(t) == w


def test_server_with_lane_groups_beyond_2_49(mps_lib, oracle):
    """Groups of lanes run the FP64 solve: a wave that reaches 2^49 takes a warp per prime."""
    spec = (3, 2, 2**49 + 1, 2**49 + 400_000, 0, 10**6, 1, 0)
    want = oracle.relations(spec[2], spec[3], oracle_item(*spec))
    with mps_lib.Server(0, tuning=mps_lib.default_tuning(table_kind=2, lanes=8)) as sv:
        t = sv.submit(mps_lib.make_item(*spec))
        assert sv.wait(t)["done"] and sv.result(t) == want
