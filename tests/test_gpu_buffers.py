"""Device memory of the work buffers."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_wave_buffers_per_odd_number(mps_lib):
    """The two wave slots together: at most 90 bytes per odd number of a chunk."""
    import torch

    torch.cuda.init()
    before = torch.cuda.mem_get_info()[0]
    with mps_lib.Siever(0, chunk_odds=1 << 27) as s:
        s.item_relations(mps_lib.make_item(2, -25, 10**6, 2 * 10**6, 0, 1000, 2, 1))
        used = before - torch.cuda.mem_get_info()[0]
    assert used <= 90 << 27


@pytest.mark.parametrize("odds", [1 << 20, 1 << 22, 1 << 23])
def test_every_prime_of_the_densest_chunk_fits(mps_lib, odds):
    """b = 2, c = -4 is solvable for every prime (n = 2): a chunk of the first odd
    numbers has as many entries as a chunk can have, and is done in one piece."""
    with mps_lib.Siever(0, chunk_odds=odds) as s:
        it = mps_lib.make_item(2, -4, 3, 3 + 2 * odds, 3, 50, 1, 0)
        s.chunk_relations(3, 3 + 2 * odds, it)
        st = s.stats()
        assert st["chunks"] == 1 and st["entries"] > 0.9 * s.count_primes(1000, 3 + 2 * odds)


def test_a_context_that_runs_out_of_memory(mps_lib, siever, oracle):
    """Chunks larger than the device: every call fails for want of the same buffer (none
    goes on with what the failed one left), and other contexts are unaffected."""
    from oracle.oracle import make_item as oracle_item

    spec = (2, -25, 10**6, 2 * 10**6, 0, 1000, 2, 1)
    it = mps_lib.make_item(*spec)
    want = oracle.relations(spec[2], spec[3], oracle_item(*spec))
    failed = set()
    with mps_lib.Siever(0, chunk_odds=1 << 36) as s:
        for call in (s.item_relations, lambda i: s.batch_relations([i, i])):
            for _ in range(2):
                with pytest.raises(mps_lib.MpsError, match="out of memory") as e:
                    call(it)
                assert e.value.code == mps_lib.MPS_E_CUDA
                failed.add(str(e.value))
                assert siever.chunk_relations(spec[2], spec[3], it) == want
    assert len(failed) == 1
    assert siever.item_relations(it) == want


def test_buffers_hold_survivors_not_odd_numbers(mps_lib, oracle):
    """At most 56 bytes an odd number for the two wave slots, and every survivor of the
    densest ranges still fits: the first odd numbers, and numbers beyond 65521^2."""
    import torch

    torch.cuda.init()
    before = torch.cuda.mem_get_info()[0]
    with mps_lib.Siever(0, chunk_odds=1 << 27) as s:
        s.item_relations(mps_lib.make_item(2, -25, 10**6, 2 * 10**6, 0, 1000, 2, 1))
        assert before - torch.cuda.mem_get_info()[0] <= 56 << 27
    for odds in (1 << 13, 1 << 18, 1 << 24):
        with mps_lib.Siever(0, chunk_odds=odds) as s:
            for lo in (3, 65521**2 + 2, 2**55 + 1):
                it = mps_lib.make_item(3, 2, lo, lo + 2 * odds, 0, 50, 1, 0)
                want = s.chunk_relations(lo, lo + 2 * odds, it)
                assert s.stats()["chunks"] == 1
                assert s.item_relations(it) == want and s.stats()["chunks"] == 1
                assert s.count_primes(lo, lo + 2 * odds) > 0
