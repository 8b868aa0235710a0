"""The hash of the baby-step tables (fq_hash), compiled for the host:
the fingerprints of residues are spread over their whole range for primes of every size."""
from __future__ import annotations

import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "arith.cuh"
#include <cstdio>
int main() {
    unsigned long long p, c;
    while (scanf("%llu %llu", &p, &c) == 2) printf("%u\n", mps::fq_hash((double)c, p < mps::kHashLow ? mps::kHashKLow : mps::kHashK));
}
"""
PRIMES = (1_000_003, 10_000_019, 100_000_007, 1_000_000_007, 1_000_000_000_039, 2**48 + 21, 2**49 - 81)


@pytest.fixture(scope="module")
def hashes(tmp_path_factory):
    d = tmp_path_factory.mktemp("hash")
    src, exe = d / "h.cu", d / "h"
    src.write_text(SRC)
    subprocess.run(["nvcc", "-std=c++17", "-I", os.path.join(ROOT, "mass-prime-siever_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True, capture_output=True)

    def run(pairs):
        text = "\n".join(f"{p} {c}" for p, c in pairs)
        out = subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True).stdout.split()
        return [int(x) for x in out]

    return run


def test_the_sum_stays_in_one_binade(hashes):
    """c k rounded to the unit 1/2, below 2^50: the hash is its 32 low bits."""
    from fractions import Fraction

    k = {True: Fraction(1.6180339887498949) * 2**19, False: Fraction(1.6180339887498949)}
    pairs = [(p, c) for p in (3, 1009, 2**20, 2**30 - 1, 2**30, 2**49 - 1) + PRIMES for c in (0, 1, p // 3, p - 1)]
    for (p, c), h in zip(pairs, hashes(pairs)):
        x = c * k[p < 2**30]
        assert x < 2**50 and h == round(2 * x) % 2**32


@pytest.mark.parametrize("p", PRIMES)
def test_fingerprints_of_baby_steps(hashes, p):
    """Of the 16,384 fingerprints, 65,536 residues leave out 1 in e^4: 16,084 are
    expected, with a deviation of 17."""
    rng = random.Random(p)
    B, x, pairs = rng.randrange(2, p), rng.randrange(1, p), []
    for _ in range(65_536):                                 # the baby steps t B^i
        pairs.append((p, x))
        x = x * B % p
    h = hashes(pairs)
    assert len({(v >> 16) & 0x3FFF for v in h}) >= 16_084 - 10 * 17
