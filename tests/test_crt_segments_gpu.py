"""Output entries that several warps recompose in segments: carries that run
through whole segments (powers of two, all ones, zero, minus one, short
results under a long bound), signs, and lengths around the segment edges.
Exact against Python integers."""
import random

import pytest

from rforest_b200 import api, packed as PK

pytestmark = pytest.mark.gpu


def _check(m, k, n, A, B):
    want = [sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
            for j in range(n)]
    assert api.matmul(m, k, n, PK.from_ints(A), PK.from_ints(B)).to_ints() == want


# bit lengths whose results lie around two and three segments of 224 words,
# around whole tiles, and well above
@pytest.mark.parametrize("bits", [7100, 7168, 7232, 10700, 10752, 10817, 16400, 50000, 131071])
def test_segment_edges(gpu, bits):
    rng = random.Random(bits)
    A = [rng.getrandbits(bits) | 1 << (bits - 1) for _ in range(4)]
    B = [-(rng.getrandbits(bits) | 1 << (bits - 1)), rng.getrandbits(bits // 3), 0,
         rng.getrandbits(bits)]
    _check(2, 2, 2, A, B)


@pytest.mark.parametrize("bits", [9000, 30001, 100000])
def test_carries_through_segments(gpu, bits):
    rng = random.Random(7 * bits)
    x, y = rng.getrandbits(bits) | 1, rng.getrandbits(bits // 2) | 1
    one = 1 << (bits - 1)
    # second column entries of x y size cancel the first term down to a short
    # value under a bound of several thousand words
    tails = [0, -1, 1, -(1 << (bits // 2)), 1 << (bits // 2), (1 << bits) - 1, -(1 << bits),
             1 - (1 << bits), -5]
    B = [y] * len(tails) + [-x * y + t for t in tails]
    _check(1, 2, len(tails), [x, 1], B)
    # powers of two, all ones, and their negatives
    A = [one, -one, 2 * one - 1, 1 - 2 * one]
    _check(4, 1, 4, A, [one, -one, 2 * one - 1, -1])


def test_long_entries_mixed_with_short(gpu):
    rng = random.Random(3)
    prods, wants = [], []
    for m, k, n, bits in [(1, 1, 1, 900000), (3, 2, 3, 300), (2, 2, 1, 40000), (1, 3, 2, 8000)]:
        A = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(m * k)]
        B = [rng.getrandbits(bits) * rng.choice((-1, 0, 1)) for _ in range(k * n)]
        prods.append((m, k, n, PK.from_ints(A), PK.from_ints(B)))
        wants.append([sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
                      for j in range(n)])
    for got, want in zip(api.matmul_batch(prods), wants):
        assert got.to_ints() == want
