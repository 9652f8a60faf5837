"""Transforms of every length and digit count through whole products: both
factors short enough for the half-zero first pass, and one long factor against
a short one (every coefficient of the transform in use); few entries (primes
cut among CTAs) and many (all primes in a CTA).  Exact against Python
integers."""
import random

import pytest

from rforest_b200 import api, packed as PK

pytestmark = pytest.mark.gpu


def _check(m, k, n, a_bits, b_bits, mode):
    rng = random.Random(a_bits * 7 + b_bits)
    A = [rng.getrandbits(a_bits) * rng.choice((-1, 1)) for _ in range(m * k)]
    B = [rng.getrandbits(b_bits) * rng.choice((-1, 1)) for _ in range(k * n)]
    before = api.contract_mode()
    api.set_contract_mode(mode)
    try:
        got = api.matmul(m, k, n, PK.from_ints(A), PK.from_ints(B)).to_ints()
    finally:
        api.set_contract_mode(before)
    assert got == [sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
                   for j in range(n)]


# equal factors: 2^2 .. 2^15 points
@pytest.mark.parametrize("bits", [40, 150, 400, 800, 1500, 3000, 6000, 12000, 25000, 50000,
                                  100000, 200000, 420000, 900000, 1900000])
@pytest.mark.parametrize("mode", [1, 2])
def test_lengths(gpu, bits, mode):
    _check(2, 1, 2, bits, bits, mode)


# a long factor against a short one
@pytest.mark.parametrize("bits", [300, 1300, 5000, 21000, 90000, 350000, 1500000])
def test_long_by_short(gpu, bits):
    _check(1, 2, 1, bits, 70, 1)


@pytest.mark.parametrize("bits,dim", [(700, 24), (9000, 14), (70000, 10)])
def test_many_entries(gpu, bits, dim):
    _check(dim, 3, dim, bits, bits, 1)
