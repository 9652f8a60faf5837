"""The tensor-core contraction of products with one frequency a group (more
than 16 rows or 32 columns): block and term remainders, terms around the
16-byte pieces, transforms shorter than the staged frequencies.  Exact against
Python integers."""
import random

import pytest

from rforest_b200 import api, packed as PK

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,bits", [
    (17, 1, 1, 120), (17, 15, 3, 700), (32, 16, 32, 300), (33, 17, 31, 300), (20, 31, 35, 90),
    (3, 33, 40, 1500), (64, 64, 64, 60), (40, 48, 65, 200), (18, 63, 5, 4000),
    (17, 20, 33, 9000)])
def test_shapes(gpu, m, k, n, bits):
    rng = random.Random(m * 100 + k)
    A = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(m * k)]
    B = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(k * n)]
    before = api.contract_mode()
    api.set_contract_mode(2)
    try:
        got = api.matmul(m, k, n, PK.from_ints(A), PK.from_ints(B)).to_ints()
    finally:
        api.set_contract_mode(before)
    assert got == [sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
                   for j in range(n)]
