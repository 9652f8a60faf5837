"""The CUDA-core contraction over shapes whose tiles are split among CTAs or
whose blocks of positions span primes: rows, columns, inner products, single
entries, edges of the 1 to 4 wide register tiles.  Exact against Python
integers."""
import random

import pytest

from rforest_b200 import api, packed as PK

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,bits", [
    (700, 1, 1, 500), (1, 1, 700, 500), (1, 300, 1, 700), (257, 2, 3, 60), (3, 2, 257, 60),
    (1, 1, 1, 20), (5, 17, 1, 3000), (1, 16, 5, 3000), (9, 31, 7, 900), (33, 3, 33, 200),
    (2, 2, 2, 300000)])
def test_shapes(gpu, m, k, n, bits):
    rng = random.Random(m * 1000 + n)
    A = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(m * k)]
    B = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(k * n)]
    before = api.contract_mode()
    api.set_contract_mode(1)
    try:
        got = api.matmul(m, k, n, PK.from_ints(A), PK.from_ints(B)).to_ints()
    finally:
        api.set_contract_mode(before)
    assert got == [sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
                   for j in range(n)]
