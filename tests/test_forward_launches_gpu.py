"""Operands of tensor-core and of CUDA-core products share the forward
launches: one for each digit count of the transforms that share a CTA."""
import random

import pytest

from rforest_b200 import api, packed as PK

pytestmark = pytest.mark.gpu


def test_one_launch_for_both_engines(gpu):
    rng = random.Random(9)
    # up to 64 terms on tensor cores, more on CUDA cores
    shapes = [(3, 16, 4, 900), (3, 16, 4, 6000), (2, 70, 3, 900), (2, 70, 3, 6000), (40, 20, 36, 900)]
    prods, wants = [], []
    for m, k, n, bits in shapes:
        A = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(m * k)]
        B = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(k * n)]
        prods.append((m, k, n, PK.from_ints(A), PK.from_ints(B)))
        wants.append([sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
                      for j in range(n)])
    before = api.contract_mode()
    api.set_contract_mode(2)
    try:
        plan = api.Plan(prods)
    finally:
        api.set_contract_mode(before)
    plan.set_timing(True)
    plan.execute()
    for got, want in zip(plan.download(), wants):
        assert got.to_ints() == want
    _, launches, _ = plan.stage_times()
    infos = [plan.info(t) for t in range(len(prods))]
    plan.close()
    assert launches[1] == 2  # both engines
    assert max(i["lgN"] for i in infos) <= 11  # several transforms a CTA
    assert launches[0] == len({(i["r"] + 29) // 30 for i in infos})
