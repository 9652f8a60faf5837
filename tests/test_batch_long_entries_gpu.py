"""Batches in chunks whose results are long: a chunk's long entries are cut
among warps (it waits for its longest one), though the whole batch has enough
entries for a warp each."""
import random

import numpy as np
import pytest

from rforest_b200 import api, packed as PK

pytestmark = pytest.mark.gpu


def test_long_entries_of_a_chunk_are_cut(gpu):
    rng = random.Random(4)
    bits, count = 459000, 800  # results of 28,690 words
    A = [rng.getrandbits(bits) | 1 << (bits - 1) for _ in range(4)]
    B = [-(rng.getrandbits(bits) | 1 << (bits - 1)) for _ in range(4)]
    want = [sum(A[2 * i + q] * B[2 * q + j] for q in range(2)) for i in range(2) for j in range(2)]
    pa, pb = PK.from_ints(A), PK.from_ints(B)
    batch = api.Batch([(2, 2, 2, pa, pb)] * count)
    limbs = count * sum(abs(int(s)) for x in (pa, pb) for s in x.sizes)
    lists, chunks = [], []
    for size in ((1 << 31) - 1, 0):  # one chunk, automatic ones
        for h in batch.holders:
            h.cl[...] = 0
        api.set_chunk_limbs(size)
        try:
            outs = batch.run()
        finally:
            api.set_chunk_limbs(0)
        assert outs[0].to_ints() == want
        for o in outs[1:]:
            assert np.array_equal(o.limbs, outs[0].limbs) and np.array_equal(o.sizes, outs[0].sizes)
        st = api.batch_stats()
        chunks.append(st["chunks"])
        lists.append(st["h2d_bytes"] - 8 * limbs)
    assert chunks[0] == 1 and chunks[1] >= 8
    # at least four pieces an entry, 24 bytes each
    assert lists[1] - lists[0] >= 4 * 24 * 4 * count
