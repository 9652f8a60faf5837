"""The work lists a batch sends to the device beside its operands: cutting the
batch into chunks, which run beside one another, must not make them longer."""
import pytest

from rforest_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [1 << 20, 300000])
def test_chunks_add_no_lists(gpu, chunk):
    prods = [W.random_product(3001, t, 2, 16, 10, 18) for t in range(160)]
    triples = [(p.m, p.k, p.n, p.A, p.B) for p in prods]
    sizes = [s for p in prods for x in (p.A, p.B) for s in x.sizes]
    limbs = sum(abs(int(s)) for s in sizes)
    lists, chunks, digests = [], [], []
    for c in (1 << 40, chunk):
        api.set_chunk_limbs(min(c, (1 << 31) - 1))
        try:
            outs = api.matmul_batch(triples)
        finally:
            api.set_chunk_limbs(0)
        st = api.batch_stats()
        chunks.append(st["chunks"])
        lists.append(st["h2d_bytes"] - 8 * limbs)
        digests.append([o.to_ints() for o in outs])
    assert chunks[0] == 1 and chunks[1] >= 4
    assert digests[0] == digests[1]
    # a chunk's own part: section alignment, the 256-byte phase of its copies
    # and its transforms' lists cut at its edges
    assert lists[1] <= lists[0] + lists[0] // 20 + 4096 * chunks[1]
