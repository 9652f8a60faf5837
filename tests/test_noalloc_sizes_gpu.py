"""mpzmm_matmul_noalloc over its transform lengths (2^2 .. 2^15 points), shapes
and pointer alignments, against Python integers."""
import ctypes as C
import random

import numpy as np
import pytest

from rforest_b200 import _lib, api, packed as PK

pytestmark = pytest.mark.gpu


def _dev(limbs, shift):
    import torch
    words = np.zeros(2 * limbs.size + 3, np.uint32)
    words[shift:shift + 2 * limbs.size] = limbs.astype("<u8").view("<u4")
    t = torch.from_numpy(words.view(np.int32)).cuda()
    return t, t.data_ptr() + 4 * shift


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("m,k,n,bits", [
    (1, 1, 1, 30), (3, 2, 2, 60), (2, 9, 2, 500), (7, 5, 3, 2500), (4, 4, 4, 9000),
    (2, 3, 2, 40000), (1, 2, 1, 300000), (2, 1, 1, 1000000)])
def test_sizes(gpu, m, k, n, bits, shift):
    import torch
    rng = random.Random(bits + shift)
    A = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(m * k)]
    B = [rng.getrandbits(bits) * rng.choice((-1, 0, 1)) for _ in range(k * n)]
    B[0] = 1 - (1 << bits)
    pa, pb = PK.from_ints(A), PK.from_ints(B)
    cap = api.output_limbs(k, 64 * pa.max_limbs(), 64 * pb.max_limbs())
    ta, da = _dev(pa.limbs, shift)
    tb, db = _dev(pb.limbs, 0)
    dc = torch.full((m * n * cap,), 5, dtype=torch.int64, device="cuda")
    dsz = torch.full((m * n,), 777, dtype=torch.int32, device="cuda")
    co, cc = np.arange(m * n, dtype=np.int64) * cap, np.full(m * n, cap, np.int64)
    i64, i32 = _lib.i64p, _lib.i32p
    arr = [np.ascontiguousarray(x) for x in (pa.offs.astype(np.int64), pa.sizes.astype(np.int32),
                                             pb.offs.astype(np.int64), pb.sizes.astype(np.int32))]
    _lib.check(_lib.lib().mpzmm_matmul_noalloc(
        m, k, n, C.c_void_p(da), arr[0].ctypes.data_as(i64), arr[1].ctypes.data_as(i32),
        C.c_void_p(db), arr[2].ctypes.data_as(i64), arr[3].ctypes.data_as(i32),
        C.c_void_p(dc.data_ptr()), co.ctypes.data_as(i64), cc.ctypes.data_as(i64),
        C.c_void_p(dsz.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    got = PK.Packed(dc.cpu().numpy().view(np.uint64), co, dsz.cpu().numpy()).to_ints()
    assert got == [sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
                   for j in range(n)]


@pytest.mark.parametrize("bits", [900, 30000, 400000, 3000000])
def test_one_product_plan_replayed(gpu, bits):
    """The same list-free launches in a plan's CUDA graph (their blocks may come
    up before the stage in front has ended), replayed back to back."""
    rng = random.Random(bits)
    A = [rng.getrandbits(bits) * rng.choice((-1, 1)) for _ in range(4)]
    B = [rng.getrandbits(bits) for _ in range(4)]
    want = [sum(A[2 * i + q] * B[2 * q + j] for q in range(2)) for i in range(2)
            for j in range(2)]
    plan = api.Plan([(2, 2, 2, PK.from_ints(A), PK.from_ints(B))])
    plan.set_graph(True)
    for _ in range(3):
        for _ in range(5):
            plan.execute()
        assert plan.download()[0].to_ints() == want
        plan.holders[0].cl[...] = 0
    plan.close()
