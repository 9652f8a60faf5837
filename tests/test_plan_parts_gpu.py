"""A plan whose results are large enough to run in parts: results, info and
times equal those of the products alone, over repeated executes, graph mode,
kept B operands, an execute captured into a caller's graph, and a capacity
error in one part."""
import ctypes as C

import pytest

from rforest_b200 import _lib, api, workloads as W

pytestmark = pytest.mark.gpu


def _products():
    # about 100 MB of results: more than the four parts' minimum
    shapes = [(12, 2, 12, 200000), (16, 1, 16, 90000), (3, 4, 2, 3000), (16, 2, 15, 240000),
              (2, 2, 2, 1500), (14, 3, 16, 250000), (16, 2, 16, 260000), (5, 5, 5, 700)]
    return [W.fixed_product(77, t, m, k, n, b, True) for t, (m, k, n, b) in enumerate(shapes * 2)]


def _same(got, want):
    return all(g.to_ints() == w.to_ints() for g, w in zip(got, want))


@pytest.fixture(scope="module")
def batch(gpu):
    ps = [(p.m, p.k, p.n, p.A, p.B) for p in _products()]
    return ps, [api.matmul(*p) for p in ps]


@pytest.mark.parametrize("graph", [False, True])
def test_parts(gpu, batch, graph):
    ps, want = batch
    plan = api.Plan(ps)
    plan.set_graph(graph)
    for _ in range(2):
        plan.execute()
        assert _same(plan.download(), want)
        for h in plan.holders:
            h.cl[...] = 0
    one = api.Plan(ps[-3:-2])
    assert [plan.info(len(ps) - 3)[x] for x in ("P", "r", "lgN")] == [
        one.info()[x] for x in ("P", "r", "lgN")]
    one.close()
    plan.set_timing(True)
    plan.execute()
    plan.download()
    ms, launches, executes = plan.stage_times()
    assert executes == 1 and all(x > 0 for x in ms)
    assert sum(launches) == plan.info()["launches"]
    plan.close()


def test_parts_kept_b(gpu, batch):
    ps, want = batch
    plan = api.Plan(ps, fixed_b=True)
    for _ in range(2):
        plan.execute()
        assert _same(plan.download(), want)
        plan.upload_a()
    plan.close()


def test_parts_captured_by_the_caller(gpu, batch):
    import torch
    ps, want = batch
    plan = api.Plan(ps)
    plan.execute()
    assert _same(plan.download(), want)
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        plan.execute(torch.cuda.current_stream())
    for h in plan.holders:
        h.cl[...] = 0
    with torch.cuda.stream(st):
        g.replay()
    assert _same(plan.download(st), want)
    plan.close()


def test_capacity_error_in_one_part(gpu, batch):
    ps, want = batch
    holders = [api.holder(*p) for p in ps]
    holders[-2].caps[...] = 3  # read when the plan is made
    arr = (_lib.Product * len(holders))(*[h.struct for h in holders])
    L, plan = _lib.lib(), C.c_void_p()
    _lib.check(L.mpzmm_plan_create(C.byref(plan), len(holders), arr, None))
    _lib.check(L.mpzmm_plan_execute(plan, None))
    assert L.mpzmm_plan_download(plan, None) == _lib.MPZMM_ERR_CAPACITY
    L.mpzmm_plan_destroy(plan)
    for t, (h, w) in enumerate(zip(holders, want)):
        if t != len(holders) - 2:
            assert h.result().to_ints() == w.to_ints()
