"""A plan in parts over the ways it is reused: new A values for kept B
operands, an execute captured and the plan then executed again, stage times
turned on and off, two plans at once, and new inputs sent between an execute
and its download."""
import pytest

from rforest_b200 import api, packed as PK, workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(12, 2, 12, 200000), (16, 1, 16, 90000), (3, 4, 2, 3000), (16, 2, 15, 240000),
          (2, 2, 2, 1500), (14, 3, 16, 250000), (16, 2, 16, 260000), (5, 5, 5, 700)] * 2


def _products(seed):
    return [W.fixed_product(seed, t, m, k, n, b, True) for t, (m, k, n, b) in enumerate(SHAPES)]


def _copy(X):
    return PK.Packed(X.limbs.copy(), X.offs, X.sizes)


def _triples(ps):
    # copies: a plan's arrays are its operands', and set_a writes into them
    return [(p.m, p.k, p.n, _copy(p.A), _copy(p.B)) for p in ps]


def _clear(plan):
    for h in plan.holders:
        h.cl[...] = 0
        h.csz[...] = -77


def _same(got, want):
    assert len(got) == len(want)
    for t, (g, w) in enumerate(zip(got, want)):
        assert PK.digest(g) == PK.digest(w), t


def _flipped(X):
    """Other values of the same signed limb counts: every limb but the top
    ones' leading bits complemented."""
    limbs = X.limbs.copy()
    for o, s in zip(X.offs, X.sizes):
        n = abs(int(s))
        if n:
            limbs[int(o):int(o) + n - 1] ^= (1 << 64) - 1
            limbs[int(o) + n - 1] ^= (1 << (int(limbs[int(o) + n - 1]).bit_length() - 1)) - 1
    return PK.Packed(limbs, X.offs, X.sizes)


@pytest.fixture(scope="module")
def two(gpu):
    a, b = _products(77), _products(78)
    return (a, [api.matmul(*t) for t in _triples(a)]), (b, [api.matmul(*t) for t in _triples(b)])


def test_kept_b_new_a_in_every_part(gpu, two):
    ps, want = two[0]
    plan = api.Plan(_triples(ps), fixed_b=True)
    plan.execute()
    _same(plan.download(), want)
    new = [_flipped(p.A) for p in ps]
    for t, A in enumerate(new):
        plan.set_a(t, A)
    _clear(plan)
    plan.upload_a()
    plan.execute()
    _same(plan.download(), [api.matmul(p.m, p.k, p.n, A, p.B) for p, A in zip(ps, new)])
    plan.close()


def test_captured_then_executed_again(gpu, two):
    import torch
    ps, want = two[0]
    plan = api.Plan(_triples(ps))
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        plan.execute(torch.cuda.current_stream())
    for replay in (True, False, True):
        _clear(plan)
        with torch.cuda.stream(st):
            if replay:
                g.replay()
            else:
                plan.execute(st)
        _same(plan.download(st), want)
    plan.close()


def test_stage_times_on_and_off(gpu, two):
    ps, want = two[0]
    plan = api.Plan(_triples(ps))
    for on in (True, False, True, False):
        plan.set_timing(on)
        _clear(plan)
        plan.execute()
        plan.set_timing(not on)
        _same(plan.download(), want)
    assert plan.stage_times()[2] == 2
    plan.close()


def test_two_plans_at_once(gpu, two):
    import torch
    streams = [torch.cuda.Stream() for _ in two]
    plans = [api.Plan(_triples(ps), stream=st) for (ps, _), st in zip(two, streams)]
    for _ in range(2):
        for p, st in zip(plans, streams):
            _clear(p)
            p.execute(st)
        for p, st, (_, want) in zip(plans, streams, two):
            _same(p.download(st), want)
    for p in plans:
        p.close()


def test_new_inputs_between_execute_and_download(gpu, two):
    ps, want = two[0]
    plan = api.Plan(_triples(ps))
    new = [_flipped(p.A) for p in ps]
    plan.execute()
    for t, A in enumerate(new):
        plan.set_a(t, A)
    plan.upload()
    _same(plan.download(), want)
    _clear(plan)
    plan.execute()
    _same(plan.download(), [api.matmul(p.m, p.k, p.n, A, p.B) for p, A in zip(ps, new)])
    plan.close()
