"""What the server counts for a request against its device budget covers what
the request's plan takes: long results carry segment records and longer work
lists."""
import re

import pytest

from rforest_b200 import _lib, api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def estimate(gpu):
    """The estimate of a request, from the refusal of a server without room."""
    srv = api.Server(budget_bytes=1, slots=1)

    def of(p):
        with pytest.raises(_lib.MpzmmError) as e:
            srv.submit(p.m, p.k, p.n, p.A, p.B)
        return int(re.search(r"needs (\d+) device bytes", str(e.value)).group(1))
    yield of
    srv.close()


# the last one splits its contraction finely (many tiles, short transforms)
@pytest.mark.parametrize("shapes", [
    [(1, 1, 1, 3000000)], [(2, 2, 2, 400000)], [(4, 3, 5, 60000)], [(2, 1, 2, 9000)],
    [(1, 1, 1, 700000), (2, 3, 1, 200000), (3, 1, 3, 40000)],
    [(40, 1, 40, 300), (3, 2, 3, 20000)]])
@pytest.mark.parametrize("mode", [1, 2])
def test_estimate_covers_the_plan(gpu, estimate, shapes, mode):
    ps = [W.fixed_product(5, t, m, k, n, b, True) for t, (m, k, n, b) in enumerate(shapes)]
    before = api.contract_mode()
    api.set_contract_mode(mode)
    try:
        counted = sum(estimate(p) for p in ps)
        plan = api.Plan([(p.m, p.k, p.n, p.A, p.B) for p in ps])
        taken = plan.info()["device_bytes"]
        plan.close()
    finally:
        api.set_contract_mode(before)
    assert taken <= counted
