"""A plan that runs in parts stays at its caller's priority: captured into a
graph, none of its kernels ranks above the stream it was executed on (a
smaller number ranks higher)."""
import pytest

from rforest_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("priority", [0, -2])
def test_no_kernel_above_the_callers_stream(gpu, priority):
    import torch
    from cuda.bindings import driver as D

    def ok(r):
        assert r[0] == D.CUresult.CUDA_SUCCESS, r[0]
        return r[1:] if len(r) > 2 else (r[1] if len(r) == 2 else None)

    shapes = [(12, 2, 12, 200000), (16, 1, 16, 90000), (16, 2, 15, 240000), (16, 2, 16, 260000)]
    ps = [W.fixed_product(77, t, m, k, n, b, True) for t, (m, k, n, b) in enumerate(shapes * 3)]
    st = torch.cuda.Stream(priority=priority)
    assert st.priority == priority
    plan = api.Plan([(p.m, p.k, p.n, p.A, p.B) for p in ps], stream=st)
    plan.execute(st)  # whatever is created on first use
    st.synchronize()
    ok(D.cuStreamBeginCapture(st.cuda_stream,
                              D.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL))
    plan.execute(st)
    graph = ok(D.cuStreamEndCapture(st.cuda_stream))
    count = ok(D.cuGraphGetNodes(graph, 0))[1]
    nodes = ok(D.cuGraphGetNodes(graph, count))[0]
    seen = []
    for node in nodes:
        if ok(D.cuGraphNodeGetType(node)) != D.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        value = ok(D.cuGraphKernelNodeGetAttribute(
            node, D.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_PRIORITY))
        seen.append(value.priority)
    ok(D.cuGraphDestroy(graph))
    plan.close()
    assert len(seen) >= 16  # four stages of several parts
    assert priority in seen and min(seen) >= priority, sorted(set(seen))
