"""tc_sched.chunk: the vertices a warp claims at a time, by the graph's size unless a caller gives a number."""
import statistics

import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


def _time(graph, out, chunk):
    import torch
    sched = N.default_sched()
    if chunk is not None:
        sched.chunk = chunk
    T, _ = graph.count(N.TC_PV_HANDLE, out, sched=sched)
    ms = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.count(N.TC_PV_HANDLE, out, sched=sched, sync=False)
        b.record()
        torch.cuda.synchronize()
        ms.append(a.elapsed_time(b))
    return T, out.clone(), statistics.median(ms)


def test_one_claim_of_every_vertex_is_one_warps_work():
    import torch
    g = G.erdos_renyi(1 << 14, 16.0 / (1 << 14), seed=1)
    graph = api.Graph.from_csr(g)
    out = torch.zeros(g.n, dtype=torch.int32, device="cuda")
    T0, pv0, base = _time(graph, out, None)
    T1, pv1, one = _time(graph, out, g.n)
    assert T1 == T0 and torch.equal(pv1, pv0)
    assert one > 4 * base  # 16384 centres in one warp after one another, against at most 5920 warps


@pytest.mark.parametrize("chunk", [-1, 0, 1, 31, 33, 64, 2**31 - 1])
def test_every_claim_size_counts_the_same(chunk):
    import torch
    g = G.rmat(11, 16, seed=4)
    graph = api.Graph.from_csr(g)
    out = torch.zeros(g.n, dtype=torch.int32, device="cuda")
    T0, pv0, _ = _time(graph, out, None)
    T1, pv1, _ = _time(graph, out, chunk)
    assert T1 == T0 and torch.equal(pv1, pv0)
