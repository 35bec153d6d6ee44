"""The meeting of the delta kernel's CTAs, made to run out at once: whichever CTAs leave, no list may be
rewritten while another CTA still counts it, and all of the phase's end must be done."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N
from tests.test_stream_gpu import edge_set, expected_after, random_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wait_ns", [1, 2000, 20000])  # before, around and after the first arrivals
@pytest.mark.parametrize("extra", [0, 1])
@pytest.mark.parametrize("size", [1, 600, 6000])
def test_a_meeting_that_runs_out_changes_no_result(size, extra, wait_ns):
    import torch
    rng = np.random.default_rng(size + extra)
    base = G.rmat(13, 16, seed=3)
    n = base.n
    graph = api.Graph.from_csr(base, slack=0.25)
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    T0, _ = graph.count(N.TC_PV_HANDLE, out)
    pv, delta = out.clone(), torch.zeros(1, dtype=torch.int64, device="cuda")
    pipe = api.Pipeline(graph, size)
    pipe.set_wait_bound(wait_ns, extra)
    cur = base
    for _ in range(3):
        s, d, x = random_batch(rng, cur, size)
        pipe.apply(*[torch.from_numpy(a).cuda() for a in (s, d, x)], per_vertex=pv, delta_dev=delta)
        try:
            pipe.sync()
            assert extra == 0
        except N.TcError as e:
            assert e.status == N.TC_ERR_TIMEOUT
        want = expected_after(n, edge_set(cur), s, d, x)
        off, ind = graph.export()
        assert np.array_equal(off, want.off) and np.array_equal(ind, want.ind)
        cur = G.Csr(n, off, ind)
    T1, _ = graph.count(N.TC_PV_HANDLE, out)
    assert T1 == T0 + int(delta.item())
    assert torch.equal(out, pv)
    pipe.close()
