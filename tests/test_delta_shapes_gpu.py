"""The delta count without a tuned plan: batches on both sides of the sizes where the default split-item
shape and the work per queue grab change, with and without hub groups, against static recounts."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hub_min", [0, 8])
@pytest.mark.parametrize("path", ["pipeline", "apply"])
@pytest.mark.parametrize("size", [1, 2, 1500, 40000, 80000])  # 70 % insertions: 28000 and 56000 of them
def test_default_shapes_match_recounts(size, path, hub_min):
    import torch
    rng = np.random.default_rng(size)
    base = G.rmat(15, 16, seed=7)
    n = base.n
    graph = api.Graph.from_csr(base, slack=0.25)
    sched = N.default_sched()
    sched.stream_hub_min = hub_min
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    T0, _ = graph.count(N.TC_PV_HANDLE, out)
    pv = out.clone()
    delta = torch.zeros(1, dtype=torch.int64, device="cuda")
    s, d = G.rmat_pairs(15, size, seed=11)
    x = np.zeros(size, np.uint8)
    k = int(0.3 * size)
    pick = rng.integers(0, base.m, k)
    s[:k] = np.repeat(np.arange(n, dtype=np.int32), base.degrees())[pick]
    d[:k] = base.ind[pick]
    x[:k] = 1
    args = [torch.from_numpy(a).cuda() for a in (s, d, x)]
    if path == "pipeline":
        pipe = api.Pipeline(graph, size, sched=sched)
        pipe.apply(*args, per_vertex=pv, delta_dev=delta)
        pipe.sync()
        pipe.close()
    else:
        graph.apply_batch(*args, per_vertex=pv, delta_dev=delta, sched=sched)
    T1, _ = graph.count(N.TC_PV_HANDLE, out)
    assert T1 == T0 + int(delta.item())
    assert torch.equal(out, pv)
