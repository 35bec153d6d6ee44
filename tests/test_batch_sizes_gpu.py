"""Batches on both sides of the sizes where a batch's kernels change (sorted by one CTA and without hub groups
up to 2048 updates, classified by warps up to 8192), and a split queue that overflows."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N
from tests.test_stream_gpu import edge_set, expected_after

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["apply", "pipeline"])  # the pipeline's last bin holds exactly `size`
@pytest.mark.parametrize("size", [2047, 2048, 2049, 8191, 8192, 8193])
def test_sizes_around_the_changes_of_path(size, path):
    import torch
    rng = np.random.default_rng(size)
    base = G.rmat(13, 16, seed=7)
    n = base.n
    graph = api.Graph.from_csr(base, slack=0.25)
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    T0, _ = graph.count(N.TC_PV_HANDLE, out)
    pv, delta = out.clone(), torch.zeros(1, dtype=torch.int64, device="cuda")
    pipe = api.Pipeline(graph, size) if path == "pipeline" else None
    cur = base
    for k in (0, size // 2, size):  # insertions only, half deletions, deletions only
        s, d = (a.astype(np.int32) for a in G.rmat_pairs(13, size, seed=size + k))
        pick = rng.choice(cur.m, k, replace=False)
        s[:k], d[:k] = np.repeat(np.arange(n, dtype=np.int32), np.diff(cur.off))[pick], cur.ind[pick]
        x = (np.arange(size) < k).astype(np.uint8)
        args = [torch.from_numpy(a).cuda() for a in (s, d, x)]
        if pipe:
            pipe.apply(*args, per_vertex=pv, delta_dev=delta)
            pipe.sync()
        else:
            graph.apply_batch(*args, per_vertex=pv, delta_dev=delta)
        want = expected_after(n, edge_set(cur), s, d, x)
        off, ind = graph.export()
        assert np.array_equal(off, want.off) and np.array_equal(ind, want.ind)
        cur = G.Csr(n, off, ind)
    T1, _ = graph.count(N.TC_PV_HANDLE, out)
    assert T1 == T0 + int(delta.item())
    assert torch.equal(out, pv)
    if pipe:
        pipe.close()


@pytest.mark.parametrize("path", ["apply", "sorted"])
def test_split_queue_overflow(path):
    """30,000 edges between lists of 2999 entries are 1.4 M items of 64 entries, of 2^20 that fit."""
    import torch
    base = G.complete(3000)
    n = base.n
    graph = api.Graph.from_csr(base)
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    T0, _ = graph.count(N.TC_PV_HANDLE, out)
    delta = torch.zeros(1, dtype=torch.int64, device="cuda")
    pick = np.random.default_rng(5).choice(n * (n - 1) // 2, 30000, replace=False)
    u, v = (a[pick].astype(np.int32) for a in np.triu_indices(n, 1))
    pv = out.clone()
    if path == "apply":
        sched = N.default_sched()
        sched.stream_hub_min = 0  # every edge by itself
        x = torch.ones(u.size, dtype=torch.uint8, device="cuda")
        graph.apply_batch(torch.from_numpy(u).cuda(), torch.from_numpy(v).cuda(), x, per_vertex=pv, delta_dev=delta,
                          sched=sched)
    else:
        s, d = (torch.from_numpy(np.concatenate(a)).cuda() for a in ((u, v), (v, u)))
        off = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        dup = torch.zeros(s.numel(), dtype=torch.int32, device="cuda")
        p = [t.data_ptr() for t in (s, d, off, dup)]
        N.check(N.lib().tc_batch_sort(n, p[0], p[1], s.numel(), p[2], p[3], None))
        N.check(N.lib().tc_count_batch(graph.handle, *p, s.numel(), -1, pv.data_ptr(), delta.data_ptr(), None, None))
        N.check(N.lib().tc_delete_sorted(graph.handle, p[0], p[1], p[3], s.numel(), None))
    T1, _ = graph.count(N.TC_PV_HANDLE, out)
    assert T1 == T0 + int(delta.item())
    assert torch.equal(out, pv)
