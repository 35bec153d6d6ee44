"""tc_count_batch on both sides of the sizes where its grid stops growing (8 and 32 CTAs of eight entries an
SM, 9472 and 37888 entries on 148 SMs): the deletion count of present edges against static recounts."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [1, 4, 4735, 4736, 4737, 18943, 18944, 18945])
def test_deletion_count_against_recounts(edges):
    import torch
    base = G.rmat(13, 16, seed=3)
    n = base.n
    graph = api.Graph.from_csr(base)
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    T0, _ = graph.count(N.TC_PV_HANDLE, out)
    before = out.clone()
    row = np.repeat(np.arange(n, dtype=np.int64), np.diff(base.off))
    up = np.flatnonzero(row < base.ind)
    pick = np.random.default_rng(edges).choice(up, edges, replace=False)
    x, y = row[pick], base.ind[pick].astype(np.int64)
    keys = np.sort(np.r_[x * n + y, y * n + x])
    s, d = (keys // n).astype(np.int32), (keys % n).astype(np.int32)
    off = np.searchsorted(s, np.arange(n + 1)).astype(np.int32)
    s, d, off, dup = (torch.from_numpy(a).cuda() for a in (s, d, off, np.zeros(len(keys), np.int32)))
    pv = torch.zeros(n, dtype=torch.int32, device="cuda")
    delta = torch.zeros(1, dtype=torch.int64, device="cuda")
    N.check(N.lib().tc_count_batch(graph.handle, s.data_ptr(), d.data_ptr(), off.data_ptr(), dup.data_ptr(), len(keys),
                                   -1, pv.data_ptr(), delta.data_ptr(), None, None))
    N.check(N.lib().tc_delete_sorted(graph.handle, s.data_ptr(), d.data_ptr(), dup.data_ptr(), len(keys), None))
    T1, _ = graph.count(N.TC_PV_HANDLE, out)
    assert T1 == T0 + int(delta.item())
    assert torch.equal(out, before + pv)
