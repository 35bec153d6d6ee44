"""tc_insert_sorted takes the caller's word for what is a duplicate: a self-loop that is not flagged goes into
its vertex's list like any other entry, also that of the last id, whose key has only ones."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 1 << 14])
def test_self_loop_of_the_last_id(n):
    import torch
    rng = np.random.default_rng(n)
    base = G.from_pairs(n, rng.integers(0, n, 4 * n).astype(np.int32), rng.integers(0, n, 4 * n).astype(np.int32))
    lists = [base.ind[base.off[v]:base.off[v + 1]] for v in range(n)]
    graph = api.Graph.from_csr(base, slack=0.0)
    # a sorted batch: entries of other vertices, some flagged, new ones of the last vertex, its self-loop
    src, dst, dup = [], [], []
    for v in (0, 1, n // 2, n - 1):
        for d in range(0, n, 3):
            if d != v:
                src.append(v), dst.append(d), dup.append(int(rng.random() < 0.5))
    src.append(n - 1), dst.append(n - 1), dup.append(0)
    src, dst, dup = (np.array(a, np.int32) for a in (src, dst, dup))
    ts, td, tdup = (torch.from_numpy(a).cuda() for a in (src, dst, dup))
    N.check(N.lib().tc_insert_sorted(graph.handle, ts.data_ptr(), td.data_ptr(), src.size, tdup.data_ptr(), None, None))
    off, ind = graph.export()
    for v in range(n):
        want = np.union1d(lists[v], dst[(src == v) & (dup == 0)])
        assert np.array_equal(ind[off[v]:off[v + 1]], want), v
