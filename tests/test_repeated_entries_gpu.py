"""Lists that repeat an id: refused, and in the time that a simple graph of the size takes. A hash set
that gave way to repeats would be built two entries at a time, hundreds of times the work."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu
LIMIT_MS = 100.0  # 2^18 entries in pieces of 768: under 400 builds of some 10 us; in pieces of 2: 131072


def _timed(fn):
    import torch
    fn()
    torch.cuda.synchronize()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    fn()
    b.record()
    torch.cuda.synchronize()
    return a.elapsed_time(b)


def _multigraph(copies):
    """A simple graph on the ids from 2 up, and vertices 0 and 1 joined `copies` times."""
    base = G.rmat(10, 8, seed=5)
    off = np.concatenate([[0, copies], 2 * copies + base.off]).astype(np.int64)
    ind = np.concatenate([np.full(copies, 1, np.int32), np.zeros(copies, np.int32), base.ind + 2]).astype(np.int32)
    return base, off, ind


@pytest.mark.parametrize("copies", [3, 100, 128, 769, 1 << 18])  # a warp's and a CTA's table
def test_repeats_are_refused_in_time(copies):
    import torch
    base, off, ind = _multigraph(copies)
    n = base.n + 2
    d_off, d_ind = torch.from_numpy(off).cuda(), torch.from_numpy(ind).cuda()
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    tri = torch.zeros(1, dtype=torch.int64, device="cuda")
    with pytest.raises(N.TcError) as ei:
        api.count_all_triangles_csr(n, d_off, d_ind, out, pv_mode=N.TC_PV_HANDLE)
    assert ei.value.status == N.TC_ERR_BAD_GRAPH
    ms = _timed(lambda: api.count_all_triangles_csr(n, d_off, d_ind, out, pv_mode=N.TC_PV_HANDLE, sync=False,
                                                    triangles_dev=tri))
    assert ms < LIMIT_MS
    # the repeated edge is in no triangle: the rest is counted as without it
    want = torch.zeros(base.n, dtype=torch.int32, device="cuda")
    T, _ = api.Graph.from_csr(base).count(N.TC_PV_HANDLE, want)
    assert int(tri.item()) == T
    assert torch.equal(out[2:], want) and not out[:2].any()


def test_repeats_at_a_batch_hub():
    """An unchecked handle: a batch whose changed edges meet at the list with the repeats."""
    import torch
    base, off, ind = _multigraph(1 << 18)
    n = base.n + 2 + 8192
    off = np.concatenate([off, np.full(8192, off[-1])])
    graph = api.Graph(n, off, ind, slack=0.25, validate=False)
    new = np.arange(n - 8192, n, dtype=np.int32)
    # the new neighbours of 0 form pairs, so that their lists have two entries and are counted
    src = np.concatenate([np.zeros(8192, np.int32), new[::2]])
    dst = np.concatenate([new, new[1::2]])
    src, dst = torch.from_numpy(src).cuda(), torch.from_numpy(dst).cuda()
    ins, rem = torch.zeros(src.numel(), dtype=torch.uint8, device="cuda"), torch.ones_like(src, dtype=torch.uint8)
    pv = torch.zeros(n, dtype=torch.int32, device="cuda")
    delta = torch.zeros(1, dtype=torch.int64, device="cuda")

    def both():
        graph.apply_batch(src, dst, ins, per_vertex=pv, delta_dev=delta)
        assert int(delta.item()) == 4096
        graph.apply_batch(src, dst, rem, per_vertex=pv, delta_dev=delta)

    assert _timed(both) < LIMIT_MS
    assert int(delta.item()) == 0 and not pv.any()
