"""The orientation's vertex tiles: lists that end and start on both sides of its 32-entry steps, empty ones
between them, and entries out of order on both sides of a step."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 0, 32, 33, 0, 0, 63, 64, 65, 2, 95, 255, 256, 257, 0, 30, 1, 1, 128, 96]


def _graph(shift):
    """Ids 0 .. 21 with planted degrees (rolled by shift) among the ids from 64 on, which form a ring of triangles."""
    rng = np.random.default_rng(shift)
    n = 32 * shift + 700
    lengths = np.roll(LENGTHS, shift)
    src, dst = [], []
    for i, k in enumerate(lengths):
        pool = rng.permutation(np.arange(64, n))[:k]
        src += [i] * len(pool)
        dst += pool.tolist()
    ring = np.arange(64, n - 1)
    src, dst = np.r_[src, ring, ring[:-1]], np.r_[dst, ring + 1, ring[:-1] + 2]
    return G.from_pairs(n, src.astype(np.int32), dst.astype(np.int32))


@pytest.mark.parametrize("entry", ["handle", "csr32", "csr64"])
@pytest.mark.parametrize("shift", [0, 1, 5, 11])
def test_planted_lengths_against_matrix_products(shift, entry):
    import torch
    g = _graph(shift)
    a = np.zeros((g.n, g.n), np.int64)
    a[np.repeat(np.arange(g.n), np.diff(g.off)), g.ind] = 1
    want = ((a @ a) * a).sum(1)  # 2 t(v)
    out = torch.zeros(g.n, dtype=torch.int32, device="cuda")
    if entry == "handle":
        T, _ = api.Graph.from_csr(g).count(N.TC_PV_HANDLE, out)
    else:
        kind = np.int32 if entry == "csr32" else np.int64
        off, ind = torch.from_numpy(g.off.astype(kind)).cuda(), torch.from_numpy(g.ind).cuda()
        T, _ = api.count_all_triangles_csr(g.n, off, ind, out, pv_mode=N.TC_PV_HANDLE)
    assert T == want.sum() // 6
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("at", [1, 31, 32, 33, 63, 64, 65, 127, 128, 199])
def test_order_is_checked_across_steps(at):
    import torch
    g = G.complete(201)  # lists of 200 entries: every list but the first starts inside a step
    for v in (0, 1, 7):
        ind = g.ind.copy()
        k = int(g.off[v]) + at
        ind[[k - 1, k]] = ind[[k, k - 1]]
        off, dev = torch.from_numpy(g.off).cuda(), torch.from_numpy(ind).cuda()
        with pytest.raises(N.TcError):
            api.count_all_triangles_csr(g.n, off, dev, None, pv_mode=N.TC_PV_NONE)
