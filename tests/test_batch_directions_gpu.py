"""tc_count_batch on batches that hold one direction of some edges and both of others, with duplicates and
absent edges, for insertions and deletions, against a plain recomputation of its definition."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


def _expected(n, adj, entries, sign):
    """Per entry (x, y) in the batch (deletions: and in the graph): each common neighbour w is kept unless
    (x, w) or (y, w) is an entry with a smaller edge; kept triangles add 1 to x, y and w, and to the
    total when x < y."""
    batch = set(entries)
    pv, total = np.zeros(n, np.int64), 0
    for x, y in sorted(batch):
        if sign < 0 and y not in adj[x]:
            continue
        key = (min(x, y), max(x, y))
        for w in adj[x] & adj[y]:
            if any((o, w) in batch and (min(o, w), max(o, w)) <= key for o in (x, y)):
                continue
            pv[[x, y, w]] += 1
            total += x < y
    return sign * pv, sign * total


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("hub", [40, 700])  # shorter lists below and above the split sizes
def test_directions(sign, hub):
    import torch
    rng = np.random.default_rng(hub)
    n = 1200
    src = np.concatenate([np.repeat([0, 1], hub), rng.integers(0, n, 6000)]).astype(np.int32)
    dst = np.concatenate([np.arange(2, hub + 2), np.arange(2, hub + 2), rng.integers(0, n, 6000)]).astype(np.int32)
    src, dst = np.append(src, 0).astype(np.int32), np.append(dst, 1).astype(np.int32)
    g = G.from_pairs(n, src, dst)
    adj = [set(g.ind[g.off[v]:g.off[v + 1]].tolist()) for v in range(n)]
    u = np.repeat(np.arange(n), np.diff(g.off))
    pick = rng.integers(0, g.m, 150)
    ent = [(int(a), int(b)) for a, b in zip(u[pick], g.ind[pick])]
    ent += [(b, a) for a, b in ent[:80]] + ent[:5] + [(0, 1), (1, 0), (0, 2), (3, 1)]
    if sign < 0:
        ent += [(5, 900), (900, 5), (7, 7)]  # mostly absent, and a self-loop
    s = torch.tensor([a for a, _ in ent], dtype=torch.int32, device="cuda")
    d = torch.tensor([b for _, b in ent], dtype=torch.int32, device="cuda")
    off = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    dup = torch.zeros(len(ent), dtype=torch.int32, device="cuda")
    lib = N.lib()
    N.check(lib.tc_batch_sort(n, s.data_ptr(), d.data_ptr(), len(ent), off.data_ptr(), dup.data_ptr(), None))
    graph = api.Graph.from_csr(g, slack=0.25)
    pv = torch.zeros(n, dtype=torch.int32, device="cuda")
    delta = torch.zeros(1, dtype=torch.int64, device="cuda")
    N.check(lib.tc_count_batch(graph.handle, s.data_ptr(), d.data_ptr(), off.data_ptr(), dup.data_ptr(), len(ent), sign,
                               pv.data_ptr(), delta.data_ptr(), None, None))
    want, total = _expected(n, adj, [e for e in ent if e[0] != e[1]], sign)
    assert np.array_equal(pv.cpu().numpy(), want)
    assert int(delta.item()) == total
