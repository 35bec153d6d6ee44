"""The static count's hash sets at the sizes where they change: tier and pass boundaries, and ids whose
hash slots collide, so that a set cannot be built over all of them at once."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

HASH = 0x9E3779B1  # the sets' multiplicative hash


def _count(g, mode, sched=None, dtype="int32"):
    import torch
    graph = api.Graph.from_csr(g)
    out = torch.zeros(g.n + 1, dtype=getattr(torch, dtype), device="cuda")
    T, _ = graph.count(mode, out, sched=sched)
    graph.close()
    return T, out[: g.n].cpu().numpy()


# out-degrees 0 .. k - 1: warp tables of every size, the warp tier's limit (64, 128), one pass (768) and two
@pytest.mark.parametrize("k", [33, 34, 65, 66, 129, 130, 769, 770])
def test_cliques_at_the_table_sizes(k):
    g = G.complete(k)
    for warp_max in (64, 128):
        s = N.default_sched()
        s.warp_max_deg = warp_max
        for mode in (N.TC_PV_NONE, N.TC_PV_HANDLE, N.TC_PV_CSR):
            T, pv = _count(g, mode, s)
            assert T == k * (k - 1) * (k - 2) // 6
            if mode == N.TC_PV_HANDLE:
                assert (pv == (k - 1) * (k - 2)).all()
            if mode == N.TC_PV_CSR:
                assert np.array_equal(pv, O.csr_per_vertex(g.n, g.off, g.ind))


@pytest.mark.parametrize("bits,n,warp_max", [(12, 1 << 16, 64), (20, 1 << 22, 2)], ids=["warp", "cta"])
def test_colliding_ids(bits, n, warp_max):
    """A clique of ids that share both slots of the set (the same leading bits of the hash), with
    other neighbours around it."""
    ids = np.arange(n, dtype=np.uint64)
    lead = ((ids * HASH) & 0xFFFFFFFF) >> (32 - bits)
    values, counts = np.unique(lead, return_counts=True)
    clique = ids[lead == values[counts.argmax()]].astype(np.int32)
    assert clique.size >= 4
    rng = np.random.default_rng(bits)
    i, j = np.triu_indices(clique.size, 1)
    other = rng.integers(0, n, 200).astype(np.int32)
    src = np.concatenate([clique[i], rng.choice(clique, 400), rng.choice(other, 300)])
    dst = np.concatenate([clique[j], rng.choice(other, 400), rng.choice(other, 300)])
    g = G.from_pairs(n, src, dst)
    tot, pv = O.fast_count(g.n, g.off, g.ind)
    s = N.default_sched()
    s.warp_max_deg = warp_max
    T, got = _count(g, N.TC_PV_HANDLE, s)
    assert 6 * T == tot and np.array_equal(got, pv)
