"""The hub-centred delta count at its table sizes: hubs around one pass (6144 entries) and its multiples,
and a hub whose neighbours' ids share both slots of the table."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


def _check(n, hub_nbrs, changed, seed):
    """Insert and delete edges between hub 0 and `changed` and compare with static recounts."""
    import torch
    rng = np.random.default_rng(seed)
    k = 3 * hub_nbrs.size
    src = np.concatenate([np.zeros(hub_nbrs.size, np.int32), rng.choice(hub_nbrs, k), rng.integers(1, n, k)])
    dst = np.concatenate([hub_nbrs, rng.choice(hub_nbrs, k), rng.choice(hub_nbrs, k)])
    src, dst = np.concatenate([src, changed]), np.concatenate([dst, rng.choice(hub_nbrs, changed.size)])
    base = G.from_pairs(n, src.astype(np.int32), dst.astype(np.int32))
    graph = api.Graph.from_csr(base, slack=0.25)
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    T0, _ = graph.count(N.TC_PV_HANDLE, out)
    pv, delta = out.clone(), torch.zeros(1, dtype=torch.int64, device="cuda")
    s = np.zeros(changed.size, np.int32)
    x = (np.isin(changed, hub_nbrs)).astype(np.uint8)  # present: deleted; absent: inserted
    graph.apply_batch(*[torch.from_numpy(a).cuda() for a in (s, changed, x)], per_vertex=pv, delta_dev=delta)
    T1, _ = graph.count(N.TC_PV_HANDLE, out)
    assert T1 == T0 + int(delta.item()) and T1 != T0
    assert torch.equal(out, pv)


@pytest.mark.parametrize("deg", [40, 6143, 6144, 6145, 12289])
def test_hub_pass_boundaries(deg):
    n = 20000
    ids = np.random.default_rng(deg).permutation(np.arange(1, n, dtype=np.int32))
    _check(n, ids[:deg], np.concatenate([ids[:20], ids[deg:deg + 20]]), deg)


def test_hub_with_colliding_ids():
    n = 1 << 22
    ids = np.arange(1, n, dtype=np.uint64)
    # a table of at most 512 slots: the two slots come from the hash's leading 16 bits
    lead = ((ids * 0x9E3779B1) & 0xFFFFFFFF) >> 16
    same = ids[lead == lead[123456]].astype(np.int32)
    assert same.size >= 16
    _check(n, np.concatenate([same[:-8], np.arange(5000, 5100, dtype=np.int32)]),
           np.concatenate([same[-8:], np.arange(5000, 5010, dtype=np.int32)]), 1)
