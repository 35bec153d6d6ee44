"""The hub-centred delta count in phases large enough for it: hubs around one pass of its table (6144 entries)
and its multiples, and a hub whose neighbours' ids share both slots of the table, so that builds fail."""
import os
import re

import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu
SRC = os.path.join(os.path.dirname(__file__), "..", "custingeralg_b200", "csrc", "tc_stream.cu")
PAD = 2600  # unrelated changed edges of each phase


def _smallest_hub_phase():
    text = open(SRC).read()
    assert "constexpr int64_t kHubBatchMin = kSmallBatch;" in text
    return int(re.search(r"constexpr int64_t kSmallBatch = (\d+);", text).group(1))


def _check(path, n, hub_nbrs, changed, seed):
    """Insert and delete edges between hub 0 and `changed`, and PAD edges apart from it in either phase;
    compare with static recounts."""
    import torch
    rng = np.random.default_rng(seed)
    k = 3 * hub_nbrs.size
    apart = np.arange(n, n + PAD, dtype=np.int32)  # a path; its chords are inserted, its edges deleted
    src = np.concatenate([np.zeros(hub_nbrs.size, np.int32), rng.choice(hub_nbrs, k), rng.integers(1, n, k), changed, apart])
    dst = np.concatenate([hub_nbrs, rng.choice(hub_nbrs, k), rng.choice(hub_nbrs, k),
                          rng.choice(hub_nbrs, changed.size), apart + 1])
    total = n + PAD + 2
    base = G.from_pairs(total, src.astype(np.int32), dst.astype(np.int32))
    graph = api.Graph.from_csr(base, slack=0.25)
    out = torch.zeros(total, dtype=torch.int32, device="cuda")
    T0, _ = graph.count(N.TC_PV_HANDLE, out)
    pv, delta = out.clone(), torch.zeros(1, dtype=torch.int64, device="cuda")
    present = np.isin(changed, hub_nbrs).astype(np.uint8)  # deleted; the others are inserted
    assert present.sum() >= 8 and (1 - present).sum() >= 8  # a hub in either phase
    s = np.concatenate([np.zeros(changed.size, np.int32), apart, apart])
    d = np.concatenate([changed, apart + 1, apart + 2])
    x = np.concatenate([present, np.ones(PAD, np.uint8), np.zeros(PAD, np.uint8)])
    args = [torch.from_numpy(a).cuda() for a in (s, d, x)]
    if path == "pipeline":
        pipe = api.Pipeline(graph, 1 << 13)
        pipe.apply(*args, per_vertex=pv, delta_dev=delta)
        info = pipe.sync()
        pipe.close()
    else:
        info = graph.apply_batch(*args, per_vertex=pv, delta_dev=delta)
    assert min(info.inserted, info.deleted) > _smallest_hub_phase()
    T1, _ = graph.count(N.TC_PV_HANDLE, out)
    assert T1 == T0 + int(delta.item()) and T1 != T0
    assert torch.equal(out, pv)


@pytest.mark.parametrize("path", ["apply", "pipeline"])
@pytest.mark.parametrize("deg", [40, 6143, 6144, 6145, 12289])
def test_hub_pass_boundaries(deg, path):
    n = 20000
    ids = np.random.default_rng(deg).permutation(np.arange(1, n, dtype=np.int32))
    _check(path, n, ids[:deg], np.concatenate([ids[:20], ids[deg:deg + 20]]), deg)


@pytest.mark.parametrize("path", ["apply", "pipeline"])
def test_hub_with_colliding_ids(path):
    n = 1 << 22
    ids = np.arange(1, n, dtype=np.uint64)
    # a table of at most 512 slots: the two slots come from the hash's leading 16 bits
    lead = ((ids * 0x9E3779B1) & 0xFFFFFFFF) >> 16
    same = ids[lead == lead[123456]].astype(np.int32)
    assert same.size >= 24
    _check(path, n, np.concatenate([same[:-8], np.arange(5000, 5100, dtype=np.int32)]),
           np.concatenate([same[-16:], np.arange(5000, 5010, dtype=np.int32)]), 1)
