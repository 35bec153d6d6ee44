"""The searched intersection of one changed edge, at list lengths around its sample counts (32, 128) and
around the two entries a lane takes at once: the edge is inserted and deleted, against set arithmetic."""
import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("short", [2, 31, 33, 64, 65, 200])
@pytest.mark.parametrize("long", [2, 31, 32, 33, 127, 128, 129, 257, 1025, 5000])
def test_one_edge_against_sets(long, short):
    import torch
    short = min(short, long)
    rng = np.random.default_rng(1000 * long + short)
    n = 2 * long + 2
    x, y = sorted(rng.choice(n, 2, replace=False).tolist())
    others = np.setdiff1d(np.arange(n), [x, y])
    nx = np.sort(rng.choice(others, long, replace=False))
    rest = np.setdiff1d(others, nx)
    hits = np.unique(np.r_[nx[0], nx[-1], rng.choice(nx, short // 2)])[:short]
    ny = np.r_[hits, rng.choice(rest, short - len(hits), replace=False)]
    src = np.r_[np.full(long, x), np.full(len(ny), y)].astype(np.int32)
    dst = np.r_[nx, ny].astype(np.int32)
    graph = api.Graph.from_csr(G.from_pairs(n, src, dst), slack=0.5)
    sched = N.default_sched()
    sched.stream_hub_min = 0
    pv = torch.zeros(n, dtype=torch.int32, device="cuda")
    delta = torch.zeros(1, dtype=torch.int64, device="cuda")
    edge = [torch.tensor([v], dtype=torch.int32, device="cuda") for v in (x, y)]
    want = np.zeros(n, np.int64)
    want[hits] = 2
    want[[x, y]] = 2 * len(hits)
    for op, total in ((0, len(hits)), (1, 0)):
        graph.apply_batch(*edge, torch.tensor([op], dtype=torch.uint8, device="cuda"), per_vertex=pv, delta_dev=delta,
                          sched=sched)
        assert int(delta.item()) == total
        np.testing.assert_array_equal(pv.cpu().numpy(), want if op == 0 else 0 * want)
