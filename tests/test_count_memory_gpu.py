"""The static count's working memory, against the arrays that it needs."""
import numpy as np
import pytest

from custingeralg_b200 import api

pytestmark = pytest.mark.gpu
MB = 1 << 20


def test_queues_of_a_large_graph_follow_its_items():
    """From 2^23 directed edges on a work item takes at least 256 neighbours and a hub's orientation
    item 2048 entries: the queues hold as many, not those of a small graph's finer items."""
    import torch
    n = 12288
    m = n * (n - 1)  # a complete graph: 151 M directed edges
    off = torch.arange(n + 1, dtype=torch.int64, device="cuda") * (n - 1)
    ind = torch.arange(n, dtype=torch.int32, device="cuda").repeat(n, 1)
    ind = ind[~torch.eye(n, dtype=torch.bool, device="cuda")]
    graph = api.Graph(n, off, ind, validate=False)
    _, _, slots = graph.info()
    del ind
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    graph.validate()  # allocates the count's working memory
    took = before - torch.cuda.mem_get_info()[0]
    items = n + m // 256 + 1
    hubs, chunks = m // 256 + 1, m // 256 + m // 2048 + 2
    need = 4 * slots + 2 * 8 * items + 3 * 4 * hubs + 2 * 4 * chunks + 16 * (n + 1)
    assert took <= need + 12 * 2 * MB  # ten arrays and the status, each rounded up to 2 MB pages
    graph.close()


@pytest.mark.parametrize("m", [(1 << 23) - 2, 1 << 23])
def test_counts_on_both_sides_of_the_finer_items(m):
    """A star forest of m directed edges with a clique: degrees of hubs, of CTA and of warp items."""
    import torch
    k = 2000  # clique on [0, k): k (k - 1) directed edges
    leaves = (m - k * (k - 1)) // 2
    n = k + leaves
    owner = np.sort(np.arange(leaves) % k).astype(np.int32)  # leaf k + i hangs on vertex owner[i]
    cnt = np.bincount(owner, minlength=k)
    off = np.concatenate([[0], np.cumsum(np.concatenate([k - 1 + cnt, np.ones(leaves, np.int64)]))]).astype(np.int64)
    ind = np.empty(off[-1], np.int32)
    first = np.concatenate([[0], np.cumsum(cnt)])
    for v in range(k):
        ind[off[v]:off[v] + v] = np.arange(v)
        ind[off[v] + v:off[v] + k - 1] = np.arange(v + 1, k)
        ind[off[v] + k - 1:off[v + 1]] = np.arange(k + first[v], k + first[v + 1])
    ind[off[k]:] = owner
    assert ind.size == m
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    T, _ = api.count_all_triangles_csr(n, torch.from_numpy(off).cuda(), torch.from_numpy(ind).cuda(), out, pv_mode=1)
    assert T == k * (k - 1) * (k - 2) // 6
    assert (out[:k] == (k - 1) * (k - 2)).all() and not out[k:].any()
