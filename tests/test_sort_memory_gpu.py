"""The working memory that tc_batch_sort keeps: one call's at a time, and given back where memory is short."""
import threading

import numpy as np
import pytest

from custingeralg_b200 import api, generators as G, native as N

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lift_cap():
    yield
    N.check(N.lib().tc_debug_alloc_cap(0))


def _sort(n, src, dst, stream=None):
    """tc_batch_sort of host arrays; the sorted pairs, offsets and duplicate flags."""
    import torch
    s, d = torch.from_numpy(src).cuda(), torch.from_numpy(dst).cuda()
    off = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    dup = torch.zeros(max(src.size, 1), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    N.check(N.lib().tc_batch_sort(n, s.data_ptr(), d.data_ptr(), src.size, off.data_ptr(), dup.data_ptr(),
                                  stream.cuda_stream if stream else None))
    return [t.cpu().numpy() for t in (s, d, off, dup[:src.size])]


def _check(n, src, dst, got):
    order = np.lexsort((dst, src))
    s, d = src[order], dst[order]
    dup = s == d
    dup[1:] |= (s[1:] == s[:-1]) & (d[1:] == d[:-1])
    off = np.concatenate([[0], np.cumsum(np.bincount(s, minlength=n))])
    for a, b in zip(got, (s, d, off, dup)):
        assert np.array_equal(a, b)


def _batch(rng, n, b):
    return rng.integers(0, n, b).astype(np.int32), rng.integers(0, n, b).astype(np.int32)


def test_a_failed_allocation_gives_the_kept_memory_back():
    import torch
    rng = np.random.default_rng(1)
    n, b = 1 << 16, 6_000_000
    src, dst = _batch(rng, n, b)
    g = G.rmat(12, 8, seed=1)
    N.check(N.lib().tc_workspace_release())
    got = _sort(n, src, dst)  # keeps 16 bytes an entry and the sort's own
    _check(n, src, dst, got)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    N.check(N.lib().tc_debug_alloc_cap(1 << 16))
    with pytest.raises(N.TcError) as ei:
        api.Graph.from_csr(g)
    assert ei.value.status == N.TC_ERR_OOM
    assert torch.cuda.mem_get_info()[0] - free >= 16 * b
    N.check(N.lib().tc_debug_alloc_cap(0))
    api.Graph.from_csr(g).close()
    _check(n, src, dst, _sort(n, src, dst))


def test_growth_that_fails_is_tried_at_the_size_of_the_call():
    rng = np.random.default_rng(2)
    big, small = _batch(rng, 1 << 10, 400_000), _batch(rng, 1 << 18, 50_000)
    N.check(N.lib().tc_workspace_release())
    _check(1 << 10, *big, _sort(1 << 10, *big))
    # the keys of 400,000 entries do not fit under the cap, those of 50,000 and 2^18 offsets do
    N.check(N.lib().tc_debug_alloc_cap(9 * (1 << 18)))
    _check(1 << 18, *small, _sort(1 << 18, *small))


def test_two_threads_sort_at_once():
    import torch
    errors = []

    def work(seed):
        try:
            torch.cuda.set_device(0)
            rng = np.random.default_rng(seed)
            stream = torch.cuda.Stream()
            for _ in range(30):
                n, b = int(rng.integers(2, 5000)), int(rng.integers(1, 200_000))
                src, dst = _batch(rng, n, b)
                _check(n, src, dst, _sort(n, src, dst, stream))
                if seed == 0 and rng.random() < 0.3:
                    N.check(N.lib().tc_workspace_release())
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors[0]
