"""The work this framework is timed on, through its public entry points.

Two kinds of case:

  count   one static triangle count: the raw-CSR calls (int32 and int64 offsets, and the
          allocation-free one) and the graph handle, with each per-vertex convention.
  stream  update batches that are applied and then taken back, as a sliding window does
          (each inverse batch deletes what its batch inserted and inserts what it deleted):
          the captured pipeline, tc_apply_batch on host arrays, and the sorted-batch calls of the
          cuStinger interface. A pass leaves the graph as it found it.

Graphs are seeded and made on the device: R-MAT (a/b/c/d = .57/.19/.19/.05), Erdos-Renyi,
Barabasi-Albert and a rewired grid, the families of the generators module. Pairs with an id of n
or more are dropped, so n need not be a power of two. The largest case is R-MAT 24 (0.5 G directed
edges), the smallest Erdos-Renyi n = 2^14.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from custingeralg_b200 import api
from custingeralg_b200 import native as N

PV = {"none": N.TC_PV_NONE, "handle": N.TC_PV_HANDLE, "csr": N.TC_PV_CSR, "handle64": N.TC_PV_HANDLE64}


def listed():
    return [
        # the smallest count a driver makes (the plain CPU-runnable workload): launches and latency
        {"name": "csr32_er14", "kind": "count", "entry": "csr32", "family": "er", "n": 1 << 14, "degree": 16,
         "pv": "csr", "read": True},
        # a mesh-like graph in a loop that must not allocate: almost no triangles, all lists tiny
        {"name": "noalloc_grid", "kind": "count", "entry": "noalloc", "family": "grid", "n": 301 * 301, "degree": 4,
         "pv": "handle", "read": False},
        # a small power-law graph recounted in a stream of work, total and counts left on the device
        {"name": "handle_rmat16", "kind": "count", "entry": "handle", "family": "rmat", "n": 1 << 16, "degree": 32,
         "pv": "handle", "read": False},
        # the benchmark's static workload through the raw-CSR call
        {"name": "csr32_rmat20", "kind": "count", "entry": "csr32", "family": "rmat", "n": 1 << 20, "degree": 32,
         "pv": "csr", "read": True},
        # the largest static workload; 2 t(v) of its hubs can pass 2^31, so int64 counts
        {"name": "handle64_rmat24", "kind": "count", "entry": "handle", "family": "rmat", "n": 1 << 24, "degree": 32,
         "pv": "handle64", "read": True},
        # the held-out graph of the scheduler: lists of 9-16 entries, few hubs
        {"name": "handle_ba22", "kind": "count", "entry": "handle", "family": "ba", "n": 1 << 22, "degree": 32,
         "pv": "handle", "read": True},
        # a total only, int64 offsets, a vertex count that divides by nothing
        {"name": "csr64_er_ragged", "kind": "count", "entry": "csr64", "family": "er", "n": 1000003, "degree": 32,
         "pv": "none", "read": True},
        # a live graph fed a trickle: batches of 3 to 1000 updates, each one's result read
        {"name": "pipe_rmat22_small", "kind": "stream", "entry": "pipeline", "family": "rmat", "n": 1 << 22,
         "degree": 32, "batch": 1000, "batches": 6, "max_batch": 1 << 20, "pv": "none", "read": True},
        # the streaming workload's largest batches, per-vertex counts kept
        {"name": "pipe_rmat22_large", "kind": "stream", "entry": "pipeline", "family": "rmat", "n": 1 << 22,
         "degree": 32, "batch": 1000003, "batches": 1, "max_batch": 1 << 20, "pv": "handle", "read": False},
        # mid-size batches on a graph with no heavy hubs
        {"name": "pipe_ba20_mid", "kind": "stream", "entry": "pipeline", "family": "ba", "n": 1 << 20, "degree": 32,
         "batch": 20011, "batches": 2, "max_batch": 1 << 15, "pv": "handle", "read": False},
        # host-resident updates into a small graph, and a recount of the updated graph
        {"name": "apply_rmat18", "kind": "stream", "entry": "apply", "family": "rmat", "n": 200003, "degree": 32,
         "batch": 5000, "batches": 1, "max_batch": 5000, "pv": "handle", "read": True},
        # the cuStinger calls: sort a symmetric batch, insert it, count, count again, delete it
        {"name": "sorted_rmat20", "kind": "stream", "entry": "sorted", "family": "rmat", "n": 1 << 20, "degree": 32,
         "batch": 50000, "batches": 1, "max_batch": 50000, "pv": "handle", "read": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.5:
        entry = rng.choice(["csr32", "csr64", "handle", "noalloc"])
        family = rng.choice(["rmat", "rmat", "er", "ba", "grid"])
        degree = 4 if family == "grid" else rng.choice([8, 16, 32, 48])
        top = {"rmat": 1 << 22, "er": 1 << 22, "ba": 1 << 21, "grid": 1 << 22}[family]
        if entry == "noalloc":
            top = min(top, N.NOALLOC_MAX_EDGES // (degree + 2))
        n = _log_int(rng, 1 << 12, top)
        if family == "grid":
            n = max(32, math.isqrt(n)) ** 2
        pv = rng.choice(["none", "handle", "csr", "handle64"])
        if family == "grid" and pv == "none":
            pv = "handle"
        return {"kind": "count", "entry": entry, "family": family, "n": n, "degree": degree, "pv": pv,
                "read": pv == "none" or rng.random() < 0.5}
    entry = rng.choice(["pipeline", "pipeline", "pipeline", "apply", "sorted"])
    n = _log_int(rng, 1 << 14, 1 << 22)
    most = min(1 << 20 if entry == "pipeline" else 1 << 17, 2 * n)
    batch = _log_int(rng, 20, most)
    return {"kind": "stream", "entry": entry, "family": rng.choice(["rmat", "rmat", "er", "ba"]), "n": n,
            "degree": rng.choice([16, 32]), "batch": batch,
            "batches": rng.choice([1, 2, 3]) if entry == "pipeline" else 1, "max_batch": batch,
            "pv": rng.choice(["none", "handle", "handle"]) if entry == "pipeline" else "handle", "read": rng.random() < 0.5}


# ---- graphs ----------------------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _ints(gen, high, count):
    return torch.randint(0, high, (count,), generator=gen, device=gen.device)


def _rmat_pairs(n, count, gen, a=0.57, b=0.19, c=0.19):
    s = torch.zeros(count, dtype=torch.int32, device=gen.device)
    d = torch.zeros_like(s)
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(count, generator=gen, device=gen.device)
        low = r >= a + b
        s.mul_(2).add_(low)
        d.mul_(2).add_(torch.where(low, r >= a + b + c, r >= a))
    keep = (s < n) & (d < n)
    return s[keep].long(), d[keep].long()


def _pairs(case, gen):
    n, family = case["n"], case["family"]
    count = n * case["degree"] // 2
    if family == "rmat":
        return _rmat_pairs(n, count, gen)
    if family == "er":
        return _ints(gen, n, count), _ints(gen, n, count)
    if family == "ba":
        # edge e joins vertex e // m + 1 to the far end of a uniformly drawn earlier edge end: end 2k
        # of edge k is its own vertex, end 2k + 1 its target, which is looked up in turn
        m = case["degree"] // 2
        e = torch.arange(count, device=gen.device)
        v = e // m + 1
        first = 2 * m * (e // m)
        t = (torch.rand(count, generator=gen, device=gen.device, dtype=torch.float64) * first).long()
        t[:m] = -1  # the first vertex's edges go to vertex 0
        while True:
            odd = (t >= 0) & (t % 2 == 1)
            if not bool(odd.any()):
                break
            t = torch.where(odd, t[(t // 2).clamp(min=0)], t)
        u = torch.where(t < 0, torch.zeros_like(t), v[(t // 2).clamp(min=0)])
        keep = v < n
        return v[keep], u[keep]
    side = math.isqrt(n)  # a grid with 5 % of its edges' far ends redrawn
    at = torch.arange(side * side, device=gen.device)
    right, down = at[at % side < side - 1], at[at < side * (side - 1)]
    s, d = torch.cat([right, down]), torch.cat([right + 1, down + side])
    redraw = torch.rand(s.numel(), generator=gen, device=gen.device) < 0.05
    return s, torch.where(redraw, _ints(gen, n, s.numel()), d)


def _graph(case, gen):
    """The symmetric, sorted, deduplicated CSR without self-loops and its directed keys src * n + dst."""
    n = case["n"]
    s, d = _pairs(case, gen)
    loop = s == d
    s, d = s[~loop], d[~loop]
    keys = torch.unique(torch.cat([s * n + d, d * n + s]))
    off = torch.searchsorted(keys, torch.arange(n + 1, device=keys.device) * n)
    return off, (keys % n).int(), keys


def _updates(case, off, keys, gen):
    """(batches, inverses): 70 % insertions (R-MAT graphs: from the graph's own distribution), 30 % deletions of
    present edges."""
    n, k = case["n"], case["batches"]
    sizes = [max(1, round(case["batch"] ** ((i + 1) / k))) for i in range(k)]
    total = sum(sizes)
    n_del = sum(int(0.3 * b) for b in sizes)
    n_ins = total - n_del
    if case["family"] == "rmat":
        s, d = _rmat_pairs(n, 2 * n_ins + 1024, gen)
        while s.numel() < n_ins:
            s, d = torch.cat([s, s]), torch.cat([d, d])
        s, d = s[:n_ins], d[:n_ins]
    else:  # half of them uniform pairs, half close a wedge u - v - w
        s, d = _ints(gen, n, n_ins), _ints(gen, n, n_ins)
        uv = keys[_ints(gen, keys.numel(), n_ins)]
        v = uv % n
        r = torch.rand(n_ins, generator=gen, device=gen.device, dtype=torch.float64)
        w = keys[off[v] + (r * (off[v + 1] - off[v])).long()] % n
        close = r * 2 % 1 < 0.5
        s, d = torch.where(close, uv // n, s), torch.where(close, w, d)
    lo, hi = torch.minimum(s, d), torch.maximum(s, d)
    ins = lo * n + hi
    # deletions: distinct present edges that no batch inserts
    pick = keys[_ints(gen, keys.numel(), n_del)] if n_del else keys[:0]
    ps, pd = pick // n, pick % n
    dele = torch.unique(torch.minimum(ps, pd) * n + torch.maximum(ps, pd))
    dele = dele[~torch.isin(dele, ins)]
    dele = dele[torch.randperm(dele.numel(), generator=gen, device=gen.device)]
    # what the insertions add to the graph: distinct, absent before, no self-loop, in the first batch that has it
    at = torch.searchsorted(keys, ins).clamp(max=keys.numel() - 1)
    fresh = (keys[at] != ins) & (lo != hi)
    seen = keys[:0]
    forward, inverse = [], []
    i0 = d0 = 0
    for b in sizes:
        nd = min(int(0.3 * b), dele.numel() - d0)
        ni = min(b - int(0.3 * b), n_ins - i0)
        bi, bd = ins[i0:i0 + ni], dele[d0:d0 + nd]
        add = torch.unique(bi[fresh[i0:i0 + ni]])
        add = add[~torch.isin(add, seen)]
        seen = torch.cat([seen, add])
        i0, d0 = i0 + ni, d0 + nd

        def batch(inserted, deleted):
            e = torch.cat([inserted, deleted])
            f = torch.cat([torch.zeros_like(inserted), torch.ones_like(deleted)])
            order = torch.randperm(e.numel(), generator=gen, device=gen.device)
            e, f = e[order], f[order]
            swap = torch.rand(e.numel(), generator=gen, device=gen.device) < 0.5
            x, y = e // n, e % n
            return torch.where(swap, y, x).int(), torch.where(swap, x, y).int(), f.to(torch.uint8)

        forward.append(batch(bi, bd))
        inverse.append(batch(bd, add))
    return forward, inverse[::-1]


# ---- the cases -------------------------------------------------------------------------------


def prepare(case, seed):
    gen = _generator(seed)
    off, ind, keys = _graph(case, gen)
    n = case["n"]
    dev = off.device
    pv = PV[case["pv"]]
    state = {"case": case, "n": n, "pv": pv}
    kind = torch.int64 if pv == N.TC_PV_HANDLE64 else torch.int32
    state["out"] = None if pv == N.TC_PV_NONE else torch.zeros(n, dtype=kind, device=dev)
    state["total"] = torch.zeros(1, dtype=torch.int64, device=dev)
    if case["kind"] == "count":
        if case["entry"] == "handle":
            state["graph"] = api.Graph(n, off, ind)
        else:
            state["off"] = off if case["entry"] == "csr64" else off.int()
            state["ind"] = ind
        return state
    state["graph"] = graph = api.Graph(n, off, ind, slack=0.25)
    forward, inverse = _updates(case, off, keys, gen)
    if case["entry"] == "pipeline":
        state["pipe"] = api.Pipeline(graph, case["max_batch"])
        state["pipe"].prepare(state["out"], state["total"])
    elif case["entry"] == "apply":
        forward, inverse = ([tuple(t.cpu().numpy() for t in b) for b in side] for side in (forward, inverse))
        state["recount"] = torch.zeros(n, dtype=torch.int32, device=dev)
    else:  # the sorted calls take both directions of every inserted edge
        src, dst, is_delete = forward[0]
        ins = is_delete == 0
        src, dst = src[ins], dst[ins]
        state["src"], state["dst"] = torch.cat([src, dst]), torch.cat([dst, src])
        state["offsets"] = torch.zeros(n + 1, dtype=torch.int32, device=dev)
        state["dup"] = torch.zeros_like(state["src"])
    state["forward"], state["inverse"] = forward, inverse
    return state


def _count(st):
    case, n, out, total, pv = st["case"], st["n"], st["out"], st["total"], st["pv"]
    if case["entry"] == "handle":
        got = st["graph"].count(pv, out, total, sync=case["read"])
    elif case["entry"] == "noalloc":
        info = N.CountInfo() if case["read"] else None
        N.check(N.lib().tc_count_csr32_noalloc(
            n, st["off"].data_ptr(), st["ind"].data_ptr(), pv, None if out is None else out.data_ptr(),
            total.data_ptr(), ctypes.byref(info) if info else None, None, torch.cuda.current_stream().cuda_stream))
        got = (info.triangles, info) if info else None
    else:
        got = api.count_all_triangles_csr(n, st["off"], st["ind"], out, pv_mode=pv, sync=case["read"],
                                          triangles_dev=total)
    res = {"total": total, "per_vertex": out}
    if got:
        T, info = got
        res["info"] = [T, info.edges_intersected, info.oriented_work, info.max_out_degree]
    return res


def _batch_info(info):
    return [info.updates, info.inserted, info.deleted, info.ignored, info.triangles_added, info.triangles_removed]


def _snapshot(st):
    return [st["total"].clone(), None if st["out"] is None else st["out"].clone()]


def _pipeline(st):
    pipe, read, infos, running = st["pipe"], st["case"]["read"], [], []
    for k, batches in enumerate((st["forward"], st["inverse"])):
        for src, dst, is_delete in batches:
            pipe.apply(src, dst, is_delete, st["out"], st["total"])
            if read:
                infos.append(_batch_info(pipe.sync()))
        running.append(_snapshot(st))  # the running counts once the window is in, and once it has left
    infos.append(_batch_info(pipe.sync()))
    return {"running": running, "infos": np.array(infos), "edges": st["graph"].info()[1]}


def _apply(st):
    graph, read, infos, running = st["graph"], st["case"]["read"], [], []
    recount = None
    for k, batches in enumerate((st["forward"], st["inverse"])):
        for src, dst, is_delete in batches:
            info = graph.apply_batch(src, dst, is_delete, st["out"], st["total"], sync=read)
            if read:
                infos.append(_batch_info(info))
        running.append(_snapshot(st))
        if k == 0:
            recount = [graph.count(N.TC_PV_HANDLE, st["recount"])[0], st["recount"]]
    return {"running": running, "infos": np.array(infos), "recount": recount, "edges": graph.info()[1]}


def _sorted(st):
    lib, g, n = N.lib(), st["graph"].handle, st["n"]
    src, dst, off, dup = st["src"].clone(), st["dst"].clone(), st["offsets"], st["dup"]
    b, stream = src.numel(), torch.cuda.current_stream().cuda_stream
    moved = ctypes.c_int64()
    s, d, o, u = src.data_ptr(), dst.data_ptr(), off.data_ptr(), dup.data_ptr()
    pv, total = st["out"].data_ptr(), st["total"].data_ptr()
    N.check(lib.tc_batch_sort(n, s, d, b, o, u, stream))
    N.check(lib.tc_insert_sorted(g, s, d, b, u, ctypes.byref(moved), stream))
    N.check(lib.tc_count_batch(g, s, d, o, u, b, 1, pv, total, None, stream))
    running = [_snapshot(st)]
    N.check(lib.tc_count_batch(g, s, d, o, u, b, -1, pv, total, None, stream))
    N.check(lib.tc_delete_sorted(g, s, d, u, b, stream))
    running.append(_snapshot(st))
    return {"running": running, "batch": [src, dst, off, dup], "edges": st["graph"].info()[1]}


def run(state):
    case = state["case"]
    if case["kind"] == "count":
        return _count(state)
    return {"pipeline": _pipeline, "apply": _apply, "sorted": _sorted}[case["entry"]](state)


# ---- what a pass cannot do without -----------------------------------------------------------


def _directed_edges(case):
    n, e = case["n"], case["n"] * case["degree"]
    if case["family"] == "rmat":  # pairs that repeat: 6 % at scale 20, fewer on larger graphs
        return e * max(0.5, 1 - 0.064 * 0.83 ** (math.log2(n) - 20))
    return e


def work(case):
    """Bytes: every list and offset of a counted graph, or the batches and the lists of their edges'
    endpoints, read once, and every output written once. The counts are integers: no flops."""
    n, m = case["n"], _directed_edges(case)
    width = {"none": 0, "handle": 4, "csr": 4, "handle64": 8}[case["pv"]]
    if case["kind"] == "count":
        return {"bytes": (8 if case["entry"] in ("csr64", "handle") else 4) * (n + 1) + 4 * m + width * n + 8, "flops": 0}
    # an edge's endpoints hold, on average, the mean degree of a neighbour each
    lists = 2 * case["degree"] * (1.27 ** math.log2(n) if case["family"] == "rmat" else 2)
    updates = sum(max(1, round(case["batch"] ** ((i + 1) / case["batches"]))) for i in range(case["batches"]))
    touched = sum(min(4 * m, 4 * lists * b) for b in
                  (max(1, round(case["batch"] ** ((i + 1) / case["batches"]))) for i in range(case["batches"])))
    return {"bytes": 2 * (9 * updates + touched + width * n), "flops": 0}


# ---- known answers ---------------------------------------------------------------------------


def _wedge_counts(n, off, ind, most):
    """t(v) per vertex and the forward counts of the raw-CSR convention, from every wedge of the degree
    orientation looked up among the oriented edges; None past `most` wedges."""
    ind = ind.long()
    deg = off[1:] - off[:-1]
    src = torch.repeat_interleave(torch.arange(n, device=off.device), deg)
    up = (deg[src] < deg[ind]) | ((deg[src] == deg[ind]) & (src < ind))
    u, v = src[up], ind[up]
    keys = u * n + v  # ascending: src ascends and its list does
    out = torch.zeros(n + 1, dtype=torch.int64, device=off.device)
    out[1:] = torch.cumsum(torch.bincount(u, minlength=n), 0)
    width = (out[1:] - out[:-1])[v]
    if int(width.sum()) > most:
        return None
    t = torch.zeros(n, dtype=torch.int64, device=off.device)
    forward = torch.zeros_like(t)
    step = 1 << 24
    e0 = 0
    total = torch.cumsum(width, 0)
    while e0 < u.numel():
        base = int(total[e0 - 1]) if e0 else 0
        e1 = max(e0 + 1, int(torch.searchsorted(total, torch.tensor(base + step, device=off.device), right=True)))
        edge = torch.repeat_interleave(torch.arange(e0, e1, device=off.device), width[e0:e1])
        k = torch.arange(edge.numel(), device=off.device) + base - (total[edge] - width[edge])
        x, y = u[edge], v[edge]
        z = v[out[y] + k]
        at = torch.searchsorted(keys, x * n + z).clamp(max=keys.numel() - 1)
        hit = keys[at] == x * n + z
        tri = torch.stack([x[hit], y[hit], z[hit]]).sort(0).values
        t += torch.bincount(tri.reshape(-1), minlength=n)
        forward += 2 * torch.bincount(tri[0], minlength=n) + torch.bincount(tri[1], minlength=n)
        e0 = e1
    return t, forward


def exact(case, seed):
    if case["kind"] != "count":
        return None  # whole numbers, compared as such
    gen = _generator(seed)
    off, ind, _ = _graph(case, gen)
    got = _wedge_counts(case["n"], off, ind, 300_000_000)
    if got is None:
        return None
    t, forward = got
    pv = {"none": None, "csr": forward.int(), "handle": (2 * t).int(), "handle64": 2 * t}[case["pv"]]
    T = t.sum().reshape(1) // 3
    res = {"total": T, "per_vertex": pv}
    if case["read"]:
        res["info"] = [int(T), None, None, None]
    return res
