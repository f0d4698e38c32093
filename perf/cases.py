"""The work a program gives this framework, as cases that can be timed.

A case is one call sequence through the public entry points on one graph:

  count   all-edge common-neighbour counts of a resident graph into the caller's
          device tensor: the default policy on the graph as it came (mode
          "direct"), or oriented on the degree-relabeled graph with the kernel
          kind the scheduler settles on there (mode "oriented")
  job     host CSR in pinned memory -> validated graph -> relabel -> oriented
          count, and either the counts back in pinned memory (out "counts") or
          the SCAN query's labels, clusters and non-core pairs (out "scan")
  query   SCAN clustering of a resident counted graph: into device tensors
          (out "device") or as the host arrays Graph.scan returns (out "host")
  edges   an undirected edge list on the host -> a sorted, deduplicated CSR
  batch   many uneven graphs: one captured count of their union and one query

Graphs are R-MAT (0.57, 0.19, 0.19, 0.05), Erdos-Renyi or Chung-Lu (power law,
exponent 2.1) draws made here from the seed: so many distinct undirected edges,
both directions of each kept ("edges" of them make 2 * edges CSR entries).
"""
import ctypes

import numpy as np
import torch

from acctricnt_gb300 import accx

RMAT = (0.57, 0.19, 0.19)


def listed():
    return [
        # a neighbourhood extracted for one request: launches and host calls are all there is
        {"name": "count_default_rmat10", "op": "count", "kind": "rmat", "n": 1 << 10, "edges": 10007, "mode": "direct",
         "policy": "heuristic"},
        # the default call on a graph that is counted once, without preparing it
        {"name": "count_default_rmat18", "op": "count", "kind": "rmat", "n": 1 << 18, "edges": 3800003,
         "mode": "direct", "policy": "heuristic"},
        # the new-graph counts a server takes between its queries (R-MAT scales 14-22)
        {"name": "count_oriented_rmat15", "op": "count", "kind": "rmat", "n": 1 << 15, "edges": 440001,
         "mode": "oriented", "policy": "bitmap"},
        # the headline workload
        {"name": "count_oriented_rmat24", "op": "count", "kind": "rmat", "n": 1 << 24, "edges": 260000000,
         "mode": "oriented", "policy": "bitmap"},
        # social graphs: a power law with a heavy head, any number of vertices
        {"name": "count_oriented_chunglu3m", "op": "count", "kind": "chunglu", "n": 3000017, "edges": 33333331,
         "mode": "oriented", "policy": "bitmap"},
        # no hubs, hardly a triangle, no locality
        {"name": "count_oriented_er5m", "op": "count", "kind": "er", "n": 5000011, "edges": 60000001,
         "mode": "oriented", "policy": "gallop"},
        # counts of a graph that arrives on the host, end to end
        {"name": "job_counts_rmat21", "op": "job", "kind": "rmat", "n": 1 << 21, "edges": 32000009, "out": "counts",
         "eps": 0.0, "mu": 0},
        # the whole SCAN job on a graph of ordinary size: what the command-line tool does between its files
        {"name": "job_scan_rmat16", "op": "job", "kind": "rmat", "n": 1 << 16, "edges": 900001, "out": "scan",
         "eps": 0.2, "mu": 5},
        # one (eps, mu) of an exploration of a large resident graph
        {"name": "query_rmat22", "op": "query", "kind": "rmat", "n": 1 << 22, "edges": 64000003, "eps": 0.2, "mu": 5,
         "out": "device"},
        # the same on a small graph, answered with host arrays
        {"name": "query_rmat13", "op": "query", "kind": "rmat", "n": 1 << 13, "edges": 100003, "eps": 0.3, "mu": 4,
         "out": "host"},
        # raw edge lists with duplicates and self loops, as converters read them
        {"name": "edges_6m", "op": "edges", "kind": "er", "n": 1000003, "edges": 6000001},
        # small graphs of many tenants, counted and clustered together
        {"name": "batch_48", "op": "batch", "k": 48, "emin": 1000, "emax": 300000, "eps": 0.3, "mu": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_graph(rng, emin, emax):
    """A graph of emin..emax edges (over the logarithm): its kind, size and number of edges."""
    e = _log_int(rng, emin, emax)
    kind = rng.choice(("rmat", "chunglu", "er"))
    if kind == "rmat":
        return {"kind": kind, "n": 1 << max(6, min(24, int(round(np.log2(e / rng.uniform(8, 24)))))), "edges": e}
    return {"kind": kind, "n": max(67, 2 * e // rng.randint(12, 32)), "edges": e}


def draw(rng):
    op = rng.choice(("count", "count", "count", "job", "query", "edges", "batch"))
    eps, mu = round(rng.uniform(0.1, 0.8), 3), rng.randint(2, 12)
    if op == "count":
        if rng.random() < 0.4:
            return {"op": op, **_draw_graph(rng, 5_000, 4_000_000), "mode": "direct", "policy": "heuristic"}
        g = _draw_graph(rng, 5_000, 100_000_000)
        return {"op": op, **g, "mode": "oriented", "policy": "gallop" if g["kind"] == "er" else "bitmap"}
    if op == "job":
        out = rng.choice(("counts", "scan"))
        return {"op": op, **_draw_graph(rng, 30_000, 32_000_000 if out == "counts" else 4_000_000), "out": out,
                "eps": eps, "mu": mu}
    if op == "query":
        out = rng.choice(("device", "host"))
        return {"op": op, **_draw_graph(rng, 30_000, 64_000_000 if out == "device" else 1_000_000), "eps": eps,
                "mu": mu, "out": out}
    if op == "edges":
        return {"op": op, **_draw_graph(rng, 20_000, 12_000_000)}
    return {"op": op, "k": rng.randint(8, 64), "emin": 1000, "emax": _log_int(rng, 20_000, 400_000), "eps": eps,
            "mu": mu}


# ---- inputs ------------------------------------------------------------------
def _draw_keys(c, k, gen, cdf):
    """k undirected draws as lo * n + hi, self loops left out."""
    n, keys = c["n"], []
    for k0 in range(0, k, 1 << 25):
        b = min(1 << 25, k - k0)
        if c["kind"] == "rmat":
            u = torch.zeros(b, dtype=torch.int64, device="cuda")
            v = torch.zeros(b, dtype=torch.int64, device="cuda")
            for _ in range(n.bit_length() - 1):
                r = torch.rand(b, device="cuda", generator=gen)
                u = 2 * u + (r >= RMAT[0] + RMAT[1])
                v = 2 * v + (((r >= RMAT[0]) & (r < RMAT[0] + RMAT[1])) | (r >= sum(RMAT)))
        elif c["kind"] == "er":
            u = torch.randint(n, (b,), device="cuda", generator=gen)
            v = torch.randint(n, (b,), device="cuda", generator=gen)
        else:
            r = torch.rand(2, b, device="cuda", generator=gen, dtype=torch.float64)
            u, v = torch.searchsorted(cdf, r).clamp_(max=n - 1)
        key = torch.minimum(u, v) * n + torch.maximum(u, v)
        keys.append(key[u != v])
    return torch.cat(keys)


def _edges(c, gen):
    """c["edges"] distinct undirected edges in random order: int64 u, v on the GPU."""
    n, e, cdf, perm = c["n"], c["edges"], None, None
    if c["kind"] == "chunglu":
        # expected degrees ~ i^(-1/(2.1-1)), at most a 20th of the vertices
        w = torch.arange(1, n + 1, device="cuda", dtype=torch.float64).pow_(-1.0 / 1.1)
        w = (w * (2 * e / w.sum())).clamp_(max=n / 20)
        cdf = torch.cumsum(w, 0)
        cdf /= cdf[-1].clone()
        perm = torch.randperm(n, device="cuda", generator=gen)
    key = torch.unique(_draw_keys(c, e + e // 10 + 64, gen, cdf))
    while key.numel() < e:
        key = torch.unique(torch.cat((key, _draw_keys(c, e // 3 + 64, gen, cdf))))
    key = key[torch.randperm(key.numel(), device="cuda", generator=gen)[:e]]
    u, v = key // n, key % n
    return (u, v) if perm is None else (perm[u], perm[v])


def _csr_of(u, v, n):
    """Sorted, deduplicated, symmetric CSR without self loops: int32 off[n+1], dst[m] on the GPU."""
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.cat((u * n + v, v * n + u)))
    del u, v, keep
    off = torch.searchsorted(key, torch.arange(n + 1, device="cuda") * n).to(torch.int32)
    return off, (key % n).to(torch.int32)


def _csr(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    off, dst = _csr_of(*_edges(c, gen), c["n"])
    torch.cuda.empty_cache()
    return off, dst


def _edge_list(c, seed):
    """The edges as a file would hold them: either direction first, an eighth of them twice, some self loops."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u, v = _edges(c, gen)
    n, e = c["n"], u.numel()
    again = torch.randint(e, (e // 8,), device="cuda", generator=gen)
    loops = torch.randint(n, (e // 64,), device="cuda", generator=gen)
    u, v = torch.cat((u, v[again], loops)), torch.cat((v, u[again], loops))
    swap = torch.rand(u.numel(), device="cuda", generator=gen) < 0.5
    order = torch.randperm(u.numel(), device="cuda", generator=gen)
    return torch.where(swap, v, u)[order], torch.where(swap, u, v)[order]


def _graph(off, dst):
    return accx.Graph.from_device(off.data_ptr(), dst.data_ptr(), off.numel() - 1, dst.numel(), validate=True)


def _batch_members(c):
    """k graphs of emin..emax edges (even over the logarithm), R-MAT and Erdos-Renyi in turn."""
    out = []
    for i in range(c["k"]):
        e = int(c["emin"] * (c["emax"] / c["emin"]) ** ((i + 0.5) / c["k"]))
        n = 1 << int(round(np.log2(e / 14))) if i % 2 else e // 8
        out.append({"kind": "rmat" if i % 2 else "er", "n": n, "edges": e})
    return out


def prepare(case, seed):
    c, op = case, case["op"]
    if op == "edges":
        u, v = _edge_list(c, seed)
        return {"case": c, "u": u.to(torch.int32).cpu().numpy().view(np.uint32),
                "v": v.to(torch.int32).cpu().numpy().view(np.uint32)}
    if op == "batch":
        seeds = np.random.default_rng(seed).integers(1 << 60, size=c["k"])
        graphs = [_graph(*_csr(m, int(s))) for m, s in zip(_batch_members(c), seeds)]
        batch = accx.Batch(graphs)
        batch.union.relabel()
        stream = torch.cuda.Stream()
        batch.capture(policy="bitmap", bias=2, stream=stream, orient=True)
        cnt = torch.empty(batch.union.m, dtype=torch.int32, device="cuda")
        return {"case": c, "batch": batch, "stream": stream, "cnt": cnt}
    off, dst = _csr(c, seed)
    n, m = off.numel() - 1, dst.numel()
    if op == "job":
        st = {"case": c, "n": n, "m": m, "off": off.cpu().pin_memory(), "dst": dst.cpu().pin_memory()}
        if c["out"] == "counts":
            st["cnt"] = torch.empty(m, dtype=torch.int32).pin_memory()
        else:
            st["pairs"] = np.full((m, 2), -1, np.int32)  # room for every entry; filled from the front
        return st
    g = _graph(off, dst)
    st = {"case": c, "g": g}
    if op == "count":
        if c["mode"] == "oriented":
            g.relabel()
        st["cnt"] = torch.empty(m, dtype=torch.int32, device="cuda")
        return st
    g.relabel()
    g.count(policy="bitmap", bias=2, out=None, orient=True)
    if c["out"] == "device":
        st["sim"] = torch.empty(m, dtype=torch.uint8, device="cuda")
        st["label"] = torch.empty(n, dtype=torch.int32, device="cuda")
        st["cluster"] = torch.empty(n, dtype=torch.int32, device="cuda")
    return st


# ---- one pass ----------------------------------------------------------------
def _stream():
    return torch.cuda.current_stream().cuda_stream


def _ok(status, what):
    if status != accx.OK:
        raise accx.AccxError(status, what)


def _summary(d):
    """The query's numbers; its digest is a hash of the labels and clusters, which are returned whole."""
    return {k: v for k, v in d.items() if k != "digest"}


class _View:
    """A graph's device array as torch takes it, keeping the graph while the tensor lives."""

    def __init__(self, graph, ptr, count):
        self.graph = graph
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def run(state):
    c = state["case"]
    op = c["op"]
    if op == "count":
        state["g"].count(policy=c["policy"], bias=2, out=state["cnt"].data_ptr(), stream=_stream(),
                         orient=c["mode"] == "oriented")
        return state["cnt"]
    if op == "query":
        g = state["g"]
        if c["out"] == "host":
            r = g.scan(c["eps"], c["mu"], stream=_stream())
            return {**r, "summary": _summary(r["summary"])}
        s = accx.ScanSummary()
        _ok(accx.lib.accx_scan_query(g._h, c["eps"], c["mu"], ctypes.c_void_p(state["sim"].data_ptr()),
                                     ctypes.c_void_p(state["label"].data_ptr()),
                                     ctypes.c_void_p(state["cluster"].data_ptr()), ctypes.byref(s),
                                     ctypes.c_void_p(_stream())), "scan_query")
        return {"sim": state["sim"], "label": state["label"], "cluster": state["cluster"],
                "summary": _summary(s.as_dict())}
    if op == "job":
        g = accx.Graph.from_device(state["off"].data_ptr(), state["dst"].data_ptr(), state["n"], state["m"],
                                   validate=True, stream=_stream())
        g.relabel(stream=_stream())
        if c["out"] == "counts":
            g.count(policy="bitmap", bias=2, out=state["cnt"].data_ptr(), stream=_stream(), orient=True)
            out = state["cnt"]
        else:
            g.count(policy="bitmap", bias=2, out=None, stream=_stream(), orient=True)
            r = g.scan(c["eps"], c["mu"], want_sim=False, stream=_stream())
            k, p = ctypes.c_uint64(), state["pairs"]
            _ok(accx.lib.accx_scan_pairs(g._h, p.ctypes.data_as(ctypes.c_void_p), len(p), ctypes.byref(k),
                                         ctypes.c_void_p(_stream())), "scan_pairs")
            out = {"label": r["label"], "cluster": r["cluster"], "pairs": p, "npairs": k.value,
                   "summary": _summary(r["summary"])}
        g.free()
        return out
    if op == "edges":
        g = accx.Graph.from_edges(state["u"], state["v"], c["n"], stream=_stream())
        off, dst, _ = g.device_ptrs()
        return [torch.as_tensor(_View(g, off, g.n + 1), device="cuda"),
                torch.as_tensor(_View(g, dst, g.m), device="cuda")]
    b, stream = state["batch"], state["stream"]
    b.launch(stream=stream)
    r = b.union.scan(c["eps"], c["mu"], want_sim=False, stream=stream)
    _ok(accx.lib.accx_cn_read(b.union._h, ctypes.c_void_p(state["cnt"].data_ptr()),
                              ctypes.c_void_p(stream.cuda_stream)), "cn_read")
    return {"counts": state["cnt"], "label": r["label"], "cluster": r["cluster"], "summary": _summary(r["summary"])}


def work(case):
    """Bytes: the input read once and the answer written once."""
    c, op = case, case["op"]
    if op == "batch":
        members = _batch_members(c)
        n, m = sum(g["n"] for g in members), 2 * sum(g["edges"] for g in members)
        return {"bytes": float(8 * m + 12 * n), "flops": 0.0}
    n, m = c["n"], 2 * c["edges"]
    csr = 4 * n + 4 * m
    if op == "edges":
        k = c["edges"] + c["edges"] // 8 + c["edges"] // 64
        return {"bytes": float(8 * k + csr), "flops": 0.0}
    if op == "count" or (op == "job" and c["out"] == "counts"):
        return {"bytes": float(csr + 4 * m), "flops": 0.0}
    if op == "job":
        return {"bytes": float(csr + 8 * n), "flops": 0.0}
    return {"bytes": float(csr + 4 * m + m + 8 * n), "flops": 0.0}  # the counts too; the similarity bytes out


# ---- the answers from the definitions, in plain torch and numpy ----------------
def _counts(off, dst):
    """2 + |N(u) and N(v)| of every entry: the shorter list's ids looked up in the longer one."""
    n, m = off.numel() - 1, dst.numel()
    off, dst = off.to(torch.int64), dst.to(torch.int64)
    deg = off[1:] - off[:-1]
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    key = src * n + dst
    cnt = torch.zeros(m, dtype=torch.int64, device="cuda")
    e = torch.nonzero(src < dst).flatten()
    s, t = src[e], dst[e]
    swap = deg[s] > deg[t]
    s, t = torch.where(swap, t, s), torch.where(swap, s, t)
    ends = torch.cumsum(deg[s], 0)
    a = 0
    while a < e.numel():
        base = int(ends[a - 1]) if a else 0
        b = max(a + 1, int(torch.searchsorted(ends, base + (1 << 26), right=True)))
        ln = deg[s[a:b]]
        which = torch.repeat_interleave(torch.arange(b - a, device="cuda"), ln)
        at = torch.arange(which.numel(), device="cuda") - (ends[a:b] - ln - base)[which] + off[s[a:b]][which]
        want = t[a:b][which] * n + dst[at]
        hit = key[torch.searchsorted(key, want).clamp_(max=m - 1)] == want
        cnt[e[a:b]] = torch.zeros(b - a, dtype=torch.int64, device="cuda").index_add_(0, which, hit.to(torch.int64))
        a = b
    rev = torch.searchsorted(key, dst[e] * n + src[e])
    cnt[rev] = cnt[e]
    return cnt + 2, src, dst, deg


def _scan(off, dst, eps, mu):
    """The reference's SCAN semantics: similarity in extended precision, clusters of similar
    cores named by their smallest vertex, hubs next to two or more clusters."""
    cnt, src, dst, deg = _counts(off, dst)
    n = off.numel() - 1
    d = (deg + 1).cpu().numpy()
    s, t = src.cpu().numpy(), dst.cpu().numpy()
    x = cnt.cpu().numpy().astype(np.longdouble) / np.sqrt((d[s] * d[t]).astype(np.longdouble))
    sim = torch.from_numpy(x.astype(np.float64) >= eps).cuda()
    core = torch.zeros(n, dtype=torch.int64, device="cuda").index_add_(0, src, sim.to(torch.int64)) >= mu
    link = sim & core[src] & core[dst]
    a, b = src[link], dst[link]
    root = torch.arange(n, device="cuda")
    while True:
        new = root.scatter_reduce(0, a, root[b], "amin")
        new = new[new]
        if torch.equal(new, root):
            break
        root = new
    near = core[dst] & ~core[src]
    r = root[dst[near]]
    lo = torch.full((n,), n, device="cuda").scatter_reduce(0, src[near], r, "amin")
    hi = torch.full((n,), -1, device="cuda").scatter_reduce(0, src[near], r, "amax")
    hub = (hi >= 0) & (lo != hi) & ~core
    label = core.to(torch.int32) + 2 * hub.to(torch.int32)
    cluster = torch.where(core, root, torch.full_like(root, -1)).to(torch.int32)
    p = sim & core[src] & ~core[dst]
    pairs = torch.unique(root[src[p]] * n + dst[p])
    pairs = torch.stack((pairs // n, pairs % n), 1).to(torch.int32)
    summary = {"cores": int(core.sum()), "clusters": int((core & (root == torch.arange(n, device="cuda"))).sum()),
               "hubs": int(hub.sum()), "outliers": int((label == 0).sum()), "similar_entries": int(sim.sum()),
               "noncore_pairs": 0}
    return sim.to(torch.uint8), label, cluster, pairs, summary


def exact(case, seed):
    c, op = case, case["op"]
    if op == "batch":
        return None
    if op == "edges":
        return list(_csr_of(*_edge_list(c, seed), c["n"]))
    # the look-ups grow faster than the edges where there are hubs
    if c["edges"] > (60_000_001 if c["kind"] == "er" else 4_000_000):
        return None
    off, dst = _csr(c, seed)
    if op == "count" or (op == "job" and c["out"] == "counts"):
        return _counts(off, dst)[0].to(torch.int32)
    sim, label, cluster, pairs, summary = _scan(off, dst, c["eps"], c["mu"])
    if op == "job":
        room = torch.full((dst.numel(), 2), -1, dtype=torch.int32, device="cuda")
        room[:len(pairs)] = pairs
        return {"label": label, "cluster": cluster, "pairs": room, "npairs": len(pairs), "summary": summary}
    return {"sim": sim, "label": label, "cluster": cluster, "summary": summary}
