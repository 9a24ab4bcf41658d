"""The workloads whose speed this repository watches, through its public entry
points (nido_b200.capi, the binding of include/nido_b200.h).

They are whole Louvain runs (one graph resident on the device, from a request
of a thousand vertices to R-MAT scale 22; many graphs in one batch; requests
through the server; upload, run and free of a host graph) and single
operators (the GraphGPU sweep, the allocation-free modularity).  Weights are
unit, integers 1..8 and FP64 (uniform, lognormal), as the generators in
nido_b200/workloads.py draw them; graphs are R-MAT (0.57, 0.19, 0.19, 0.05),
stochastic block models with power-law communities and planted partitions.
Inputs are drawn on the GPU from the seed alone.
"""
import numpy as np
import torch

from nido_b200 import capi, workloads

DEV = "cuda:0"


# ---- cases -------------------------------------------------------------------

def listed():
    return [
        # the smallest request of the serving stream: launches and round trips
        {"name": "run_sbm_1k_uniform", "op": "run", "kind": "sbm", "nv": 1000, "degree": 32.0, "weights": "uniform",
         "batches": 2},
        # a small graph of the many-graph set run alone, ragged size, integer weights
        {"name": "run_rmat_20k_int", "op": "run", "kind": "rmat", "nv": 20011, "degree": 32.0, "weights": "int",
         "batches": 2},
        # the planted-partition configuration: 65,536 vertices, 256 blocks, one batch
        {"name": "run_planted_64k_uniform", "op": "run", "kind": "planted", "nv": 65536, "degree": 32.0,
         "weights": "uniform", "batches": 1},
        # the command line's -c: conflict-free colour-class batches
        {"name": "run_colors_sbm_100k_int", "op": "colors", "kind": "sbm", "nv": 100003, "degree": 32.0,
         "weights": "int", "batches": 2},
        # the reference's tie rule (--tie=nido), used for parity with it
        {"name": "run_tie_rmat18_unit", "op": "tie", "kind": "rmat", "nv": 1 << 18, "degree": 32.0,
         "weights": "unit", "batches": 2},
        # -b 32 on power-law communities with lognormal weights (the batched-partition configuration's shape)
        {"name": "run_sbm_2m_lognormal_b32", "op": "run", "kind": "sbm", "nv": 1 << 21, "degree": 32.0,
         "weights": "lognormal", "batches": 32},
        # the R-MAT scale 22 configuration, unit weights: the largest
        {"name": "run_rmat22_unit", "op": "run", "kind": "rmat", "nv": 1 << 22, "degree": 32.0, "weights": "unit",
         "batches": 2},
        # the many-graph configuration at an eighth of its graphs: uneven SBM / R-MAT mix, integer weights
        {"name": "batch_512_graphs_int", "op": "batch", "kind": "many", "graphs": 512, "edges": 60000000,
         "weights": "int", "batches": 2},
        # a host graph uploaded, run and freed, as the command line does
        {"name": "oneshot_rmat_300k_uniform", "op": "oneshot", "kind": "rmat", "nv": 300007, "degree": 32.0,
         "weights": "uniform", "batches": 2},
        # requests of mixed sizes through the server
        {"name": "serve_12_mixed_uniform", "op": "serve", "kind": "many", "graphs": 12, "nv": 100000,
         "weights": "uniform", "batches": 2},
        # GraphGPU's operators called one by one: four sweeps and their modularity
        {"name": "sweeps_sbm_250k_lognormal", "op": "sweeps", "kind": "sbm", "nv": 250007, "degree": 32.0,
         "weights": "lognormal", "batches": 2},
        # modularity of a partition in caller-owned device arrays, no allocation
        {"name": "noalloc_rmat20_uniform", "op": "noalloc", "kind": "rmat", "nv": 1 << 20, "degree": 32.0,
         "weights": "uniform", "batches": 1},
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    op = rng.choice(["run", "run", "run", "run", "batch", "batch", "colors", "tie", "oneshot", "serve", "sweeps",
                     "noalloc"])
    if op == "batch":
        return {"op": op, "kind": "many", "graphs": _log(rng, 16, 512), "edges": _log(rng, 1000000, 60000000),
                "weights": "int", "batches": rng.randint(1, 3)}
    if op == "serve":
        return {"op": op, "kind": "many", "graphs": rng.randint(4, 12), "nv": _log(rng, 5000, 100000),
                "weights": "uniform", "batches": 2}
    lo, hi = {"run": (1000, 1 << 21), "colors": (5000, 150000), "tie": (5000, 1 << 18), "oneshot": (5000, 400000),
              "sweeps": (10000, 400000), "noalloc": (1000, 1 << 20)}[op]
    case = {"op": op, "kind": rng.choice(["sbm", "rmat"]), "nv": _log(rng, lo, hi),
            "degree": round(rng.uniform(8.0, 64.0 if op != "run" else 40.0), 2),
            "weights": rng.choice(["unit", "int", "uniform", "lognormal"]), "batches": rng.choice([1, 2, 2, 3, 8])}
    if op in ("colors", "tie"):
        case["weights"] = rng.choice(["unit", "int"])
    if op == "sweeps" or op == "noalloc":
        case["weights"] = rng.choice(["int", "uniform", "lognormal"])
    return case


# ---- graphs, drawn on the GPU --------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rmat_pairs(gen, nv, n):
    scale = max(1, int(nv - 1).bit_length())
    got_u, got_v, have = [], [], 0
    while have < n:
        m = n - have if have == 0 else 2 * (n - have) + 64
        u = torch.zeros(m, dtype=torch.int64, device=DEV)
        v = torch.zeros(m, dtype=torch.int64, device=DEV)
        for _ in range(scale):
            r = torch.rand(m, generator=gen, device=DEV)
            hi = r >= 0.76  # quadrants (0,0) .57, (0,1) .19, (1,0) .19, (1,1) .05
            lo = ((r >= 0.57) & ~hi) | (r >= 0.95)
            u.mul_(2).add_(hi)
            v.mul_(2).add_(lo)
        ok = (u < nv) & (v < nv)
        u, v = u[ok][:n - have], v[ok][:n - have]
        got_u.append(u)
        got_v.append(v)
        have += int(u.numel())
    return torch.cat(got_u), torch.cat(got_v)


def _block_pairs(gen, nv, n, intra, start, size):
    """Pairs whose second end is in the first end's block with probability
    `intra`; start and size: first vertex and vertices of every vertex's block."""
    u = torch.randint(0, nv, (n,), generator=gen, device=DEV)
    r = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)
    inside = torch.rand(n, generator=gen, device=DEV) < intra
    v = torch.where(inside, start[u] + (r * size[u]).long(), (r * nv).long())
    return u, v


def _pairs(gen, kind, nv, degree):
    n = max(1, int(round(nv * degree / 2)))
    if kind == "rmat":
        return _rmat_pairs(gen, nv, n)
    if kind == "planted":
        size = torch.full((nv,), 256, dtype=torch.int64, device=DEV)
        start = torch.arange(nv, device=DEV) // 256 * 256
        return _block_pairs(gen, nv, n, 0.8, start, torch.minimum(size, nv - start))
    # community sizes: power law of exponent 2.5 clipped to 16..65,536
    r = torch.rand(nv // 16 + 1, generator=gen, device=DEV, dtype=torch.float64)
    lo, hi = 16.0 ** -1.5, 65536.0 ** -1.5
    sizes = ((lo - r * (lo - hi)) ** (-1.0 / 1.5)).long()
    ends = torch.cumsum(sizes, 0)
    block = torch.searchsorted(ends, torch.arange(nv, device=DEV), right=True)
    start = (ends - sizes)[block]
    u, v = _block_pairs(gen, nv, n, 0.7, start, torch.minimum(sizes[block], nv - start))
    perm = torch.randperm(nv, generator=gen, device=DEV)
    return perm[u], perm[v]


def _weights(gen, mode, n):
    if mode == "unit":
        return torch.ones(n, dtype=torch.float64, device=DEV)
    if mode == "int":
        return torch.randint(1, 9, (n,), generator=gen, device=DEV).double()
    if mode == "uniform":
        return 0.5 + torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)
    return torch.exp(0.5 * torch.randn(n, generator=gen, device=DEV, dtype=torch.float64))


def _device_csr(seed, kind, nv, degree, weights):
    """Symmetric CSR without self-loops and duplicates, rows sorted by id."""
    gen = _generator(seed)
    u, v = _pairs(gen, kind, nv, degree)
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.minimum(u, v) * nv + torch.maximum(u, v))
    w = _weights(gen, weights, key.numel())
    lo, hi = key // nv, key % nv
    key, order = torch.sort(torch.cat([key, hi * nv + lo]))
    w = torch.cat([w, w])[order]
    off = torch.searchsorted(key, torch.arange(nv + 1, device=DEV) * nv)
    return off, key % nv, w


def _host_csr(seed, kind, nv, degree, weights):
    off, adj, w = _device_csr(seed, kind, nv, degree, weights)
    return capi.Csr(off.cpu().numpy(), adj.cpu().numpy(), w.cpu().numpy())


def _many(case, seed):
    """(vertex bases, packed CSR) of the many-graph law: vertex counts
    log-uniform, SBM or R-MAT, degrees uniform in 8..64, scaled to the edges.
    The sizes are the case's, the edges and weights the seed's."""
    V, d, kind = workloads.many_graph_plan(case["graphs"], 4, float(case["edges"]))
    parts = [_host_csr(seed * 100003 + i, "rmat" if k else "sbm", int(n), float(x), case["weights"])
             for i, (n, x, k) in enumerate(zip(V, d, kind))]
    return capi.pack_graphs(parts)


# ---- what a program has in hand before the call ----------------------------------

class _Held(dict):
    """Inputs and handles of one prepared case; handles are closed with it."""

    def __del__(self):
        for k in ("graph", "batch", "server"):
            if self.get(k) is not None:
                self[k].close()
        if self.get("pinned") is not None:
            capi.host_unregister(self["pinned"])


_context = None


def _ctx():
    """The program's one context (one device, one stream)."""
    global _context
    if _context is None:
        _context = capi.Context(0)
    return _context


def _registered(n):
    a = np.zeros(n, np.int64)
    capi.host_register(a)
    return a


def prepare(case, seed):
    op, s = case["op"], _Held()
    s["op"], s["batches"] = op, case["batches"]
    if op == "batch":
        s["batch"] = capi.Batch(_ctx(), nbatches=case["batches"], packed=_many(case, seed))
        s["pinned"] = _registered(s["batch"].nv)
    elif op == "serve":
        rng = np.random.default_rng(5)  # the sizes are the case's
        sizes = np.exp(rng.uniform(np.log(1000), np.log(case["nv"]), case["graphs"])).astype(np.int64)
        s["requests"] = [_host_csr(seed * 1009 + i, "rmat" if i % 2 else "sbm", int(n), 32.0, case["weights"])
                         for i, n in enumerate(sizes)]
        s["server"] = capi.Server(0, 0, 4)
    elif op == "noalloc":
        off, adj, w = _device_csr(seed, case["kind"], case["nv"], case["degree"], case["weights"])
        nv = case["nv"]
        comm = torch.randint(0, nv // 40 + 1, (nv,), generator=_generator(seed + 1), device=DEV)
        row = torch.repeat_interleave(torch.arange(nv, device=DEV), off[1:] - off[:-1])
        a = torch.zeros(nv, dtype=torch.float64, device=DEV).index_add_(0, comm[row], w)
        s.update(off=off, adj=adj, w=w, comm=comm, a=a, m=float(w.sum()) / 2, nv=nv,
                 q=torch.zeros(1, dtype=torch.float64, device=DEV))
    else:
        g = _host_csr(seed, case["kind"], case["nv"], case["degree"], case["weights"])
        if op == "oneshot":
            s["csr"] = g
        else:
            s["graph"] = capi.Graph(_ctx(), g, case["batches"])
            if op != "sweeps":
                s["pinned"] = _registered(g.nv)
    return s


# ---- one pass ---------------------------------------------------------------------

def _answer(part, st):
    # the statistics' per-phase arrays have a fixed length; phases not reached are zero
    return {"partition": part, "q": st.final_q, "phases": int(st.phases), "q_phase": np.array(st.q_phase[:]),
            "loops_phase": np.array(st.loops_phase[:], np.int64), "nv_phase": np.array(st.nv_phase[:], np.int64)}


def run(state):
    op = state["op"]
    if op in ("run", "colors", "tie"):
        tie = capi.NIDO_TIE_NIDO if op == "tie" else capi.NIDO_TIE_SMALLEST_ID
        return _answer(*state["graph"].run(tie=tie, color_batches=op == "colors", out=state["pinned"]))
    if op == "batch":
        _, q, phases, loops, _ = state["batch"].run(out=state["pinned"])
        return {"partition": state["pinned"], "q": q, "phases": phases, "loops": loops}
    if op == "oneshot":
        with capi.Graph(_ctx(), state["csr"], state["batches"]) as g:
            return _answer(*g.run())
    if op == "serve":
        server = state["server"]
        tickets = [server.submit(g, state["batches"]) for g in state["requests"]]
        done = [server.wait(t) for t in tickets]
        return {"partitions": [p for p, _ in done], "q": np.array([i.final_q for _, i in done])}
    if op == "sweeps":
        g = state["graph"]
        g.singleton_partition()
        qs = []
        for _ in range(4):
            for b in range(state["batches"]):
                g.louvain_update(b)
                g.update_community_weights(b)
                g.update_community_ids(b)
            qs.append(g.compute_modularity())
        comm, old, a = g.state()
        return {"q": np.array(qs), "comm": comm, "old": old, "a": a}
    capi._check(capi.lib().nido_modularity_noalloc(
        torch.cuda.current_stream().cuda_stream, state["nv"], state["off"].data_ptr(), state["adj"].data_ptr(),
        state["w"].data_ptr(), state["comm"].data_ptr(), state["a"].data_ptr(), state["m"], state["q"].data_ptr()))
    return {"q": state["q"]}


def work(case):
    """The graph read once (4-byte ids, 8-byte weights and offsets on the
    device; 8-byte ids where the caller's arrays are read) and the partition
    written once; two operations an edge."""
    if case["op"] == "batch":
        ne, nv = case["edges"], case["edges"] / 36.0
    elif case["op"] == "serve":
        nv = case["graphs"] * (case["nv"] - 1000) / np.log(case["nv"] / 1000)
        ne = 32.0 * nv
    else:
        nv, ne = case["nv"], case["nv"] * case["degree"]
    ids = 8 if case["op"] in ("oneshot", "serve", "noalloc") else 4
    out = 8.0 if case["op"] == "noalloc" else 8.0 * nv
    state = 24.0 * nv if case["op"] == "noalloc" else 8.0 * nv  # offsets (and communities and degrees)
    return {"bytes": (ids + 8.0) * ne + state + out, "flops": 2.0 * ne}


# ---- the same numbers from plain torch in 64 bits ------------------------------------

def _cuts(off, nb):
    """The -b cut rule: each batch ends at the first vertex past the average edge count."""
    nv = len(off) - 1
    ave, parts = int(off[nv]) // nb, [0]
    while len(parts) <= nb + 1:
        i = int(np.searchsorted(off, off[parts[-1]] + ave, side="right"))
        i = max(i, parts[-1] + 1)
        parts.append(min(i, nv))
        if i >= nv:
            break
    if len(parts) > nb + 1:
        extra = (nv - parts[nb]) // nb
        parts = [0] + [p + extra for p in parts[1:nb]] + [nv]
    return parts[:nb + 1] + [nv] * (nb + 1 - len(parts))


def _modularity(row, adj, w, comm, a, m):
    return float((w * (comm[row] == comm[adj])).sum() / (2 * m) - (a * a).sum() / (4 * m * m))


def _sweeps_exact(case, seed):
    off, adj, w = _device_csr(seed, case["kind"], case["nv"], case["degree"], case["weights"])
    nv = case["nv"]
    row = torch.repeat_interleave(torch.arange(nv, device=DEV), off[1:] - off[:-1])
    k = torch.zeros(nv, dtype=torch.float64, device=DEV).index_add_(0, row, w)
    m = float(k.sum()) / 2
    cuts = _cuts(off.cpu().numpy(), case["batches"])
    comm, a, qs = torch.arange(nv, device=DEV), k.clone(), []
    for _ in range(4):
        for v0, v1 in zip(cuts[:-1], cuts[1:]):
            e0, e1 = int(off[v0]), int(off[v1])
            key, inv = torch.unique(row[e0:e1] * nv + comm[adj[e0:e1]], return_inverse=True)
            e = torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, inv, w[e0:e1])
            v, c = key // nv, key % nv
            own = comm[v] == c
            eown = torch.zeros(nv, dtype=torch.float64, device=DEV)
            eown[v[own]] = e[own]
            gain = (e - k[v] * a[c] / (2 * m)) / m
            gain = torch.where(own, torch.full_like(gain, -1e308), gain)
            best = torch.full((nv,), -1e308, dtype=torch.float64, device=DEV).scatter_reduce_(0, v, gain, "amax")
            cand = torch.full((nv,), nv, device=DEV).scatter_reduce_(
                0, v, torch.where((gain == best[v]) & ~own, c, torch.full_like(c, nv)), "amin")
            self_gain = (eown - k * (a[comm] - k) / (2 * m)) / m
            go = (cand < nv) & (best - self_gain > 0)
            go[:v0] = False
            go[v1:] = False
            a.index_add_(0, comm[go], -k[go]).index_add_(0, cand[go], k[go])
            comm = torch.where(go, cand, comm)
        qs.append(_modularity(row, adj, w, comm, a, m))
    return {"q": np.array(qs), "comm": None, "old": None, "a": a.cpu().numpy()}


def exact(case, seed):
    if case["op"] == "noalloc":
        s = prepare(case, seed)
        row = torch.repeat_interleave(torch.arange(s["nv"], device=DEV), s["off"][1:] - s["off"][:-1])
        q = _modularity(row, s["adj"], s["w"], s["comm"], s["a"], s["m"])
        return {"q": torch.tensor([q], dtype=torch.float64)}
    if case["op"] == "sweeps":
        return _sweeps_exact(case, seed)
    return None  # the partition a whole run reaches has no closed value
