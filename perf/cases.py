"""Performance cases: exact group Steiner tree queries through the public API.

A user of this engine keeps one graph and its group index resident
(`engine.Engine`) and asks queries of it in one of five ways, the modes here:

  plain    `Engine.query`, one query after another (the reference's way);
  batch    `Engine.query_batch`, many queries sharing device rounds;
  serve    `engine.Server`: requests submitted together, polled until done;
  noalloc  `Engine.query_noalloc`, everything in the library's static scratch;
  load     a new `Engine` from host CSR arrays, then its first query: what
           every start of a program pays.

The graph belongs to the case (the handle that a program keeps; it is made once
from the case's sizes), the queries to the seed.  Graphs are Chung-Lu power-law
or R-MAT with weights uniform in [1, 100], groups have truncated Zipf sizes and
cover every vertex, as in `gpugst_b200.gen`, but are generated with torch on the
GPU: the largest takes seconds instead of minutes.

A query's optimal cost is unique, its optimal tree is not (ties are frequent
with weights up to 100 and are broken by the order in which the GPU's threads
arrive), so a pass returns every query's status and cost, and the weight of the
tree it was given.
"""
import time

import numpy as np
import torch

from gpugst_b200 import engine

NO_HOPS = -1  # no hop bound


def listed():
    def case(name, mode, n, k, D, share, graph="chung_lu", V=10_000, E=50_000, gamma=2.5, groups=2_000, zipf=1.5,
             smax=50):
        return {"name": name, "mode": mode, "n": n, "k_lo": k[0], "k_hi": k[1], "D_lo": D[0], "D_hi": D[1],
                "hop_share": share, "graph": graph, "V": V, "E": E, "gamma": gamma, "groups": groups, "zipf": zipf,
                "smax": smax}

    g170k = dict(V=170_000, E=6_800_000, gamma=2.3, groups=200_000, smax=200)
    rmat = dict(graph="rmat", V=1 << 20, E=10_000_000, groups=500_000, smax=200)
    g3m = dict(V=3_000_000, E=117_000_000, gamma=2.1, groups=1_000_000, zipf=1.3, smax=500)
    none = (NO_HOPS, NO_HOPS)
    return [
        # the smallest call: one query on a graph that fits the caches, where launches and latency count
        case("plain_10k", "plain", 1, (3, 3), none, 0.0),
        # the same graph under hop bounds, as in an interactive exploration
        case("plain_10k_hop", "plain", 4, (3, 5), (3, 5), 1.0),
        # a host that may not allocate device memory while it answers
        case("noalloc_10k", "noalloc", 1, (4, 4), none, 0.0),
        # an odd mid-size graph with the largest queries: merges of many subsets
        case("plain_54k_k7", "plain", 2, (6, 7), none, 0.0, V=54_321, E=400_003, groups=30_011, smax=100),
        # one query at a time on the social-network-sized graph
        case("plain_170k", "plain", 6, (3, 5), none, 0.0, **g170k),
        # an experiment's query file in one batch
        case("batch_170k", "batch", 90, (3, 5), none, 0.0, **g170k),
        # a service with mixed requests in flight
        case("serve_170k", "serve", 64, (3, 6), (2, 4), 0.5, **g170k),
        # the start of a program on that graph, up to its first answer
        case("load_170k", "load", 1, (3, 3), none, 0.0, **g170k),
        # hop-bounded queries on the R-MAT graph, one at a time and as a batch
        case("plain_rmat_hop", "plain", 6, (3, 5), (2, 4), 1.0, **rmat),
        case("batch_rmat_hop", "batch", 48, (3, 5), (2, 4), 1.0, **rmat),
        # the largest graph: mixed queries one at a time and batched
        case("plain_3m", "plain", 6, (3, 6), (2, 4), 0.5, **g3m),
        case("batch_3m", "batch", 48, (3, 6), (2, 4), 0.5, **g3m),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    mode = rng.choice(["plain", "plain", "batch", "batch", "serve", "noalloc", "load"])
    graph = "rmat" if mode != "noalloc" and rng.random() < 0.25 else "chung_lu"
    if graph == "rmat":
        V = 1 << rng.randint(12, 20)
        degree = log_int(6, 24)
    else:
        V = log_int(2_000, 20_000 if mode == "noalloc" else 800_000)
        degree = log_int(6, 80)
    E = max(V, min(V * degree // 2, 9_000_000) + rng.randint(0, 999))
    hops = rng.choice([0.0, 0.0, 0.5, 1.0])
    k_lo = rng.randint(2, 5)
    k_hi = min(k_lo + rng.randint(0, 2), 4 if mode == "noalloc" else 6)
    D_lo = rng.randint(2, 4)
    n = {"plain": log_int(1, 8), "batch": log_int(8, 96), "serve": log_int(8, 64), "noalloc": rng.randint(1, 3),
         "load": 1}[mode]
    return {"mode": mode, "n": n, "k_lo": min(k_lo, k_hi), "k_hi": k_hi, "D_lo": D_lo if hops else NO_HOPS,
            "D_hi": min(D_lo + rng.randint(0, 2), 4) if hops else NO_HOPS, "hop_share": hops, "graph": graph, "V": V,
            "E": E, "gamma": round(rng.uniform(2.1, 2.6), 2), "groups": max(64, int(V * rng.uniform(0.2, 1.2))),
            "zipf": round(rng.uniform(1.3, 1.6), 2), "smax": rng.choice([20, 50, 100, 200])}


# ---------------------------------------------------------------------------
# Graphs and groups
# ---------------------------------------------------------------------------

def _endpoints(case, n, gen):
    """n vertex pairs of the case's degree distribution."""
    V = case["V"]
    if case["graph"] == "rmat":  # initiator (0.57, 0.19, 0.19, 0.05), labels permuted
        u = torch.zeros(n, dtype=torch.int64, device="cuda")
        v = torch.zeros_like(u)
        for _ in range(V.bit_length() - 1):
            r = torch.rand(n, device="cuda", generator=gen)
            u = u * 2 + (r >= 0.76)
            v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        perm = torch.randperm(V, device="cuda", generator=gen)
        return perm[u], perm[v]
    # Chung-Lu: vertex i has weight (i + i0)^(-1/(gamma-1)), i0 such that the
    # largest expected degree is about 2 sqrt(2E)
    i = torch.arange(V, dtype=torch.float64, device="cuda")
    beta = 1.0 / (case["gamma"] - 1.0)
    target = min(2.0 * (2.0 * case["E"]) ** 0.5, V / 2.0) / (2.0 * case["E"] / V)
    lo, hi = 0.0, float(V)
    for _ in range(50):
        mid = 0.5 * (lo + hi)
        w = (i + mid) ** -beta
        lo, hi = (mid, hi) if float(w[0] / w.mean()) > target else (lo, mid)
    cdf = torch.cumsum((i + lo) ** -beta, 0)
    cdf /= cdf[-1].clone()

    def ends():
        return torch.searchsorted(cdf, torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)).clamp_(max=V - 1)

    return ends(), ends()


def _csr(case, gen):
    """(beg_pos, csr, weight): a symmetric CSR of about E undirected edges without loops or duplicates."""
    V, E = case["V"], case["E"]
    u, v = _endpoints(case, int(1.15 * E) + 1024, gen)
    key = torch.unique((torch.minimum(u, v) * V + torch.maximum(u, v))[u != v])
    del u, v
    if len(key) > E:
        key = key[torch.randperm(len(key), device="cuda", generator=gen)[:E]]
    w = torch.randint(1, 101, (len(key),), device="cuda", generator=gen)
    lo, hi = key // V, key % V
    del key
    both = torch.cat([lo * V + hi, hi * V + lo]) * 128 + torch.cat([w, w])
    del lo, hi, w
    both = both.sort().values
    w = (both % 128).to(torch.int32).cpu().numpy()
    both //= 128
    beg = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    beg[1:] = torch.cumsum(torch.bincount(both // V, minlength=V), 0)
    csr = (both % V).to(torch.int32).cpu().numpy().view(np.uint32)
    return beg.cpu().numpy().astype(np.uint32), csr, w


def _groups(case, gen):
    """(ptr, members): truncated Zipf sizes, members uniform; vertices left over join random groups."""
    V, n = case["V"], case["groups"]
    smax = min(case["smax"], V // 4)
    p = torch.arange(1, smax + 1, dtype=torch.float64, device="cuda") ** -case["zipf"]
    size = torch.multinomial(p, n, replacement=True, generator=gen) + 1
    gid = torch.repeat_interleave(torch.arange(n, device="cuda"), size)
    mem = torch.randint(0, V, (len(gid),), device="cuda", generator=gen)
    covered = torch.zeros(V, dtype=torch.bool, device="cuda")
    covered[mem] = True
    left = torch.nonzero(~covered).flatten()
    gid = torch.cat([gid, torch.randint(0, n, (len(left),), device="cuda", generator=gen)])
    key = torch.unique(gid * V + torch.cat([mem, left]))
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(key // V, minlength=n), 0)
    return ptr.cpu().numpy().astype(np.uint64), (key % V).cpu().numpy().astype(np.uint32)


class Resident:
    """A graph with its groups: the host arrays, and the engine and server that a program keeps open on them."""

    def __init__(self, case):
        gen = torch.Generator("cuda")
        gen.manual_seed(case["V"] * 31 + case["E"])
        self.arrays = (*_csr(case, gen), *_groups(case, gen))
        torch.cuda.empty_cache()  # the engine allocates from the device, beside torch's pool
        self._engine = self._server = None

    def engine(self):
        if self._engine is None:
            self._engine = engine.Engine(*self.arrays)
        return self._engine

    def server(self):
        if self._server is None:
            self._server = engine.Server(self.engine(), hbm_budget=24 << 30)
        return self._server

    def __del__(self):
        if self._server is not None:
            self._server.close()
        if self._engine is not None:
            self._engine.close()


GRAPH_KEYS = ("graph", "V", "E", "gamma", "groups", "zipf", "smax")
_resident = {}  # the graph used last: a program's one resident graph


def _graph_of(case):
    key = tuple(case[k] for k in GRAPH_KEYS)
    if key not in _resident:
        _resident.clear()
        _resident[key] = Resident(case)
    return _resident[key]


# ---------------------------------------------------------------------------
# The measured interface
# ---------------------------------------------------------------------------

def _queries(case, seed):
    rng = np.random.default_rng(seed)
    queries, Ds = [], []
    for i in range(case["n"]):
        k = int(rng.integers(case["k_lo"], case["k_hi"] + 1))
        queries.append(rng.choice(case["groups"], size=k, replace=False).astype(np.uint32))
        hop = int(rng.integers(case["D_lo"], case["D_hi"] + 1))
        # a share of 1/2 alternates, so that every seed has the same mix
        Ds.append(hop if int((i + 1) * case["hop_share"]) > int(i * case["hop_share"]) else NO_HOPS)
    return queries, Ds


def prepare(case, seed):
    graph = _graph_of(case)
    if case["mode"] == "serve":
        graph.server()
    elif case["mode"] != "load":
        graph.engine()
    queries, Ds = _queries(case, seed)
    return {"mode": case["mode"], "graph": graph, "queries": queries, "Ds": Ds}


def run(state):
    graph, queries, Ds, mode = state["graph"], state["queries"], state["Ds"], state["mode"]
    if mode == "plain":
        res = [graph.engine().query(q, D=D) for q, D in zip(queries, Ds)]
    elif mode == "noalloc":
        res = [graph.engine().query_noalloc(q, D=D) for q, D in zip(queries, Ds)]
    elif mode == "batch":
        res = graph.engine().query_batch(queries, Ds)
    elif mode == "load":
        eng = engine.Engine(*graph.arrays)
        res = [eng.query(q, D=D) for q, D in zip(queries, Ds)]
        eng.close()
    else:
        server = graph.server()
        for i, (q, D) in enumerate(zip(queries, Ds)):
            server.submit(i, q, D)
        got = {}
        while len(got) < len(queries):
            new = server.poll(max_results=64, max_edges=256)
            got.update(new)
            if not new:
                time.sleep(0.0001)
        res = [got[i] for i in range(len(queries))]
    return {"status": np.array([r.status for r in res], dtype=np.int32),
            "cost": np.array([r.cost for r in res], dtype=np.int32),
            "tree_weight": np.array([int(r.edges[:, 2].sum()) for r in res], dtype=np.int64)}


def work(case):
    """The graph read once ({neighbour, weight} 8 bytes an arc, an offset a vertex); for each query one distance a
    group and vertex written and read once, which its bounds need; additions: one an arc and group."""
    arcs, n, k = 2 * case["E"], case["n"], 0.5 * (case["k_lo"] + case["k_hi"])
    return {"bytes": 8.0 * arcs + 4.0 * (case["V"] + 1) + n * k * 8.0 * case["V"], "flops": n * k * arcs}


def exact(case, seed):
    """Subset dynamic programming over all vertices, 64-bit integers, in plain torch."""
    queries, Ds = _queries(case, seed)
    steps = sum(3 ** len(q) * case["V"] + 12 * 2 ** len(q) * 2 * case["E"] * (1 if D < 0 else D) for q, D in zip(queries, Ds))
    if steps > 4e10:
        return None
    beg, csr, w, ptr, mem = _graph_of(case).arrays
    V, inf = case["V"], 1 << 40
    src = torch.repeat_interleave(torch.arange(V), torch.from_numpy(np.diff(beg.astype(np.int64)))).cuda()
    dst = torch.from_numpy(csr.astype(np.int64)).cuda()
    w = torch.from_numpy(w.astype(np.int64)).cuda()

    def grown(row):  # one step along every arc
        return torch.full_like(row, inf).scatter_reduce_(0, dst, (row[src] + w).clamp_(max=inf), "amin")

    status, cost = [], []
    for q, D in zip(queries, Ds):
        table = {}  # (subset, height) -> cost of a tree rooted at each vertex; height 0 throughout without a hop bound
        for d in range(max(D, 0) + 1):
            for S in range(1, 1 << len(q)):
                row = torch.full((V,), inf, dtype=torch.int64, device="cuda")
                if d == 0 and S & (S - 1) == 0:
                    g = int(q[S.bit_length() - 1])
                    row[torch.from_numpy(mem[int(ptr[g]):int(ptr[g + 1])].astype(np.int64)).cuda()] = 0
                A = (S - 1) & S
                while A:
                    for e in range(min(d, max(D, 0) - d) + 1):
                        row = torch.minimum(row, (table[A, d] + table[S ^ A, e]).clamp_(max=inf))
                    A = (A - 1) & S
                if D >= 0 and d > 0:
                    row = torch.minimum(row, grown(table[S, d - 1]))
                while D < 0:
                    new = torch.minimum(row, grown(row))
                    if torch.equal(new, row):
                        break
                    row = new
                table[S, d] = row
        full = (1 << len(q)) - 1
        best = min(int(table[full, d].min()) for d in range(max(D, 0) + 1))
        status.append(0 if best < inf else 1)  # solved / no solution
        cost.append(best if best < inf else -1)
    return {"status": np.array(status, dtype=np.int32), "cost": np.array(cost, dtype=np.int32),
            "tree_weight": np.maximum(np.array(cost, dtype=np.int64), 0)}
