"""Paths of the round kernels that depend on sizes, against the CPU oracle:
every hop bound (which rounds relax and which gather, and the buffers their
rows are kept in), hub vertices around the chunking threshold, every number of
groups, and batches around the numbers of slots at which the control step and
the small-round cluster change their ways (8 descriptors staged, 32 slots in
one warp); and adjacency lists around the sizes at which the graph's creation
sorts them differently (256 and 4096 arcs, and the merges of longer ones)."""
import numpy as np
import pytest

from gpugst_b200 import gen

pytestmark = pytest.mark.gpu


def _hub_instance(seed, V=700, hubs=(255, 256, 289, 640)):
    """A sparse random graph plus hubs whose degrees straddle the chunking
    threshold (256 arcs) and the chunk size (32 + 256 arcs)."""
    rng = np.random.default_rng(seed)
    pairs = {(int(a), int(b)) for a, b in rng.integers(0, V, size=(2 * V, 2)) if a < b}
    for h, deg in enumerate(hubs):
        pairs = {(a, b) for a, b in pairs if h not in (a, b)}
    for h, deg in enumerate(hubs):
        for v in rng.choice(np.arange(len(hubs), V), size=deg, replace=False):
            pairs.add((h, int(v)))
    u, v = (np.array(x, dtype=np.int64) for x in zip(*sorted(pairs)))
    g = gen.csr_from_edges(V, u, v, rng.integers(1, 60, size=len(u)).astype(np.int32))
    assert sorted(np.diff(g.beg_pos.astype(np.int64))[:len(hubs)]) == sorted(hubs)
    return g, gen.zipf_groups(V, 120, 1.5, 8, seed=seed + 1)


def _check(eng, O, g, gr, q, D, r):
    want = O.prunedpp(g, gr, q, 0) if D < 0 else O.hop(g, gr, q, D)
    if want.status != 0:
        return [] if r.status == eng.GST_NO_SOLUTION else [(q.tolist(), D, "want no solution", r.status, r.cost)]
    if r.status != eng.GST_OK or r.cost != want.cost:
        return [(q.tolist(), D, want.cost, r.status, r.cost)]
    v = O.validate(g, gr, q, D, r.cost, r.root, r.edges)
    return [(q.tolist(), D, "invalid tree", v)] if v else []


@pytest.mark.parametrize("D", range(-1, 8))
def test_every_hop_bound_on_hubs(gst_lib, oracle_mod, D):
    eng, O = gst_lib, oracle_mod
    bad = []
    for seed in (1, 2):
        g, gr = _hub_instance(seed)
        E = eng.Engine.from_instance(g, gr)
        rng = np.random.default_rng(seed)
        for k in (1, 2, 3, 4, 5):
            q = rng.choice(gr.n_groups, size=k, replace=False).astype(np.uint32)
            bad += _check(eng, O, g, gr, q, D, E.query(q, D=D))
            bad += _check(eng, O, g, gr, q, D, E.query_noalloc(q, D=D))
        E.close()
    assert not bad, bad[:10]


@pytest.mark.parametrize("persistent", (0, 1))
@pytest.mark.parametrize("n", (1, 8, 9, 31, 32, 33, 70))
def test_batch_sizes(gst_lib, oracle_mod, n, persistent):
    eng, O = gst_lib, oracle_mod
    g, gr = _hub_instance(3)
    rng = np.random.default_rng(n)
    queries = [rng.choice(gr.n_groups, size=int(rng.integers(1, 5)), replace=False).astype(np.uint32)
               for _ in range(n)]
    Ds = [int(rng.integers(-1, 6)) for _ in range(n)]
    E = eng.Engine.from_instance(g, gr)
    E.set_tuning(persistent=persistent)
    res = E.query_batch(queries, Ds)
    E.close()
    bad = []
    for q, D, r in zip(queries, Ds, res):
        bad += _check(eng, O, g, gr, q, D, r)
    assert not bad, bad[:10]


@pytest.mark.parametrize("n", (1, 2, 31, 33, 255, 256, 257, 4095, 4096, 4097, 8192, 8193, 12289, 70001))
def test_star_of_every_list_size(gst_lib, n):
    """A star of n leaves with heavy and equal weights: the tree of two leaves
    costs the sum of their two arcs, so an arc that the sort of the hub's list
    lost or misplaced shows as a wrong cost."""
    eng = gst_lib
    rng = np.random.default_rng(n)
    w = rng.choice([1, 2, 3, 64, 128, 129, 255, 256, 257, 3000], size=n).astype(np.int32)
    g = gen.csr_from_edges(n + 1, np.zeros(n, dtype=np.int64), np.arange(1, n + 1), w)
    # one group a leaf, and one of the hub
    gr = gen.Groups(np.arange(n + 2, dtype=np.uint64), np.concatenate([np.arange(1, n + 1), [0]]).astype(np.uint32))
    pairs = [(int(a), int(b)) for a, b in rng.integers(0, n + 1, size=(60, 2)) if a != b]
    pairs += [(0, n), (n - 1, n), (int(w.argmax()), n), (int(w.argmin()), n)]
    E = eng.Engine.from_instance(g, gr)
    res = E.query_batch([np.array(p, dtype=np.uint32) for p in pairs])
    E.close()
    cost = np.append(w, 0)
    for (a, b), r in zip(pairs, res):
        assert r.status == eng.GST_OK and r.cost == cost[a] + cost[b], (a, b, r.status, r.cost, cost[a] + cost[b])
        assert sorted(r.edges[:, 2].tolist()) == sorted(int(c) for c in (cost[a], cost[b]) if c)


def test_staging_grows_for_large_member_lists(gst_lib, oracle_mod):
    """Member lists larger than the staging a runner starts with (2 MB a half):
    it grows for them, alone and behind others, and small queries go on."""
    eng, O = gst_lib, oracle_mod
    V = 900_000
    rng = np.random.default_rng(4)
    u = np.arange(1, V)
    g = gen.csr_from_edges(V, u, (u * rng.random(V - 1)).astype(np.int64), rng.integers(1, 9, V - 1).astype(np.int32))
    big = [np.arange(i, V, 2) for i in range(2)]  # 1.8 MB of members each
    ptr = np.cumsum([0, len(big[0]), len(big[1]), 1, 1, 1]).astype(np.uint64)
    gr = gen.Groups(ptr, np.concatenate([*big, [5, 70_000, 899_999]]).astype(np.uint32))
    E = eng.Engine.from_instance(g, gr)
    small = np.array([2, 3, 4], dtype=np.uint32)
    want = O.prunedpp(g, gr, small, 0).cost
    queries = [small, np.array([0, 1], dtype=np.uint32), small, np.array([0, 1, 2], dtype=np.uint32), small]
    for batch in (queries, queries[1:2], queries):
        res = E.query_batch(batch)
        for q, r in zip(batch, res):
            assert r.status == eng.GST_OK
            if len(q) == 3 and q[0] == 2:
                assert r.cost == want
            else:
                assert not O.validate(g, gr, q, -1, r.cost, r.root, r.edges)
    E.close()


def _subset_dp(g, gr, q):
    """Optimal cost by subset dynamic programming over all vertices, 64-bit (the
    oracle's programs take costs from 100000 on for infinite); None: not connected."""
    inf = 1 << 60
    src = np.repeat(np.arange(g.V), np.diff(g.beg_pos.astype(np.int64)))
    table = {}
    for S in range(1, 1 << len(q)):
        row = np.full(g.V, inf, dtype=np.int64)
        if S & (S - 1) == 0:
            row[gr.group(int(q[S.bit_length() - 1]))] = 0
        A = (S - 1) & S
        while A:
            row = np.minimum(row, table[A] + table[S ^ A])
            A = (A - 1) & S
        while True:
            new = np.minimum(row, inf)
            np.minimum.at(new, g.csr, row[src] + g.weight)
            if (new == row).all():
                break
            row = new
        table[S] = row
    best = int(table[(1 << len(q)) - 1].min())
    return best if best < inf // 2 else None


@pytest.mark.parametrize("wmax", (3, 40, 300, 1_000_000))
def test_weights_beyond_the_reach(gst_lib, oracle_mod, wmax):
    """Distances that end inside the first windows, beyond the reach of the first
    rounds (two widths: every vertex then relaxes again), far beyond it, and
    groups that are not connected at all (no incumbent ever ends the windows)."""
    eng, O = gst_lib, oracle_mod
    rng = np.random.default_rng(wmax)
    V = 400
    a, b = rng.integers(0, V - 20, size=(2, 1000))
    keep = a != b
    pairs = np.unique(np.stack([np.minimum(a, b), np.maximum(a, b)], 1)[keep], axis=0)
    chain = np.stack([np.arange(V - 20, V - 1), np.arange(V - 19, V)], 1)  # a component of its own
    pairs = np.concatenate([pairs, chain])
    g = gen.csr_from_edges(V, pairs[:, 0], pairs[:, 1], rng.integers(1, wmax + 1, len(pairs)).astype(np.int32))
    gr = gen.zipf_groups(V, 60, 1.5, 4, seed=wmax)
    E = eng.Engine.from_instance(g, gr)
    queries = [rng.choice(gr.n_groups, size=int(k), replace=False).astype(np.uint32)
               for k in rng.integers(2, 6, size=24)]
    res = E.query_batch(queries) + [E.query(q) for q in queries[:6]]
    E.close()
    bad = []
    for q, r in zip(queries + queries[:6], res):
        want = _subset_dp(g, gr, q)
        if want is None:
            bad += [] if r.status == eng.GST_NO_SOLUTION else [(q.tolist(), "want no solution", r.status, r.cost)]
        elif r.status != eng.GST_OK or r.cost != want:
            bad.append((q.tolist(), want, r.status, r.cost))
        elif O.validate(g, gr, q, -1, r.cost, r.root, r.edges):
            bad.append((q.tolist(), "invalid tree"))
    assert not bad, bad[:10]
