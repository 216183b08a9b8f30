"""Paths of the round kernels that depend on sizes, against the CPU oracle:
every hop bound (which rounds relax and which gather, and the buffers their
rows are kept in), hub vertices around the chunking threshold, every number of
groups, and batches around the numbers of slots at which the control step and
the small-round cluster change their ways (8 descriptors staged, 32 slots in
one warp)."""
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
