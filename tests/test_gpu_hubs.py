"""Chunk thresholds (hub_min_deg) below the arcs that a DP grow keeps for its own
warp (128), on vertices around both, the graph's last one among them: a tuning
changes no result."""
import numpy as np
import pytest

from gpugst_b200 import gen

pytestmark = pytest.mark.gpu

DEGREES = (31, 32, 33, 63, 64, 65, 100, 127, 128, 129, 160, 257)


def _instance(seed, V=500):
    """A sparse random graph whose last vertices have the given degrees."""
    rng = np.random.default_rng(seed)
    n = V - len(DEGREES)
    pairs = {(int(a), int(b)) for a, b in rng.integers(0, n, size=(V, 2)) if a < b}
    for i, deg in enumerate(np.roll(DEGREES, seed)):
        pairs |= {(int(v), n + i) for v in rng.choice(n, size=deg, replace=False)}
    u, v = (np.array(x, dtype=np.int64) for x in zip(*sorted(pairs)))
    g = gen.csr_from_edges(V, u, v, rng.integers(1, 60, size=len(u)).astype(np.int32))
    assert sorted(np.diff(g.beg_pos.astype(np.int64))[n:]) == sorted(DEGREES)
    return g, gen.zipf_groups(V, 100, 1.5, 6, seed=seed + 1)


@pytest.mark.parametrize("persistent", (0, 1))
@pytest.mark.parametrize("hub_min_deg", (32, 64, 100, 127, 128, 129))
def test_low_chunk_thresholds(gst_lib, oracle_mod, hub_min_deg, persistent):
    eng, O = gst_lib, oracle_mod
    bad = []
    for seed in range(4):
        g, gr = _instance(seed)
        E = eng.Engine.from_instance(g, gr)
        E.set_tuning(hub_min_deg=hub_min_deg, persistent=persistent)
        rng = np.random.default_rng(seed)
        qs = [rng.choice(gr.n_groups, size=k, replace=False).astype(np.uint32) for k in (2, 3, 4, 5)] * 4
        Ds = [D for D in (-1, 2, 3, 5) for _ in range(4)]
        for q, D, r in zip(qs, Ds, E.query_batch(qs, Ds)):
            want = O.prunedpp(g, gr, q, 0) if D < 0 else O.hop(g, gr, q, D)
            if want.status != 0:
                if r.status != eng.GST_NO_SOLUTION:
                    bad.append((seed, q.tolist(), D, "want no solution", r.status, r.cost))
            elif r.status != eng.GST_OK or r.cost != want.cost or O.validate(g, gr, q, D, r.cost, r.root, r.edges):
                bad.append((seed, q.tolist(), D, want.cost, r.status, r.cost))
        E.close()
    assert not bad, bad[:10]
