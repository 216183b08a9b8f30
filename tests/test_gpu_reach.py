"""Weights inside the first distance window, beyond the reach of the first rounds
and far beyond it, and groups that are not connected, through the ways to ask that
run the rounds differently: serving, persistent launches, a profiled batch (no
round inside the control kernel), the allocation-free query, hop bounds and
progressive mode.  Against a subset dynamic program over all vertices in 64
bits."""
import time

import numpy as np
import pytest

from gpugst_b200 import gen

pytestmark = pytest.mark.gpu

INF = 1 << 60


def _instance(wmax, V=300):
    rng = np.random.default_rng(wmax)
    a, b = rng.integers(0, V - 20, size=(2, 800))
    pairs = np.unique(np.stack([np.minimum(a, b), np.maximum(a, b)], 1)[a != b], axis=0)
    chain = np.stack([np.arange(V - 20, V - 1), np.arange(V - 19, V)], 1)  # a component of its own
    pairs = np.concatenate([pairs, chain])
    g = gen.csr_from_edges(V, pairs[:, 0], pairs[:, 1], rng.integers(1, wmax + 1, len(pairs)).astype(np.int32))
    gr = gen.zipf_groups(V, 60, 1.5, 4, seed=wmax)
    queries = [rng.choice(gr.n_groups, size=int(k), replace=False).astype(np.uint32)
               for k in rng.integers(2, 6, size=16)]
    return g, gr, queries


def _optimum(g, gr, q, D):
    """Optimal cost, None if there is no tree (D < 0: no hop bound)."""
    src = np.repeat(np.arange(g.V), np.diff(g.beg_pos.astype(np.int64)))

    def grown(row):
        new = np.full(g.V, INF, dtype=np.int64)
        np.minimum.at(new, g.csr, np.minimum(row[src] + g.weight, INF))
        return new

    table = {}  # (subset, height); height 0 throughout without a hop bound
    for d in range(max(D, 0) + 1):
        for S in range(1, 1 << len(q)):
            row = np.full(g.V, INF, dtype=np.int64)
            if d == 0 and S & (S - 1) == 0:
                row[gr.group(int(q[S.bit_length() - 1]))] = 0
            A = (S - 1) & S
            while A:
                for e in range(min(d, max(D, 0) - d) + 1):
                    row = np.minimum(row, np.minimum(table[A, d] + table[S ^ A, e], INF))
                A = (A - 1) & S
            if D >= 0 and d > 0:
                row = np.minimum(row, grown(table[S, d - 1]))
            while D < 0:
                new = np.minimum(row, grown(row))
                if (new == row).all():
                    break
                row = new
            table[S, d] = row
    best = min(int(table[(1 << len(q)) - 1, d].min()) for d in range(max(D, 0) + 1))
    return best if best < INF else None


def _faults(eng, O, g, gr, name, queries, Ds, want, results, ratio=1.0):
    bad = []
    for q, D, w, r in zip(queries, Ds, want, results):
        if w is None:
            ok = r.status == eng.GST_NO_SOLUTION
        else:
            ok = (r.status == eng.GST_OK and w <= r.cost <= ratio * w and r.stats["lower_bound"] <= w
                  and not O.validate(g, gr, q, D, r.cost, r.root, r.edges))
        if not ok:
            bad.append((name, q.tolist(), D, w, r.status, r.cost))
    return bad


def _served(eng, E, queries, Ds):
    S = eng.Server(E, max_inflight=6)
    for i, (q, D) in enumerate(zip(queries, Ds)):
        assert S.submit(i, q, D=D) == eng.GST_OK
    got, t0 = {}, time.time()
    while len(got) < len(queries) and time.time() - t0 < 60:
        got.update(S.poll(max_edges=256))
    S.close()
    return [got[i] for i in range(len(queries))]


@pytest.mark.parametrize("wmax", (3, 40, 300, 1_000_000))
def test_weights_beyond_the_reach_in_every_mode(gst_lib, oracle_mod, wmax):
    eng, O = gst_lib, oracle_mod
    g, gr, queries = _instance(wmax)
    Ds = [(-1, 3, -1, 4, -1, 2, -1, 6)[i % 8] for i in range(len(queries))]
    want = [_optimum(g, gr, q, D) for q, D in zip(queries, Ds)]
    E = eng.Engine.from_instance(g, gr)
    bad = []

    def check(name, results, ratio=1.0):
        bad.extend(_faults(eng, O, g, gr, name, queries, Ds, want, results, ratio))

    check("noalloc", [E.query_noalloc(q, D=D) for q, D in zip(queries, Ds)])
    check("served", _served(eng, E, queries, Ds))
    E.profile(True)
    check("profiled", E.query_batch(queries, Ds))
    E.profile(False)
    for ratio in (1.25, 3.0):
        check(f"ratio {ratio}", [E.query(q, D=D, ratio=ratio) for q, D in zip(queries, Ds)], ratio)
        check(f"batch ratio {ratio}", E.query_batch(queries, Ds, ratios=[ratio] * len(queries)), ratio)
    E.set_tuning(persistent=1)
    check("persistent", E.query_batch(queries, Ds))
    check("persistent served", _served(eng, E, queries, Ds))
    check("persistent ratio", E.query_batch(queries, Ds, ratios=[2.0] * len(queries)), 2.0)
    E.close()
    assert not bad, (len(bad), bad[:10])
