"""Dense graphs: in one round many threads lower the same vertex before any of
them sees its pending flag, so a frontier list gets it many times over and can
outgrow a list of one entry a vertex.  Every entry point still answers."""
import numpy as np
import pytest

from gpugst_b200 import gen

pytestmark = pytest.mark.gpu


def _complete(V, groups, seed):
    u, v = np.triu_indices(V, 1)
    w = np.random.default_rng(seed).integers(1, 101, len(u)).astype(np.int32)
    cut = np.linspace(0, V, groups + 1).astype(np.uint64)
    return gen.csr_from_edges(V, u, v, w), gen.Groups(cut, np.arange(V, dtype=np.uint32))


@pytest.mark.parametrize("V,groups", ((200, 4), (500, 4), (500, 500), (1000, 1000), (2000, 4)))
def test_complete_graph(gst_lib, oracle_mod, V, groups):
    eng, O = gst_lib, oracle_mod
    g, gr = _complete(V, groups, V)
    E = eng.Engine.from_instance(g, gr)
    qs = [(np.arange(k, dtype=np.uint32), D) for k in (2, 3, 4) for D in (-1, 2, 4)]
    batch = E.query_batch([q for q, _ in qs], [D for _, D in qs])
    bad = []
    for (q, D), b in zip(qs, batch):
        want = (O.prunedpp(g, gr, q, 0) if D < 0 else O.hop(g, gr, q, D)).cost
        for name, r in (("query", E.query(q, D=D)), ("batch", b), ("noalloc", E.query_noalloc(q, D=D))):
            if r.status != eng.GST_OK or r.cost != want or O.validate(g, gr, q, D, r.cost, r.root, r.edges):
                bad.append((name, len(q), D, want, r.status, r.cost))
    E.close()
    assert not bad, bad
