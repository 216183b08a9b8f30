"""What gst_graph_create builds on the device, read back and compared word for
word with a host sort: every list by (weight, neighbour), and the weight index;
and that it needs no device memory beside the graph's own."""
import numpy as np
import pytest
import torch

from gpugst_b200 import gen

pytestmark = pytest.mark.gpu


def _mismatches(E, beg, csr, w):
    """Numbers of adjacency pairs and index words that differ from a host sort's."""
    beg = beg.astype(np.int64)
    V = len(beg) - 1
    src = np.repeat(np.arange(V, dtype=np.int64), np.diff(beg))
    order = np.lexsort((csr, w, src))
    pairs, index = E.adjacency()
    bad = int((pairs[:, 0] != csr[order]).sum()) + int((pairs[:, 1] != w[order].astype(np.uint32)).sum())
    for b in range(7):
        light = np.bincount(src[w <= 1 << b], minlength=V)
        bad += int((index[:, b] != beg[:-1] + light).sum())
    return bad + int((index[:, 7] != beg[:-1]).sum())


def _star(n, w):
    """A hub with n leaves: (beg_pos, csr, weight)."""
    beg = np.concatenate([[0], np.arange(n, 2 * n + 1)]).astype(np.uint32)
    csr = np.concatenate([np.arange(1, n + 1), np.zeros(n)]).astype(np.uint32)
    return beg, csr, np.concatenate([w, w]).astype(np.int32)


def _parallel(n, w):
    """Two vertices with n parallel edges."""
    return (np.array([0, n, 2 * n], dtype=np.uint32), np.repeat(np.array([1, 0], dtype=np.uint32), n),
            np.concatenate([w, w]).astype(np.int32))


@pytest.mark.parametrize("n", (1, 2, 3, 31, 33, 255, 256, 257, 4095, 4096, 4097, 8192, 8193, 12289, 16385, 70001))
@pytest.mark.parametrize("shape", (_star, _parallel))
def test_every_list_size(gst_lib, shape, n):
    rng = np.random.default_rng(n)
    # few distinct weights, so that the neighbour decides, and heavy ones beyond the index
    graph = shape(n, rng.choice([1, 2, 3, 64, 65, 128, 129, 3000], size=n))
    E = gst_lib.Engine(*graph)
    bad = _mismatches(E, *graph)
    E.close()
    assert bad == 0


@pytest.mark.parametrize("V,E,gamma", ((1, 0, 2.5), (5, 0, 2.5), (60, 200, 2.5), (20_000, 900_000, 2.1)))
def test_power_law_graphs(gst_lib, V, E, gamma):
    g = gen.chung_lu(V, E, gamma, seed=V) if E else gen.csr_from_edges(V, *np.zeros((3, 0), dtype=np.int64))
    eng = gst_lib.Engine(g.beg_pos, g.csr, g.weight)
    bad = _mismatches(eng, g.beg_pos, g.csr, g.weight)
    eng.close()
    assert bad == 0


def test_many_long_lists(gst_lib):
    """A complete graph of 4200 vertices: every list is merged, in more groups than
    the index's memory is used for."""
    V = 4200
    u, v = np.triu_indices(V, 1)
    g = gen.csr_from_edges(V, u, v, np.random.default_rng(1).integers(1, 101, len(u)).astype(np.int32))
    E = gst_lib.Engine(g.beg_pos, g.csr, g.weight)
    bad = _mismatches(E, g.beg_pos, g.csr, g.weight)
    E.close()
    assert bad == 0


@pytest.mark.parametrize("shape,n", ((_star, 8_000_000), (_parallel, 6_000_000)))
def test_created_in_the_memory_it_keeps(gst_lib, shape, n):
    """With the device full but for the graph's own arrays (offsets, adjacency and
    index) and 16 MB, its creation succeeds: the caller's arrays (128 and 96 MB of
    arcs) and the merge (64 and 48 MB a list) find their place in what is there."""
    rng = np.random.default_rng(n)
    graph = shape(n, rng.integers(1, 101, n))
    small = _star(3, np.ones(3))
    gst_lib.Engine(*small).close()  # the kernels are loaded
    V, arcs = len(graph[0]) - 1, len(graph[1])
    own = 4 * (V + 1) + 8 * arcs + 32 * V
    free = torch.cuda.mem_get_info()[0]
    rest = torch.empty(free - own - (16 << 20), dtype=torch.uint8, device="cuda")
    try:
        E = gst_lib.Engine(*graph)
        bad = _mismatches(E, *graph)
        E.close()
    finally:
        del rest
        torch.cuda.empty_cache()
    assert bad == 0
