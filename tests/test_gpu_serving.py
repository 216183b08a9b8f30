"""The serving loop and batches while requests are rerun, withdrawn or arrive:
what the host keeps about a request has to survive its being staged again, and
what the control steps know about the queries in flight has to survive an
admission."""
import time

import numpy as np
import pytest

from gpugst_b200 import gen

pytestmark = pytest.mark.gpu


def _poll_all(S, n, timeout=60.0):
    got = {}
    t0 = time.time()
    while len(got) < n and time.time() - t0 < timeout:
        for rid, r in S.poll():
            got[rid] = r
        time.sleep(0.0005)
    return got


def _rerun_instance():
    """A path of 3000 vertices: its ends, and every other vertex, as groups.  The
    1500 members outgrow the smallest frontier list (1024 entries) in the first
    round, so the query is rerun; the rerun takes 1500 rounds or more, a distance
    from either end growing by one vertex a round."""
    V = 3000
    u = np.arange(V - 1)
    g = gen.csr_from_edges(V, u, u + 1, np.full(V - 1, 100, dtype=np.int32))
    even = np.arange(0, V, 2)
    ptr = np.array([0, 1, 2, 2 + len(even)], dtype=np.uint64)
    return g, gen.Groups(ptr, np.concatenate([[0, V - 1], even]).astype(np.uint32))


def test_cancel_of_a_request_that_is_rerun(gst_lib, monkeypatch):
    """A cancel that the server accepted ends the request wherever it is taken:
    in the run whose list overflows, while it waits for its rerun, in the
    iteration that stages it again, or in the rerun."""
    eng = gst_lib
    g, gr = _rerun_instance()
    monkeypatch.setenv("GSTB_QUEUE_CAP", "1")
    E = eng.Engine.from_instance(g, gr)
    E.set_tuning(delta_sssp=1, delta_dp=1, cap_pct=100)
    S = eng.Server(E, max_inflight=2)
    q = np.array([0, 1, 2], dtype=np.uint32)
    rng = np.random.default_rng(3)
    lost, n = [], 120
    for i in range(n):
        assert S.submit(i, q) == eng.GST_OK
        t0 = time.perf_counter()
        while S.stats()["inflight"] < 1 and time.perf_counter() - t0 < 10:
            pass
        t1 = time.perf_counter() + float(rng.uniform(0, 8e-4))
        while time.perf_counter() < t1:
            pass
        assert S.cancel(i) == eng.GST_OK
        got = _poll_all(S, 1)
        if got[i].status != eng.GST_CANCELLED:
            lost.append((i, got[i].status))
    st = S.stats()
    assert S.submit(n, q) == eng.GST_OK  # one that nobody cancels is still answered
    last = _poll_all(S, 1)[n]
    S.close()
    E.close()
    assert not lost, (len(lost), lost[:10])
    assert st["cancelled"] == n and st["completed"] == n and st["inflight"] == 0
    assert last.status == eng.GST_OK and last.stats["retries"] > 0 and last.cost == 100 * (g.V - 1)


def test_bytes_in_use_of_rerun_requests(gst_lib, monkeypatch):
    """A rerun's workspace is larger than the one the request was admitted with;
    once all is done, nothing is in use."""
    eng = gst_lib
    g, gr = _rerun_instance()
    monkeypatch.setenv("GSTB_QUEUE_CAP", "1")
    E = eng.Engine.from_instance(g, gr)
    S = eng.Server(E, max_inflight=4)
    q = np.array([0, 1, 2], dtype=np.uint32)
    for i in range(8):
        assert S.submit(i, q) == eng.GST_OK
    got = _poll_all(S, 8)
    st = S.stats()
    S.close()
    E.close()
    assert all(r.status == eng.GST_OK and r.stats["retries"] > 0 for r in got.values()) and len(got) == 8
    assert st["inflight"] == 0 and st["in_use_bytes"] == 0


def test_windows_count_every_live_query(gst_lib):
    """The distance windows widen after a window with few items over all live
    queries.  Two queries whose every window is too large for that, with a third
    kept busy by small ones that come and go, run exactly the rounds that they run
    without them.

    The graph is 40 layers of 12000 vertices, 16 apart, and each window (16 wide
    at the start) holds one layer: 12000 items are few, 24000 are not.  The large
    queries have no solution, so nothing but the windows paces them."""
    eng = gst_lib
    n, layers = 12000, 40
    V = n * layers + 1
    a = np.arange(n * (layers - 1))
    nxt = (a // n + 1) * n
    u = np.concatenate([a, a])
    v = np.concatenate([nxt + a % n, nxt + (a + 1) % n])
    g = gen.csr_from_edges(V, u, v, np.full(len(u), 16, dtype=np.int32))
    gr = gen.Groups(np.array([0, n, n + 1, n + 2], dtype=np.uint64),
                    np.concatenate([np.arange(n), [V - 1, V // 2]]).astype(np.uint32))
    E = eng.Engine.from_instance(g, gr)
    E.set_tuning(rounds_per_launch=1)
    large, small = np.array([0, 1], dtype=np.uint32), np.array([2], dtype=np.uint32)
    alone = E.query_batch([large, large])
    # small ones of 5 to 7 rounds, so that their admissions meet the windows' ends too
    mixed = E.query_batch([large, large] + [small] * 40, [-1, -1] + [-1, 0, 1, 2] * 10, max_concurrent=3)
    E.close()
    assert [r.status for r in alone + mixed[:2]] == [eng.GST_NO_SOLUTION] * 4
    assert all(r.status == eng.GST_OK and r.cost == 0 for r in mixed[2:])
    rounds = [r.stats["rounds"] for r in alone + mixed[:2]]
    assert rounds[0] == rounds[1] > 2 * layers - 10, rounds
    assert rounds[2:] == rounds[:2], rounds
