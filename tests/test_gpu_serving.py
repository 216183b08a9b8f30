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
