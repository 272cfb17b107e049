"""What the serving loop asks of its device slots: a batch's share of the
resident blocks of its motif size's kernels."""
import pytest

from everest_b200 import serve
from tests.test_serve_cpu import FakeBackend, graph  # noqa: F401


@pytest.mark.parametrize("share,want", [(0.5, {3: 5, 4: 3, 5: 2}), (0.1, {3: 1, 4: 1, 5: 1}), (1.0, {})])
def test_batch_share(graph, share, want):  # noqa: F811
    be = FakeBackend({"g": graph}, free_bytes=1 << 40)
    make, asked = be.Batch, {}

    def batch(device, max_q):
        b = make(device, max_q)

        def set_tuning(tile_roots=256, blocks_per_sm=0, steal_interval=16, min_split=2, use_graph=True):
            if blocks_per_sm:
                asked[len(b.q[0][1])] = blocks_per_sm
        b.set_tuning = set_tuning
        return b
    be.Batch = batch
    srv = serve.Server(max_batch=4, inflight_batches=2, enum_slots=1, mem_reserve=0, backend=be, batch_share=share)
    srv.add_graph("g", "g")
    for mu, mv in (([0, 1, 2], [1, 2, 0]), ([0, 1, 2, 3], [1, 2, 3, 0]), ([0, 1, 2, 3, 4], [1, 2, 3, 4, 0])):
        srv.submit("g", mu, mv, 300)
        srv.drain(60)
    srv.close()
    assert asked == want


def test_slots_are_tuned_before_each_job(graph):  # noqa: F811
    # a job reads the interval when it is taken: every job of an enumeration
    # or heavy slot runs by the rule, the first as the later ones
    be = FakeBackend({"g": graph}, free_bytes=1 << 40)
    make, calls = be.Worker, {}

    def worker(device):
        w = make(device)
        log = calls.setdefault(id(w), [])
        tune, take = w.set_tuning, w.take
        w.keep = w  # (the id stays its own)

        def set_tuning(**kw):
            log.append(kw["steal_interval"])
            tune(**kw)

        def taken(*a, **kw):
            log.append("take")
            take(*a, **kw)
        w.set_tuning, w.take = set_tuning, taken
        return w
    be.Worker = worker
    srv = serve.Server(max_batch=4, inflight_batches=1, enum_slots=1, mem_reserve=0, backend=be, limit=1, heavy_slots=1)
    srv.add_graph("g", "g")
    for _ in range(3):
        srv.submit("g", [0, 1, 2], [1, 2, 0], 2000, enum_cap=10)
        srv.submit("g", [0, 1, 2], [1, 2, 0], 3000)
        srv.drain(60)
    srv.close()
    logs = [x for x in calls.values() if x]
    assert len(logs) == 2  # the enumeration slot's and the heavy slot's
    for x in logs:
        assert len(x) >= 6 and x == [-1, "take"] * (len(x) // 2)
