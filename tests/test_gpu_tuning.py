"""A worker's tuning values: the interval may be left to the rule (-1), and
what was refused stays refused."""
import pytest

from everest_b200 import capi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_interval_by_rule():
    u, v, t = synth.generate(synth.GraphSpec("tuning", "zipf", 200, 6_000, seed=4, t_max=60_000))
    dg = capi.DeviceGraph(capi.graph_build_host(u, v, t), 0)
    g = O.Graph(u, v, t, 200)
    w = capi.Worker(0)
    for mu, mv in (([0, 1, 2], [1, 2, 0]), ([0, 1, 1], [1, 2, 3]), ([0, 1, 2, 3], [1, 2, 3, 0])):
        want = O.count(g, mu, mv, 2000)[0]
        for interval in (16, -1, 0, 1, 4):
            w.set_tuning(steal_interval=interval)
            w.take(dg, mu, mv, 2000)
            assert w.run() == want
        for interval in (-2, -4, 3, 12, -(2**31)):
            with pytest.raises(capi.EvxError):
                w.set_tuning(steal_interval=interval)
    w.close()
    dg.free()


@pytest.mark.parametrize("strict", [0, capi.FLAG_STRICT_TS])
def test_window_bound_asked_for_and_refused(strict):
    # three edges by range arithmetic (off by rule), by the pair table and four
    # edges (on by rule): the same counts either way, alone and in a batch
    u, v, t = synth.generate(synth.GraphSpec("bound", "bursty", 500, 12_000, seed=6, t_span=200_000))
    dg = capi.DeviceGraph(capi.graph_build_host(u, v, t), 0)
    g = O.Graph(u, v, t, 500)
    w, b = capi.Worker(0), capi.Batch(0, 32)
    want = []
    for mu, mv in (([0, 1, 0], [1, 2, 1]), ([0, 1, 1], [1, 2, 3]), ([0, 0, 0], [1, 2, 2]), ([0, 1, 2], [1, 2, 1]),
                   ([0, 1, 2], [1, 2, 0]), ([0, 1, 2, 3], [1, 2, 3, 0])):
        c = O.count(g, mu, mv, 3000, strict_ts=bool(strict))[0]
        for flags in (0, capi.FLAG_ROOT_BOUND, capi.FLAG_NO_ROOT_BOUND, capi.FLAG_ROOT_BOUND | capi.FLAG_NO_ROOT_BOUND):
            w.take(dg, mu, mv, 3000, 0, -1, 0, flags | strict)
            assert w.run() == c
            b.add(dg, mu, mv, 3000, 0, -1, flags | strict)
            want.append(c)
    assert b.run() == want
    b.close()
    w.close()
    dg.free()
