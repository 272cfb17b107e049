"""A batch with a bound on its blocks per SM keeps to it: one launch per motif
size, one after the other on its own stream, with the counts of a batch that
has the whole GPU."""
import pytest

from everest_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
def test_bounded_batch(graph):
    u, v, t = synth.generate(synth.GraphSpec("share", "bursty", 5_000, 40_000, seed=8, t_span=800_000))
    dg = capi.DeviceGraph(capi.graph_build_host(u, v, t), 0)
    qs = [([a for a, _ in p], [b for _, b in p]) for p in synth.random_patterns(40, (2, 6), (2, 4), seed=5)]
    sizes = len({len(mu) for mu, _ in qs})
    b = capi.Batch(0, 64)
    for mu, mv in qs:
        b.add(dg, mu, mv, 2000)
    want = b.run()
    assert b.last_stats()["kernel_launches"] > sizes
    for bps in (1, 4, 100):
        b.set_tuning(blocks_per_sm=bps, use_graph=graph)
        assert b.run() == want and b.run() == want
        assert b.last_stats()["kernel_launches"] == sizes
    b.set_tuning(use_graph=graph)
    assert b.run() == want
    assert b.last_stats()["kernel_launches"] > sizes
    b.close()
    dg.free()
