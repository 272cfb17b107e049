"""Launches on both sides of the root count below which a search takes the
kernel that holds every way of counting the last edge, alone and in a batch
(where a size's queries count together), against the oracle."""
import pytest

from everest_b200 import capi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FEW = 148 * 16
MOTIFS = [
    ([0, 1, 2, 3], [1, 2, 3, 0]), ([0, 0, 0, 0], [1, 2, 3, 4]), ([0, 1, 0, 1], [1, 0, 2, 3]), ([0, 1, 2, 1], [1, 2, 0, 2]),
    ([0, 1, 2, 2, 3], [1, 0, 1, 1, 2]), ([0, 1, 2, 1, 3], [1, 0, 0, 3, 0]), ([0, 0, 1, 2, 2], [1, 1, 0, 0, 3]),
    ([0, 1, 1, 2, 2], [1, 2, 0, 3, 3]), ([0, 1, 1, 2, 3], [1, 2, 0, 3, 2]), ([0, 1, 2, 0, 1], [1, 2, 3, 1, 0]),
]


@pytest.mark.parametrize("strict", [False, True])
@pytest.mark.parametrize("n", [FEW - 1, FEW, FEW + 1])
def test_both_sides(n, strict):
    u, v, t = synth.generate(synth.GraphSpec("few", "bursty", 120, 6_000, seed=12, t_span=600_000))
    host = capi.graph_build_host(u, v, t)
    dg = capi.DeviceGraph(host, 0)
    g = O.Graph(host.eg[0::3], host.eg[1::3], host.eg[2::3], host.num_vertices)
    flags = capi.FLAG_STRICT_TS if strict else 0
    w, whole = capi.Worker(0), capi.Batch(0, 16)
    want = []
    for mu, mv in MOTIFS:
        c = O.count(g, mu, mv, 2000, roots=(1000, 1000 + n), strict_ts=strict)[0]
        w.take(dg, mu, mv, 2000, 1000, 1000 + n, 0, flags)
        assert w.run() == c, (mu, mv)
        parts = capi.Batch(0, 8)  # the same roots as three queries of one size
        for a, b in ((1000, 1007), (1007, 1000 + n // 2), (1000 + n // 2, 1000 + n)):
            parts.add(dg, mu, mv, 2000, a, b, flags)
        assert sum(parts.run()) == c, (mu, mv)
        parts.close()
        whole.add(dg, mu, mv, 2000, 1000, 1000 + n, flags)
        want.append(c)
    assert whole.run() == want and sum(want) > 0
    whole.close()
    w.close()
    dg.free()
