"""Root ranges of every size a tile and a batch can take: fewer roots than
warps (one-root tiles whose roots are shared between lanes), ranges around a
tile's and a batch's edge, counted and enumerated, against the oracle."""
import numpy as np
import pytest

from everest_b200 import capi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MOTIFS = {
    "2e": ([0, 1], [1, 2]), "closing-2e": ([0, 1], [1, 0]),
    "triangle": ([0, 1, 2], [1, 2, 0]), "reverse-pair": ([0, 1, 2], [1, 2, 1]), "same-pair": ([0, 0, 0], [1, 2, 2]),
    "fixed-pair": ([0, 1, 0], [1, 2, 1]), "star": ([0, 0, 0, 0], [1, 2, 3, 4]), "4-cycle": ([0, 1, 2, 3], [1, 2, 3, 0]),
    "5e": ([0, 1, 2, 2, 3], [1, 0, 1, 1, 2]),
}


@pytest.fixture(scope="module")
def graph():
    spec = synth.GraphSpec("tiles", "bursty", 300, 30_000, seed=31, t_span=3_000_000)
    u, v, t = synth.generate(spec)
    host = capi.graph_build_host(u, v, t)
    dg = capi.DeviceGraph(host, 0)
    w = capi.Worker(0)
    yield dg, w, O.Graph(host.eg[0::3], host.eg[1::3], host.eg[2::3], host.num_vertices)
    w.close()
    dg.free()


@pytest.mark.parametrize("strict", [False, True])
@pytest.mark.parametrize("name", MOTIFS)
def test_root_ranges_of_every_size(graph, name, strict):
    dg, w, g = graph
    mu, mv = MOTIFS[name]
    flags = capi.FLAG_STRICT_TS if strict else 0
    b = capi.Batch(0, 64)
    want = []
    for n in (1, 2, 3, 16, 17, 31, 32, 33, 63, 64, 65, 1000, 30_000 - len(mu) + 1):
        beg = (7 * n) % max(1, 30_000 - n)
        end = min(30_000, beg + n)
        c = O.count(g, mu, mv, 3000, roots=(beg, end), strict_ts=strict)[0]
        w.take(dg, mu, mv, 3000, beg, end, 0, flags)
        assert w.run() == c, (n, beg)
        if c <= 200_000:
            w.take(dg, mu, mv, 3000, beg, end, c + 1, flags)
            assert w.run() == c
            rows = w.enum_rows(c)
            ref = O.enumerate_rows(g, mu, mv, 3000, c, roots=(beg, end), strict_ts=strict)[0]
            assert np.array_equal(rows[np.lexsort(rows.T)], ref[np.lexsort(ref.T)]), (n, beg)
        b.add(dg, mu, mv, 3000, beg, end, flags)
        want.append(c)
    assert b.run() == want
    b.close()
