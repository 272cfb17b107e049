"""The device build of the pair index: long and short runs, one vertex pair
holding most edges, ids around a power of two, vertices without out-edges, and
in-lists that are not in (target, edge id) order, through two-edge queries that
the pair index alone counts."""
import numpy as np
import pytest

from everest_b200 import capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu

PAIR_QUERIES = [([0, 1], [1, 0]), ([0, 0], [1, 1])]  # reverse pair, same pair


def edges(kind, n, seed=3):
    r = np.random.default_rng(seed)
    if kind == "one-pair":
        u, v = np.zeros(n, np.int32), np.ones(n, np.int32)
        u[::7], v[::7] = 1, 0
        u[::11], v[::11] = r.integers(2, 40, u[::11].size), 0
    elif kind == "bipartite":
        u, v = r.integers(0, 16, n), r.integers(16, 257, n)
        back = r.random(n) < 0.3
        u, v = np.where(back & (v < 32), v, u), np.where(back & (v < 32), u, v)
    else:
        u = r.integers(0, 128, n)
        v = (u + r.integers(1, 128, n)) % 128
    return u.astype(np.int32), v.astype(np.int32), np.sort(r.integers(0, 20 * n, n)).astype(np.int32)


@pytest.mark.parametrize("kind", ["one-pair", "bipartite", "spread"])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 20_011])
def test_pair_queries(kind, n):
    u, v, t = edges(kind, n)
    host = capi.graph_build_host(u, v, t)
    g = O.Graph(u, v, t, int(max(u.max(), v.max())) + 1)
    turned = capi.HostGraph(host.num_edges, host.num_vertices, host.eg, host.out_v, host.in_v.copy(), host.out_r,
                            host.in_r, host.euid)
    for x in range(host.num_vertices):  # every in-list backwards
        a, b = host.in_r[x], host.in_r[x + 1]
        turned.in_v[a:b] = host.in_v[a:b][::-1]
    w = capi.Worker(0)
    for h in (host, turned):
        dg = capi.DeviceGraph(h, 0)
        for mu, mv in PAIR_QUERIES:
            for delta in (0, 60, 5000):
                w.take(dg, mu, mv, delta)
                assert w.run() == O.count(g, mu, mv, delta)[0], (h is turned, mu, mv, delta)
        dg.free()
    w.close()
