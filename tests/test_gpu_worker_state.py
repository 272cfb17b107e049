"""A worker made while the default stream is busy: its first searches find
their device state cleared, whatever that stream still has to do."""
import pytest
import torch

from everest_b200 import capi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_first_searches_beside_a_busy_default_stream():
    u, v, t = synth.generate(synth.GraphSpec("state", "zipf", 300, 8_000, seed=5, t_max=80_000))
    dg = capi.DeviceGraph(capi.graph_build_host(u, v, t), 0)
    g = O.Graph(u, v, t, 300)
    queries = [([0, 1, 2], [1, 2, 0], 2000), ([0, 1, 2, 3], [1, 2, 3, 0], 1500)]
    want = [O.count(g, *q)[0] for q in queries]
    a = torch.randn(4096, 4096, device="cuda")
    w = capi.Worker(0)  # (kernels loaded and the graph resident before the timing matters)
    for mu, mv, d in queries:
        w.take(dg, mu, mv, d)
        w.run()
    w.close()
    for _ in range(4):
        for _ in range(8):
            a = torch.tanh(a @ a)  # some milliseconds of work that nothing waits for
        w = capi.Worker(0)
        got = []
        for mu, mv, d in queries * 2:
            w.take(dg, mu, mv, d)
            got.append(w.run())
        assert got == want * 2
        w.close()
    torch.cuda.synchronize()
    dg.free()
