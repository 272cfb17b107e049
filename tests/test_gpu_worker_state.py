"""A worker made while the default stream is busy: its first searches find
their device state cleared, whatever that stream still has to do."""
import numpy as np
import pytest
import torch

from everest_b200 import capi, synth
from everest_b200.constraints import Constraints
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


def test_a_captured_search_that_never_runs():
    # a job that leaves the state as it ended (the per-lane constrained search),
    # a plain search captured behind it and dropped, and a plain search that runs
    u, v, t = synth.generate(synth.GraphSpec("state", "zipf", 300, 8_000, seed=5, t_max=80_000))
    host = capi.graph_build_host(u, v, t)
    dg = capi.DeviceGraph(host, 0)
    dg.set_features(np.arange(host.num_vertices) % 7, np.arange(host.num_edges) % 5)
    g = O.Graph(u, v, t, 300)
    mu, mv = [0, 1, 2], [1, 2, 0]
    cons = Constraints.from_yaml({"filter": "e0 + e2 > 3"}, mu, mv)
    stream = torch.cuda.Stream()
    w = capi.Worker(0, stream.cuda_stream)
    w.take(dg, mu, mv, 2000)
    want = w.run()
    assert want == O.count(g, mu, mv, 2000)[0]
    w.take(dg, mu, mv, 2000, constraints=cons)
    w.run()
    w.take(dg, mu, mv, 2000)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        w.launch()
        graph.capture_end()
    for _ in range(2):
        w.take(dg, mu, mv, 2000)
        assert w.run() == want
    with torch.cuda.stream(stream):
        graph.replay()
    assert w.run() == want
    w.close()
    dg.free()
