"""Graph arrays whose out- or in-list names an edge twice (and so lacks
another): refused before anything searches them, from host and device arrays;
a list in another order than the builder's is not."""
import numpy as np
import pytest
import torch

from everest_b200 import capi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[2, 255, 20_000])
def host(request):
    u, v, t = synth.generate(synth.GraphSpec("lists", "zipf", 60, request.param, seed=9, t_max=60_000))
    return capi.graph_build_host(u, v, t)


def changed(host, **lists):
    return capi.HostGraph(host.num_edges, host.num_vertices, host.eg, lists.get("out_v", host.out_v),
                          lists.get("in_v", host.in_v), host.out_r, host.in_r, host.euid)


@pytest.mark.parametrize("which", ["out_v", "in_v"])
@pytest.mark.parametrize("at,like", [(0, 1), (-1, 0)])
def test_a_list_that_lacks_an_edge_is_refused(host, which, at, like):
    x = getattr(host, which).copy()
    x[at] = x[like]
    bad = changed(host, **{which: x})
    with pytest.raises(capi.EvxError) as ei:
        capi.DeviceGraph(bad, 0)
    assert ei.value.code == -1
    arrays = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
              for a in (bad.eg, bad.out_v, bad.in_v, bad.out_r, bad.in_r, bad.euid)]
    torch.cuda.synchronize()
    with pytest.raises(capi.EvxError):
        capi.DeviceGraph.from_device(0, bad.num_edges, bad.num_vertices, *(a.data_ptr() for a in arrays))


def test_whole_lists_are_taken(host):
    g = O.Graph(host.eg[0::3], host.eg[1::3], host.eg[2::3], host.num_vertices)
    w = capi.Worker(0)
    dg = capi.DeviceGraph(host, 0)
    w.take(dg, [0, 1], [1, 0], 500)
    assert w.run() == O.count(g, [0, 1], [1, 0], 500)[0]
    w.close()
    dg.free()
