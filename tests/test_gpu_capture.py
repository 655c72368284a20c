"""Trees made, grown and dropped while another stream is being captured: a
relaxed capture allows allocations and frees beside it, but nothing may wait
for the whole device, which would invalidate it."""
import gc

import pytest
import torch

from conftest import uniform

pytestmark = pytest.mark.gpu


def make(ob, n, seed):
    tns = ob.TNS(torch.float32)
    ob.set_search_radius_(tns, 0.1)
    sid = ob.add_point_set_(tns, torch.from_numpy(uniform(n, 3, seed)).cuda().t())
    ob.set_active_search_(tns, sid, sid)
    ob.run_(tns)
    ob.build_edges(tns, sid, sid)
    return tns


@pytest.mark.parametrize("what", ["dropped", "grown", "made"])
def test_beside_a_capture(ob, what):
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.arange(1000, device="cuda", dtype=torch.float32)
    tns = make(ob, 3000, 1301)
    big = torch.from_numpy(uniform(20_000, 3, 1302)).cuda().t()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side, capture_error_mode="relaxed"):
        y = x + 1
        if what == "dropped":
            del tns
            gc.collect()
        else:
            with torch.cuda.stream(other):
                if what == "made":
                    tns = ob.TNS(torch.float32)
                    ob.set_search_radius_(tns, 0.1)
                    ob.add_point_set_(tns, big)
                else:
                    ob.resize_point_set_(tns, 1, big)
                ob.run_(tns)
        z = y * 2
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(z, (x + 1) * 2)
    if what != "dropped":
        assert tns.trees[0].n_nodes > 1
