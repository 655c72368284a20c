"""Device memory of dropped trees goes back when the caller asks, when one of
the host's own allocations would fail, and at once on a nearly full device."""
import gc

import pytest
import torch

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def drop_a_tree(ob, n=12_000_000):
    tns = ob.TNS(torch.float32)
    ob.set_search_radius_(tns, 0.01)
    ob.add_point_set_(tns, torch.rand((n, 3), device="cuda").t())
    ob.run_(tns)
    del tns
    gc.collect()


def test_release_memory(ob):
    ob.api._Context.get(torch.cuda.current_device())
    ob.release_memory()
    before = free()
    drop_a_tree(ob)
    held = before - free()
    assert held > 500 * MB  # kept for the next tree
    ob.release_memory()
    assert before - free() < 64 * MB


def test_nothing_is_kept_on_a_nearly_full_device(ob):
    ob.api._Context.get(torch.cuda.current_device())
    ob.release_memory()
    total = torch.cuda.mem_get_info()[1]
    rest = torch.empty(free() - total // 16, dtype=torch.uint8, device="cuda")
    before = free()
    drop_a_tree(ob)
    assert before - free() < 64 * MB
    del rest
    free()


def test_own_allocations_give_it_back(ob):
    """About 1.5 GB of edges for a set of 30,000 points where only the kept memory can
    hold them."""
    x = torch.rand((30_000, 3), device="cuda")
    tns = ob.TNS(torch.float32)
    ob.set_search_radius_(tns, 0.27)
    sid = ob.add_point_set_(tns, x.t())
    ob.set_active_search_(tns, sid, sid)
    ob.run_(tns)
    for _ in range(3):  # (until the hit records' size has settled)
        n = ob.build_edges_(tns, sid, sid).n_edges
    need = 24 * (n + n // 4)
    assert 900 * MB < need < 2200 * MB
    tns.edge_buffers[0] = ob.EdgeBuffer(torch.float32, 3, torch.cuda.current_device())
    ob.release_memory()
    drop_a_tree(ob, 32_000_000)  # (2 GB and more)
    rest = torch.empty(free() - 200 * MB, dtype=torch.uint8, device="cuda")
    e = ob.build_edges(tns, sid, sid)
    assert e.senders.numel() == n
    del rest, e, tns
    free()
