"""Device memory kept for the next tree: trees made after others were dropped
take their buffers (stale contents included) and are exact, on one stream, on
several, and from several threads; what is held stays within its bound."""
import gc
import threading

import numpy as np
import pytest
import torch

from conftest import uniform
from test_gpu_parity import assert_edges_equal, assert_tree_equal, gpu_run

pytestmark = pytest.mark.gpu


def check(ob, oracle_mod, n, r, seed, ndims=3):
    x = uniform(n, ndims, seed)
    r = np.float32(r)
    tns, sid = gpu_run(ob, x, r)
    ot = oracle_mod.build_tree(x, r)
    assert_tree_equal(tns.trees[sid - 1], ot)
    assert_edges_equal(ob.build_edges(tns, sid, sid), oracle_mod.build_edges(ot, x, exclude_self=True))


def test_trees_in_the_buffers_of_dropped_ones(ob, oracle_mod):
    for k, (n, ndims) in enumerate([(20_000, 3), (1, 3), (20_000, 2), (19_000, 3), (40, 2), (30_000, 3), (15_000, 3)]):
        check(ob, oracle_mod, n, 0.05 if ndims == 3 else 0.02, 1000 + k, ndims)
        gc.collect()


def test_buffers_pass_between_streams(ob, oracle_mod):
    streams = [torch.cuda.Stream() for _ in range(3)]
    for k in range(6):
        with torch.cuda.stream(streams[k % 3]):
            check(ob, oracle_mod, 12_000 + 500 * k, 0.05, 1100 + k)
        gc.collect()


def test_trees_made_and_dropped_by_threads(ob):
    """Each thread makes and drops trees of its own (the library's calls of one
    context are serialized by a lock here, as its users must)."""
    lock = threading.Lock()
    ctx = ob.api._Context.get(torch.cuda.current_device())
    failed = []

    def work(seed):
        try:
            for k in range(5):
                x = torch.from_numpy(uniform(5000 + 700 * k, 3, seed + k)).cuda()
                with lock:
                    tns = ob.TNS(torch.float32)
                    ob.set_search_radius_(tns, 0.06)
                    sid = ob.add_point_set_(tns, x.t())
                    ob.set_active_search_(tns, sid, sid)
                    ob.run_(tns)
                    n = ob.build_edges(tns, sid, sid).senders.numel()
                    d = torch.cdist(x, x)
                    near = int((d < 0.06 - 1e-5).sum()) - len(x), int((d < 0.06 + 1e-5).sum()) - len(x)
                    if not near[0] <= n <= near[1]:
                        failed.append((seed, k, n, near))
                del tns
        except Exception as e:  # noqa: BLE001
            failed.append((seed, repr(e)))

    threads = [threading.Thread(target=work, args=(1200 + 100 * t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    assert ctx.handle is not None


def test_held_memory_is_bounded(ob):
    """Dropping trees of 12 million points (over 1 GB each) one after another
    leaves no more than the bound (4 GiB) beyond one context's own buffers."""
    torch.cuda.empty_cache()
    free0, _ = torch.cuda.mem_get_info()
    for k in range(3):
        sets = []
        for j in range(3):
            tns = ob.TNS(torch.float32)
            ob.set_search_radius_(tns, 0.01)
            ob.add_point_set_(tns, torch.rand((12_000_000 + 1_000_000 * j, 3), device="cuda").t())
            ob.run_(tns)
            sets.append(tns)
        del sets, tns
        gc.collect()
        torch.cuda.empty_cache()
    free1, _ = torch.cuda.mem_get_info()
    assert free0 - free1 < (4 << 30) + (64 << 20)
