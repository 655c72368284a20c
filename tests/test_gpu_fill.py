"""The fill into arrays that are aligned to their element only, and from record
lists longer than its shared-memory list, against the oracle's COO."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import clustered, uniform
from test_gpu_parity import assert_edges_equal, gpu_run, torch_dtype

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndims", [2, 3])
def test_fill_into_arrays_off_their_vector_alignment(ob, oracle_mod, ndims, dtype, offset):
    x = uniform(4001, ndims, 771, dtype=dtype)
    r = dtype(0.07 if ndims == 3 else 0.03)
    tns, sid = gpu_run(ob, x, r)
    want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
    ctx, h, T = tns._ctx, tns.trees[sid - 1].handle, torch_dtype(x)
    ne = C.c_int64()
    ctx.check(ctx.lib.oct_edges_count(ctx.handle, h, h, 1, C.byref(ne)), "count")
    m = int(ne.value)
    assert m == len(want["senders"])
    snd, rcv = (torch.full((m + 8,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    disp, dist = torch.full((ndims * m + 8,), -1, dtype=T, device="cuda"), torch.full((m + 8,), -1, dtype=T, device="cuda")
    part = [t[offset:offset + k] for t, k in ((snd, m), (rcv, m), (disp, ndims * m), (dist, m))]
    ctx.check(ctx.lib.oct_edges_fill(ctx.handle, h, h, 1, *(C.c_void_p(t.data_ptr()) for t in part), m), "fill")
    ob.synchronize(tns)
    assert np.array_equal(part[0].cpu().numpy(), want["senders"])
    assert np.array_equal(part[1].cpu().numpy(), want["receivers"])
    assert np.array_equal(part[2].cpu().numpy().reshape(m, ndims), want["rel_displacement"])
    assert np.array_equal(part[3].cpu().numpy(), want["rel_dist_norm"])
    for whole, k in ((snd, m), (rcv, m), (disp, ndims * m), (dist, m)):
        assert (whole[:offset] == -1).all() and (whole[offset + k:] == -1).all()


@pytest.mark.parametrize("ndims", [2, 3])
@pytest.mark.parametrize("n", [33, 64, 700, 2500])
def test_every_point_a_neighbor_of_every_other(ob, oracle_mod, n, ndims):
    """Records of 32 hits: 1,024 per batch of records, more than the list holds."""
    x = (0.5 + 0.01 * clustered(n, ndims, 781 + n)).astype(np.float32)
    r = np.float32(0.1)
    tns, sid = gpu_run(ob, x, r)
    want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
    assert len(want["senders"]) == n * (n - 1)
    assert_edges_equal(ob.build_edges(tns, sid, sid), want)
    ob.materialize_all_neighbors_(tns)
    assert np.array_equal(tns.neighbor_buffers[0].flat.cpu().numpy(), want["senders"])
