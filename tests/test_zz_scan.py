"""The offset scan at the edges of a thread's eight items, of the one-block form
(8,192 counts) and of its 2,048-count tiles, over arrays that start on a 32-byte
boundary or not, through the allocation-free count (whose arrays are the
caller's).  Collected after the file that expects that count's first call."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048, 2049, 8191, 8192, 8193, 10241, 2048 * 70 + 3])
def test_offsets(ob, n):
    x = uniform(n, 3, 1501)
    r = np.float32(1.2 / max(n, 2) ** (1 / 3))
    tns = ob.TNS(torch.float32)
    ob.set_search_radius_(tns, r)
    sid = ob.add_point_set_(tns, torch.from_numpy(x).cuda().t())
    ob.set_active_search_(tns, sid, sid)
    ob.run_(tns)
    e = ob.build_edges(tns, sid, sid)
    want = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    want[1:] = torch.cumsum(torch.bincount(e.receivers.long() - 1, minlength=n), 0)
    ctx = tns._ctx
    for shift_in, shift_out in ((0, 0), (1, 0), (0, 1), (3, 2)):
        counts = torch.full((n + 16,), -7, dtype=torch.int32, device="cuda")
        offsets = torch.full((n + 17,), -7, dtype=torch.int64, device="cuda")
        total = C.c_int64(-1)
        ctx.bind_stream()
        tree = tns.trees[sid - 1].handle
        ctx.check(ctx.lib.oct_edges_count_noalloc(ctx.handle, tree, tree, 1, C.c_void_p(counts[shift_in:].data_ptr()),
                                                  C.c_void_p(offsets[shift_out:].data_ptr()), C.byref(total)), "count")
        assert total.value == e.senders.numel()
        assert torch.equal(offsets[shift_out:shift_out + n + 1], want)
        assert torch.equal(counts[shift_in:shift_in + n].long(), want[1:] - want[:-1])
        # nothing outside the two arrays
        assert (counts[:shift_in] == -7).all() and (counts[shift_in + n:] == -7).all()
        assert (offsets[:shift_out] == -7).all() and (offsets[shift_out + n + 1:] == -7).all()
