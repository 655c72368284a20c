"""The searching adjoint's segments and mirror scans at their edges: few edges,
edge counts off the four-receiver runs and the eight-entry scan blocks, points
without edges, and edge arrays that do not start on a 16- or 32-byte boundary."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import uniform

pytestmark = pytest.mark.gpu


def off_boundary(t, words):
    """A copy of t that starts `words` elements into its allocation."""
    buf = torch.empty(t.numel() + words, dtype=t.dtype, device=t.device)
    buf[words:] = t.reshape(-1)
    return buf[words:]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,r", [(2, 2.0), (3, 2.0), (9, 0.4), (33, 0.2), (257, 0.05), (1023, 0.12)])
def test_adjoint_segments(ob, oracle_mod, dtype, n, r):
    x = uniform(n, 3, 9100 + n, dtype=dtype)
    r = dtype(r)
    T = torch.from_numpy(x).dtype
    tns = ob.TNS(T, ndims=3)
    ob.set_search_radius_(tns, r)
    sid = ob.add_point_set_(tns, torch.from_numpy(x).cuda().t())
    ob.set_active_search_(tns, sid, sid)
    ob.run_(tns)
    e = ob.build_edges(tns, sid, sid)
    # without the edges of two points (both directions, so that the mirrors stay)
    drop = torch.tensor([1, n // 2 + 1], device="cuda") if n > 8 else torch.tensor([0], device="cuda")
    keep = ~(torch.isin(e.senders, drop) | torch.isin(e.receivers, drop))
    snd, rcv = e.senders[keep], e.receivers[keep]
    rd = e.rel_displacement.t()[keep].contiguous()
    rn = e.rel_dist_norm.reshape(-1)[keep].contiguous()
    gd, gn = torch.sin(rd * 7), torch.cos(rn * 3)
    m = snd.numel()
    lc = tns._ctx
    lc.bind_stream()
    p = lambda t: C.c_void_p(t.data_ptr())
    grads = []
    for words in (0, 1, 4):
        s, q = off_boundary(snd, words), off_boundary(rcv, words)
        grad = torch.empty(n, 3, dtype=T, device="cuda")
        lc.check(lc.lib.oct_edges_diff_backward(lc.handle, 3, 0 if dtype == np.float32 else 1, n, m, p(s), p(q), p(rd),
                                                p(rn), p(gd), p(gn), float(r), p(grad)), "adjoint")
        grads.append(grad)
    assert torch.equal(grads[0], grads[1]) and torch.equal(grads[0], grads[2])
    want = oracle_mod.diff_backward(n, snd.cpu().numpy(), rcv.cpu().numpy(), rd.cpu().numpy(), rn.cpu().numpy(),
                                    gd.cpu().numpy(), gn.cpu().numpy(), r)
    tol = 1e-12 if dtype == np.float64 else 2e-5
    assert np.abs(grads[0].cpu().numpy() - want).max() <= tol * max(np.abs(want).max(), 1e-30)
