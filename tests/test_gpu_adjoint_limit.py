"""The adjoint at the largest edge count that the entry points take, 2^31 - 1:
a ring of 2^28 - 1 points with eight neighbors each, and seven more edges on
the last point, so that the last segment ends where Int32 does."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

OFFSETS = (-4, -3, -2, -1, 1, 2, 3, 4)


def test_two_to_the_31_edges(ob):
    torch.cuda.empty_cache()
    ob.release_memory()
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GB of device memory")
    n = (1 << 28) - 1
    m = (1 << 31) - 1
    snd = torch.empty(m, dtype=torch.int32, device="cuda")
    rcv = torch.empty(m, dtype=torch.int32, device="cuda")
    d_dist = torch.empty(m, dtype=torch.float32, device="cuda")
    i = torch.arange(n, device="cuda")
    for c, off in enumerate(OFFSETS):
        snd[:8 * n].view(n, 8)[:, c] = ((i + off) % n + 1).int()
        rcv[:8 * n].view(n, 8)[:, c] = (i + 1).int()
        d_dist[:8 * n].view(n, 8)[:, c] = (i % 13).float() / 16 + c
    del i
    snd[8 * n:] = snd[8 * n - 8:8 * n - 1].clone()
    rcv[8 * n:] = n
    d_dist[8 * n:] = 0.25
    x = torch.rand((n, 3), device="cuda")
    grad = torch.empty((n, 3), device="cuda")
    lib = ob._lib.load()
    ctx = C.c_void_p()
    assert lib.oct_ctx_create(torch.cuda.current_device(), C.byref(ctx)) == 0
    p = lambda t: C.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    st = lib.oct_edges_diff_backward_recompute(ctx, 3, 0, n, m, p(snd), p(rcv), p(x), None, p(d_dist), 1.0, p(grad))
    torch.cuda.synchronize()
    msg = lib.oct_ctx_last_error(ctx)
    lib.oct_ctx_destroy(ctx)
    assert st == 0, msg
    # 64-bit gradients of the first, middle and last points: the edge j -> q and
    # its mirror each pull along (x_q - x_j) / |x_q - x_j|
    for lo in (0, n // 2, n - 6):
        qs = torch.arange(lo, lo + 6, device="cuda")
        win = (torch.arange(lo - 4, lo + 10, device="cuda") % n)
        xs = dict(zip(win.tolist(), x[win].double().cpu().numpy()))
        d = dict(zip(win.tolist(), d_dist[:8 * n].view(n, 8)[win].double().cpu().numpy()))
        for q, got in zip(qs.tolist(), grad[qs].double().cpu().numpy()):
            want = np.zeros(3)
            for c, off in enumerate(OFFSETS):
                j = (q + off) % n
                own = [d[q][c]] + ([0.25] if q == n - 1 and c < 7 else [])
                u = (xs[q] - xs[j]) / np.linalg.norm(xs[q] - xs[j])
                want += sum((w + d[j][7 - c]) * u for w in own)
            # 15 edges and mirrors of up to 8 each, six Float32 roundings per term
            assert np.abs(got - want).max() <= 2 * 15 * 8 * 6 * 2.0 ** -24, (q, got, want)
