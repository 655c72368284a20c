"""Senders outside 1..n all over a large COO: the blocks that meet them set the
status while others read it, and the call ends with an argument error every
time, on a context that goes on working."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [0, -5, 400_001, 2**31 - 1])
@pytest.mark.parametrize("every", [1, 97, 50_000, 3_199_999])
def test_bad_senders(ob, every, bad):
    n, deg = 400_000, 8
    i = torch.arange(n, device="cuda")
    off = torch.tensor([-4, -3, -2, -1, 1, 2, 3, 4], device="cuda")
    good = ((i[:, None] + off) % n + 1).int().reshape(-1)
    rcv = (i + 1).int().repeat_interleave(deg)
    m = n * deg
    snd = good.clone()
    snd[every - 1::every] = bad
    x = torch.rand((n, 3), device="cuda")
    d = torch.ones(m, device="cuda")
    grad = torch.empty((n, 3), device="cuda")
    lc = ob.api._Context.get(torch.cuda.current_device())
    lc.bind_stream()
    p = lambda t: C.c_void_p(t.data_ptr())

    def backward(s):
        lc.check(lc.lib.oct_edges_diff_backward_recompute(lc.handle, 3, 0, n, m, p(s), p(rcv), p(x), None, p(d), 1.0,
                                                          p(grad)), "adjoint")

    for _ in range(3):
        with pytest.raises(ob.ArgumentError):
            backward(snd)
    backward(good)
    # each edge and its mirror pull with 1 along the line between the points
    j = 12_345
    u = x[j].double() - x[(j + off) % n].double()
    want = 2 * (u / u.norm(dim=1, keepdim=True)).sum(0)
    assert (grad[j].double() - want).abs().max() <= 2 * 8 * 6 * 2.0 ** -24
