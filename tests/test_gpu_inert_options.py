"""The options that belonged to a walk of the tree (max_seg, multi_pop,
sub_boxes, prefetch) are accepted and reported and change no work."""
import ctypes as C

import pytest
import torch

from conftest import uniform
from test_gpu_parity import gpu_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,value", [("OPT_MAX_SEG", 4), ("OPT_MULTI_POP", 2), ("OPT_SUB_BOXES", 4), ("OPT_PREFETCH", 2)])
def test_inert_option(ob, name, value):
    ctx = ob.api._Context.get(torch.cuda.current_device())
    opt = getattr(ob._lib, name)
    work = ob._lib.TRAVERSAL_STATS.index("cycles_total")  # the counts before the cycles

    def run():
        tns, _ = gpu_run(ob, uniform(6000, 3, 1701), 0.06)
        v = (C.c_uint64 * len(ob._lib.TRAVERSAL_STATS))()
        h = tns.trees[0].handle
        ctx.check(ctx.lib.oct_edges_traversal_stats(ctx.handle, h, h, 1, v, len(v)), "stats")
        return list(v)[:work]

    base = run()
    try:
        ctx.check(ctx.lib.oct_ctx_set_option(ctx.handle, opt, value), name)
        got = C.c_int64()
        ctx.check(ctx.lib.oct_ctx_get_option(ctx.handle, opt, C.byref(got)), name)
        assert got.value == value
        assert run() == base
    finally:
        ctx.check(ctx.lib.oct_ctx_set_option(ctx.handle, opt, 0), name)
