"""Device memory of a built tree: uniform Float32 points took 82 bytes each
when the search walked the tree's nodes; the search layout may not take more."""
import ctypes as C
import gc

import numpy as np
import pytest
import torch

from test_gpu_parity import assert_edges_equal, assert_tree_equal

pytestmark = pytest.mark.gpu


def test_bytes_per_point(ob):
    n = 24_000_000
    x = torch.rand((n, 3), device="cuda")
    ob.api._Context.get(torch.cuda.current_device())
    gc.collect()
    ob.release_memory()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    tns = ob.TNS(torch.float32)
    ob.set_search_radius_(tns, 0.01)
    ob.add_point_set_(tns, x.t())
    ob.run_(tns)
    torch.cuda.empty_cache()
    used = before - torch.cuda.mem_get_info()[0]
    assert used <= 83 * n, used / n


def sparse_chunks(cells, ndims, seed):
    """Cells of four radii whose octants (quadrants) hold 33 points in two
    sub-cells (17 and 16, two chunks) and one point (a chunk of its own) in
    turn: 12 chunks per 136 points, more than two per 32."""
    rng = np.random.default_rng(seed)
    base = np.stack(np.meshgrid(*[np.arange(cells)] * ndims, indexing="ij"), -1).reshape(-1, ndims) * 4.0
    parts = []
    for slot in range(2 ** ndims):
        at = base + 2.0 * np.array([slot >> d & 1 for d in range(ndims)])
        for k, m in ((0, 17), (2 ** ndims - 1, 16)) if slot % 2 == 0 else ((0, 1),):
            sub = np.array([k >> d & 1 for d in range(ndims)], float)
            parts.append(np.repeat(at + sub, m, axis=0) + 0.05 + 0.9 * rng.random((m * len(at), ndims)))
    x = np.concatenate(parts)
    return x[rng.permutation(len(x))]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndims,cells", [(3, 9), (2, 40)])
def test_more_chunks_than_expected(ob, oracle_mod, ndims, cells, dtype):
    """The first build is laid out again with the counted capacity, a later one of
    the same tree is not; a step with unchanged keys between them (which builds
    no topology, so its attempts are not counted) uses that capacity too."""
    x = sparse_chunks(cells, ndims, 1501).astype(dtype)
    r = dtype(1.0)
    tns = ob.TNS(torch.from_numpy(x).dtype, ndims)
    ob.set_search_radius_(tns, r)
    ob.set_refit_mode_(tns, True)
    sid = ob.add_point_set_(tns, torch.from_numpy(x).cuda().t())
    ob.set_active_search_(tns, sid, sid)
    ctx = tns._ctx
    attempts = C.c_int64()
    # (the 2D set has more nodes than expected too, which takes an attempt of its own)
    for build, want_attempts in enumerate((3 if ndims == 2 else 2, None, 1)):
        if build:
            x = x + dtype(0.01) * np.random.default_rng(build).random(x.shape).astype(dtype) * (build == 2)
            ob.update_point_set_(tns, sid, torch.from_numpy(x).cuda().t())
        ob.run_(tns)
        ctx.check(ctx.lib.oct_ctx_get_option(ctx.handle, ob._lib.STAT_BUILD_ATTEMPTS, C.byref(attempts)), "attempts")
        assert want_attempts is None or attempts.value == want_attempts
        assert (tns.trees[0].last_build()[0] == 2) == (build == 1)
        ot = oracle_mod.build_tree(x, r)
        assert_tree_equal(tns.trees[0], ot)
        assert_edges_equal(ob.build_edges(tns, sid, sid), oracle_mod.build_edges(ot, x, exclude_self=True))


def test_pullback_after_each_kind_of_build(ob):
    """apply_zsort's gradient needs the inverse order, which shares the run
    boxes' memory: after a sort, after a merge, after unchanged keys, and for
    points of a single cell."""
    g = torch.Generator(device="cuda").manual_seed(3)
    for n, r in ((50_000, 0.02), (500, 5.0)):
        x = torch.rand((n, 3), device="cuda", generator=g)
        tns = ob.TNS(torch.float32)
        ob.set_search_radius_(tns, r)
        ob.set_refit_mode_(tns, True)
        sid = ob.add_point_set_(tns, x.t())
        for step in range(5):
            if step in (1, 2):
                x = x.clone()
                x[::97] = (x[::97] + 0.03) % 1
            ob.update_point_set_(tns, sid, x.t())
            ob.run_(tns)
            perm = tns.permutation[0].long() - 1
            assert torch.equal(perm.sort().values, torch.arange(n, device="cuda"))
            a = torch.rand((4, n), device="cuda", generator=g, requires_grad=True)
            y = ob.apply_zsort(tns, sid, a)
            assert torch.equal(y.detach(), a.detach()[:, perm])
            w = torch.rand((4, n), device="cuda", generator=g)
            grad, = torch.autograd.grad(y, a, w)
            want = torch.empty_like(w)
            want[:, perm] = w
            assert torch.equal(grad, want)
