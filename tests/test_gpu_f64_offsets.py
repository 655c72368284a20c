"""Float64 points far from the origin and at large scales: the search keeps its
COO and tests no more targets than the same points at the origin."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_parity import assert_edges_equal, gpu_run

pytestmark = pytest.mark.gpu


def points(n, ndims, seed):
    """Multiples of 2^-20 in the unit cube: shifted by up to 2^30 or scaled by a
    power of two they are the same points exactly, pair for pair."""
    return np.random.default_rng(seed).integers(0, 1 << 20, (n, ndims)).astype(np.float64) / (1 << 20)


def work(ob, tns, sid):
    lib, ctx = tns._ctx.lib, tns._ctx
    names = ob._lib.TRAVERSAL_STATS
    v = (C.c_uint64 * len(names))()
    ctx.bind_stream()
    h = tns.trees[sid - 1].handle
    ctx.check(lib.oct_edges_traversal_stats(ctx.handle, h, h, 1, v, len(names)), "stats")
    return dict(zip(names, v))


@pytest.mark.parametrize("ndims,n,r", [(3, 20_003, 1 / 16), (2, 20_003, 1 / 64)])
@pytest.mark.parametrize("offset,log2_scale", [(1e5, 0), (3e6, 0), (float(1 << 30), 0), (0.0, 70), (0.0, 400)])
def test_work_and_coo_do_not_depend_on_the_offset(ob, oracle_mod, offset, log2_scale, ndims, n, r):
    x0 = points(n, ndims, 1401)
    near, sid = gpu_run(ob, x0, np.float64(r))
    base = work(ob, near, sid)
    x = np.ldexp(x0, log2_scale) + offset
    rad = np.float64(np.ldexp(r, log2_scale))
    far, sid = gpu_run(ob, x, rad)
    e = ob.build_edges(far, sid, sid)
    assert_edges_equal(e, oracle_mod.build_edges(oracle_mod.build_tree(x, rad), x, exclude_self=True))
    assert e.senders.numel() == ob.build_edges(near, 1, 1).senders.numel()
    # Only the cells' origin (the minimum less 1e-6, rounded) differs, by at most
    # 1e-6 of a cell side of 1/64 or more: fewer than one point in ten thousand
    # changes its cell.
    got = work(ob, far, sid)
    for name in ("children_tested", "leaf_chunks", "targets_staged", "pair_tests"):
        assert got[name] <= 1.05 * base[name], (name, got[name], base[name])


@pytest.mark.parametrize("ndims,r", [(3, 1 / 8), (2, 1 / 32)])
def test_cross_pair_and_batch_far_from_the_origin(ob, oracle_mod, ndims, r):
    """Queries and targets of different extents, and clouds at different places."""
    a, b = points(3001, ndims, 1402) * 2 + 5e6, points(9001, ndims, 1403) + 5e6
    tns = ob.TNS(torch.float64, ndims)
    ob.set_search_radius_(tns, r)
    ia = ob.add_point_set_(tns, torch.from_numpy(a).cuda().t())
    ib = ob.add_point_set_(tns, torch.from_numpy(b).cuda().t())
    ob.set_active_search_(tns, ia, ib)
    ob.run_(tns)
    want = oracle_mod.build_edges(oracle_mod.build_tree(b, np.float64(r)), a, exclude_self=False)
    assert_edges_equal(ob.build_edges(tns, ia, ib), want)
    from test_gpu_batch import check_against_oracle, run_batch
    clouds = [points(n, ndims, 1410 + n) + place for n, place in [(700, 1e9), (1, -3e6), (2500, 0.0), (999, 4.5e6)]]
    radii = np.array([r, 2 * r, r, r / 2])
    e = run_batch(ob, clouds, np.array([len(c) for c in clouds], np.int64), radii, np.float64)
    check_against_oracle(e, clouds, radii, oracle_mod)


@pytest.mark.parametrize("log2_width", [13, 16, 24, 29, 31])
def test_sets_many_radii_wide(ob, oracle_mod, log2_width):
    """Two dense spots and a line of points between them, up to just under 2^31
    radii apart: the box units per radius fall from 2^14 to 1/4."""
    rng = np.random.default_rng(1420)
    width = np.ldexp(1.0, log2_width) - 4
    spots = [rng.random((600, 3)) * 3 + np.array([k * (width - 3), 0, 0]) for k in (0, 1)]
    line = np.sort(rng.random(300)) * width
    x = np.concatenate(spots + [np.stack([line, 0 * line, 0 * line], 1)])[rng.permutation(1500)] - 12345.0
    r = np.float64(1.0)
    tns, sid = gpu_run(ob, x, r)
    want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
    assert_edges_equal(ob.build_edges(tns, sid, sid), want)
    # few queries are one group, whose far members lie beyond the targets' units
    up, down = np.ldexp(1.0, 30) - width / 2, np.ldexp(1.0, 29) - width / 4  # all together below 2^31 radii wide
    far = [x[:4] + up, x[4:8] - down] if log2_width < 31 else []
    for q in (np.concatenate([x[:20] + 0.25, *far]), np.concatenate([x[::3] - 0.25, *far])):
        pair = ob.TNS(torch.float64, 3)
        ob.set_search_radius_(pair, 1.0)
        iq = ob.add_point_set_(pair, torch.from_numpy(q).cuda().t())
        it = ob.add_point_set_(pair, torch.from_numpy(x).cuda().t())
        ob.set_active_search_(pair, iq, it)
        ob.run_(pair)
        want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), q, exclude_self=False)
        assert_edges_equal(ob.build_edges(pair, iq, it), want)


def test_time_steps_far_from_the_origin(ob, oracle_mod):
    """Refit-mode steps (a sort, merges that do not wait for the bounds, unchanged
    keys) whose extremes move, so that the units' origin differs between the
    steps; the kernels derive it on the device, the search from the host's copy."""
    rng = np.random.default_rng(1430)
    x = points(8000, 3, 1431) + 3e6
    r = np.float64(1 / 16)
    tns = ob.TNS(torch.float64, 3)
    ob.set_search_radius_(tns, r)
    ob.set_refit_mode_(tns, True)
    sid = ob.add_point_set_(tns, torch.from_numpy(x).cuda().t())
    ob.set_active_search_(tns, sid, sid)
    paths = []
    for step in range(7):
        if step:
            x = x.copy()
            if step == 4:
                x[5] = x[5]  # nothing moves
            else:
                move = rng.choice(len(x), 150, replace=False)
                x[move] += 0.02 * rng.standard_normal((150, 3))
            if step == 5:
                x[x[:, 0].argmin(), 0] -= 1e-4  # the origin, by less than a cell
            ob.update_point_set_(tns, sid, torch.from_numpy(x).cuda().t())
        ob.run_(tns)
        paths.append(tns.trees[0].last_build()[0])
        want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
        assert_edges_equal(ob.build_edges(tns, sid, sid), want)
    assert paths[0] == 0 and 1 in paths and paths[4] == 2
