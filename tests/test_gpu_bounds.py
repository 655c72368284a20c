"""The bounds fold at the edges of its vector groups (two, four points per
16-byte words), blocks (2,048 points) and grid, from a point array that starts
on a 16-byte boundary or not: extremes in the first, last and a random point,
-0.0 beside 0.0, non-finite values anywhere."""
import numpy as np
import pytest
import torch

from conftest import uniform
from test_gpu_parity import assert_edges_equal, assert_tree_equal, torch_dtype

pytestmark = pytest.mark.gpu


def run(ob, x, r, shift):
    """The tree of x, whose device array starts `shift` points into an allocation."""
    T = torch_dtype(x)
    buf = torch.empty((len(x) + shift, x.shape[1]), dtype=T, device="cuda")
    buf[shift:] = torch.from_numpy(x).cuda()
    tns = ob.TNS(T, ndims=x.shape[1])
    ob.set_search_radius_(tns, r)
    sid = ob.add_point_set_(tns, buf[shift:].t())
    ob.set_active_search_(tns, sid, sid)
    ob.run_(tns)
    return tns, sid


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndims", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 2047, 2048, 2049, 4 * 148 * 2048 + 5])
def test_bounds(ob, oracle_mod, n, ndims, dtype):
    big = n > 100000
    r = dtype(0.01 if big else 0.1)
    for at in {0, n - 1, (7 * n) // 11}:
        x = uniform(n, ndims, 1301, -0.5, 0.5, dtype=dtype)
        x[at] = np.resize([-0.75, 0.875], ndims)
        if n > 4:
            x[:, 0] = np.abs(x[:, 0])
            x[2, 0], x[n // 2, 0] = -0.0, 0.0  # the minimum of the first axis
            x[at, 0] = 0.75
        ot = oracle_mod.build_tree(x, r, nthreads=0)
        for shift in (0, 1):
            tns, sid = run(ob, x, r, shift)
            assert_tree_equal(tns.trees[sid - 1], ot)
            if not big:
                assert_edges_equal(ob.build_edges(tns, sid, sid), oracle_mod.build_edges(ot, x, exclude_self=True))
        if big:
            break


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,at", [(1, 0), (5, 4), (2049, 2048), (2049, 1000)])
def test_non_finite(ob, n, at, dtype, value):
    x = uniform(n, 3, 1302, dtype=dtype)
    x[at, 1] = value
    for shift in (0, 1):
        with pytest.raises(Exception):
            run(ob, x, dtype(0.1), shift)
