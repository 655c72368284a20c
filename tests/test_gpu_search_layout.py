"""The search over the visiting-order layout where its fast pair test cannot
decide alone, where its box hierarchy has its most levels, and in orders that
mix ascending and descending parts, against the oracle's COO."""
import numpy as np
import pytest
import torch

from conftest import uniform
from test_gpu_parity import assert_edges_equal, gpu_run

pytestmark = pytest.mark.gpu


def grid(per, ndims, dtype):
    g = np.stack(np.meshgrid(*[np.arange(per)] * ndims, indexing="ij"), -1).reshape(-1, ndims)
    return g.astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndims,per", [(2, 90), (3, 21)])
@pytest.mark.parametrize("h,origin", [(0.25, 0.0), (0.1, 0.0), (0.01, 100.0), (1e-4, -3.0)])
def test_pairs_at_exactly_the_radius(ob, oracle_mod, h, origin, ndims, per, dtype):
    """A regular lattice searched with r = 2 h: every query has pairs at
    distance r up to the coordinates' own rounding, so their membership is
    decided by the rounded squared distance alone."""
    x = (grid(per, ndims, np.float64) * h + origin).astype(dtype)
    r = dtype(2 * h)
    tns, sid = gpu_run(ob, x, r)
    want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
    assert_edges_equal(ob.build_edges(tns, sid, sid), want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("scale", [1e-13, 1e-6, 1.0, 1e6, 1e17])
def test_scales_of_the_radius(ob, oracle_mod, scale, dtype):
    """The same points at scales whose squared radii run from 6e-29 (where the
    fast test still applies) to 6e31."""
    x = (uniform(3000, 3, 811, dtype=np.float64) * scale).astype(dtype)
    r = dtype(0.08 * scale)
    tns, sid = gpu_run(ob, x, r)
    want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
    assert_edges_equal(ob.build_edges(tns, sid, sid), want)


@pytest.mark.parametrize("ndims", [2, 3])
def test_groups_wide_against_the_radius(ob, oracle_mod, ndims):
    """Sparse points (leaves of 32 spanning many cells): the fast test does not
    apply; and a few dense spots among them, where it does."""
    rng = np.random.default_rng(821)
    sparse = rng.random((6000, ndims)) * 100
    dense = np.concatenate([rng.random((1, ndims)) * 100 + 0.05 * rng.standard_normal((700, ndims))
                            for _ in range(4)])
    x = np.concatenate([sparse, dense]).astype(np.float32)
    r = np.float32(0.03)
    tns, sid = gpu_run(ob, x, r)
    want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
    assert_edges_equal(ob.build_edges(tns, sid, sid), want)


def test_four_level_hierarchy(ob):
    """35,152,000 points (more than 64 x 512 x 32 x 32): pairs 0.25 apart on a
    lattice of spacing 1, so with r = 0.3 every point's only neighbor is its
    partner."""
    per = 260
    axis = torch.arange(per, device="cuda", dtype=torch.float32)
    site = torch.stack(torch.meshgrid(axis, axis, axis, indexing="ij"), -1).reshape(-1, 3)
    m = site.shape[0]
    order = torch.randperm(2 * m, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    x = torch.cat([site, site + torch.tensor([0.25, 0.0, 0.0], device="cuda")])[order]
    place = torch.empty_like(order)
    place[order] = torch.arange(2 * m, device="cuda")
    partner = place[(order + m) % (2 * m)]
    tns = ob.TNS(torch.float32)
    ob.set_search_radius_(tns, 0.3)
    sid = ob.add_point_set_(tns, x.t())
    ob.set_active_search_(tns, sid, sid)
    ob.run_(tns)
    e = ob.build_edges(tns, sid, sid)
    assert e.senders.numel() == 2 * m
    assert torch.equal(e.receivers, torch.arange(1, 2 * m + 1, device="cuda", dtype=torch.int32))
    assert torch.equal(e.senders.long(), partner + 1)
