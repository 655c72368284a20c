"""Node numbering, ranges and bounds at the edges of the topology passes' tiles
(512 positions per block, 64 per warp, strips of 32) and of the one-block scan
(8,192 inputs), against the oracle's tree."""
import numpy as np
import pytest
import torch

from conftest import uniform
from test_gpu_parity import assert_edges_equal, assert_tree_equal, gpu_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndims", [2, 3])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 96, 511, 512, 513, 1023, 1025, 8191, 8192, 8193])
def test_tree_at_tile_edges(ob, oracle_mod, n, ndims):
    """Uniform points, and the same with most of them in a few cells (leaves
    of far more than 32 points next to single points)."""
    x = uniform(n, ndims, 700 + n)
    tied = x.copy()
    tied[: 3 * n // 4] = x[np.random.default_rng(n).integers(0, 3, 3 * n // 4) % n]
    for y in (x, tied):
        tns, sid = gpu_run(ob, y, np.float32(0.04))
        ot = oracle_mod.build_tree(y, np.float32(0.04))
        assert_tree_equal(tns.trees[sid - 1], ot)
        assert_edges_equal(ob.build_edges(tns, sid, sid), oracle_mod.build_edges(ot, y, exclude_self=True))


@pytest.mark.parametrize("n", [372 * 512, 372 * 512 + 1])
def test_tree_around_the_one_block_scan(ob, oracle_mod, n):
    """22 levels x 372 and 373 blocks of node counts: 8,184 and 8,206 inputs."""
    x = uniform(n, 3, 731)
    tns, sid = gpu_run(ob, x, np.float32(0.02))
    assert_tree_equal(tns.trees[sid - 1], oracle_mod.build_tree(x, np.float32(0.02), nthreads=0))
