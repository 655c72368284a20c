"""The layout pass at the edges of its rounds: leaves of one point up to the
eight of a round, the 32 of all rounds and beyond (cells that cannot split),
next to one another below one parent, against the oracle's tree and COO."""
import numpy as np
import pytest

from test_gpu_parity import assert_edges_equal, assert_tree_equal, gpu_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndims", [2, 3])
@pytest.mark.parametrize("sizes", [(1, 2, 7, 8, 9), (31, 32, 33, 1), (8, 40, 64, 65, 300), (16, 17, 0, 24, 25)])
def test_leaf_sizes(ob, oracle_mod, sizes, ndims, dtype):
    """A grid of cells of side 1 (the radius) holding sizes[k % len] points each,
    some cells empty, in shuffled order."""
    rng = np.random.default_rng(911 + sum(sizes))
    per = 24 if ndims == 2 else 9
    cells = np.stack(np.meshgrid(*[np.arange(per)] * ndims, indexing="ij"), -1).reshape(-1, ndims)
    cells = cells[rng.random(len(cells)) < 0.7]
    counts = rng.permutation(np.resize(np.asarray(sizes), len(cells)))
    at = np.repeat(cells, counts, axis=0)
    x = (at + 0.05 + 0.9 * rng.random(at.shape)).astype(dtype)[rng.permutation(len(at))]
    r = dtype(1.0)
    tns, sid = gpu_run(ob, x, r)
    ot = oracle_mod.build_tree(x, r)
    assert_tree_equal(tns.trees[sid - 1], ot)
    assert_edges_equal(ob.build_edges(tns, sid, sid), oracle_mod.build_edges(ot, x, exclude_self=True))
