"""The fill's two ways of listing hits, and sets that change between them: all
points neighbors of all (full masks), dense spots among sparse points, masks
around sixteen hits, and neighbor lists, in 2D and 3D and both types."""
import numpy as np
import pytest
import torch

from conftest import uniform
from test_gpu_parity import assert_edges_equal, gpu_run

pytestmark = pytest.mark.gpu


def sets(ndims, dtype):
    rng = np.random.default_rng(1601)
    spots = [rng.random((1, ndims)) * 50 + 0.02 * rng.standard_normal((m, ndims)) for m in (1, 15, 16, 17, 31, 32, 33, 400)]
    return {
        "all": (uniform(701, ndims, 1602, dtype=dtype), dtype(2.0)),
        "spots": (np.concatenate([rng.random((900, ndims)) * 50, *spots])[rng.permutation(1445)].astype(dtype), dtype(0.2)),
        "half": (uniform(3000, ndims, 1603, dtype=dtype), dtype(0.2)),
        "repeated": (np.repeat(uniform(90, ndims, 1604, dtype=dtype), 40, axis=0)[rng.permutation(3600)], dtype(0.05)),
    }


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndims", [2, 3])
@pytest.mark.parametrize("name", ["all", "spots", "half", "repeated"])
def test_dense_fill(ob, oracle_mod, name, ndims, dtype):
    x, r = sets(ndims, dtype)[name]
    tns, sid = gpu_run(ob, x, r)
    want = oracle_mod.build_edges(oracle_mod.build_tree(x, r), x, exclude_self=True)
    for _ in range(2):  # (the second count has room for every record)
        assert_edges_equal(ob.build_edges(tns, sid, sid), want)
    ob.materialize_all_neighbors_(tns)
    assert torch.equal(tns.neighbor_buffers[0].flat.cpu(), torch.from_numpy(want["senders"]))
