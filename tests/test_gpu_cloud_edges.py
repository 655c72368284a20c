"""Clouds at the edges of the batch's tiles: sizes around the 512 threads and
4,096 points of a bounds round and the 2,048-point sort tiles, many tiny and
empty clouds in one tile, extremes (and -0.0, non-finite values) in the last
point of a cloud."""
import numpy as np
import pytest
import torch

from test_gpu_batch import check_against_oracle, run_batch

pytestmark = pytest.mark.gpu

SIZES = {
    "rounds": [0, 1, 511, 512, 513, 4095, 4096, 4097, 8193, 3, 0, 2048],
    "tiny": [k % 4 for k in range(3000)] + [2049],
}


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndims", [2, 3])
@pytest.mark.parametrize("name", list(SIZES))
def test_cloud_sizes(ob, oracle_mod, name, ndims, dtype):
    rng = np.random.default_rng(1201)
    clouds = []
    for n in SIZES[name]:
        x = rng.random((n, ndims)) - 0.5
        if n > 2:
            x[-1] = rng.choice([-0.75, 0.75], ndims)  # the last point is an extreme of the box
            x[0, 0] = -0.0
        clouds.append((x + rng.integers(-3, 3)).astype(dtype))
    radii = np.array([float(dtype(r)) for r in rng.uniform(0.05, 0.1, len(clouds))])
    e = run_batch(ob, clouds, np.array(SIZES[name], np.int64), radii, dtype)
    check_against_oracle(e, clouds, radii, oracle_mod)


@pytest.mark.parametrize("n", [1, 512, 4097])
def test_non_finite_last_point(ob, n):
    clouds = [np.random.default_rng(k).random((n, 3)).astype(np.float32) for k in range(3)]
    clouds[1][-1, 2] = np.nan
    with pytest.raises(Exception):
        run_batch(ob, clouds, np.full(3, n, np.int64), np.full(3, 0.25), np.float32)
