"""The radii of a batch, one per cloud: the shapes that are taken and refused,
and their rounding to the element type."""
import numpy as np
import pytest
import torch


@pytest.mark.parametrize("radii", [[0.1, 0.2, 0.3], np.array([[0.1], [0.2], [0.3]]), (0.1, 0.2, 0.3)])
@pytest.mark.parametrize("T", [torch.float32, torch.float64])
def test_one_radius_per_cloud(ob, T, radii):
    got = ob.api._cloud_radii(radii, 3, T)
    want = [float(torch.tensor(r, dtype=T).item()) for r in (0.1, 0.2, 0.3)]
    assert got.shape == (3,) and got.flags.c_contiguous and got.tolist() == want


def test_out_of_range_rounds_as_torch_does(ob):
    r = [1e300, 1e-50, 3.5e38, 1.0 + 2.0 ** -24]
    assert ob.api._cloud_radii(r, 4, torch.float32).tolist() == [torch.tensor(v, dtype=torch.float32).item() for v in r]


@pytest.mark.parametrize("radii,error", [
    (np.full((3, 2), 0.1), TypeError), (np.empty((3, 0)), TypeError), (np.full((3, 1, 2), 0.1), TypeError),
    ([0.1, 0.2], "DimensionMismatch"), ([], "DimensionMismatch")])
def test_refused_shapes(ob, radii, error):
    with pytest.raises(getattr(ob, error) if isinstance(error, str) else error):
        ob.api._cloud_radii(radii, 3, torch.float32)
