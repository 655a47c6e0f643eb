"""voxelize takes the density as two arrays: a call without the second is an error, whatever the first one is
(a complex density taken whole is TileVoxelizer's form)."""
import pytest
import torch

import gs_tmi_b200
from gs_tmi_b200 import synthetic


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64])
def test_density_i_is_required(dtype):
    pos, scl, rot, dr, _ = synthetic.random_gaussians(10, (16, 16, 16)).tensors()
    with pytest.raises((TypeError, AttributeError)):
        gs_tmi_b200.voxelize(pos, scl, rot, dr.to(dtype), None, (16, 16, 16))
