"""The separating-plane cull on an axis of more than 2^23 voxels, which the reference-signature kernels take
with a caller's own lists: a block's centre (first voxel + 1.5) is no FP32 number there.  Centres and
coefficients are chosen so that the block's first voxel, and no other, is inside the cutoff
(m = 8.95), while half a voxel more would have ruled the block out."""
import math

import pytest
import torch

import gs_tmi_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts", [8, 4])
def test_included_voxel_past_2_to_the_23(ts, cuda_device):
    w0 = 1 << 23
    shape, r = (1, 1, w0 + 8), 10.0
    q = 8.95 / (2 * 1.5 ** 2 + r ** 2)
    f = lambda x: torch.tensor(x, dtype=torch.float32, device=cuda_device)
    ps = [f([[1.5, 1.5, w0 - r]]), f([[[q, 0, 0], [0, q, 0], [0, 0, q]]]), f([2.0]), f([-3.0])]
    ps = [p.requires_grad_(True) for p in ps]
    ranges = torch.zeros((shape[2] // ts, 2), dtype=torch.int32, device=cuda_device)
    ranges[w0 // ts, 1] = 1
    ids = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    vr, vi = gs_tmi_b200._TileVoxelizeCUDA.apply(*ps, ranges, ids, f([1.0, 1.0, 1.0]), ts, *shape)
    up = torch.zeros_like(vr)
    up[w0] = 1.0
    grads = torch.autograd.grad((vr, vi), ps, (up, torch.zeros_like(up)))
    weight = math.exp(-8.95 / 2)
    assert vr[w0].item() == pytest.approx(2 * weight, rel=1e-5) and vi[w0].item() == pytest.approx(-3 * weight, rel=1e-5)
    assert vr.count_nonzero() == 1
    assert grads[2].item() == pytest.approx(weight, rel=1e-5)
    # dL/dcenter = rho w Q e, e the voxel's offset from the centre
    assert grads[0][0].tolist() == pytest.approx([2 * weight * q * e for e in (-1.5, -1.5, r)], rel=1e-5)
