"""The reference-signature backward with Gaussians whose inverse covariance is NaN or infinite: they
include no voxel, so all their gradients are exactly zero and nobody else's change.  Tile edges of
every kernel (8, 4 and the generic one)."""
import numpy as np
import pytest
import torch

import gs_tmi_b200
from gs_tmi_b200 import synthetic
from oracle import oracle as O
from tests.helpers import rel
from tests.test_gpu_parity import _cov_inv_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts", [8, 4, 5])
def test_gaussian_without_a_voxel_has_zero_gradient(ts, cuda_device):
    shape, n = (21, 18, 19), 300
    gs, gv = synthetic.random_gaussians(n, shape, seed=ts), synthetic.upstream_grad(shape, seed=1)
    center, radius, _ = O.preprocess_f32(*(t.numpy() for t in gs.tensors()[:3]), shape)
    lists = [torch.tensor(x, device=cuda_device) for x in O.build_tile_pairs(center, radius, shape, ts)]
    half = torch.tensor([0.5 * s for s in shape], device=cuda_device)
    cov = _cov_inv_f32(gs.scales, gs.rotations)
    bad = cov.clone()
    bad[57, 0, 1] = float("nan")
    bad[91] = torch.diag(torch.full((3,), float("inf")))
    bad[92] = float("nan")

    def grads(m):
        ps = [t.to(cuda_device).requires_grad_(True)
              for t in (torch.tensor(center), m, gs.density_r.clone(), gs.density_i.clone())]
        vol = gs_tmi_b200._TileVoxelizeCUDA.apply(*ps, *lists, half, ts, *shape)
        up = gv.reshape(-1).to(cuda_device)
        return [g.cpu().numpy() for g in torch.autograd.grad(vol, ps, (up.real.contiguous(), up.imag.contiguous()))]

    want, got = grads(cov), grads(bad)
    gone = np.isin(np.arange(n), [57, 91, 92])
    for a, b in zip(got, want):
        assert (a[gone] == 0).all()
        assert rel(a[~gone], b[~gone]) < 1e-5  # the order of the atomics
