"""The deterministic gather takes 4 or 32 Gaussians a warp by their number; a Gaussian's gradients are the same
bits either way: those of a set, and of the same set with more Gaussians behind it."""
import pytest
import torch

import gs_tmi_b200
from gs_tmi_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total", [57343, 57344, 60001])
def test_gradients_do_not_depend_on_the_warp_share(total, cuda_device):
    shape, n = (48, 40, 44), 3001
    sets = [synthetic.random_gaussians(n, shape, seed=5).tensors(),
            synthetic.random_gaussians(total - n, shape, seed=7).tensors()]
    gv = synthetic.upstream_grad(shape, seed=6).to(cuda_device)
    grads = []
    for parts in (sets[:1], sets):
        ps = [torch.cat(x).to(cuda_device).requires_grad_(True) for x in zip(*parts)]
        vol = gs_tmi_b200.voxelize(*ps, shape, 8, deterministic=True)
        grads.append(torch.autograd.grad(vol, ps, gv))
    for a, b in zip(*grads):
        assert torch.equal(a, b[:n])
