"""A complex density goes to the library whole (interleaved, read and written two floats apart): the same
volume and gradients, bit for bit in the deterministic mode, as its parts passed as two arrays, in every
form a caller may hold it."""
import pytest
import torch

import gs_tmi_b200
from gs_tmi_b200 import synthetic

pytestmark = pytest.mark.gpu

SHAPE = (24, 20, 18)


def _parts(dev, n=700):
    gs = synthetic.random_gaussians(n, SHAPE, seed=n)
    return [t.to(dev) for t in gs.tensors()], synthetic.upstream_grad(SHAPE, seed=n + 1).to(dev)


def _reference(ps, gv):
    leaves = [t.clone().requires_grad_(True) for t in ps]
    vol = gs_tmi_b200.voxelize(*leaves, SHAPE, 8, deterministic=True)
    return vol.detach(), torch.autograd.grad(vol, leaves, gv)


FORMS = {
    "plain": lambda r, i: torch.complex(r, i),
    "complex128": lambda r, i: torch.complex(r, i).to(torch.complex128),
    "strided": lambda r, i: torch.stack([torch.complex(r, i)] * 3, 1)[:, 1],
    "conjugated": lambda r, i: torch.complex(r, -i).conj(),
    "one_column": lambda r, i: torch.complex(r, i)[:, None],
}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("static", [False, True])
def test_complex_density_forms(form, static, cuda_device):
    ps, gv = _parts(cuda_device)
    vol0, g0 = _reference(ps, gv)
    geo = [t.clone().requires_grad_(True) for t in ps[:3]]
    den = FORMS[form](ps[3], ps[4]).detach().requires_grad_(True)
    vox = gs_tmi_b200.TileVoxelizer(SHAPE, deterministic=True, device=str(cuda_device))
    if static:
        vox = vox.static(ps[0].shape[0], vox.count_pairs(ps[0], ps[1]))
    vol = vox(*geo, den)
    grads = torch.autograd.grad(vol, [*geo, den], gv)
    assert torch.equal(vol.detach(), vol0)
    for a, b in zip(grads[:3], g0[:3]):
        assert torch.equal(a, b)
    assert grads[3].shape == den.shape and grads[3].dtype == den.dtype
    d = grads[3].reshape(-1).to(torch.complex64)
    assert torch.equal(d.real, g0[3]) and torch.equal(d.imag, g0[4])


def test_real_and_empty_densities(cuda_device):
    ps, gv = _parts(cuda_device, 300)
    vox = gs_tmi_b200.TileVoxelizer(SHAPE, deterministic=True, device=str(cuda_device))
    zero = [*ps[:4], torch.zeros_like(ps[4])]
    vol0, g0 = _reference(zero, gv)
    leaves = [t.clone().requires_grad_(True) for t in ps[:4]]
    vol = vox(*leaves)
    assert torch.equal(vol.detach(), vol0)
    for a, b in zip(torch.autograd.grad(vol, leaves, gv), g0):
        assert torch.equal(a, b)
    none = [t[:0] for t in ps[:3]] + [torch.complex(ps[3], ps[4])[:0].requires_grad_(True)]
    vol = vox(*none)
    assert not vol.any()
    assert torch.autograd.grad(vol, none[3], gv)[0].shape == (0,)


def test_density_may_change_before_the_backward(cuda_device):
    """The densities' values of the forward count: a later change of the tensor changes no gradient."""
    ps, gv = _parts(cuda_device, 300)
    _, g0 = _reference(ps, gv)
    pos = ps[0].clone().requires_grad_(True)
    den = torch.complex(ps[3], ps[4])
    vol = gs_tmi_b200.TileVoxelizer(SHAPE, deterministic=True, device=str(cuda_device))(pos, ps[1], ps[2], den)
    den.mul_(3.0)
    assert torch.equal(torch.autograd.grad(vol, pos, gv)[0], g0[0])
