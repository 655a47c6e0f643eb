"""The SENSE and TV kernels at the forms their dispatch tells apart: rows of one and of two voxels per
thread (row length a multiple of four, aligned arrays), coil counts around the unrolled four, ragged
volumes.  Against torch in 64 bits; the bar is the rounding of a sum of
nc terms (data term) or of a quotient (TV)."""
import pytest
import torch

from gs_tmi_b200 import sense, synthetic

pytestmark = pytest.mark.gpu


def _crand(shape, g, dev):
    return torch.complex(torch.randn(shape, generator=g), torch.randn(shape, generator=g)).to(dev)


@pytest.mark.parametrize("shape", [(8, 8, 8), (5, 7, 12), (6, 5, 10), (9, 8, 7), (1, 1, 4), (2, 3, 1), (17, 9, 36)])
@pytest.mark.parametrize("nc", [1, 3, 4, 5, 9])
@pytest.mark.parametrize("offset", [0, 1])
def test_data_term_forms(shape, nc, offset, cuda_device):
    """offset 1: the coil maps start 8 bytes past a 16-byte boundary."""
    g = torch.Generator().manual_seed(nc)
    vol = _crand(shape, g, cuda_device)
    S = _crand((nc, *shape), g, cuda_device)
    flat = torch.empty(S.numel() + 2, dtype=torch.complex64, device=cuda_device)
    S = flat[offset:offset + S.numel()].view_as(S).copy_(S)
    mask = (torch.rand(shape, generator=g) < 0.5).float().to(cuda_device)
    ku = _crand((nc, *shape), g, cuda_device)
    v1 = vol.clone().requires_grad_(True)
    l1 = sense.sense_data_term(v1, S, mask, ku)
    g1, = torch.autograd.grad(3.0 * l1, v1)
    v2 = vol.to(torch.complex128).requires_grad_(True)
    diff = synthetic.fft3c(v2.unsqueeze(0) * S.to(torch.complex128)) * mask.double() - ku.to(torch.complex128)
    l2 = diff.real.square().sum() + diff.imag.square().sum()
    g2, = torch.autograd.grad(3.0 * l2, v2)
    assert abs(float(l1.detach()) - float(l2.detach())) <= 1e-5 * float(l2.detach())
    assert float((g1 - g2).abs().norm()) <= 1e-5 * float(g2.abs().norm())


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 5), (8, 8, 32), (9, 9, 33), (17, 7, 31), (16, 24, 70), (2, 65, 64)])
def test_tv_forms(shape, cuda_device):
    g = torch.Generator().manual_seed(sum(shape))
    vol = _crand(shape, g, cuda_device)
    vol[0, 0, 0] = 0.0
    v1 = vol.clone().requires_grad_(True)
    l1 = sense.magnitude_tv_fused(v1)
    g1, = torch.autograd.grad(l1, v1)
    v2 = vol.to(torch.complex128).requires_grad_(True)
    m = v2.abs()
    l2 = sum(torch.diff(m, dim=a).abs().sum() for a in range(3))
    g2, = torch.autograd.grad(l2, v2)
    assert abs(float(l1.detach()) - float(l2.detach())) <= 1e-5 * max(float(l2.detach()), 1e-30)
    assert float((g1 - g2).abs().norm()) <= 1e-5 * max(float(g2.abs().norm()), 1e-30)
