"""Flat and needle-shaped Gaussians: the cull still leaves out most of the blocks they do not reach, for the
native path (counted) and the reference-signature one (its kernels take less than twice the native
kernels' time; without its own cull four times), and both agree with the FP64 oracle."""
import ctypes

import numpy as np
import pytest
import torch

import gs_tmi_b200
from gs_tmi_b200 import synthetic
from gs_tmi_b200._lib import GsvGrads, GsvParams, check, lib
from gs_tmi_b200.tile_voxelizer import _ptr, _shape, prepare_and_bin, work_census
from oracle import oracle as O
from tests.helpers import rel
from tests.test_gpu_parity import _cov_inv_f32

pytestmark = pytest.mark.gpu

FORMS = {"pancake": (0.4, 6.0, 6.0), "needle": (0.3, 0.3, 10.0), "thin": (0.2, 6.0, 6.0)}


def _set(form, n, shape, dev, seed=0):
    g = torch.Generator().manual_seed(seed)
    half = torch.tensor([0.5 * s for s in shape])
    gs = synthetic.GaussianSet(torch.rand(n, 3, generator=g) * 2 - 1, (torch.tensor(FORMS[form]) / half).repeat(n, 1),
                               torch.randn(n, 4, generator=g), 0.1 * torch.randn(n, generator=g), 0.1 * torch.randn(n, generator=g))
    return gs, tuple(t.to(dev).contiguous() for t in gs.tensors())


def _compat_inputs(gs, shape, ts, dev):
    center, radius, _ = O.preprocess_f32(*(t.numpy() for t in gs.tensors()[:3]), shape)
    lists = [torch.tensor(x, device=dev) for x in O.build_tile_pairs(center, radius, shape, ts)]
    cov = _cov_inv_f32(gs.scales, gs.rotations).reshape(-1, 9).contiguous()
    half = torch.tensor([0.5 * s for s in shape], device=dev)
    return torch.tensor(center, device=dev), cov.to(dev), lists, half


@pytest.mark.parametrize("form", list(FORMS))
def test_kept_blocks(form, cuda_device):
    shape = (64, 60, 68)
    _, ps = _set(form, 3000, shape, cuda_device)
    plan = prepare_and_bin(ps, _shape(shape, 8))
    on, off = work_census(plan), work_census(plan, cull=False)
    assert on["included"] == off["included"] > 0
    assert on["empty_kept_slots"] < on["evaluated"] / 64 / 3  # of the kept blocks, two thirds hold an included voxel


@pytest.mark.parametrize("ts", [8, 4])
@pytest.mark.parametrize("form", list(FORMS))
def test_reference_signature_agrees(form, ts, cuda_device):
    shape, n = (21, 30, 26), 400
    gs, _ = _set(form, n, shape, cuda_device, seed=1)
    center, cov, lists, half = _compat_inputs(gs, shape, ts, cuda_device)
    gv = synthetic.upstream_grad(shape, seed=2)
    ps = [t.requires_grad_(True) for t in (center, cov.reshape(-1, 3, 3), gs.density_r.to(cuda_device), gs.density_i.to(cuda_device))]
    vr, vi = gs_tmi_b200._TileVoxelizeCUDA.apply(*ps, *lists, half, ts, *shape)
    up = gv.reshape(-1).to(cuda_device)
    grads = torch.autograd.grad((vr, vi), ps, (up.real.contiguous(), up.imag.contiguous()))
    tr, pid = (t.cpu().numpy() for t in lists)
    cp = (center.detach().cpu().numpy(), cov.cpu().numpy(), None, gs.density_r.numpy(), gs.density_i.numpy())
    hs = half.cpu().numpy()
    ovol, _ = O.forward(cp, shape, ts, tr, pid, compat=True, half_shape=hs)
    assert rel((vr + 1j * vi).detach().cpu().numpy().reshape(shape), ovol) < 1e-5
    og = O.backward(cp, shape, ts, tr, pid, gv.numpy(), compat=True, half_shape=hs)
    for a, b in zip(grads, (og[0], og[1], og[3], og[4])):
        assert rel(a.cpu().numpy().reshape(b.shape), b) < 1e-4


def _best(fn, reps=8):
    times = []
    for _ in range(reps + 2):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times[2:])


def test_reference_signature_needles_are_culled(cuda_device):
    shape, n = (100, 84, 60), 20_000
    gs, native = _set("needle", n, shape, cuda_device)
    center, cov, (tr, pid), half = _compat_inputs(gs, shape, 8, cuda_device)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    voxels = shape[0] * shape[1] * shape[2]
    vr, vi, gr, gi = (torch.randn(voxels, device=cuda_device) for _ in range(4))
    outs = [torch.empty_like(t) for t in (center, cov, native[3], native[4])]
    args = (_ptr(center), _ptr(cov), _ptr(native[3]), _ptr(native[4]), _ptr(tr), _ptr(pid), _ptr(half))

    def compat():
        check(lib.gsv_tile_forward(*args, n, int(tr.shape[0]), 8, *shape, _ptr(vr), _ptr(vi), st), "forward")
        check(lib.gsv_tile_backward(*args, _ptr(gr), _ptr(gi), n, int(tr.shape[0]), 8, *shape, *(_ptr(o) for o in outs), st),
              "backward")

    plan = prepare_and_bin(native, _shape(shape, 8))
    vol = torch.randn(shape, device=cuda_device, dtype=torch.complex64)
    gp = GsvParams(*(t.data_ptr() for t in native), n)
    nouts = [torch.empty_like(t) for t in native]
    gg = GsvGrads(*(o.data_ptr() for o in nouts))
    out = torch.empty_like(vol)

    def fused():
        check(lib.gsv_forward(plan.shape, n, _ptr(plan.ws_gauss), _ptr(plan.ws_pairs), plan.capacity, _ptr(out), st), "forward")
        check(lib.gsv_backward(ctypes.byref(gp), plan.shape, _ptr(plan.ws_gauss), _ptr(plan.ws_pairs), plan.capacity,
                               _ptr(vol), ctypes.byref(gg), plan.flags, st), "backward")

    assert _best(compat) < 2 * _best(fused)
