"""The block walks of the tile-8 and tile-4 kernels where their bookkeeping can go wrong: list lengths
around a warp, a staged chunk and a full queue in one tile, ragged volumes, infinite and NaN densities
and gradients, and the counting sort's rows.  Against the FP64 oracle, with the
suite's tolerances."""
import numpy as np
import pytest
import torch

import gs_tmi_b200
from gs_tmi_b200 import synthetic
from oracle import oracle as O
from tests.helpers import FWD_TOL, GRAD_TOL, rel

pytestmark = pytest.mark.gpu


def _dense(n, shape, seed):
    """n Gaussians of 1 to 2 voxels inside the volume's first tile."""
    g = torch.Generator().manual_seed(seed)
    half = torch.tensor([0.5 * s for s in shape])
    pos = (torch.rand(n, 3, generator=g) * 7 + 0.5) / half - 1
    scl = (1 + torch.rand(n, 3, generator=g)) / half
    return synthetic.GaussianSet(pos, scl, torch.randn(n, 4, generator=g), 0.1 * torch.randn(n, generator=g),
                                 0.1 * torch.randn(n, generator=g))


def _run(gs, shape, ts, gv, dev, deterministic):
    ps = [t.to(dev).requires_grad_(True) for t in gs.tensors()]
    vol = gs_tmi_b200.voxelize(*ps, shape, ts, deterministic=deterministic)
    grads = torch.autograd.grad(vol, ps, gv.to(dev))
    return vol.detach().cpu().numpy(), [t.cpu().numpy() for t in grads]


def _oracle(gs, shape, ts, gv):
    p = tuple(t.numpy() for t in gs.tensors())
    c, r, _ = O.preprocess_f32(*p[:3], shape)
    tr, pid = O.build_tile_pairs(c, r, shape, ts)
    return O.forward(p, shape, ts, tr, pid)[0], O.backward(p, shape, ts, tr, pid, gv.numpy())


@pytest.mark.parametrize("ts", [8, 4])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 32, 33, 64, 65, 127, 129, 255, 257, 511, 513, 1025])
def test_list_lengths(n, ts, cuda_device):
    shape = (11, 9, 13)
    gs, gv = _dense(n, shape, n), synthetic.upstream_grad(shape, seed=n)
    ovol, og = _oracle(gs, shape, ts, gv)
    for det in (False, True):
        vol, grads = _run(gs, shape, ts, gv, cuda_device, det)
        assert rel(vol, ovol) < FWD_TOL
        for a, b in zip(grads, og):
            assert rel(a, b) < GRAD_TOL


@pytest.mark.parametrize("ts", [8, 4])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e30])
def test_one_wild_density_or_gradient_stays_where_it_is(value, ts, cuda_device):
    """A density or an upstream gradient that is infinite, NaN or huge reaches exactly the voxels and the
    Gaussians that include it; every other value is the one without it."""
    shape = (24, 20, 18)
    gs, gv = synthetic.random_gaussians(400, shape, seed=8), synthetic.upstream_grad(shape, seed=9)
    vol, grads = _run(gs, shape, ts, gv, cuda_device, True)
    one = synthetic.GaussianSet(*(t[57:58] for t in gs.tensors()))
    one.density_r.fill_(1.0)
    touched = _run(one, shape, ts, gv, cuda_device, True)[0] != 0
    wild = synthetic.GaussianSet(*(t.clone() for t in gs.tensors()))
    wild.density_r[57] = value
    v2, g2 = _run(wild, shape, ts, gv, cuda_device, True)
    assert touched.any() and not touched.all()
    assert np.array_equal(v2[~touched], vol[~touched])
    assert not np.isclose(v2[touched].real, vol[touched].real).any()
    rest = np.arange(400) != 57
    for a, b in zip(g2, grads):
        assert rel(a[rest], b[rest]) < 1e-6 and np.isfinite(a[rest]).all()
    # the gradient of one voxel
    at = np.unravel_index(np.argmax(touched), shape)
    gw = gv.clone()
    gw[at] = complex(value, 0.0)
    _, g3 = _run(gs, shape, ts, gw, cuda_device, True)
    lone = torch.zeros(shape, dtype=torch.complex64)
    lone[at] = 1.0
    hit = _run(gs, shape, ts, lone, cuda_device, True)[1][3] != 0
    assert hit[57] and not hit.all()
    for a, b in zip(g3, grads):
        assert rel(a[~hit], b[~hit]) < 1e-6
    assert not np.isclose(g3[3][hit], grads[3][hit]).any()


@pytest.mark.parametrize("shape,ts,n", [((128, 128, 96), 8, 300_000), ((256, 256, 144), 8, 2_000), ((256, 256, 144), 8, 100_000),
                                        ((50, 61, 47), 4, 9_001), ((64, 64, 64), 4, 400_000), ((64, 64, 64), 8, 257),
                                        ((160, 160, 152), 8, 511)])
def test_counting_sort_rows(shape, ts, n, cuda_device):
    """Rows of 64 and of 256 Gaussians, their last ones cut anywhere, up to the largest tile count and the
    largest number of row counts: the lists of the radix sort."""
    from tests.test_gpu_binning_modes import _params, _prepare, _same_lists

    from gs_tmi_b200.tile_voxelizer import _shape

    gs = synthetic.random_gaussians(n, shape, seed=2, log_scale_mean_vox=-0.5 if n > 10_000 else 0.6)
    _same_lists(_prepare(_params(gs, cuda_device), _shape(shape, ts)))


@pytest.mark.parametrize("ts", [8, 4, 5])
def test_deterministic_backward_over_capacity_stays_in_its_buffers(ts, cuda_device):
    """A static deterministic plan whose capacity is half the pairs: the overflow is flagged, and the
    marks and partials of pairs past the capacity are dropped (guard bytes behind the pair workspace
    stay as they were)."""
    import ctypes

    from gs_tmi_b200 import _lib
    from gs_tmi_b200._lib import GsvGrads, GsvParams, check, lib
    from gs_tmi_b200.tile_voxelizer import StaticPlan, TileVoxelizer, _ptr, _shape, _stream

    shape = (40, 40, 40)
    gs = synthetic.random_gaussians(3000, shape, seed=3)
    ps = [t.to(cuda_device) for t in gs.tensors()]
    total = TileVoxelizer(shape, ts).count_pairs(ps[0], ps[1])
    plan = StaticPlan(_shape(shape, ts), 3000, cuda_device, total // 2, flags=_lib.GSV_BACKWARD_DETERMINISTIC)
    guarded = torch.full((plan.pair_bytes + (1 << 22),), 77, dtype=torch.uint8, device=cuda_device)
    plan.ws_pairs = guarded
    gv = synthetic.upstream_grad(shape, seed=4).to(cuda_device)
    outs = [torch.empty_like(t) for t in ps]
    gp, gg, st = GsvParams(*(t.data_ptr() for t in ps), 3000), GsvGrads(*(o.data_ptr() for o in outs)), _stream(cuda_device)
    check(lib.gsv_prepare(ctypes.byref(gp), plan.shape, _ptr(plan.ws_gauss), plan.gauss_bytes, None, st), "prepare")
    check(lib.gsv_bin(plan.shape, 3000, _ptr(plan.ws_gauss), _ptr(guarded), plan.pair_bytes, plan.capacity, st), "bin")
    check(lib.gsv_backward(ctypes.byref(gp), plan.shape, _ptr(plan.ws_gauss), _ptr(guarded), plan.capacity, _ptr(gv),
                           ctypes.byref(gg), plan.flags, st), "backward")
    assert plan.read_status(st)[1] & _lib.GSV_FLAG_CAPACITY_OVERFLOW
    assert all(torch.isfinite(o).all() for o in outs)
    assert (guarded[plan.pair_bytes:] == 77).all()
