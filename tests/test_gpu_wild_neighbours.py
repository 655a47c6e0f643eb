"""One Gaussian with an infinite, NaN or huge density takes the guarded loop of the backward; the other
Gaussians' deterministic gradients keep every bit, whichever of them are evaluated beside it: with the cull
on and off, other chunks and more CTAs per list."""
import numpy as np
import pytest
import torch

from gs_tmi_b200 import synthetic
from gs_tmi_b200._lib import GSV_BACKWARD_DETERMINISTIC, GSV_TUNE_NO_CULL, GsvTuning
from gs_tmi_b200.tile_voxelizer import _shape, prepare_and_bin
from tests.test_gpu_autotune import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts", [8, 4])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e30])
def test_neighbours_keep_their_bits(value, ts, cuda_device):
    shape, n, at = (24, 20, 18), 400, 57
    gs, gv = synthetic.random_gaussians(n, shape, seed=8), synthetic.upstream_grad(shape, seed=9).to(cuda_device)

    def grads(tune):
        params = tuple(t.to(cuda_device) for t in gs.tensors())
        plan = prepare_and_bin(params, _shape(shape, ts), flags=GSV_BACKWARD_DETERMINISTIC)
        return _run(plan, params, gv, GsvTuning(*tune))[1]

    want = grads((2, 32, 0, 1))
    gs.density_r[at] = value
    rest = np.arange(n) != at
    for tune in [(2, 32, 0, 1), (2, 32, GSV_TUNE_NO_CULL, 1), (2, 7, 0, 1), (2, 32, 0, 4)]:
        for a, b in zip(grads(tune), want):
            assert np.array_equal(a[rest].view(np.int32), b[rest].view(np.int32))
