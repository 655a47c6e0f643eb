"""Which sort gsv_bin takes: the lists are the oracle's whichever it is, on either side of every line of the
rule (grids just above the ones that always count, few pairs, many row counts for the pairs, parked rows, a
repeated bin, a capacity above the total), and on grids where the two sorts differ it is not the slow one."""
import ctypes

import numpy as np
import pytest
import torch

from gs_tmi_b200 import _lib, synthetic
from gs_tmi_b200._lib import check, lib
from gs_tmi_b200.tile_voxelizer import _ptr, _shape
from oracle import oracle as O
from tests.test_gpu_binning_modes import _bin, _params, _prepare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n,size", [((128, 128, 96), 300, -1.0), ((128, 136, 96), 300, -1.0), ((128, 136, 96), 2000, 0.0),
                                         ((192, 192, 256), 700, -1.0), ((192, 192, 256), 1500, 0.0),
                                         ((192, 192, 192), 60000, -1.5), ((192, 192, 192), 60000, 0.6),
                                         ((61, 200, 250), 257, 1.6)])
def test_lists(dims, n, size, cuda_device):
    gs = synthetic.random_gaussians(n, dims, seed=5, log_scale_mean_vox=size)
    params = _params(gs, cuda_device)
    for live in (None, n // 3):
        count = n if live is None else live
        plan = _prepare(params, _shape(dims, 8), None if live is None else torch.tensor([live], dtype=torch.int32, device=cuda_device))
        center, radius, _ = O.preprocess_f32(*(t[:count].numpy() for t in gs.tensors()[:3]), dims)
        ranges, ids = O.build_tile_pairs(center, radius, dims, 8)
        for mode, cap in [(_lib.GSV_BIN_AUTO, plan.total), (_lib.GSV_BIN_RADIX, plan.total), (_lib.GSV_BIN_AUTO, 4 * plan.total),
                          (_lib.GSV_BIN_COUNTING, plan.total), (_lib.GSV_BIN_AUTO, plan.total)]:
            got = _bin(plan, mode, cap)
            assert np.array_equal(got[0], ranges) and np.array_equal(got[1], ids) and got[2] == 0


def _time(plan, mode):
    """Least time of a binning in a replayed graph of ten, us."""
    stream = torch.cuda.Stream()

    def once():
        check(lib.gsv_bin_ex(plan.shape, plan.n, _ptr(plan.ws_gauss), _ptr(plan.ws_pairs), plan.pair_bytes, plan.total, mode,
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "gsv_bin_ex")

    with torch.cuda.stream(stream):
        once()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(10):
                once()
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 100)
    return min(times)


@pytest.mark.parametrize("dims,n,size", [((192, 192, 256), 500, -1.0), ((192, 192, 256), 100_000, -1.0),
                                         ((192, 192, 192), 100_000, -1.0), ((192, 192, 256), 30_000, 1.6),
                                         ((144, 128, 96), 30_000, 0.6)])
def test_not_the_slow_one(dims, n, size, cuda_device):
    plan = _prepare(_params(synthetic.random_gaussians(n, dims, seed=5, log_scale_mean_vox=size), cuda_device), _shape(dims, 8))
    plan.alloc_pairs(plan.total)
    both = [_time(plan, mode) for mode in (_lib.GSV_BIN_RADIX, _lib.GSV_BIN_COUNTING)]
    assert _time(plan, _lib.GSV_BIN_AUTO) < 1.25 * min(both)
