"""Host threads that bin grids of different sizes at the same time, each on a stream of its own: every
launch is accepted and every list is the one a lone thread gets."""
import threading

import pytest
import torch

from gs_tmi_b200 import _lib, synthetic
from gs_tmi_b200._lib import lib
from gs_tmi_b200.tile_voxelizer import _ptr, _shape
from tests.test_gpu_binning_modes import _bin, _params, _prepare

pytestmark = pytest.mark.gpu


def _lists(plan):
    tiles = int(lib.gsv_num_tiles(plan.shape))
    tr, ids = plan.views()
    tr, ids = tr - plan.ws_gauss.data_ptr(), ids - plan.ws_pairs.data_ptr()
    return (plan.ws_gauss[tr:tr + 8 * tiles].view(torch.int32).reshape(tiles, 2).cpu().numpy(),
            plan.ws_pairs[ids:ids + 4 * plan.total].view(torch.int32).cpu().numpy())


def test_threads_with_different_grids(cuda_device):
    work = []
    for i in range(8):
        dims = [(192, 192, 256), (160, 160, 152)][i % 2]  # 18432 and 7600 tiles
        params = _params(synthetic.random_gaussians(50, dims, seed=i, log_scale_mean_vox=0.5), cuda_device)
        plan = _prepare(params, _shape(dims, 8))
        work.append((plan, params, _bin(plan, _lib.GSV_BIN_COUNTING, plan.total)))
    torch.cuda.synchronize()
    codes, start = [set() for _ in work], threading.Barrier(len(work))

    def loop(i):
        plan = work[i][0]
        with torch.cuda.device(cuda_device):
            stream = torch.cuda.Stream()
            args = (plan.shape, plan.n, _ptr(plan.ws_gauss), _ptr(plan.ws_pairs), plan.pair_bytes, plan.total,
                    _lib.GSV_BIN_COUNTING, stream.cuda_stream)
            start.wait()
            for k in range(3000):
                codes[i].add(lib.gsv_bin_ex(*args))
                if k % 200 == 199:
                    stream.synchronize()
            stream.synchronize()

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [{0}] * len(work)
    for plan, _, want in work:
        for a, b in zip(_lists(plan), want):
            assert (a == b).all()
