"""The counting sort against the oracle's lists, bit for bit, where its row length
and its lanes per Gaussian change: rows of 64 and of 256 on either side of as
many rows as tiles, rows whose mean is a few pairs, some twenty and many, and a
last row with few Gaussians."""
import ctypes

import numpy as np
import pytest
import torch

from gs_tmi_b200 import _lib
from gs_tmi_b200._lib import GsvParams, check, lib
from gs_tmi_b200.tile_voxelizer import BinPlan, _ptr, _shape, _stream
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.004, 0.05, 0.13])
@pytest.mark.parametrize("dims,n", [((64, 64, 64), 8191), ((64, 64, 64), 32511), ((64, 64, 64), 32512),
                                    ((9, 7, 5), 300), ((200, 72, 90), 65)])
def test_rows_and_lanes(dims, n, scale, cuda_device):
    g = torch.Generator().manual_seed(n)
    pos = torch.rand(n, 3, generator=g) * 2 - 1
    scl = torch.full((n, 3), scale)
    scl[n // 3:n // 3 + 70] = 0.3  # a stretch of wide ones: one row's mean differs from the others'
    rot, den = torch.randn(n, 4, generator=g), torch.randn(2, n, generator=g)
    center, radius = O.preprocess_f32(pos.numpy(), scl.numpy(), rot.numpy(), dims)[:2]
    want_ranges, want_ids = O.build_tile_pairs(center, radius, dims, 8)

    dev = [t.to(cuda_device).contiguous() for t in (pos, scl, rot, den[0], den[1])]
    plan = BinPlan(_shape(dims, 8), n, torch.device(cuda_device))
    gp = GsvParams(*(t.data_ptr() for t in dev), n)
    total = ctypes.c_int64(0)
    check(lib.gsv_prepare(ctypes.byref(gp), plan.shape, _ptr(plan.ws_gauss), plan.gauss_bytes, ctypes.byref(total),
                          _stream(plan.device)), "gsv_prepare")
    cap = int(total.value)
    plan.alloc_pairs(cap)
    check(lib.gsv_bin_ex(plan.shape, n, _ptr(plan.ws_gauss), _ptr(plan.ws_pairs), plan.pair_bytes, cap,
                         _lib.GSV_BIN_COUNTING, _stream(plan.device)), "gsv_bin_ex")
    torch.cuda.synchronize()
    tiles = int(lib.gsv_num_tiles(plan.shape))
    tr, pid = plan.views()
    tr, pid = tr - plan.ws_gauss.data_ptr(), pid - plan.ws_pairs.data_ptr()
    ranges = plan.ws_gauss[tr:tr + 8 * tiles].view(torch.int32).reshape(tiles, 2).cpu().numpy()
    ids = plan.ws_pairs[pid:pid + 4 * cap].view(torch.int32).cpu().numpy()
    assert np.array_equal(ranges, want_ranges) and np.array_equal(ids, want_ids)
