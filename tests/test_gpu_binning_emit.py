"""The radix path's emission and range pass against the oracle's lists, bit for
bit: pair counts around the range pass's four keys a thread and 128 a warp,
Gaussians without pairs, a box that is the whole grid, and a grid of more than
four million tiles (where pair indices outgrow single precision)."""
import ctypes

import numpy as np
import pytest
import torch

from gs_tmi_b200 import _lib
from gs_tmi_b200._lib import GsvParams, check, lib
from gs_tmi_b200.tile_voxelizer import BinPlan, _ptr, _shape, _stream
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,tile,n,wide,cut", [
    ((64, 64, 64), 8, 1, 0, 0), ((64, 64, 64), 8, 2, 0, 1), ((64, 64, 64), 8, 33, 1, 0), ((61, 50, 47), 5, 300, 2, 5),
    ((128, 96, 130), 4, 3000, 1, 0), ((96, 96, 96), 3, 5000, 0, 1000), ((330, 322, 324), 2, 40, 1, 0)])
def test_radix_lists(dims, tile, n, wide, cut, cuda_device):
    g = torch.Generator().manual_seed(n)
    pos = torch.rand(n, 3, generator=g) * 2.2 - 1.1  # some outside: no pairs, or clamped boxes
    scl = torch.rand(n, 3, generator=g) * 0.02 + 0.002
    scl[n // 2:n // 2 + wide] = 3.0
    rot = torch.randn(n, 4, generator=g)
    den = torch.randn(2, n, generator=g)
    center, radius = O.preprocess_f32(pos.numpy(), scl.numpy(), rot.numpy(), dims)[:2]
    want_ranges, want_ids = O.build_tile_pairs(center, radius, dims, tile)[:2]

    dev = [t.to(cuda_device).contiguous() for t in (pos, scl, rot, den[0], den[1])]
    plan = BinPlan(_shape(dims, tile), n, torch.device(cuda_device))
    gp = GsvParams(*(t.data_ptr() for t in dev), n)
    total = ctypes.c_int64(0)
    check(lib.gsv_prepare(ctypes.byref(gp), plan.shape, _ptr(plan.ws_gauss), plan.gauss_bytes, ctypes.byref(total),
                          _stream(plan.device)), "gsv_prepare")
    assert total.value == len(want_ids)
    cap = max(int(total.value) + 7 - cut, 1)
    plan.alloc_pairs(cap)
    check(lib.gsv_bin_ex(plan.shape, n, _ptr(plan.ws_gauss), _ptr(plan.ws_pairs), plan.pair_bytes, cap,
                         _lib.GSV_BIN_RADIX, _stream(plan.device)), "gsv_bin_ex")
    _, flags = plan.read_status(_stream(plan.device))
    assert bool(flags & _lib.GSV_FLAG_CAPACITY_OVERFLOW) == (cap < total.value)
    tiles = int(lib.gsv_num_tiles(plan.shape))
    tr, pid = plan.views()
    tr, pid = tr - plan.ws_gauss.data_ptr(), pid - plan.ws_pairs.data_ptr()
    ranges = plan.ws_gauss[tr:tr + 8 * tiles].view(torch.int32).reshape(tiles, 2).cpu().numpy()
    k = min(int(total.value), cap)
    ids = plan.ws_pairs[pid:pid + 4 * k].view(torch.int32).cpu().numpy()
    if cap >= total.value:
        assert np.array_equal(ranges, want_ranges) and np.array_equal(ids, want_ids)
        return
    # the first `cap` pairs in Gaussian order are kept, and their lists are whole
    assert ranges[:, 1].max() == cap and (ranges[:, 1] - ranges[:, 0]).sum() == cap
    for t in np.flatnonzero(ranges[:, 1]):
        a, b = ranges[t]
        wa = want_ranges[t, 0]
        assert np.array_equal(ids[a:b], want_ids[wa:wa + (b - a)])
