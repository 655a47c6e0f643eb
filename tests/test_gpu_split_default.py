"""gsv_tuning.split = 0 means one CTA per (half) tile in the backward, as it always has; only a call without a
gsv_tuning leaves the number to the library.  Read from the launched grid."""
import ctypes
import json

import pytest
import torch

from gs_tmi_b200 import synthetic
from gs_tmi_b200._lib import GsvGrads, GsvParams, GsvTuning, check, lib
from gs_tmi_b200.tile_voxelizer import _ptr, _shape, prepare_and_bin

pytestmark = pytest.mark.gpu


def _grids(run, kernel, path):
    """Grid sizes of the launches of `kernel` in run()."""
    run()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    events = json.loads(path.read_text())["traceEvents"]
    return [e["args"]["grid"][0] for e in events if e.get("cat") == "kernel" and kernel in e["name"]]


@pytest.mark.parametrize("tuning,ctas", [(None, 2), (GsvTuning(2, 32, 0, 0), 1), (GsvTuning(2, 32, 0, 1), 1),
                                         (GsvTuning(2, 32, 0, 4), 4)])
def test_ctas_per_tile(tuning, ctas, tmp_path, cuda_device):
    shape = (32, 32, 32)
    ps = tuple(t.to(cuda_device) for t in synthetic.random_gaussians(500, shape, seed=3).tensors())
    plan = prepare_and_bin(ps, _shape(shape, 8))
    gv = synthetic.upstream_grad(shape, seed=4).to(cuda_device)
    outs = [torch.empty_like(p) for p in ps]
    gp, gg = GsvParams(*(p.data_ptr() for p in ps), plan.n), GsvGrads(*(o.data_ptr() for o in outs))
    st = ctypes.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)

    def run():
        check(lib.gsv_backward_ex(ctypes.byref(gp), plan.shape, _ptr(plan.ws_gauss), _ptr(plan.ws_pairs), plan.capacity,
                                  _ptr(gv), ctypes.byref(gg), 0, None if tuning is None else ctypes.byref(tuning), st),
              "gsv_backward_ex")

    assert _grids(run, "k_backward8", tmp_path / "trace.json") == [64 * ctas]
