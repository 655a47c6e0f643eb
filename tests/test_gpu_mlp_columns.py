"""gsv_mlp_gemm's plain and summed outputs with transposed rows, where a lane of the epilogue's warp may
hold a row past the last one while its neighbours read tensor memory: against FP32 products of the same
BF16 inputs (only the order of summation differs: relative error 1e-5), and nothing is written past
the last row."""
import pytest
import torch

from tests.test_gpu_mlp_tiles import ATOMIC, F32, gemm, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64, 200])
@pytest.mark.parametrize("M,N", [(19001, 256), (1003, 512), (257, 48), (33, 16), (31, 256), (1, 16)])
def test_transposed_outputs(M, N, K, cuda_device):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    ref = a.float() @ b.float().t()
    out = torch.full((N, M + 3), 7.0, device="cuda")  # columns of pitch M + 3
    gemm(a, b, (1, M + 3), M, N, K, F32, f32=out, bias=bias)
    assert rel(out[:, :M].t(), ref + bias) < 1e-5 and (out[:, M:] == 7.0).all()
    acc = torch.zeros(N, M + 3, device="cuda")
    gemm(a, b, (1, M + 3), M, N, K, ATOMIC, f32=acc, splits=2)
    assert rel(acc[:, :M].t(), ref) < 1e-5 and (acc[:, M:] == 0).all()
