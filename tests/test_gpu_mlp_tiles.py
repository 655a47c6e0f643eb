"""gsv_mlp_gemm over more tiles than SMs, each way an operand can be copied and
each way the output can be written, against FP32 products of the same BF16
inputs.  Products of BF16 values are exact in FP32 and the sums have at most
2,000 terms, so only the order of summation differs: relative error 1e-5."""
import ctypes

import pytest
import torch

from gs_tmi_b200._lib import check, lib

pytestmark = pytest.mark.gpu

F32, BIAS_GELU, GELU_GRAD, ATOMIC = 0, 1, 2, 3


def _p(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def gemm(a, b, c_strides, M, N, K, epi, f32=None, bf16=None, z=None, bias=None, col_sum=None, splits=1):
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    check(lib.gsv_mlp_gemm(_p(a), a.stride(0), a.stride(1), _p(b), b.stride(0), b.stride(1), M, N, K, splits,
                           _p(bias), _p(f32), _p(bf16), _p(z), *c_strides, epi, _p(col_sum), _p(err),
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "gsv_mlp_gemm")
    torch.cuda.synchronize()
    assert int(err.item()) == 0


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def operand(rows, K, form, g):
    """rows x K in BF16: K-major, rows contiguous, overlapping rows (TMA takes
    no stride below the row's length), and strides that only element-wise
    copies take."""
    if form == "k":
        return torch.randn(rows, K, device="cuda", generator=g).bfloat16()
    if form == "mn":
        pitch = (rows + 7) // 8 * 8
        return torch.randn(K, pitch, device="cuda", generator=g).bfloat16()[:, :rows].t()
    if form == "overlap":
        return torch.randn(rows * 8 + K, device="cuda", generator=g).bfloat16().as_strided((rows, K), (8, 1))
    return torch.randn(rows, K * 3, device="cuda", generator=g).bfloat16()[:, ::3]


@pytest.mark.parametrize("fa", ["k", "mn", "overlap", "odd"])
@pytest.mark.parametrize("fb", ["k", "mn", "odd"])
@pytest.mark.parametrize("M,N,K", [(19100, 512, 72), (300, 48, 200), (1, 256, 8), (129, 16, 2000)])
def test_operand_forms(M, N, K, fa, fb, cuda_device):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = operand(M, K, fa, g), operand(N, K, fb, g)
    ref = a.float() @ b.float().t()
    out = torch.full((M, N), float("nan"), device="cuda")
    gemm(a, b, (N, 1), M, N, K, F32, f32=out)
    assert rel(out, ref) < 1e-5
    acc = torch.zeros(M, N, device="cuda")
    gemm(a, b, (N, 1), M, N, K, ATOMIC, f32=acc, splits=3)
    assert rel(acc, ref) < 1e-5


@pytest.mark.parametrize("M,N", [(19000, 256), (130, 512), (257, 48), (31, 16)])
@pytest.mark.parametrize("layout", ["rows", "odd rows", "columns"])
def test_output_forms(M, N, layout, cuda_device):
    """Whole rows, rows at an odd pitch and transposed; z equals the product
    plus bias, the BF16 outputs the rounded GELU and GELU' of that z (one BF16
    unit in the last place), the column sums those of what was stored."""
    K = 64
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = (torch.randn(N, K, device="cuda", generator=g) * 0.2).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)

    def new(dtype):
        if layout == "columns":
            return torch.full((N, M), 7.0, device="cuda", dtype=dtype).t()
        return torch.full((M, N + (layout == "odd rows")), 7.0, device="cuda", dtype=dtype)[:, :N]

    z, y, d = new(torch.float32), new(torch.bfloat16), new(torch.bfloat16)
    strides = z.stride()
    prod = a.float() @ b.float().t()
    gemm(a, b, strides, M, N, K, BIAS_GELU, bf16=y, z=z, bias=bias)
    assert rel(z, prod + bias) < 1e-5
    want = torch.nn.functional.gelu(z, approximate="tanh")
    assert ((y.float() - want).abs() <= 2 ** -7 * want.abs() + 1e-3).all()  # 1e-3: tanh.approx
    col = torch.zeros(N, device="cuda") if strides[1] == 1 else None
    gemm(a, b, strides, M, N, K, GELU_GRAD, bf16=d, z=z, col_sum=col)
    zz = z.detach().clone().requires_grad_(True)
    torch.nn.functional.gelu(zz, approximate="tanh").backward(prod)
    assert ((d.float() - zz.grad).abs() <= 2 ** -7 * zz.grad.abs() + 2e-3 * prod.abs() + 1e-5).all()
    if col is not None:
        assert float((col - d.float().sum(0)).abs().max()) <= 1e-5 * float(d.float().abs().sum(0).max())
