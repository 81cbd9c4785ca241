"""fp16 and bfloat16 linears of 65 to 256 tokens where clusters share a feature tile (csrc/gemm_f16.cu, f16_cluster_us): calls on both sides of the line to the SM
pairs, edges of the token tiles, few feature tiles and a last one that is short, bias.  Reference: float64.

Tolerance: the result rounds to its type (2^-11, 2^-8 of it) and its fp32 sums of K products to K 2^-24 of the sum of their absolute values at the most."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("K,N", [(5632, 2048), (4096, 4096), (11008, 4096), (20480, 5120), (8192, 1000), (520, 200)])
@pytest.mark.parametrize("T", [65, 96, 128, 129, 200, 256])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_against_float64(K, N, T, dtype):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops, ops_seq
    g = torch.Generator(device=DEV).manual_seed(K + N + T)
    x = torch.randn(T, K, generator=g, device=DEV).to(dtype)
    w = (torch.randn(N, K, generator=g, device=DEV) * 0.05).to(dtype)
    bias = torch.randn(N, generator=g, device=DEV).to(dtype)
    call = (lambda: ops.gemm_f16(x, w, bias)) if dtype == torch.float16 else (lambda: ops_seq.linear(x, w, bias, out_dtype=torch.bfloat16))
    y = call()
    assert torch.equal(call(), y)
    ref, size = x.double() @ w.double().T + bias.double(), x.double().abs() @ w.double().abs().T + bias.double().abs()
    tol = (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * ref.abs() + K * 2.0 ** -24 * size + 1e-7
    assert bool(((y.double() - ref).abs() <= tol).all())
