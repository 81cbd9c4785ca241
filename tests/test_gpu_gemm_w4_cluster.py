"""Super-tiles of an int4 linear that a cluster of CTAs shares (csrc/gemm_w4a16.cu, launch_plan_w4): clusters of 2, 3 and 8, parts of k that are not all as
long, a last super-tile short of columns, bias, the fused SiLU, results off any four halves, token tiles at their edges, and no workspace at all.
Reference: float64 over the format's fp16 weights.  Tolerance: as test_gpu_gemm_w4_whole.py's."""
import ctypes

import pytest
import torch
from .test_gpu_gemm_w4_few import DEV, _near, _weights
from .test_gpu_gemm_w4_whole import _whole

pytestmark = pytest.mark.gpu


def _cluster(T, N, K, workspace=1):
    """CTAs that share a super-tile of such a call on this device"""
    from tgis_b200 import _lib
    out = (ctypes.c_int32 * 8)()
    assert _lib.load().b200_debug_w4_plan(T, N, K, torch.cuda.get_device_properties(0).multi_processor_count, workspace, None, out) == 0
    return out[3]


# 44 k-blocks over clusters of 8: parts of 5 and 6; a last super-tile of 32 features; clusters of 3 and 2
@pytest.mark.parametrize("N,K,gs,cluster", [(2048, 5632, 128, 8), (1312, 4384, 32, 8), (11264, 2048, 64, 3), (12288, 4096, 128, 2)])
@pytest.mark.parametrize("T", [9, 16, 17, 33, 64, 65, 128])
def test_shared_super_tiles(N, K, gs, cluster, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    assert _cluster(T, N, K) == cluster
    g = torch.Generator(device=DEV).manual_seed(N + K + T)
    qweight, qzeros, scales, w = _weights(g, N, K, gs)
    x, bias = torch.randn(T, K, generator=g, device=DEV).half(), torch.randn(N, generator=g, device=DEV).half()
    packed = ops.gptq_pack(qweight, qzeros, scales, gs)
    got = ops.gemm_w4a16(x, packed, N, gs, bias)
    _near(got, x, w, bias)
    assert torch.equal(ops.gemm_w4a16(x, packed, N, gs, bias), got)   # sums in the order of the ranks
    _near(ops.gemm_w4a16(x, packed, N, gs), x, w)
    _near(_whole(x, packed, torch.empty_like(got), N, gs, bias), x, w, bias)
    room = torch.full((T * N + 2,), 7.0, dtype=torch.float16, device=DEV)
    off = room[1:-1].view(T, N)
    _near(_whole(x, packed, off, N, gs, bias), x, w, bias)
    assert float(room[0]) == 7.0 == float(room[-1])


@pytest.mark.parametrize("T", [9, 17, 64, 128])
def test_without_a_workspace(T):
    """clusters of six share super-tiles that eight CTAs share through a workspace"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    N = K = 4096
    assert (_cluster(T, N, K), _cluster(T, N, K, workspace=0)) == (0, 6)
    g = torch.Generator(device=DEV).manual_seed(T)
    qweight, qzeros, scales, w = _weights(g, N, K, 128)
    x, bias = torch.randn(T, K, generator=g, device=DEV).half(), torch.randn(N, generator=g, device=DEV).half()
    packed = ops.gptq_pack(qweight, qzeros, scales, 128)
    _near(_whole(x, packed, torch.empty(T, N, dtype=torch.float16, device=DEV), N, 128, bias), x, w, bias)


@pytest.mark.parametrize("I,K", [(1024, 5632), (5632, 2048)])
@pytest.mark.parametrize("T", [9, 17, 64, 128])
def test_gate_and_up_with_silu(I, K, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    assert _cluster(T, 2 * I, K) == (8 if I == 1024 else 3)
    g = torch.Generator(device=DEV).manual_seed(I + K + T)
    qweight, qzeros, scales, w = _weights(g, 2 * I, K, 128)
    x = torch.randn(T, K, generator=g, device=DEV).half()
    pairs = ops.gptq_pack(qweight, qzeros, scales, 128, ops.W4_LAYOUT_GATE_UP)
    both = ops.gemm_w4a16(x, pairs, 2 * I, 128, layout=ops.W4_LAYOUT_GATE_UP)
    _near(both, x, w)
    assert torch.equal(ops.gemm_w4a16(x, pairs, 2 * I, 128, layout=ops.W4_LAYOUT_GATE_UP, silu_mul=True), ops.silu_mul(both))
