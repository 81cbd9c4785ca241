"""Super-tiles of an int4 linear that one CTA has alone (csrc/gemm_w4a16.cu, w4_finish): the last of a CTA's is written by all threads, those before it by
the epilogue warps.  Without a workspace every CTA has whole super-tiles, one or several, the last of them short of columns; with one, some are shared.
9 and 16 tokens take that end with the SiLU only; 17, 64, 65 and 128 are the edges of the token tiles above.  Reference: float64 over the format's fp16 weights.

Tolerance: the result rounds to fp16 (2^-11 of it) and its fp32 sums of K products to K 2^-24 of the sum of their absolute values at the most."""
import ctypes

import pytest
import torch
from .test_gpu_gemm_w4_few import DEV, _near, _weights

pytestmark = pytest.mark.gpu
TOKENS = [9, 16, 17, 33, 64, 65, 128]


def _whole(x, packed, y, N, gs, bias=None, layout=0, act=0):
    """y = x W with no workspace"""
    from tgis_b200 import _lib
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())  # noqa: E731
    rc = _lib.load().b200_gemm_w4a16_ex(p(x), p(packed), p(bias), p(y), x.shape[0], N, x.shape[1], gs, layout, act, None, st)
    assert rc == 0
    return y


# 288: the second super-tile is an eighth full; 38048: 149 super-tiles, so that one CTA has two
@pytest.mark.parametrize("N,K,gs", [(288, 96, 32), (512, 256, 64), (38048, 128, 128)])
@pytest.mark.parametrize("T", TOKENS)
def test_whole_super_tiles(N, K, gs, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N + K + T)
    qweight, qzeros, scales, w = _weights(g, N, K, gs)
    x, bias = torch.randn(T, K, generator=g, device=DEV).half(), torch.randn(N, generator=g, device=DEV).half()
    packed = ops.gptq_pack(qweight, qzeros, scales, gs)
    got = _whole(x, packed, torch.empty(T, N, dtype=torch.float16, device=DEV), N, gs, bias)
    _near(got, x, w, bias)
    _near(_whole(x, packed, torch.empty_like(got), N, gs), x, w)
    _near(ops.gemm_w4a16(x, packed, N, gs, bias), x, w, bias)
    room = torch.full((T * N + 2,), 7.0, dtype=torch.float16, device=DEV)   # a y that starts off any four halves
    off = room[1:-1].view(T, N)
    assert torch.equal(_whole(x, packed, off, N, gs, bias), got) and float(room[0]) == 7.0 == float(room[-1])


@pytest.mark.parametrize("I,K", [(128, 96), (2048, 512), (14336, 256)])
@pytest.mark.parametrize("T", TOKENS)
def test_gate_and_up_with_silu(I, K, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(I + K + T)
    qweight, qzeros, scales, w = _weights(g, 2 * I, K, 32)
    x, bias = torch.randn(T, K, generator=g, device=DEV).half(), torch.randn(2 * I, generator=g, device=DEV).half()
    pairs = ops.gptq_pack(qweight, qzeros, scales, 32, ops.W4_LAYOUT_GATE_UP)
    both = _whole(x, pairs, torch.empty(T, 2 * I, dtype=torch.float16, device=DEV), 2 * I, 32, bias, ops.W4_LAYOUT_GATE_UP)
    _near(both, x, w, bias)
    one = _whole(x, pairs, torch.empty(T, I, dtype=torch.float16, device=DEV), 2 * I, 32, bias, ops.W4_LAYOUT_GATE_UP, 1)
    assert torch.equal(one, ops.silu_mul(both))
    room = torch.full((T * I + 2,), 7.0, dtype=torch.float16, device=DEV)
    assert torch.equal(_whole(x, pairs, room[1:-1].view(T, I), 2 * I, 32, bias, ops.W4_LAYOUT_GATE_UP, 1), one)
    assert float(room[0]) == 7.0 == float(room[-1])


# 16 super-tiles of eight CTAs each, 81 that 148 CTAs straddle, and gate and up
@pytest.mark.parametrize("N,K,act", [(4096, 4096, 0), (20736, 4096, 0), (4096, 4096, 1)])
@pytest.mark.parametrize("T", [4, 9, 64])
def test_shared_super_tiles_off_any_four_halves(N, K, act, T):
    """with a workspace, so that CTAs share super-tiles: a y that starts off any four halves gets the bits of one that does not"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib, ops
    lib, g = _lib.load(), torch.Generator(device=DEV).manual_seed(N + K + T)
    qweight, qzeros, scales, w = _weights(g, N, K, 128)
    x, bias = torch.randn(T, K, generator=g, device=DEV).half(), torch.randn(N, generator=g, device=DEV).half()
    layout = ops.W4_LAYOUT_GATE_UP if act else 0
    packed = ops.gptq_pack(qweight, qzeros, scales, 128, layout)
    ws = torch.zeros(lib.b200_gemm_workspace_bytes(T, N, K), dtype=torch.uint8, device=DEV)
    cols = N // 2 if act else N
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731

    def call(y, x):
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.b200_gemm_w4a16_ex(p(x), p(packed), p(bias), p(y), T, N, K, 128, layout, act, p(ws), st) == 0
        return y
    room = torch.full((T * cols + 2,), 7.0, dtype=torch.float16, device=DEV)
    off = call(room[1:-1].view(T, cols), x)
    assert float(room[0]) == 7.0 == float(room[-1])
    if T > 8:   # (up to eight tokens a y on four halves goes to another kernel)
        assert torch.equal(off, call(torch.empty(T, cols, dtype=torch.float16, device=DEV), x))
    if not act:
        return _near(off, x, w, bias)
    sums, size = x.double() @ w + bias.double(), x.double().abs() @ w.abs()
    (gate, up), (d_gate, d_up) = sums.chunk(2, 1), (2 ** -11 * sums.abs() + K * 2 ** -24 * size).chunk(2, 1)
    silu = torch.nn.functional.silu(gate)   # its slope is 1.1 at the most; it and the product round once each
    assert bool(((off.double() - silu * up).abs() <= 1.1 * d_gate * (up.abs() + d_up) + silu.abs() * d_up + 2 ** -10 * (silu * up).abs() * 1.01 + 2 ** -20).all())
