"""SiLU(x Wg^T) * (x Wu^T) of a prompt in one kernel on SM pairs (b200_gemm_f16_silu, csrc/gemm_pair.cuh): the bits of the product and the activation by
themselves, whose sums and roundings it has.  Tokens at the edges of token tiles and of 32 of them, features that fill no tile, bias, and what it refuses."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _call(x, w, bias, y):
    from tgis_b200 import _lib
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())  # noqa: E731
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    return _lib.load().b200_gemm_f16_silu(p(x), p(w), p(bias), p(y), x.shape[0], w.shape[0] // 2, x.shape[1], st)


@pytest.mark.parametrize("I,K", [(5632, 256), (200, 64), (136, 72), (8, 128), (704, 520)])
@pytest.mark.parametrize("T", [257, 288, 300, 511, 513, 1100])
@pytest.mark.parametrize("with_bias", [False, True])
def test_bits_of_the_two_kernels(I, K, T, with_bias):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(I + K + T)
    x, w = torch.randn(T, K, generator=g, device=DEV).half(), (torch.randn(2 * I, K, generator=g, device=DEV) * 0.1).half()
    bias = torch.randn(2 * I, generator=g, device=DEV).half() if with_bias else None
    room = torch.full((T + 2, I), 7.0, dtype=torch.float16, device=DEV)
    assert _call(x, w, bias, room[1:-1]) == 0
    both = ops.gemm_f16(x, w, bias)
    assert torch.equal(room[1:-1], ops.silu_mul(both))
    assert bool((room[0] == 7.0).all()) and bool((room[-1] == 7.0).all())
    ref = (x.double() @ w.double().T + (bias.double() if with_bias else 0)).half()   # each factor within one rounding of its sum
    gate, up = ref[:, :I].double(), ref[:, I:].double()
    err = (room[1:-1].double() - torch.nn.functional.silu(gate) * up).abs()
    # roundings to fp16 (2^-11 each): of the gate (the SiLU's slope is at most 1.1), of the up factor, of the SiLU and of the product
    assert bool((err <= 2.0 ** -11 * (2.2 * gate.abs() * up.abs() + 4 * (torch.nn.functional.silu(gate) * up).abs()) + 2.0 ** -10).all())


def test_what_it_refuses():
    import tgis_b200  # noqa: F401
    x, w = torch.zeros(300, 128, dtype=torch.float16, device=DEV), torch.zeros(32, 128, dtype=torch.float16, device=DEV)
    y = torch.zeros(300 * 16 + 8, dtype=torch.float16, device=DEV)
    assert _call(x, w, None, y[8:]) == 0
    assert _call(x, w, None, y[4:]) != 0                  # y off 16 bytes
    assert _call(x[:256], w, None, y) != 0                # 256 tokens
    assert _call(x, w[:24], None, y) != 0                 # 12 outputs
    assert _call(x[:, :60].contiguous(), w[:, :60].contiguous(), None, y) != 0
