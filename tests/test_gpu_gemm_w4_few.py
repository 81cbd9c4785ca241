"""int4 linears of up to eight tokens and few k-blocks per SM (csrc/gemm_w4_few.cuh): clusters of one to eight CTAs, parts of one k-block and of
several, k that ends inside a block, a last super-tile that is half empty, every group size, both layouts, SiLU * up, bias, a deferred result; calls on
the far side of the rule beside them.  Reference: float64 over the format's fp16 weights.

Tolerance: the result rounds to fp16 (2^-11 of it) and its fp32 sums of K products to K 2^-24 of the sum of their absolute values at the most; SiLU * up
rounds three times more."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (N, K): super-tiles x k-blocks.  6144 x 4096 clusters of five, 4096 x 4096 six, 2560 x 2048 and below eight; 96 x 160 one CTA per k-block, two of them, the
# second a quarter full; 288: the second super-tile has one tile of 32 features; 2048 x 1120: nine k-blocks over eight CTAs, the last of them short
SHAPES = [(6144, 4096, 128), (4096, 4096, 64), (2560, 2048, 32), (96, 160, 32), (288, 128, 64), (2048, 1120, 32), (1024, 5632, -1)]


def _weights(g, N, K, gs):
    groups = 1 if gs <= 0 else (K + gs - 1) // gs
    size = K if gs <= 0 else gs
    qweight = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device=DEV, dtype=torch.int64).int()
    zeros = torch.randint(0, 16, (groups, N // 8, 8), generator=g, device=DEV, dtype=torch.int64)
    packed = (zeros << (4 * torch.arange(8, device=DEV))).sum(-1)
    qzeros = torch.where(packed >= 2 ** 31, packed - 2 ** 32, packed).int()
    scales = (torch.rand(groups, N, generator=g, device=DEV) * 0.01 + 0.001).half()
    shift = 4 * torch.arange(8, device=DEV, dtype=torch.int32)
    q = ((qweight[:, None, :] >> shift[None, :, None]) & 15).reshape(K, N)
    z = zeros.reshape(groups, N) + 1
    at = torch.arange(K, device=DEV) // size
    w = (scales[at].double() * (q - z[at]).double()).half().double()
    return qweight, qzeros, scales, w


def _near(got, x, w, bias=None):
    want = x.double() @ w + (0 if bias is None else bias.double())
    room = 2 ** -11 * want.abs() + x.shape[1] * 2 ** -24 * (x.double().abs() @ w.abs()) + 2 ** -24
    assert bool(((got.double() - want).abs() <= room).all()), float(((got.double() - want).abs() / room).max())


@pytest.mark.parametrize("N,K,gs", SHAPES)
@pytest.mark.parametrize("T", [1, 7, 8, 9])
def test_few_tokens(N, K, gs, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N + K + T)
    qweight, qzeros, scales, w = _weights(g, N, K, gs)
    x, bias = torch.randn(T, K, generator=g, device=DEV).half(), torch.randn(N, generator=g, device=DEV).half()
    packed = ops.gptq_pack(qweight, qzeros, scales, gs)
    _near(ops.gemm_w4a16(x, packed, N, gs), x, w)
    for _ in range(2):   # the workspace is left as it was found
        got = ops.gemm_w4a16(x, packed, N, gs, bias)
        _near(got, x, w, bias)
        _near(ops.splitk_reduce(ops.gemm_w4a16_deferred(x, packed, N, gs, bias=bias)), x, w, bias)   # (goes the other way)


@pytest.mark.parametrize("I,K", [(256, 512), (2048, 2048), (128, 96)])
@pytest.mark.parametrize("T", [1, 8])
def test_gate_and_up_beside_each_other(I, K, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(I + K + T)
    qweight, qzeros, scales, w = _weights(g, 2 * I, K, 32)
    x = torch.randn(T, K, generator=g, device=DEV).half()
    pairs = ops.gptq_pack(qweight, qzeros, scales, 32, ops.W4_LAYOUT_GATE_UP)
    both = ops.gemm_w4a16(x, pairs, 2 * I, 32, layout=ops.W4_LAYOUT_GATE_UP)
    _near(both, x, w)
    assert torch.equal(both, ops.gemm_w4a16(x, ops.gptq_pack(qweight, qzeros, scales, 32), 2 * I, 32))
    assert torch.equal(ops.gemm_w4a16(x, pairs, 2 * I, 32, layout=ops.W4_LAYOUT_GATE_UP, silu_mul=True), ops.silu_mul(both))


def test_a_token_alone_and_among_others():
    """columns of a product are independent: what is not finite stays with its token, and padding never shows"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    N, K = 2560, 2048
    g = torch.Generator(device=DEV).manual_seed(3)
    qweight, qzeros, scales, _ = _weights(g, N, K, 128)
    packed, x = ops.gptq_pack(qweight, qzeros, scales, 128), torch.randn(5, K, generator=g, device=DEV).half()
    alone = torch.cat([ops.gemm_w4a16(x[i:i + 1].contiguous(), packed, N, 128) for i in range(5)])
    x2 = torch.cat([x, torch.full((1, K), float("nan"), device=DEV).half(), x[:1]])
    got = ops.gemm_w4a16(x2, packed, N, 128)
    assert torch.equal(got[:5], alone) and torch.equal(got[6], alone[0]) and bool(got[5].isnan().all())
