"""fp16 and bfloat16 linears whose feature tiles are shared by clusters of CTAs (csrc/gemm_f16.cu): every element format, token counts at the edges of the
token tiles, clusters of two to eight with parts of unlike length, k that ends inside a block, features that end inside a tile and inside four; wide outputs of
17 to 64 tokens that go to the SM pairs, and their neighbours; no workspace.

Tolerance: fp32 sums of K products, K 2^-24 of the sum of their absolute values at the most, and the result's own rounding (2^-11 fp16, 2^-8 bfloat16)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _near(got, x, w, bias, rounding):
    want = x.double() @ w.double().T + (0 if bias is None else bias.double())
    room = rounding * want.abs() + x.shape[1] * 2 ** -24 * (x.double().abs() @ w.double().abs().T) + 2 ** -24
    assert bool(((got.double() - want).abs() <= room).all()), float(((got.double() - want).abs() / room).max())


def _data(T, N, K, dtype):
    g = torch.Generator(device=DEV).manual_seed(T + N + K)
    return (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((T, K), (N, K), (N,)))


# feature tiles: 1 and 2 (clusters of eight), 20 (six), 30 (four), 40 (three), 74 (two), 75 (none); k-blocks that the clusters cut unevenly, one with eight of 64
SHAPES = [(40, 520), (250, 2056), (2560, 2048), (3840, 1096), (5120, 776), (9472, 512), (9600, 512), (1023, 576)]


@pytest.mark.parametrize("N,K", SHAPES)
@pytest.mark.parametrize("T", [1, 16, 17, 33, 64, 65])
def test_fp16(N, K, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    x, w, bias = _data(T, N, K, torch.float16)
    first = ops.gemm_f16(x, w, bias)
    _near(first, x, w, bias, 2 ** -11)
    assert torch.equal(ops.gemm_f16(x, w, bias), first)
    _near(ops.gemm_f16(x, w), x, w, None, 2 ** -11)


@pytest.mark.parametrize("N,K", [(250, 2056), (2560, 2048), (9600, 512)])
@pytest.mark.parametrize("T", [1, 64, 128, 129, 256])
def test_bfloat16(N, K, T):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    x, w, bias = _data(T, N, K, torch.bfloat16)
    _near(ops.linear(x, w, bias, out_dtype=torch.float32), x, w, bias, 2 ** -24)
    _near(ops.linear(x, w, bias), x, w, bias, 2 ** -8)
    squared = ops.linear(x, w, act=ops.ACT_RELU2).double()
    want = (x.double() @ w.double().T).clamp(min=0).square()
    assert bool(((squared - want).abs() <= 2 ** -7 * want + 1e-3).all())


def test_tokens_do_not_mix():
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    x, w, _ = _data(24, 2560, 2048, torch.float16)
    want = ops.gemm_f16(x, w)
    x[5] = float("inf")
    got = ops.gemm_f16(x, w)
    keep = torch.arange(24, device=DEV) != 5
    assert torch.equal(got[keep], want[keep]) and not bool(got[5].isfinite().any())


@pytest.mark.parametrize("T", [16, 17, 64])
@pytest.mark.parametrize("N", [11264, 22016, 32000])
def test_wide_outputs(N, T):
    """one wave of the SM pairs, a wave and a sixth, two waves"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    x, w, bias = _data(T, N, 512, torch.float16)
    _near(ops.gemm_f16(x, w, bias), x, w, bias, 2 ** -11)


def test_without_workspace():
    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib, ops
    for T, N, K in ((8, 2560, 2048), (40, 32000, 256)):
        x, w, bias = _data(T, N, K, torch.float16)
        y = torch.empty(T, N, dtype=torch.float16, device=DEV)
        _lib.check(_lib.load().b200_gemm_f16(x.data_ptr(), w.data_ptr(), bias.data_ptr(), y.data_ptr(), T, N, K, None, ops._stream()), "gemm_f16")
        _near(y, x, w, bias, 2 ** -11)


@pytest.mark.parametrize("T", [8, 24, 64])
def test_a_result_off_any_eight_bytes(T):
    """a result that starts one element into its memory: equal to the aligned one, and nothing beside it is touched"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib, ops
    N, K = 2560, 2048
    x, w, bias = _data(T, N, K, torch.float16)
    got = []
    for off in (0, 1):
        room = torch.full((T * N + 2,), 7.0, dtype=torch.float16, device=DEV)
        _lib.check(_lib.load().b200_gemm_f16(x.data_ptr(), w.data_ptr(), bias.data_ptr(), room[off:].data_ptr(), T, N, K, None, ops._stream()), "gemm_f16")
        got.append(room[off:off + T * N].clone())
        assert all(float(v) == 7.0 for v in torch.cat([room[:off], room[off + T * N:]]))
    assert torch.equal(*got)


# 32 feature tiles of four CTAs each, 172 that 148 CTAs straddle; clusters of four
@pytest.mark.parametrize("T,N,K", [(4, 4096, 4096), (16, 22016, 1024), (16, 4096, 4096)])
def test_results_off_any_eight_bytes(T, N, K):
    """with a workspace, so that CTAs share feature tiles through it or in clusters: the bits of a y on eight bytes"""
    import ctypes
    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib
    lib, (x, w, bias) = _lib.load(), _data(T, N, K, torch.float16)
    ws = torch.zeros(lib.b200_gemm_workspace_bytes(T, N, K), dtype=torch.uint8, device=DEV)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731

    def call(y):
        assert lib.b200_gemm_f16(p(x), p(w), p(bias), p(y), T, N, K, p(ws), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        return y
    room = torch.full((T * N + 2,), 7.0, dtype=torch.float16, device=DEV)
    want = call(torch.empty(T, N, dtype=torch.float16, device=DEV))
    _near(want, x, w, bias, 2 ** -11)
    assert torch.equal(call(room[1:-1].view(T, N)), want) and float(room[0]) == 7.0 == float(room[-1])
