"""Linears of prompt size (csrc/gemm_pair.cuh: SM pairs) against the same product in float64: token counts around the tile steps of 32, the cut
last tile, the change from the decode kernels and the groups of sixteen token tiles; feature counts that end inside a tile, a CTA's half and
an eight-feature piece; k that ends inside a k-block; every element type, group size and epilogue.

Tolerance: operands are exact, sums are fp32.  |error| <= rounding of the result (2^-11 of it in fp16, 2^-8 in bfloat16, none in fp32) plus that
of an fp32 sum in any order, sqrt(K) 2^-23 sum |x w| (its typical size is below a tenth of that)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _bound(ref, x, w, unit):
    spread = x.double().abs() @ w.double().abs().t()
    return unit * ref.abs() + x.shape[1] ** 0.5 * 2.0 ** -23 * spread + 1e-7


SHAPES = [(65, 256, 64), (96, 96, 72), (97, 264, 200), (128, 512, 1000), (129, 520, 128), (160, 8, 64), (256, 300, 192), (257, 2560, 320),
          (385, 130, 4096), (700, 4096, 256), (4129, 264, 128), (9001, 96, 64)]


@pytest.mark.parametrize("T,N,K", SHAPES)
@pytest.mark.parametrize("kind", ["fp16", "bf16", "bf16->fp32", "bf16 relu2"])
def test_dense(T, N, K, kind):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops, ops_seq
    g = torch.Generator(device=DEV).manual_seed(T + N + K)
    dtype = torch.float16 if kind == "fp16" else torch.bfloat16
    x = torch.randn(T, K, generator=g, device=DEV).to(dtype)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(dtype)
    for bias in (None, torch.randn(N, generator=g, device=DEV).to(dtype)):
        ref = x.double() @ w.double().t() + (0 if bias is None else bias.double())
        tol = _bound(ref, x, w, {"fp16": 2.0 ** -11, "bf16->fp32": 0.0}.get(kind, 2.0 ** -8))
        if kind == "fp16":
            y = ops.gemm_f16(x, w, bias)
        elif kind == "bf16 relu2":
            y = ops_seq.linear(x, w, bias, act=ops_seq.ACT_RELU2)
            tol = 2.0 ** -8 * ref.square() + 2 * ref.abs() * _bound(ref, x, w, 0.0) + 1e-7
            ref = ref.clamp(min=0).square()
        else:
            y = ops_seq.linear(x, w, bias, out_dtype=torch.float32 if kind == "bf16->fp32" else None)
        assert bool(((y.double() - ref).abs() <= tol).all()), float(((y.double() - ref).abs() - tol).max())


def test_dense_rows_that_are_not_aligned():
    """an output whose rows are not 16-byte pieces is stored by value, and nothing beside it is touched"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(3)
    for T, N, K, offset in ((130, 129, 128, 0), (300, 264, 64, 1)):
        x, w = torch.randn(T, K, generator=g, device=DEV).half(), torch.randn(N, K, generator=g, device=DEV).half()
        buf = torch.full((T * N + 16,), 7.0, dtype=torch.float16, device=DEV)
        out = buf[offset:offset + T * N].view(T, N)
        ops.gemm_f16(x, w, out=out)
        ref = x.double() @ w.double().t()
        assert bool(((out.double() - ref).abs() <= _bound(ref, x, w, 2.0 ** -11)).all())
        assert bool((buf[:offset] == 7).all()) and bool((buf[offset + T * N:] == 7).all())


def _weight(g, K, N, group):
    qw = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device=DEV).to(torch.int32)
    groups = -(-K // group)
    qz = torch.randint(-2 ** 31, 2 ** 31, (groups, N // 8), generator=g, device=DEV).to(torch.int32)
    sc = (torch.rand(groups, N, generator=g, device=DEV) * 0.02 + 0.001).half()
    shift = 4 * torch.arange(8, device=DEV, dtype=torch.int32)
    q = ((qw[:, None] >> shift[None, :, None]) & 15).reshape(K, N)
    z = ((qz[:, :, None] >> shift) & 15).reshape(groups, N) + 1
    of = torch.arange(K, device=DEV) // group
    return qw, qz, sc, (sc[of].double() * (q - z[of]).double()).half()   # [K, N], fp16 as the format defines its weights


@pytest.mark.parametrize("T,N,K,group", [(129, 256, 128, 128), (160, 96, 32, 32), (161, 288, 320, 64), (256, 512, 224, 32), (257, 768, 1024, 1024),
                                         (300, 4096, 384, 128), (385, 544, 4096, 64), (4129, 256, 128, 128)])
@pytest.mark.parametrize("bias", [False, True])
def test_int4(T, N, K, group, bias):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T + N + K)
    qw, qz, sc, W = _weight(g, K, N, group)
    x = torch.randn(T, K, generator=g, device=DEV).half()
    b = torch.randn(N, generator=g, device=DEV).half() if bias else None
    ref = x.double() @ W.double() + (b.double() if bias else 0)
    tol = _bound(ref, x, W.t(), 2.0 ** -11)
    for layout in (ops.W4_LAYOUT_PLAIN, ops.W4_LAYOUT_GATE_UP):
        if layout == ops.W4_LAYOUT_GATE_UP and N % 256:
            continue
        packed = ops.gptq_pack(qw, qz, sc, group, layout=layout)
        y = ops.gemm_w4a16(x, packed, N, group, b, layout=layout)
        assert bool(((y.double() - ref).abs() <= tol).all()), (layout, float(((y.double() - ref).abs() - tol).max()))
        if layout == ops.W4_LAYOUT_GATE_UP:
            y = ops.gemm_w4a16(x, packed, N, group, b, layout=layout, silu_mul=True)
            gate, up = ref.chunk(2, 1)
            want = gate * torch.sigmoid(gate) * up
            # both factors and the product are rounded: |d(silu)/dgate| <= 1.1
            slack = 1.1 * tol[:, :N // 2] * up.abs() + (gate * torch.sigmoid(gate)).abs() * tol[:, N // 2:] + 2 * 2.0 ** -11 * want.abs() + 1e-6
            assert bool(((y.double() - want).abs() <= slack).all()), float(((y.double() - want).abs() - slack).max())


@pytest.mark.parametrize("T,N,K", [(100, 520, 20480), (129, 300, 16384), (65, 2048, 1088), (256, 9600, 4096), (250, 40, 600), (96, 19000, 640), (200, 2560, 520)])
@pytest.mark.parametrize("kind", ["fp16", "bf16", "bf16 relu2"])
def test_sums_in_pieces(T, N, K, kind):
    """calls of 65 to 256 tokens add pieces of k in fp32: deep sums, pieces that end unevenly, token tiles of every width, more tiles than pairs"""
    test_dense(T, N, K, kind)


@pytest.mark.parametrize("T,N,K", [(100, 512, 20480), (200, 512, 20480), (256, 4096, 8192)])
def test_a_deep_sum_is_as_good_as_its_rounding(T, N, K):
    """against float64 the result is off by the rounding to fp16 and hardly more: the same sum in one tensor-core accumulator is 0.5 % further off at k = 20480"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(K)
    x, w = torch.randn(T, K, generator=g, device=DEV).half(), (torch.randn(N, K, generator=g, device=DEV) * 0.02).half()
    ref = x.double() @ w.double().t()
    off, rounding = (ops.gemm_f16(x, w).double() - ref).norm(), (ref.half().double() - ref).norm()
    assert float(off / rounding) < 1.002


def test_first_calls_inside_a_capture():
    """a process whose first prompt linear and first prompt attention are captured into a graph (where a kernel reports a wait that ran out is set up
    then): replays give what a call gives"""
    import os
    import subprocess
    import sys
    code = """
import torch, tgis_b200
from tgis_b200 import ops
D = 'cuda:0'
x, w = torch.randn(300, 256, device=D).half(), torch.randn(384, 256, device=D).half()
q, kp, vp = torch.randn(300, 4, 64, device=D).half(), torch.randn(20, 2, 16, 64, device=D).half(), torch.randn(20, 2, 16, 64, device=D).half()
table, lens, cu = torch.arange(20, device=D, dtype=torch.int32)[None].contiguous(), torch.tensor([300], dtype=torch.int32, device=D), torch.tensor([0, 300], dtype=torch.int32, device=D)
ws = ops.gemm_workspace(x.device, 300, 384, 256)
call = lambda: (ops.gemm_f16(x, w), ops.attn_prefill_paged(q, kp, vp, table, lens, cu, 300, 0.125))
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    a = call()
for _ in range(2):
    for t in a:
        t.zero_()
    g.replay()
    torch.cuda.synchronize()
    b = call()
    assert all(torch.equal(s, t) and bool(s.abs().sum() > 0) for s, t in zip(a, b))
print('ok')
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]
