"""Products over weights that the launch just before has written, on the same stream and without waiting for it: the same bits as after a wait.  A kernel may
begin while the one before it ends, when that one's stores are not all in place yet; so weights are read behind the wait for it, or were settled when they were
packed.  The weights' memory holds another matrix before, so that what is read too early shows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _differs(call, write, rounds):
    """how many of so many products right behind `write` differ from the product after a wait; write(i) leaves other weights for every i"""
    n = 0
    for i in range(rounds):
        torch.cuda.synchronize()
        write(i)
        at_once = call()
        torch.cuda.synchronize()
        n += not torch.equal(at_once, call())
    return n


@pytest.mark.parametrize("T", [1, 8, 16, 64, 129, 1000])
@pytest.mark.parametrize("K,N,gate_up", [(4096, 6144, False), (1024, 2048, True)])
def test_packed_records(T, K, N, gate_up):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    from .test_gpu_gemm_w4_few import _weights
    g = torch.Generator(device=DEV).manual_seed(T)
    some = [_weights(g, N, K, 128)[:3] for _ in range(3)]
    x, layout, held = torch.randn(T, K, generator=g, device=DEV).half(), int(gate_up), {}

    def write(i):
        held.pop("packed", None)   # the next one takes its memory
        held["packed"] = ops.gptq_pack(*some[i % 3], 128, layout)
    assert _differs(lambda: ops.gemm_w4a16(x, held["packed"], N, 128, layout=layout, silu_mul=gate_up), write, 60) == 0


@pytest.mark.parametrize("T", [1, 8, 64, 200, 1000])
@pytest.mark.parametrize("K,N", [(4096, 4096), (2048, 32000), (512, 384)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_matrix_that_was_just_computed(T, K, N, dtype):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops, ops_seq
    g = torch.Generator(device=DEV).manual_seed(T)
    a, x = torch.randn(N, K, generator=g, device=DEV).to(dtype), torch.randn(T, K, generator=g, device=DEV).to(dtype)
    w, gamma = torch.empty_like(a), torch.ones(K, dtype=torch.float16, device=DEV)
    call = (lambda: ops.gemm_f16(x, w)) if dtype == torch.float16 else (lambda: ops_seq.linear(x, w, out_dtype=torch.float32))
    assert _differs(call, lambda i: torch.mul(a, 0.25 + i, out=w), 40) == 0

    def write(i):   # a kernel of this library in between, which itself begins early
        torch.mul(a, 0.25 + i, out=w)
        ops.rmsnorm_residual(gamma[None], None, gamma, 1e-5)
    assert _differs(call, write, 40) == 0


def test_heads():
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq
    g = torch.Generator(device=DEV).manual_seed(1)
    T, Z, N, K = 20, 16, 512, 128
    a, x = torch.randn(Z, N, K, generator=g, device=DEV).bfloat16(), torch.randn(T, Z, K, generator=g, device=DEV).bfloat16()
    w = torch.empty_like(a)

    def call():
        out = torch.empty(T, Z, N, dtype=torch.float32, device=DEV)
        ops_seq.linear_per_head(x, w, out)
        return out
    assert _differs(call, lambda i: torch.mul(a, 0.25 + i, out=w), 100) == 0


@pytest.mark.parametrize("T", [1, 16, 64, 200])
@pytest.mark.parametrize("K,N", [(4096, 4096), (2048, 11264), (512, 384)])
def test_held_weights(T, K, N):
    """the entries for weights that were settled: the bits of the plain ones, also right behind the launch that settles"""
    import ctypes
    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib, ops
    g = torch.Generator(device=DEV).manual_seed(T)
    a, x = torch.randn(N, K, generator=g, device=DEV).half(), torch.randn(T, K, generator=g, device=DEV).half()
    w, y, lib = torch.empty_like(a), torch.empty(T, N, dtype=torch.float16, device=DEV), _lib.load()
    ws = ops.gemm_workspace(w.device, T, N, K)

    def write(i):
        torch.mul(a, 0.25 + i, out=w)
        ops.settle()

    def held():
        _lib.check(lib.b200_gemm_f16_held(x.data_ptr(), w.data_ptr(), None, y.data_ptr(), T, N, K, ws.data_ptr(), ops._stream()), "held")
        desc = _lib.B200SplitK()
        _lib.check(lib.b200_gemm_f16_deferred_held(x.data_ptr(), w.data_ptr(), None, T, N, K, ws.data_ptr(), ctypes.byref(desc), ops._stream()), "held")
        return torch.stack([y, ops.splitk_reduce(ops.SplitK(desc, ws, None))])
    assert _differs(held, write, 20) == 0
    assert torch.equal(held(), torch.stack([ops.gemm_f16(x, w), ops.splitk_reduce(ops.gemm_f16_deferred(x, w))]))
