"""The native per-call host side (csrc/host/host_calls.cpp): the calls that it serves give what the Python path gives, and calls that it leaves to
Python end as they would without it - the same results for the unusual ones, the same errors for the wrong ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class _Nothing:
    """a native side that serves no call"""

    def __getattr__(self, name):
        return lambda *a: None


@pytest.fixture(params=["ops", "ops_seq"])
def both(request, monkeypatch):
    """runs a call with the native side and without it"""
    import tgis_b200
    from tgis_b200 import ops, ops_seq

    mod = {"ops": ops, "ops_seq": ops_seq}[request.param]
    native = mod._native()

    def run(call):
        got = []
        for side in (native, _Nothing()):
            monkeypatch.setattr(mod, "_host", side)
            try:
                got.append(call(mod))
            except Exception as e:
                got.append((type(e), str(e)))
        monkeypatch.setattr(mod, "_host", native)
        a, b = got
        assert type(a) is type(b) and (torch.equal(a, b) and a.dtype == b.dtype and a.stride() == b.stride() if isinstance(a, torch.Tensor) else a == b), (a, b)
        return a
    run.name = request.param
    return run


def _r(*shape, dtype=torch.float16):
    return torch.randn(*shape, device=DEV, dtype=torch.float32).to(dtype)


def test_linears(both):
    x, w, b = _r(5, 256), _r(96, 256), _r(96)
    if both.name == "ops_seq":
        x, w, b = (t.bfloat16() for t in (x, w, b))
        for dt in (None, torch.bfloat16, torch.float32):
            assert both(lambda m: m.linear(x, w, b, out_dtype=dt)).dtype == (dt or torch.bfloat16)
            both(lambda m: m.linear(x, w, None, out_dtype=dt))
        both(lambda m: m.linear(x.float(), w.float(), b.float()))                      # a true 32-bit product
        wide = _r(5, 300).bfloat16()
        both(lambda m: m.linear(wide[:, :256], w))                                     # row-strided
        both(lambda m: m.linear(x[:, :40].contiguous(), w[:, :40].contiguous()))       # small k
        both(lambda m: m.linear(x, w, act=m.ACT_RELU2))
        both(lambda m: m.linear(x[:0], w))
        assert both(lambda m: m.linear(x.cpu(), w))[0].__name__ == "B200Error"
        assert both(lambda m: m.linear(x, w[:, :128]))[0] is AssertionError
        return
    out, ws = torch.empty(5, 96, dtype=torch.float16, device=DEV), torch.zeros(1 << 24, dtype=torch.uint8, device=DEV)
    both(lambda m: m.gemm_f16(x, w, b))
    both(lambda m: m.gemm_f16(x, torch.nn.Parameter(w, requires_grad=False)))
    assert both(lambda m: m.gemm_f16(x, w, b, out)).data_ptr() == out.data_ptr()
    both(lambda m: m.gemm_f16(x, w, workspace=ws))
    both(lambda m: m.gemm_f16(x[:0], w))
    assert both(lambda m: m.gemm_f16(x.float(), w))[0].__name__ == "B200Error"
    assert both(lambda m: m.gemm_f16(x.cpu(), w))[0].__name__ == "B200Error"
    assert both(lambda m: m.gemm_f16(x.t(), w))[0] is AssertionError
    assert both(lambda m: m.gemm_f16(x[0], w))[0] is ValueError
    assert both(lambda m: m.gemm_f16(_r(5, 100), _r(96, 100)))[0].__name__ == "B200Error"   # refused by the entry


@pytest.mark.parametrize("both", ["ops"], indirect=True)
def test_int4(both):
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    K, N = 256, 512
    qweight = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device=DEV).int()
    qzeros, scales = torch.full((K // 128, N // 8), 0x77777777, device=DEV).int(), torch.rand(K // 128, N, device=DEV).half() * 0.01
    plain, pairs = ops.gptq_pack(qweight, qzeros, scales, 128), ops.gptq_pack(qweight, qzeros, scales, 128, ops.W4_LAYOUT_GATE_UP)
    x, b = _r(3, K), _r(N)
    both(lambda m: m.gemm_w4a16(x, plain, N, 128))
    both(lambda m: m.gemm_w4a16(x, plain, N, 128, b, torch.empty(3, N, dtype=torch.float16, device=DEV)))
    assert both(lambda m: m.gemm_w4a16(x, pairs, N, 128, layout=1, silu_mul=True)).shape == (3, N // 2)
    assert both(lambda m: m.gemm_w4a16(x, plain, N, 128, silu_mul=True))[0].__name__ == "B200Error"   # needs the other layout
    assert both(lambda m: m.gemm_w4a16(x.bfloat16(), plain, N, 128))[0].__name__ == "B200Error"


@pytest.mark.parametrize("both", ["ops"], indirect=True)
def test_attention(both):
    lens = torch.tensor([20, 3], dtype=torch.int32, device=DEV)
    table = torch.tensor([[0, 2], [1, 0]], dtype=torch.int32, device=DEV)
    k, v = _r(3, 2, 16, 64), _r(3, 2, 16, 64)
    qkv = _r(2, 8 * 64)
    q = qkv[:, :4 * 64].unflatten(1, (4, 64))
    both(lambda m: m.attn_decode_paged(q, k, v, table, lens, 20, 0.125, 2))
    both(lambda m: m.attn_decode_paged(q, k, v, table, lens, 20, 0.125, 2, torch.empty(2, 4, 64, dtype=torch.float16, device=DEV)))
    assert both(lambda m: m.attn_decode_paged(q, k, v, table, lens, 4000, 0.125, 2, workspace=lens))[0].__name__ == "B200Error"
    assert both(lambda m: m.attn_decode_paged(q, k, v, table.long(), lens, 20, 0.125, 2))[0].__name__ == "B200Error"
    assert both(lambda m: m.attn_decode_paged(q.transpose(0, 1), k, v, table, lens, 20, 0.125, 2))[0] is AssertionError
    cu = torch.tensor([0, 1, 2], dtype=torch.int32, device=DEV)
    both(lambda m: m.attn_prefill_paged(q, k, v, table, lens, cu, 1, 0.125))
    assert both(lambda m: m.attn_prefill_paged(q, k[:, :, ::2], v, table, lens, cu, 1, 0.125))[0] is AssertionError
    assert both(lambda m: m.attn_prefill_paged(q, k, v, table, lens, cu.long(), 1, 0.125))[0].__name__ == "B200Error"


def _forget_workspaces(m, monkeypatch):
    """as in a process that has made no call yet"""
    from tgis_b200 import _lib
    monkeypatch.setattr(m, "_gemm_ws", {})
    if not isinstance(m._host, _Nothing):
        m._host = None
        m._native()


def test_first_calls_inside_a_capture(both, monkeypatch):
    """A workspace that has to be made while a stream is captured belongs to the graph, whose replays zero its counters: a call ahead of the first replay gets
    another one."""
    x = _r(4, 2048) if both.name == "ops" else _r(4, 2048, dtype=torch.bfloat16)
    w = _r(2048, 2048, dtype=x.dtype)

    def call(m):
        f = m.gemm_f16 if both.name == "ops" else m.linear
        _forget_workspaces(m, monkeypatch)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y, z = f(x, w), f(x, w)
        assert not m._gemm_ws
        eager = f(x, w)
        graph.replay()
        torch.cuda.synchronize()
        assert len(m._gemm_ws) == 1 and torch.equal(y, eager) and torch.equal(z, eager)
        return y.clone()
    both(call)


def test_a_workspace_grows(both, monkeypatch):
    x = _r(4, 2048) if both.name == "ops" else _r(4, 2048, dtype=torch.bfloat16)
    wide, narrow = _r(20480, 2048, dtype=x.dtype), _r(128, 2048, dtype=x.dtype)

    def call(m):
        f = m.gemm_f16 if both.name == "ops" else m.linear
        _forget_workspaces(m, monkeypatch)
        got, sizes = [], []
        for w in (narrow, wide, narrow):
            got.append(f(x, w))
            sizes.append([t.numel() for t in m._gemm_ws.values()])
        assert len(sizes[0]) == 1 and sizes[0][0] < sizes[1][0] == sizes[2][0] and torch.equal(got[0], got[2])
        return torch.cat(got, 1)
    both(call)


def test_calls_from_several_threads(both, monkeypatch):
    """each thread on a stream of its own, with workspaces of its own, sizes that differ"""
    import threading
    dt = torch.float16 if both.name == "ops" else torch.bfloat16
    xs, ws = [_r(2 + i, 2048, dtype=dt) for i in range(4)], [_r(128 << i, 2048, dtype=dt) for i in range(4)]
    torch.cuda.synchronize()

    def call(m):
        got, wrong = [None] * 4, []
        want = [m.gemm_f16(x, w) if both.name == "ops" else m.linear(x, w) for x, w in zip(xs, ws)]
        torch.cuda.synchronize()

        def work(i):
            try:
                with torch.cuda.stream(torch.cuda.Stream()):
                    mine = m.gemm_workspace(torch.device(DEV), 8, 1024, 2048).clone() if both.name == "ops" else None
                    for _ in range(50):
                        got[i] = m.gemm_f16(xs[i], ws[i], workspace=mine) if both.name == "ops" else m.linear(xs[i].float(), ws[i].float())
                    torch.cuda.current_stream().synchronize()
            except Exception as e:
                wrong.append(e)
        threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong
        if both.name == "ops":
            assert all(torch.equal(a, b) for a, b in zip(got, want))
        return torch.cat([g.flatten() for g in got])
    both(call)


@pytest.mark.parametrize("entry", ["gemm_f16", "gemm_w4a16", "linear_bf16", "attn_decode_paged"])
def test_workspace_lives_until_the_entry_returns(entry):
    """While an entry runs, other threads may make a call that needs a larger workspace, which replaces the first: its memory is not given to
    anybody else before the entry has returned.  The entries are functions of this test, which launch nothing."""
    import ctypes

    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib, ops, ops_seq
    which = int(entry == "linear_bf16")
    seen = []
    need = [1 << 20]

    def run(*a):
        ws = {"gemm_f16": 7, "gemm_w4a16": 10, "linear_bf16": 8, "attn_decode_paged": 9}[entry]
        if need[0] == 1 << 20:
            need[0] = 1 << 21
            call()                                                                       # as another thread's larger call
            others = [torch.empty(1 << 20, dtype=torch.uint8, device=DEV) for _ in range(64)]   # who asks now must not get the first one's memory
            seen.append((a[ws], [t.data_ptr() for t in others]))
        return 0

    P, L, I, F = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int, ctypes.c_float
    types = {"gemm_f16": [P, P, P, P, L, L, L, P, P], "gemm_w4a16": [P, P, P, P, L, L, L, I, I, I, P, P], "linear_bf16": [P, P, P, P, I, L, L, L, P, P],
             "attn_decode_paged": [P, L, P, P, P, L, P, P, L, P, L, I, I, I, I, I, F, P]}[entry]
    fns = [ctypes.CFUNCTYPE(I, *types)(run), ctypes.CFUNCTYPE(L, L, L)(lambda n, k: 1 << 20 if n == 64 else 1 << 21),
           ctypes.CFUNCTYPE(L, I, I, I, I)(lambda b, h, d, most: need[0])]
    names = [{"gemm_f16": "b200_gemm_f16", "gemm_w4a16": "b200_gemm_w4a16_ex", "linear_bf16": "b200_gemm_bf16", "attn_decode_paged": "b200_attn_decode_paged"}[entry],
             "b200_gemm_workspace_bytes_max", "b200_attn_decode_workspace_bytes"]
    host = (ops_seq if which else ops)._native()
    held = {}

    def make(like, *a):
        held["ws"] = torch.zeros(a[0] if len(a) == 1 else 1 << 20 if a[0] == 64 else 1 << 21, dtype=torch.uint8, device=DEV)
        return held["ws"]

    x, q = _r(2, 64), _r(2, 4, 64)
    pool, table, lens = _r(3, 2, 16, 64), torch.zeros(2, 2, dtype=torch.int32, device=DEV), torch.ones(2, dtype=torch.int32, device=DEV)

    def call():
        N = 64 if need[0] == 1 << 20 else 128
        w = _r(N, 64)
        if entry == "gemm_f16":
            return host.gemm_f16(x, w, None, None, None)
        if entry == "gemm_w4a16":
            return host.gemm_w4a16(x, torch.empty(64, dtype=torch.uint8, device=DEV), N, 64, None, None, None, 0, False)
        if entry == "linear_bf16":
            return host.linear_bf16(x.bfloat16(), w.bfloat16(), None, 0)
        return host.attn_decode_paged(q, pool, pool, table, lens, 20, 0.125, 2, None, None)

    try:
        torch.cuda.empty_cache()
        host.bind(which, {n: ctypes.cast(f, P).value for n, f in zip(names, fns)}, make, make)
        assert call() is not None
    finally:
        for m in (ops, ops_seq):
            m._host = None
            m._native()
    (used, taken), = seen
    assert not [t for t in taken if abs(t - used) < 1 << 20]
