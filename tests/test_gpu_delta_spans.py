"""Gated delta rule in spans of sixteen tokens (csrc/delta_spans.cuh): steps of 96 or more tokens per sequence (192 on grids that fill the chip), key sizes 64 and 128, values in
multiples of 32.  Sequences that end inside, with and behind a span, behind cached tokens and fresh on slots full of garbage, more than 32 sequences, an odd
number of heads, a decay per head or per key channel with zeros and ones, values that are not finite, records in several parts.  Reference: float64.

Tolerance: that of the chain over four tokens (test_gpu_delta_prompts.py)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(g, lens, H, G, dk, dv, channels):
    T, n_dec = sum(lens), H * dk if channels else H
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, dk, generator=g, device=DEV), dim=-1) for _ in range(2))
    v, decay, beta = torch.randn(T, H, dv, generator=g, device=DEV), torch.rand(T, n_dec, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV)
    decay[:, ::5], decay[:, 1::7] = 0.0, 1.0
    decay[torch.rand(T, n_dec, generator=g, device=DEV) < 0.7] = 0.99
    return q, k, v, decay, beta


def _rows(q, k, v, decay, beta):
    x = torch.cat([q.flatten(1), k.flatten(1), v.flatten(1), decay, beta], 1)
    return torch.nn.functional.pad(x, (0, -x.shape[1] % 4)).contiguous()


def _step(starts, lens, slots):
    from tgis_b200 import ops_seq
    return ops_seq.RaggedStep(T=sum(lens), B=len(lens), position_ids=torch.cat([torch.arange(s, s + n, device=DEV) for s, n in zip(starts, lens)]),
                              cu_q=torch.tensor([0] + list(lens), device=DEV).cumsum(0).int(), slot_mapping=torch.zeros(sum(lens), dtype=torch.int64, device=DEV),
                              seq_of_token=torch.repeat_interleave(torch.arange(len(lens), device=DEV, dtype=torch.int32), torch.tensor(lens, device=DEV)),
                              block_table=torch.zeros(len(lens), 1, dtype=torch.int32, device=DEV), state_slots=torch.tensor(slots, dtype=torch.int32, device=DEV))


def _exact(q, k, v, decay, beta, S0, lens):
    """float64, all sequences side by side -> y [T, H, dv], S [B, H, dk, dv]; tokens behind a sequence's end neither decay nor write"""
    B, L, H = len(lens), max(lens), v.shape[1]
    live = torch.arange(L, device=DEV)[None] < torch.tensor(lens, device=DEV)[:, None]

    def padded(x, fill):
        out = torch.full((B, L, *x.shape[1:]), fill, dtype=torch.float64, device=DEV)
        out[live] = x.double()
        return out

    rep = H // q.shape[1]
    Q, K = padded(q, 0.0).repeat_interleave(rep, 2), padded(k, 0.0).repeat_interleave(rep, 2)
    V, D, Bt = padded(v, 0.0), padded(decay, 1.0).unflatten(2, (H, -1)), padded(beta, 0.0)
    S, y = S0.double(), torch.zeros(B, L, H, v.shape[2], dtype=torch.float64, device=DEV)
    for t in range(L):
        S = D[:, t, :, :, None] * S
        S = S + K[:, t, :, :, None] * (Bt[:, t, :, None] * (V[:, t] - (K[:, t, :, None] @ S)[:, :, 0]))[:, :, None]
        y[:, t] = (Q[:, t, :, None] @ S)[:, :, 0]
    return y[live], S


def _scan(x, S, st, H, G, dk, dv, channels):
    from tgis_b200 import _lib, ops_seq as ops
    assert _lib.load_seq().b200_seq_delta_rows_scan_bytes(st.T, st.B, H, dk, dv) > 0
    return ops.delta_rows_scan(_rows(*x), S, st, H, G, dk, dv, channels).unflatten(1, (H, dv)).double()


def _close(got, want):
    return float((got - want).abs().max()) < 2e-5 * max(1.0, float(want.abs().max()))


SOME = [1, 15, 16, 17, 260, 4, 500, 31]
MANY = [5, 33, 900, 16] * 10


@pytest.mark.parametrize("H,G,dk,dv,channels,lens", [(3, 1, 64, 32, True, SOME), (2, 2, 128, 128, True, SOME), (4, 2, 128, 64, False, SOME), (3, 3, 64, 96, False, SOME),
                                                     (1, 1, 128, 32, True, MANY), (2, 1, 64, 64, False, [257])])
def test_spans(H, G, dk, dv, channels, lens):
    import tgis_b200  # noqa: F401
    g = torch.Generator(device=DEV).manual_seed(H + dk + dv)
    x, B = _inputs(g, lens, H, G, dk, dv, channels), len(lens)
    slots = [B + 1 - i for i in range(B)]
    S0 = torch.randn(B + 2, H, dk, dv, generator=g, device=DEV)
    starts = [0 if i % 3 == 1 else 16 + i for i in range(B)]
    for i in range(B):
        if starts[i] == 0:
            S0[slots[i]] = float("nan")   # a fresh sequence never reads its slot
    S = S0.clone()
    y = _scan(x, S, _step(starts, lens, slots), H, G, dk, dv, channels)
    want, S_want = _exact(*x, S0[slots].nan_to_num(0.0), lens)
    assert _close(y, want) and _close(S[slots].double(), S_want)
    assert torch.equal(S[0], S0[0]) and torch.equal(S[1], S0[1])


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_value_reaches_its_own_column_from_its_token_on(bad):
    import tgis_b200  # noqa: F401
    H, G, dk, dv, lens, at = 2, 1, 128, 64, [250, 130], 37
    g = torch.Generator(device=DEV).manual_seed(5)
    x, S0 = _inputs(g, lens, H, G, dk, dv, True), torch.randn(2, H, dk, dv, generator=g, device=DEV)
    clean, S = S0.clone(), S0.clone()
    want = _scan(x, clean, _step([16, 16], lens, [0, 1]), H, G, dk, dv, True)
    x[2][at, 1, 9] = bad
    y = _scan(x, S, _step([16, 16], lens, [0, 1]), H, G, dk, dv, True)
    hit = torch.zeros_like(y, dtype=torch.bool)
    hit[at:250, 1, 9] = True
    assert torch.equal(y[~hit], want[~hit]) and not bool(y[at, 1, 9].isfinite())
    assert torch.equal(S[1], clean[1])


def test_records_in_parts():
    """one prompt whose records take more than the room for them: the second part goes on where the first ended"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib
    H, G, dk, dv, lens = 256, 1, 64, 32, [9500]
    bytes_of = _lib.load_seq().b200_seq_delta_rows_scan_bytes
    assert bytes_of(9500, 1, H, dk, dv) == bytes_of(12000, 1, H, dk, dv) > bytes_of(8000, 1, H, dk, dv) > 0
    g = torch.Generator(device=DEV).manual_seed(7)
    x, S = _inputs(g, lens, H, G, dk, dv, False), torch.full((1, H, dk, dv), float("nan"), device=DEV)
    y = _scan(x, S, _step([0], lens, [0]), H, G, dk, dv, False)
    want, S_want = _exact(*x, torch.zeros(1, H, dk, dv, device=DEV), lens)
    assert _close(y, want) and _close(S.double(), S_want)


def _scan_in(x, S, st, H, G, dk, dv, channels, spans):
    """with room for so many spans' records"""
    import ctypes
    from tgis_b200 import _lib
    lib, rows = _lib.load_seq(), _rows(*x)
    room = spans * (lib.b200_seq_delta_rows_scan_bytes(500, 1, H, dk, dv) // (500 // 16 + 1))
    ws, y = torch.empty(room, dtype=torch.uint8, device=DEV), torch.full((st.T, H * dv), 9.0, device=DEV)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check_seq(lib.b200_seq_delta_rows_scan_in(p(rows), int(channels), p(S), p(st.state_slots), p(st.cu_q), p(st.position_ids), p(y), H * dv, st.T, st.B, H, G, dk,
                                                   dv, p(ws), room, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "rows_scan_in")
    return y


@pytest.mark.parametrize("lens", [[1, 1030, 16, 0, 2100, 17, 1020, 500], [5, 33, 900, 16, 0] * 9, [3000, 1], [1, 1, 1, 1700]])
@pytest.mark.parametrize("H,G,dk,dv,channels", [(3, 1, 64, 32, True), (2, 1, 128, 64, False)])
def test_parts_of_several_sequences(lens, H, G, dk, dv, channels):
    """sequences that end in an earlier part, go over from one to the next, or begin in the last: the same bits as in one part, states included"""
    import tgis_b200  # noqa: F401
    g = torch.Generator(device=DEV).manual_seed(len(lens))
    x, B = _inputs(g, lens, H, G, dk, dv, channels), len(lens)
    S0 = torch.randn(B, H, dk, dv, generator=g, device=DEV)
    starts = [0 if i % 3 == 1 else 16 + i for i in range(B)]
    st = _step(starts, lens, list(range(B)))
    whole = S0.clone()
    want = _scan_in(x, whole, st, H, G, dk, dv, channels, sum(lens) // 16 + B)
    assert _close(want.unflatten(1, (H, dv)).double(), _exact(*x, torch.where(torch.tensor([s == 0 for s in starts], device=DEV)[:, None, None, None], 0.0, S0), lens)[0])
    for spans in (64, 65, 100, sum(lens) // 16 + B - 1):
        S = S0.clone()
        assert torch.equal(_scan_in(x, S, st, H, G, dk, dv, channels, spans), want) and torch.equal(S, whole)
    S = S0.clone()   # too little room: four tokens at a time
    assert _close(_scan_in(x, S, st, H, G, dk, dv, channels, 63).double(), want.double()) and _close(S.double(), whole.double())


def test_no_room_at_all(monkeypatch):
    """a step whose records cannot be had goes four tokens at a time, as it did before there were any"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq
    H, G, dk, dv, lens = 2, 1, 128, 64, [250, 130]
    g = torch.Generator(device=DEV).manual_seed(5)
    x, S0 = _inputs(g, lens, H, G, dk, dv, True), torch.randn(2, H, dk, dv, generator=g, device=DEV)
    st, got, empty, asked = _step([16, 0], lens, [0, 1]), [], torch.empty, []
    for most in (1 << 40, 0):
        def some(*a, **k):
            if k.get("dtype") == torch.uint8:
                asked.append(a[0])
                if a[0] > most:
                    raise torch.cuda.OutOfMemoryError("out of memory")
            return empty(*a, **k)
        monkeypatch.setattr(ops_seq.torch, "empty", some)
        S = S0.clone()
        got.append((_scan(x, S, st, H, G, dk, dv, True), S.double()))
        monkeypatch.undo()
    assert len(asked) == 3 and asked[0] == asked[1] == 8 * asked[2]
    (a, Sa), (b, Sb) = got
    assert _close(b, a) and _close(Sb, Sa)
