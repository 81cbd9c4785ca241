"""Gated delta rule over steps of prompts (csrc/seq_delta.cu): the preparation over runs of sixteen tokens (steps of 384 tokens on, key sizes 64 and
128, up to four taps) with runs that end with their sequence, one token alone, inputs from the state behind cached tokens, two heads in a span,
dead lanes, a decay per head or per key channel; and the memory on both sides of the grid size that decides over its lanes.  Reference: float64.

Tolerances.  Preparation: a convolution of `taps` products, SiLU and a unit vector over dk channels, all fp32: (taps + dk / 32 + 16) 2^-24 of a value,
relative, and 4e-6 where the products of a convolution cancel (16 2^-22); decays are exp(-exp(a) softplus(x)), whose argument (up to ~40 here before the result vanishes) carries 4 * 2^-24: 2e-5 covers both.  Memory: the
bound of test_gpu_nomalorn.py's test_delta_memory_alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(spans, slots):
    from tgis_b200 import ops_seq
    new = [n for _, n in spans]
    return ops_seq.RaggedStep(T=sum(new), B=len(new), position_ids=torch.cat([torch.arange(s, s + n, device=DEV) for s, n in spans]),
                              cu_q=torch.tensor([0] + new, device=DEV).cumsum(0).int(), slot_mapping=torch.zeros(sum(new), dtype=torch.int64, device=DEV),
                              seq_of_token=torch.repeat_interleave(torch.arange(len(new), device=DEV, dtype=torch.int32), torch.tensor(new, device=DEV)),
                              block_table=torch.zeros(len(new), 1, dtype=torch.int32, device=DEV), state_slots=torch.tensor(slots, dtype=torch.int32, device=DEV))


def _prepared(u, raw, dec, conv_w, A_log, dt_bias, H, G, dk, channels):
    """a whole sequence's rows in float64: q | k | v | decays | write strengths"""
    L, taps = u.shape[0], conv_w.shape[0]
    padded = torch.cat([torch.zeros(taps - 1, u.shape[1], dtype=torch.float64, device=DEV), u.double()])
    c = sum(padded[j:j + L] * conv_w[j].double() for j in range(taps))
    c = c * torch.sigmoid(c)

    def unit(x):
        x = x.unflatten(1, (G, dk))
        return (x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)).flatten(1)

    rate = -A_log.double().exp()
    rate = rate.repeat_interleave(dk) if channels else rate
    decay = torch.exp(rate * torch.nn.functional.softplus(dec.double() + dt_bias.double()))
    return torch.cat([unit(c[:, :G * dk]) * dk ** -0.5, unit(c[:, G * dk:2 * G * dk]), c[:, 2 * G * dk:], decay, torch.sigmoid(raw.double())], 1)


SHAPES = [(4, 2, 64, 40, True), (3, 1, 64, 20, True), (3, 3, 128, 44, True), (4, 2, 128, 64, False), (3, 1, 64, 36, False)]


@pytest.mark.parametrize("H,G,dk,dv,channels", SHAPES)
@pytest.mark.parametrize("taps", [1, 2, 3, 4])
def test_preparation_over_runs(H, G, dk, dv, channels, taps):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    g = torch.Generator(device=DEV).manual_seed(taps * 100 + dk + dv)
    C, n_dec = 2 * G * dk + H * dv, H * dk if channels else H
    lens = [1, 15, 16, 17, 31, 5, 385, 50]
    conv_w, A_log, dt_bias = torch.randn(taps, C, generator=g, device=DEV), torch.randn(H, generator=g, device=DEV) * 0.5, torch.randn(n_dec, generator=g, device=DEV)
    # what the kernel is given: columns inside wider rows, at multiples of four
    wide = [torch.randn(n, 8 + C + 4 + n_dec + H, generator=g, device=DEV) for n in lens]
    want = [_prepared(w[:, 8:8 + C], w[:, 12 + C + n_dec:], w[:, 12 + C:12 + C + n_dec], conv_w, A_log, dt_bias, H, G, dk, channels) for w in wide]
    slots = [9, 0, 3, 7, 1, 2, 8, 5]
    # cut into two steps: the second one begins behind the state that the first one left
    for cuts in ([0] * 8, [1, 13, 0, 16, 2, 4, 3, 1], [0, 15, 1, 1, 30, 1, 1, 49]):
        state = torch.full((10, max(taps - 1, 1), C), float("nan"), device=DEV)
        got = [[] for _ in lens]
        for which in (0, 1):
            spans = [(0, c) if which == 0 else (c, n - c) for c, n in zip(cuts, lens)]
            at = [i for i, (_, n) in enumerate(spans) if n > 0]
            if not at:
                continue
            x = torch.cat([wide[i][spans[i][0]:sum(spans[i])] for i in at])
            st = _step([spans[i] for i in at], [slots[i] for i in at])
            x4 = torch.empty(x.shape[0], (x.shape[1] + 3) // 4 * 4, device=DEV)   # rows of a multiple of four columns
            x4[:, :x.shape[1]] = x
            rows = ops.delta_prepare(x4, 8, conv_w, state, x4, 12 + C + n_dec, x4, 12 + C, A_log, dt_bias, dk ** -0.5, st, H, G, dk, dv, channels)
            assert which == 0 or st.T >= 384
            row = 0
            for i in at:
                got[i].append(rows[row:row + spans[i][1], :want[i].shape[1]])
                row += spans[i][1]
        for i, n in enumerate(lens):
            y = torch.cat(got[i]).double()
            assert bool(((y - want[i]).abs() <= 2e-5 * want[i].abs() + 4e-6).all()), (cuts, i, float((y - want[i]).abs().max()))
            if taps > 1:
                last = torch.cat([torch.zeros(taps - 1, C, device=DEV), wide[i][:, 8:8 + C]])[-(taps - 1):]
                known = min(n, taps - 1)   # (entries before a sequence's first token are never read)
                assert torch.equal(state[slots[i], taps - 1 - known:], last[taps - 1 - known:]), (cuts, i)


@pytest.mark.parametrize("H,G,dk,dv", [(16, 8, 64, 128), (16, 4, 128, 128), (16, 16, 200, 128), (37, 1, 128, 64), (19, 1, 44, 126)])
@pytest.mark.parametrize("channels", [True, False])
def test_memory_on_both_sides_of_the_grid_rule(H, G, dk, dv, channels):
    """B H ceil(dv / 32) blocks of 32 columns: 32 lanes per memory column group up to 296, 16 above; the same sequences alone and among others"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    g = torch.Generator(device=DEV).manual_seed(H + dk + dv)
    per = H * ((dv + 31) // 32)
    many = 296 // per + 1
    assert many * per > 296 >= (many - 1) * per
    lens = [(3, 70, 1, 16, 29, 4, 18, 33)[i % 8] for i in range(many)]
    lay_v, n_dec = 2 * G * dk, H * dk if channels else H
    lib_width = (lay_v + H * dv + n_dec + H + 3) // 4 * 4
    T = sum(lens)
    rows = torch.zeros(T, lib_width, device=DEV)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, dk, generator=g, device=DEV), dim=-1) for _ in range(2))
    v, decay, beta = torch.randn(T, H, dv, generator=g, device=DEV), torch.rand(T, n_dec, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV)
    decay[:, ::5], decay[:, 1::7] = 0.0, 1.0
    rows[:, :lay_v + H * dv + n_dec + H] = torch.cat([q.flatten(1), k.flatten(1), v.flatten(1), decay, beta], 1)
    S0 = torch.randn(many, H, dk, dv, generator=g, device=DEV)
    # float64, all sequences side by side; tokens behind a sequence's end neither decay nor write
    L = max(lens)
    live = torch.arange(L, device=DEV)[None] < torch.tensor(lens, device=DEV)[:, None]

    def padded(x, fill):
        out = torch.full((many, L, *x.shape[1:]), fill, dtype=torch.float64, device=DEV)
        out[live] = x.double()
        return out

    rep = H // G
    Q, K = padded(q, 0.0).repeat_interleave(rep, 2), padded(k, 0.0).repeat_interleave(rep, 2)
    V, D, Bt = padded(v, 0.0), padded(decay, 1.0).unflatten(2, (H, -1)), padded(beta, 0.0)
    S, want = S0.double(), torch.zeros(many, L, H, dv, dtype=torch.float64, device=DEV)
    for t in range(L):
        S = D[:, t, :, :, None] * S
        S = S + K[:, t, :, :, None] * (Bt[:, t, :, None] * (V[:, t] - (K[:, t, :, None] @ S)[:, :, 0]))[:, :, None]
        want[:, t] = (Q[:, t, :, None] @ S)[:, :, 0]
    top = float(want.abs().max())
    for B in (many, many - 1):
        if B == 0:
            continue
        n = sum(lens[:B])
        state = S0.clone()
        st = _step([(16, m) for m in lens[:B]], list(range(B)))
        y = ops.delta_rows_scan(rows[:n].contiguous(), state, st, H, G, dk, dv, channels).unflatten(1, (H, dv)).double()
        assert float((y - want[live][:n]).abs().max()) < 2e-5 * max(1.0, top), B
        assert float((state[:B].double() - S[:B]).abs().max()) < 2e-5 * max(1.0, float(S.abs().max())), B
        assert torch.equal(state[B:], S0[B:])
