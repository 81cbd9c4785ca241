"""Attention of few queries over runs of keys (csrc/seq_talk_attn.cu, talk_attn_mma_kernel and its merge): up to 32 runs, more runs than there are keys,
chunks and windows that leave some of them empty, sinks that count once, several tokens of unlike sequences, with and without a mix of heads, queries that
are not 16-byte aligned.  Reference: float64.

Tolerance: queries, keys' products and weights round to bfloat16 (2^-9 each); 4e-3 of the result's 2-norm is twice what one of them alone can do."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 16


def _step(new, past):
    from tgis_b200 import ops_seq
    ends = [p + n for p, n in zip(past, new)]
    pages = [(e + PAGE - 1) // PAGE for e in ends]
    table = torch.zeros(len(new), max(pages), dtype=torch.int32, device=DEV)
    perm, at = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(3)).int().to(DEV), 0
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    return ops_seq.RaggedStep(T=sum(new), B=len(new), position_ids=torch.cat([torch.arange(p, e, device=DEV) for p, e in zip(past, ends)]),
                              cu_q=torch.tensor([0] + new, device=DEV).cumsum(0).int(), block_table=table, slot_mapping=torch.zeros(sum(new), dtype=torch.int64, device=DEV),
                              seq_of_token=torch.repeat_interleave(torch.arange(len(new), device=DEV, dtype=torch.int32), torch.tensor(new, device=DEV)),
                              state_slots=torch.arange(len(new), dtype=torch.int32, device=DEV)), sum(pages)


def _exact(q, cache, step, new, past, G, d, scale, chunk, window, sink, talk):
    H, out, at = q.shape[1], torch.empty(q.shape, dtype=torch.float64, device=DEV), 0
    for b, (n, p0) in enumerate(zip(new, past)):
        L = p0 + n
        rows = cache[step.block_table[b].long()].flatten(0, 1)[:L].double()
        K, V = (rows[:, o:o + G * d].unflatten(1, (G, d)).repeat_interleave(H // G, 1) for o in (0, G * d))
        s = torch.einsum("thd,jhd->htj", q[at:at + n].double(), K) * scale
        if talk is not None:
            s = torch.einsum("hg,gtj->htj", talk.double(), s)
        p, j = torch.arange(p0, L, device=DEV)[:, None], torch.arange(L, device=DEV)[None]
        ok = j <= p
        if chunk:
            ok = ok & (j // chunk == p // chunk)
        if window:
            ok = ok & (j > p - window)
        s = s.masked_fill(~ok, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None, None].expand(H, n, 1)], 2)
        out[at:at + n] = torch.einsum("htj,jhd->thd", torch.softmax(s, -1)[:, :, :L], V)
        at += n
    return out


@pytest.mark.parametrize("new,past", [([1], [0]), ([1], [40]), ([1], [1000]), ([1, 1, 1], [5, 700, 64]), ([3, 6, 4], [1500, 90, 31]), ([7], [513]), ([1] * 30, [60] * 30)])
@pytest.mark.parametrize("chunk,window,with_sink", [(0, 0, False), (512, 0, True), (0, 100, False), (0, 33, True)])
@pytest.mark.parametrize("H,G,d", [(16, 4, 128), (8, 8, 64), (32, 8, 128)])
def test_runs(new, past, chunk, window, with_sink, H, G, d):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    g = torch.Generator(device=DEV).manual_seed(sum(new) + sum(past) + H)
    step, blocks = _step(new, past)
    cache = torch.randn(blocks, PAGE, 2 * G * d, generator=g, device=DEV).bfloat16()
    q = torch.randn(sum(new), H, d, generator=g, device=DEV)
    sink = torch.randn(H, generator=g, device=DEV) if with_sink else None
    talk = torch.eye(H, device=DEV) + 0.2 * torch.randn(H, H, generator=g, device=DEV)
    shifted = torch.empty(q.numel() + 1, device=DEV)[1:].view(q.shape).copy_(q)
    for mix in (None, talk):
        want = _exact(q, cache, step, new, past, G, d, d ** -0.5, chunk, window, sink, mix)
        for x in (q, shifted):
            got = ops.talk_attn(x, cache, step, kv_heads=G, vdim=d, k_off=0, v_off=G * d, scale=d ** -0.5, talk=mix, chunk=chunk, window=window, sink=sink).double()
            assert float((got - want).norm()) <= 4e-3 * float(want.norm()) * (1.5 if mix is not None else 1.0)


@pytest.mark.parametrize("new,past", [([1], [1000]), ([2, 1], [900, 90])])
@pytest.mark.parametrize("chunk,window", [(0, 0), (512, 0), (0, 100)])
@pytest.mark.parametrize("which", ["keys", "one head's keys", "values"])
def test_what_is_not_a_number_shows(new, past, chunk, window, which):
    """Keys of four whole pages, which are whole runs, are NaN: every row that sees one of them is NaN, the others are as without."""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    H, G, d = 16, 4, 128
    g = torch.Generator(device=DEV).manual_seed(7)
    step, blocks = _step(new, past)
    cache = torch.randn(blocks, PAGE, 2 * G * d, generator=g, device=DEV).bfloat16()
    q = torch.randn(sum(new), H, d, generator=g, device=DEV)
    at = {"keys": slice(0, G * d), "one head's keys": slice(d, 2 * d), "values": slice(G * d, 2 * G * d)}[which]
    cache[step.block_table[0, 40:44].long(), :, at] = float("nan")   # tokens 640 .. 703 of the first sequence
    call = lambda mix: ops.talk_attn(q, cache, step, kv_heads=G, vdim=d, k_off=0, v_off=G * d, scale=d ** -0.5, talk=mix, chunk=chunk, window=window).double()  # noqa: E731
    sees = window == 0   # the window of the first sequence's queries starts behind them
    for mix in (None, torch.eye(H, device=DEV) + 0.2 * torch.randn(H, H, generator=g, device=DEV)):
        nan = torch.zeros(sum(new), H, dtype=torch.bool, device=DEV)
        if sees:
            nan[:new[0]] = torch.ones(H, dtype=torch.bool, device=DEV) if which != "one head's keys" or mix is not None else torch.arange(H, device=DEV) // (H // G) == 1
        got = call(mix)
        assert torch.equal(got.isnan().all(-1), nan) and torch.equal(got.isnan().any(-1), nan)
        want = _exact(q, cache.nan_to_num(), step, new, past, G, d, d ** -0.5, chunk, window, None, mix)
        assert float((got - want)[~nan].norm()) <= 6e-3 * float(want[~nan].norm())
