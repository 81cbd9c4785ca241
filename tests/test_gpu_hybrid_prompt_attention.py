"""Prompts over token-major bfloat16 pages (csrc/attn_prompt.cuh behind ops_seq.talk_attn): tiles of 128 (token, head) rows for every head ratio, chunk
borders inside a tile, windows whose first key tile some rows do not see, sinks, portions behind cached tokens, single tokens among prompts, more
items than SMs, and the forms beside it that stay with the general kernels.  Reference: float64.

Tolerance: queries are given as bfloat16 values, so products are exact; a weight is rounded to bfloat16 once (2^-9 of it) and the sum adds the
rounded weights: 2 * 2^-9 of the weighted mean of |v|, and d 2^-24 of the largest score times the weight's slope for the fp32 sums."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(new, past, H, G, d, chunk=0, window=0, sink=None, page=16, dv=None, pad=0, seed=0, key_scale=1.0, width=0):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq
    g = torch.Generator(device=DEV).manual_seed(seed)
    dv = dv or d
    starts = past if isinstance(past, list) else [past] * len(new)
    L = [s + n for s, n in zip(starts, new)]
    pages = [(n + page - 1) // page for n in L]
    perm = torch.randperm(sum(pages) + 2, generator=g, device=DEV).int()
    table, at = torch.zeros(len(new), max(max(pages), width), dtype=torch.int32, device=DEV), 0
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    k_off, v_off = pad, pad + G * d + pad
    width = v_off + G * dv + pad
    cache = (torch.randn(sum(pages) + 2, page, width, generator=g, device=DEV) * key_scale).bfloat16()
    T = sum(new)
    q = torch.randn(T, H, d, generator=g, device=DEV).bfloat16().float()
    pos = torch.cat([torch.arange(s, s + n, device=DEV) for s, n in zip(starts, new)])
    cu = torch.tensor([0] + new, device=DEV).cumsum(0).int()
    seq = torch.repeat_interleave(torch.arange(len(new), device=DEV, dtype=torch.int32), torch.tensor(new, device=DEV))
    step = ops_seq.RaggedStep(T=T, B=len(new), position_ids=pos, cu_q=cu, seq_of_token=seq, slot_mapping=pos, block_table=table, state_slots=None)
    out = ops_seq.talk_attn(q, cache, step, kv_heads=G, vdim=dv, k_off=k_off, v_off=v_off, scale=d ** -0.5, chunk=chunk, window=window, sink=sink)
    row = 0
    for b, (n, s0, Lb) in enumerate(zip(new, starts, L)):
        rows = cache[table[b, :pages[b]].long()].flatten(0, 1)[:Lb].double()
        K, V = rows[:, k_off:k_off + G * d].unflatten(1, (G, d)), rows[:, v_off:v_off + G * dv].unflatten(1, (G, dv))
        p, j = s0 + torch.arange(n, device=DEV)[:, None], torch.arange(Lb, device=DEV)[None]
        ok = j <= p
        if chunk:
            ok = ok & (j // chunk == p // chunk)
        if window:
            ok = ok & (j > p - window)
        for h in range(H):
            s = (q[row:row + n, h].double() @ K[:, h * G // H].T * d ** -0.5).masked_fill(~ok, -math.inf)
            top = s.masked_fill(~ok, 0).abs().amax(1, keepdim=True)
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(n, 1)], 1)
            w = torch.softmax(s, 1)[:, :Lb]
            ref, spread = w @ V[:, h * G // H], w @ V[:, h * G // H].abs()
            tol = (2 * 2.0 ** -9 + 2 * d * 2.0 ** -24 * (1 + top)) * spread + 1e-6
            err = (out[row:row + n, h].double() - ref).abs()
            assert bool((err <= tol).all()), (b, h, float((err / tol).max()), int((err > tol).sum()))
        row += n


@pytest.mark.parametrize("H,G,d", [(4, 4, 64), (4, 2, 128), (16, 4, 128), (8, 1, 64), (16, 1, 128), (6, 2, 64)])   # (6, 2): three heads a key head, the general kernel
def test_head_ratios(H, G, d):
    _run([1, 31, 32, 33, 64, 65, 129, 200], 0, H, G, d)
    _run([100, 3, 77], [5, 400, 128], H, G, d, seed=1)


@pytest.mark.parametrize("chunk,window", [(64, 0), (100, 0), (0, 1), (0, 40), (0, 130), (200, 50), (2048, 0)])
def test_masks(chunk, window):
    _run([300, 90], [0, 170], 8, 2, 64, chunk=chunk, window=window, seed=2)
    _run([150], 2000, 4, 1, 128, chunk=chunk, window=window, seed=3)


def test_sinks():
    g = torch.Generator(device=DEV).manual_seed(4)
    sink = torch.randn(8, generator=g, device=DEV) * 3
    sink[0], sink[1], sink[2] = 40.0, -40.0, -math.inf
    _run([70, 200], [0, 300], 8, 2, 128, sink=sink, seed=5)
    _run([140], 0, 8, 2, 64, window=30, sink=sink, seed=6)


def test_more_items_than_sms():
    _run([25 + 13 * (i % 7) for i in range(60)], [17 * (i % 5) for i in range(60)], 16, 8, 64, chunk=128, seed=7)


def test_long_items_and_short_ones_in_turn():
    _run([1500, 1, 700, 130, 40, 900], 0, 16, 4, 64, seed=13)   # items of one key tile and of many, several to a block
    _run([300] * 9 + [1], [0, 900] * 5, 8, 8, 64, chunk=512, seed=14)


@pytest.mark.parametrize("past,window,chunk", [(0, 33, 0), (31, 64, 0), (65, 95, 0), (96, 0, 160), (33, 130, 288)])
def test_borders_inside_a_key_tile(past, window, chunk):
    _run([33, 97, 160, 1], past, 8, 2, 64, chunk=chunk, window=window, seed=15)
    _run([130, 63], past, 16, 1, 128, chunk=chunk, window=window, seed=16)


def test_maxima_that_leap():
    _run([700], 0, 4, 2, 128, key_scale=6.0, seed=8)


@pytest.mark.parametrize("kw", [dict(page=32), dict(dv=128), dict(pad=4), dict(pad=8)])   # other pages, value sizes, offsets (the last one stays with the tcgen05 kernel)
def test_forms_beside_it(kw):
    _run([60, 130], [0, 20], 4, 2, 64, seed=9, **kw)


@pytest.mark.parametrize("d,H,G", [(64, 8, 2), (128, 16, 4)])
@pytest.mark.parametrize("new,past,chunk,window", [([1, 40, 128, 150], [0, 0, 0, 0], 0, 0), ([70, 33, 300], [5, 1003, 130], 0, 0), ([100, 40], [500, 37], 0, 45),
                                                   ([90, 200], [333, 1000], 128, 0), ([60, 24], [2041, 700], 200, 77)])
def test_what_no_query_sees_does_not_matter(d, H, G, new, past, chunk, window):
    """slots that no query of the step sees - behind a sequence's last key, ahead of its first visible one, blocks of no sequence - and table
    entries of pages without a visible key: NaN and Inf there change no bit of the result"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq
    g = torch.Generator(device=DEV).manual_seed(d + sum(new))
    L = [s + n for s, n in zip(past, new)]
    pages = [(n + 15) // 16 for n in L]
    blocks = sum(pages) + 3
    perm = torch.randperm(blocks, generator=g, device=DEV).int()
    spare = perm[-1]
    table, at = torch.full((len(new), max(pages) + 2), int(spare), dtype=torch.int32, device=DEV), 0
    seen = torch.zeros(blocks, 16, dtype=torch.bool, device=DEV)
    for b, n in enumerate(pages):
        p = past[b]
        lo = max(p // chunk * chunk if chunk else 0, p - window + 1 if window else 0)
        first = lo // 16
        table[b, first:n] = perm[at + first:at + n]
        at += n
        j = torch.arange(lo, L[b], device=DEV)
        seen[table[b, j // 16].long(), j % 16] = True
    cache = torch.randn(blocks, 16, 2 * G * d, generator=g, device=DEV).bfloat16()
    q = torch.randn(sum(new), H, d, generator=g, device=DEV)
    pos = torch.cat([torch.arange(s, e, device=DEV) for s, e in zip(past, L)])
    cu = torch.tensor([0] + new, device=DEV).cumsum(0).int()
    seq = torch.repeat_interleave(torch.arange(len(new), device=DEV, dtype=torch.int32), torch.tensor(new, device=DEV))
    step = ops_seq.RaggedStep(T=sum(new), B=len(new), position_ids=pos, cu_q=cu, seq_of_token=seq, slot_mapping=pos, block_table=table, state_slots=None)

    def run(c):
        return ops_seq.talk_attn(q, c, step, kv_heads=G, vdim=d, k_off=0, v_off=G * d, scale=d ** -0.5, chunk=chunk, window=window)

    clean = run(cache)
    assert bool(clean.isfinite().all())
    for bad in (math.nan, math.inf):
        assert torch.equal(run(torch.where(seen[..., None], cache, torch.full_like(cache, bad))), clean)


def _fp32_case(H, G, d, new, seed, held=False):
    """queries that bfloat16 does not hold (`held`: that it does); -> call, largest difference to float64, the same relative to the weighted mean of |v|"""
    from tgis_b200 import ops_seq
    g = torch.Generator(device=DEV).manual_seed(seed)
    pages = [(n + 15) // 16 for n in new]
    table, at = torch.zeros(len(new), max(pages), dtype=torch.int32, device=DEV), 0
    for b, n in enumerate(pages):
        table[b, :n] = torch.arange(at, at + n, device=DEV, dtype=torch.int32)
        at += n
    cache = torch.randn(at, 16, 2 * G * d, generator=g, device=DEV).bfloat16()
    q = torch.randn(sum(new), H, d, generator=g, device=DEV)
    q = q.bfloat16().float() if held else q
    pos = torch.cat([torch.arange(n, device=DEV) for n in new])
    seq = torch.repeat_interleave(torch.arange(len(new), device=DEV, dtype=torch.int32), torch.tensor(new, device=DEV))
    step = ops_seq.RaggedStep(T=sum(new), B=len(new), position_ids=pos, cu_q=torch.tensor([0] + new, device=DEV).cumsum(0).int(), seq_of_token=seq,
                              slot_mapping=pos, block_table=table, state_slots=None)
    out = ops_seq.talk_attn(q, cache, step, kv_heads=G, vdim=d, k_off=0, v_off=G * d, scale=d ** -0.5).double()
    worst, row = 0.0, 0
    for b, n in enumerate(new):
        rows = cache[table[b, :pages[b]].long()].flatten(0, 1)[:n].double()
        K, V = rows[:, :G * d].unflatten(1, (G, d)).repeat_interleave(H // G, 1), rows[:, G * d:].unflatten(1, (G, d)).repeat_interleave(H // G, 1)
        s = torch.einsum("nhd,lhd->hnl", q[row:row + n].double(), K) * d ** -0.5
        w = torch.softmax(s.masked_fill(torch.arange(n, device=DEV)[None] > torch.arange(n, device=DEV)[:, None], -math.inf), -1)
        ref, spread = torch.einsum("hnl,lhd->nhd", w, V), torch.einsum("hnl,lhd->nhd", w, V.abs())
        worst = max(worst, float(((out[row:row + n] - ref).abs() / spread).max()))
        row += n
    return worst


@pytest.mark.parametrize("H,G,d", [(16, 16, 128), (32, 16, 128), (24, 24, 64), (64, 16, 128), (32, 32, 64)])
def test_shapes_that_are_computed_in_fp32(H, G, d):
    """shapes that the m16n8k16 kernel does not take keep fp32 queries, weights and sums on the general kernel.  Bound: d 2^-24 of a score of size
    up to ~6 (its error is the weight's relative one), and the sums over 150 keys"""
    import tgis_b200  # noqa: F401
    assert _fp32_case(H, G, d, [150, 40], H + d) < (6 * d + 150) * 2.0 ** -24 * 2


@pytest.mark.parametrize("H,G,d", [(16, 4, 128), (8, 2, 64), (32, 8, 128)])
def test_weights_are_not_rounded_to_bfloat16(H, G, d):
    """queries that bfloat16 holds leave the weights as the only 16-bit operand: two bfloat16 values each, 2^-17 off, beside the fp32 terms above"""
    import tgis_b200  # noqa: F401
    assert _fp32_case(H, G, d, [300, 40], d, held=True) < 2 * 2.0 ** -17 + (6 * d + 300) * 2.0 ** -24 * 2


def test_the_switch_for_fp32():
    """B200_SEQ_ATTN_MMA=0 selects the fp32 form for prompts as well (read once per process: a process of its own)"""
    import os
    import subprocess
    import sys
    code = "import torch, tests.test_gpu_hybrid_prompt_attention as t; import tgis_b200; print(t._fp32_case(16, 4, 128, [150, 40], 1))"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    worst = [float(subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, B200_SEQ_ATTN_MMA=v), check=True, capture_output=True, text=True).stdout)
             for v in ("0", "1")]
    assert worst[0] < (6 * 128 + 150) * 2.0 ** -24 * 2 < worst[1]


@pytest.mark.parametrize("new,H,G", [([600, 500], 16, 4), ([560, 600], 16, 4), ([31, 33, 64, 65, 1, 96], 16, 4), ([40] * 11, 8, 8), ([40] * 9, 8, 8)])
def test_around_one_tile_per_sm(new, H, G):
    """steps whose tiles each have an item to themselves, and steps just above that"""
    _run(new, 0, H, G, 64, seed=10)
    _run(new, 100, H, G, 64, chunk=256, seed=11)


@pytest.mark.parametrize("chunk,window,sink", [(0, 0, False), (512, 0, True), (0, 300, False)])
def test_few_queries_over_a_long_cache(chunk, window, sink):
    """the same steps on both sides of the rule that leaves few items over many keys to the kernel that cuts the keys into runs (the host takes the
    block table's width for the number of keys)"""
    s = torch.linspace(-2, 2, 8, device=DEV) if sink else None
    for width in (0, 4000):
        _run([64, 24], [3000, 700], 8, 2, 64, chunk=chunk, window=window, sink=s, seed=12, width=width)
        _run([30], [5000], 8, 2, 128, chunk=chunk, window=window, sink=s, seed=13, width=width)
