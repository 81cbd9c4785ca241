"""Prompt attention over the paged pool (csrc/attn_prefill_paged.cu) where its schedule could go wrong: more items than SMs, head groups that
pair heads and that pair query tiles (with and without a second tile), maxima that grow slowly, by leaps and late, scores of any sign of the
scale, and rows whose weights are all alike.  Reference: float64.

Tolerance: a weight is rounded to fp16 once (2^-11 of it), the sum normalises the rounded weights, so an output is off by at most 2 * 2^-11 of the
weighted mean of |v|, plus its own rounding; scores are fp32 sums of d products (d 2^-24 of the largest, times the weight's slope 1)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(lens, past, H, G, d, scale, shape_keys=None, seed=0):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(seed)
    L = [n + past for n in lens]
    pages = [(n + 15) // 16 for n in L]
    perm = torch.randperm(sum(pages) + 3, generator=g, device=DEV).int()
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32, device=DEV)
    shape = (sum(pages) + 3, G, 16, d)
    kp, vp = torch.randn(shape, generator=g, device=DEV).half(), torch.randn(shape, generator=g, device=DEV).half()
    T = sum(lens)
    q = torch.randn(T, (H + 2 * G) * d, generator=g, device=DEV).half()[:, :H * d].unflatten(1, (H, d))
    t, c = torch.arange(16, device=DEV)[:, None], torch.arange(d // 8, device=DEV)[None, :]
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
        if shape_keys is not None:   # a factor per key position
            f = shape_keys(torch.arange(n * 16, device=DEV)).view(n, 1, 16, 1)
            idx = table[b, :n].long()
            kp[idx] = (kp[idx].float() * f).half()
    out = torch.full((T, H, d), float("nan"), dtype=torch.float16, device=DEV)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    ops.attn_prefill_paged(q, kp, vp, table, torch.tensor(L, dtype=torch.int32, device=DEV), cu, max(lens), scale, out=out)
    plain = [p.unflatten(-1, (-1, 8))[..., t, c ^ (t & 7), :].flatten(-2) for p in (kp, vp)]
    row = 0
    for b, (n, Lb) in enumerate(zip(lens, L)):
        K, V = (p[table[b, :pages[b]].long()].transpose(1, 2).flatten(0, 1)[:Lb].double() for p in plain)
        ok = torch.arange(Lb, device=DEV)[None] <= past + torch.arange(n, device=DEV)[:, None]
        for h in range(H):
            s = q[row:row + n, h].double() @ K[:, h * G // H].T
            top = (s * scale).masked_fill(~ok, 0).abs().amax(1, keepdim=True)
            w = torch.softmax((s * scale).masked_fill(~ok, -math.inf), 1)
            ref, spread = w @ V[:, h * G // H], w @ V[:, h * G // H].abs()
            tol = 2.0 ** -11 * ref.abs() + (2 * 2.0 ** -11 + 2 * d * 2.0 ** -24 * (1 + top)) * spread + 1e-6
            err = (out[row:row + n, h].double() - ref).abs()
            assert bool((err <= tol).all()), (b, h, float((err / tol).max()), int((err > tol).sum()))
        row += n


@pytest.mark.parametrize("H,G,d", [(8, 2, 128), (6, 2, 128), (3, 3, 64), (7, 1, 64), (12, 2, 64)])
def test_head_and_tile_pairs(H, G, d):
    _run([1, 128, 129, 255, 256, 257, 385, 40], 0, H, G, d, d ** -0.5)
    _run([130, 3, 300], 77, H, G, d, d ** -0.5, seed=1)


def test_more_items_than_sms():
    _run([33 + 17 * (i % 9) for i in range(40)], 0, 16, 4, 64, 0.125, seed=2)


@pytest.mark.parametrize("grow", ["slow", "leaps", "late", "falling", "flat"])
def test_maxima_that_move(grow):
    f = {"slow": lambda p: 0.2 + p / 300.0, "leaps": lambda p: 4.0 ** (p // 300).clamp(max=3), "late": lambda p: torch.where(p > 1300, 12.0, 0.05),
         "falling": lambda p: 6.0 / (1 + p / 100.0), "flat": lambda p: 0.0 * p}[grow]
    _run([1500, 700], 0, 4, 2, 128, 128 ** -0.5, shape_keys=f, seed=3)
    _run([40], 1490, 4, 4, 64, 0.125, shape_keys=f, seed=4)


@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_scales_that_are_not_positive(scale):
    _run([300, 20], 50, 4, 2, 64, scale, seed=5)


def test_scores_of_minus_infinity():
    """keys that a query must not weigh at all: a first key tile of nothing else, single ones among others; a query that sees no other key gives zeros"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(6)
    H, G, d, L = 4, 2, 64, 400
    kp, vp = torch.randn(26, G, 16, d, generator=g, device=DEV).half(), torch.randn(26, G, 16, d, generator=g, device=DEV).half()
    t, c = torch.arange(16, device=DEV)[:, None], torch.arange(d // 8, device=DEV)[None, :]
    table = torch.randperm(26, generator=g, device=DEV).int()[None, :25].contiguous()
    dead = torch.zeros(25 * 16, dtype=torch.bool, device=DEV)
    dead[:150], dead[200], dead[300:310] = True, True, True
    K = torch.randn(25 * 16, G, d, generator=g, device=DEV).half()
    K[dead, :, 0] = -math.inf
    kp[table[0].long()] = K.unflatten(0, (25, 16)).transpose(1, 2).unflatten(-1, (-1, 8))[..., t, c ^ (t & 7), :].flatten(-2)   # the swizzle is its own inverse
    V = vp[table[0].long()].unflatten(-1, (-1, 8))[..., t, c ^ (t & 7), :].flatten(-2).transpose(1, 2).flatten(0, 1).double()
    q = torch.randn(L, H, d, generator=g, device=DEV).half()
    q[..., 0] = q[..., 0].abs() + 0.5
    out = ops.attn_prefill_paged(q, kp, vp, table, torch.tensor([L], dtype=torch.int32, device=DEV), torch.tensor([0, L], dtype=torch.int32, device=DEV), L, 0.125)
    assert bool((out[:150] == 0).all())
    ok = (torch.arange(L, device=DEV)[None] <= torch.arange(L, device=DEV)[:, None]) & ~dead[None]
    for h in range(H):
        s = q[:, h].double() @ K[:, h * G // H].double().nan_to_num(neginf=0.0).T * 0.125
        w = torch.softmax(s.masked_fill(~ok, -math.inf), 1)[150:]
        ref, spread = w @ V[:, h * G // H], w @ V[:, h * G // H].abs()
        top = s.abs().amax(1, keepdim=True)[150:]
        tol = 2.0 ** -11 * ref.abs() + (2 * 2.0 ** -11 + 2 * d * 2.0 ** -24 * (1 + top)) * spread + 1e-6
        assert bool(((out[150:, h].double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("lens,H,G", [([100] * 4, 37, 37), ([100] * 3, 50, 50), ([100] * 5, 30, 15), ([130, 20], 36, 12), ([130, 20], 38, 38), ([1], 71, 1), ([300], 32, 8)])
def test_around_one_tile_per_sm(lens, H, G):
    """up to 148 tiles each has an item to itself; above, items are two tiles: two heads, or two query tiles"""
    _run(lens, 0, H, G, 64, 0.125, seed=7)
    _run(lens, 200, H, G, 64, 0.125, seed=8)


@pytest.mark.parametrize("spread", [0.3, 1.0, 3.0])
def test_the_largest_weight_is_exact(spread):
    """behind 1500 keys the result is no further from float64 than weights in fp16 must be: the largest one of a row is exactly 1, all others are
    rounded once.  The bound is that of the same sums with weights rounded so, and its half percent for fp32 scores, sums and exponentials"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(9)
    H, G, d, n, L = 16, 4, 128, 200, 1700
    pages = (L + 15) // 16
    kp, vp = torch.randn(pages, G, 16, d, generator=g, device=DEV).half(), torch.randn(pages, G, 16, d, generator=g, device=DEV).half()
    q = (torch.randn(n, H, d, generator=g, device=DEV) * spread).half()
    table = torch.arange(pages, device=DEV, dtype=torch.int32)[None].contiguous()
    out = ops.attn_prefill_paged(q, kp, vp, table, torch.tensor([L], dtype=torch.int32, device=DEV), torch.tensor([0, n], dtype=torch.int32, device=DEV), n, d ** -0.5)
    t, c = torch.arange(16, device=DEV)[:, None], torch.arange(d // 8, device=DEV)[None, :]
    K, V = (p.unflatten(-1, (-1, 8))[..., t, c ^ (t & 7), :].flatten(-2).transpose(1, 2).flatten(0, 1)[:L].double() for p in (kp, vp))
    ok = torch.arange(L, device=DEV)[None] <= L - n + torch.arange(n, device=DEV)[:, None]
    got = must = 0.0
    for h in range(H):
        s = (q[:, h].double() @ K[:, h * G // H].T * d ** -0.5).masked_fill(~ok, -math.inf)
        w = torch.exp(s - s.amax(1, keepdim=True))
        ref, rounded = w @ V[:, h * G // H] / w.sum(1, keepdim=True), w.half().double()
        best = (rounded @ V[:, h * G // H] / rounded.sum(1, keepdim=True)).half().double()
        got, must = got + float((out[:, h].double() - ref).square().sum()), must + float((best - ref).square().sum())
    assert (got / must) ** 0.5 < 1.005, (got / must) ** 0.5


@pytest.mark.parametrize("past", [0, 1, 31, 32, 33, 95, 127])
def test_borders_inside_a_key_tile(past):
    """the mask is looked at 32 keys at a time"""
    _run([1, 31, 32, 33, 63, 65, 97, 127, 160], past, 4, 2, 64, 0.125, seed=6 + past)
    _run([97, 129, 33], past, 4, 2, 128, 128 ** -0.5, seed=6 + past)
