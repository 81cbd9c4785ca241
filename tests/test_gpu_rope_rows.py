"""Rotation and cache write on both sides of the line to 16-byte accesses (csrc/elementwise.cu, kRopeVecRows): as many tokens, heads enough to cross it, and a
cache that starts off any eight halves, which stays with the other form.  Reference: the rotation in fp32 (two products and a sum, fp16 result: 2^-10 of the
larger operand), the cache holds the bits of the rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("T,h,kv", [(64, 32, 16), (64, 32, 15), (41, 96, 2), (40, 96, 2), (9, 448, 8), (255, 8, 4), (256, 4, 2)])
@pytest.mark.parametrize("off", [0, 4])
def test_both_forms(d, T, h, kv, off):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(d + T + h)
    rows = h + 2 * kv
    x = torch.randn(T, rows * d, generator=g, device=DEV).half()
    angle = torch.arange(300, device=DEV)[:, None] * 10000.0 ** (-torch.arange(d // 2, device=DEV) / (d // 2))
    cos, sin = angle.cos().half(), angle.sin().half()
    pos = torch.randint(0, 300, (T,), generator=g, device=DEV)
    slots = torch.randperm((T + 40) // 16 * 16, generator=g, device=DEV)[:T].long()
    slots[T // 2] = -1
    n = (T + 40) // 16 * kv * 16 * d
    room = [torch.full((n + 8,), 7.0, dtype=torch.float16, device=DEV) for _ in range(2)]
    k_pool, v_pool = (r[off:off + n].view(-1, kv, 16, d) for r in room)
    out = x.clone()
    ops.rope_kv_write_paged(out, cos, sin, pos, slots, k_pool, v_pool, h, kv, d)
    q = x.view(T, rows, d).float()
    a, b, c, s = q[:, :h + kv, :d // 2], q[:, :h + kv, d // 2:], cos[pos].float()[:, None], sin[pos].float()[:, None]
    want = torch.cat([torch.cat([a * c - b * s, a * s + b * c], -1), q[:, h + kv:]], 1)
    got = out.view(T, rows, d)
    big = torch.maximum(q[..., :d // 2].abs(), q[..., d // 2:].abs()).repeat(1, 1, 2)
    assert bool(((got.float() - want).abs() <= 2.0 ** -10 * big + 1e-7).all())
    assert torch.equal(got[:, h + kv:], x.view(T, rows, d)[:, h + kv:])
    t, ch = torch.arange(16, device=DEV)[:, None], torch.arange(d // 8, device=DEV)[None, :]
    for pool, part in ((k_pool, got[:, h:h + kv]), (v_pool, got[:, h + kv:])):
        plain = pool.unflatten(-1, (-1, 8))[..., t, ch ^ (t & 7), :].flatten(-2).transpose(1, 2).flatten(0, 1)   # [slot][kv][d]
        live = slots >= 0
        assert torch.equal(plain[slots[live]], part[live])
        other = torch.ones(plain.shape[0], dtype=torch.bool, device=DEV)
        other[slots[live]] = False
        assert bool((plain[other] == 7.0).all())
    for r in room:
        assert bool((r[:off] == 7.0).all()) and bool((r[off + n:] == 7.0).all())
