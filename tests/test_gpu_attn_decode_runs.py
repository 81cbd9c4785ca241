"""Decode attention over runs of keys (csrc/attn_decode.cu): one run that writes its result itself, two to eight runs merged by a cluster, grids too
large for that and contexts of more than eight runs merged by a second kernel; lengths of no key, of one, at the edges of pages and runs, unlike lengths in a
batch, group sizes of 1 to 16.  Reference: float64.

Tolerance: fp16 probabilities (2^-11 of a value's share), fp32 sums, an fp16 result: 2^-10 of the largest value is room for all of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(lens, heads, kv, d, most):
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + heads + d)
    pages = [(n + 15) // 16 for n in lens]
    perm = torch.randperm(sum(pages) + 3, generator=g, device=DEV).int()
    table = torch.zeros(len(lens), max(1, (most + 15) // 16), dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    k, v = (torch.randn(sum(pages) + 3, kv, 16, d, generator=g, device=DEV).half() for _ in range(2))
    qkv = torch.randn(len(lens), (heads + 2 * kv) * d, generator=g, device=DEV).half()
    return qkv[:, :heads * d].unflatten(1, (heads, d)), k, v, table, torch.tensor(lens, dtype=torch.int32, device=DEV)


def _plain(pool):
    """pages whose 16-byte chunks sit at chunk ^ (token & 7) -> the plain order, [blocks, kv, 16, d]"""
    c = pool.unflatten(-1, (-1, 8))
    t, j = torch.arange(16, device=DEV)[:, None], torch.arange(c.shape[-2], device=DEV)[None]
    return c[..., t, j ^ (t & 7), :].flatten(-2)


def _exact(q, k, v, table, lens, scale):
    k, v, out = _plain(k).double(), _plain(v).double(), torch.zeros(q.shape, dtype=torch.float64, device=DEV)
    r = q.shape[1] // k.shape[1]
    for b, n in enumerate(lens.tolist()):
        if n > 0:
            at = table[b, :(n + 15) // 16].long()
            K, V = (x[at].transpose(1, 2).flatten(0, 1)[:n].repeat_interleave(r, 1) for x in (k, v))
            p = torch.softmax(torch.einsum("hd,lhd->hl", q[b].double(), K) * scale, -1)
            out[b] = torch.einsum("hl,lhd->hd", p, V)
    return out


@pytest.mark.parametrize("heads,kv,d", [(8, 2, 128), (4, 4, 64), (16, 1, 64), (5, 1, 128)])
@pytest.mark.parametrize("lens", [[1], [16, 0, 17], [128, 127, 1], [129, 300, 5, 0], [1000, 15, 16, 17, 33, 512, 513, 999], [2047, 1, 0], [4096], [5000, 70]])
def test_runs(heads, kv, d, lens):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    case = _case(lens, heads, kv, d, max(lens))
    want = _exact(*case, d ** -0.5)
    for most in (max(lens), max(lens) + 700):   # the bound that a program knows may be larger than any length
        table = torch.nn.functional.pad(case[3], (0, 44))
        got = ops.attn_decode_paged(case[0], case[1], case[2], table, case[4], most, d ** -0.5, kv)
        assert float((got.double() - want).abs().max()) <= 2 ** -10 * float(want.abs().max()), most


@pytest.mark.parametrize("most", [100, 400, 900])
def test_more_blocks_than_the_chip_holds(most):
    """75 sequences of 8 key heads: a run each, and several"""
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    lens = [1 + (most - 1) * i // 74 for i in range(75)]
    case = _case(lens, 16, 8, 64, most)
    want = _exact(*case, 0.125)
    out = torch.full((75, 16, 64), float("nan"), dtype=torch.float16, device=DEV)
    ops.attn_decode_paged(*case, most, 0.125, 8, out)
    assert float((out.double() - want).abs().max()) <= 2 ** -10 * float(want.abs().max())
