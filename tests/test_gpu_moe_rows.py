"""Routed products of few rows per expert (csrc/seq_moe.cu, moe_linear_mma_kernel): experts with no row, one, 15 to 17, 48, 63 to 65 and 130, steps on both
sides of the rule for the pipeline's depth, k that is shorter than the pipeline, ends inside a step, features that end inside a tile, compact and gathered
rows, the square of ReLU.  Reference: float64.

Tolerance: fp32 sums of K products (K 2^-24 of the sum of absolute values), a bfloat16 result 2^-8 of itself; the square of ReLU doubles both."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _routing(rows):
    """one pick per token: expert e takes rows[e] tokens, in an order that mixes them"""
    from tgis_b200 import ops_seq as ops
    E, T = len(rows), sum(rows)
    expert = torch.cat([torch.full((n,), e, device=DEV) for e, n in enumerate(rows)])[torch.randperm(T, generator=torch.Generator().manual_seed(T)).to(DEV)]
    logits = torch.zeros(T, E, device=DEV)
    logits[torch.arange(T, device=DEV), expert] = 5.0
    r = ops.moe_route(logits, 1)
    at = 2 * E + 2 + 2 * ((T + 63) // 64 + E) + T   # the plan: counts, offsets, tiles' number, experts and first rows, places, then the row of every pick
    return r, expert, r.plan[at:at + T].long()


@pytest.mark.parametrize("rows", [[0, 1, 0, 2], [15, 16, 0, 17], [3, 0, 48, 1, 7], [63, 0, 64, 65], [130, 1, 0, 0]])
@pytest.mark.parametrize("N,K", [(64, 64), (72, 136), (200, 1032)])
def test_rows_of_experts(rows, N, K):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    r, expert, row_of = _routing(rows)
    assert sorted(row_of.tolist()) == list(range(sum(rows)))
    g = torch.Generator(device=DEV).manual_seed(N + K)
    w, a = (torch.randn(*s, generator=g, device=DEV).bfloat16() for s in ((len(rows), N, K), (sum(rows), K)))
    want = torch.einsum("tk,tnk->tn", a.double(), w.double()[expert])
    room = K * 2 ** -24 * torch.einsum("tk,tnk->tn", a.double().abs(), w.double().abs()[expert]) + 1e-9
    compact = torch.empty_like(a)
    compact[row_of] = a
    for x, gather in ((a, True), (compact, False)):
        got = ops.moe_linear(x, w, r, gather=gather, out_dtype=torch.float32)[row_of].double()
        assert bool(((got - want).abs() <= room).all())
        got = ops.moe_linear(x, w, r, gather=gather, out_dtype=torch.bfloat16)[row_of].double()
        assert bool(((got - want).abs() <= room + 2 ** -8 * want.abs()).all())
        got = ops.moe_linear(x, w, r, gather=gather, out_dtype=torch.bfloat16, act=ops.ACT_RELU2)[row_of].double()
        top = want.clamp(min=0)
        assert bool(((got - top.square()).abs() <= 2 * top * room + room.square() + 2 ** -8 * top.square()).all())


def test_what_is_not_finite_stays_in_its_row():
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    r, _, row_of = _routing([17, 5])
    g = torch.Generator(device=DEV).manual_seed(1)
    w, a = (torch.randn(*s, generator=g, device=DEV).bfloat16() for s in ((2, 64, 200), (22, 200)))
    want = ops.moe_linear(a, w, r, gather=True, out_dtype=torch.float32)[row_of]
    a[3] = float("inf")
    got = ops.moe_linear(a, w, r, gather=True, out_dtype=torch.float32)[row_of]
    keep = torch.arange(22, device=DEV) != 3
    assert torch.equal(got[keep], want[keep]) and not bool(got[3].isfinite().any())
