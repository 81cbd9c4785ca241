"""Grouped products of routed experts on SM pairs (csrc/gemm_pair.cuh behind ops_seq.experts_linear): experts without rows, with one row, with exactly and
just over a row tile, all rows with one expert, picks of identity outputs (rows that no expert has), features that end inside a tile, k that ends
inside a k-block, more tiles than pairs.  Reference: float64; tolerance as in test_gpu_gemm_pair."""
import pytest
import torch

from tests.test_gpu_gemm_pair import _bound

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _routing(counts, identity_rows=0):
    """one pick per token; expert e has counts[e] tokens, dealt out in a scattered order"""
    from tgis_b200 import ops_seq
    E = len(counts)
    pick = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)] + [torch.full((identity_rows,), E)])
    pick = pick[torch.randperm(len(pick), generator=torch.Generator().manual_seed(len(pick)))].to(DEV)
    logits = torch.zeros(len(pick), E + 1, device=DEV)
    logits[torch.arange(len(pick), device=DEV), pick] = 5.0
    return ops_seq.moe_route(logits, 1, softmax_scores=True, identity=1), pick


@pytest.mark.parametrize("counts,identity", [([40, 0, 1, 31, 256, 257, 533, 200], 20), ([0, 0, 700, 0], 0), ([600, 513, 1, 64], 3), ([161] * 20, 0)])
@pytest.mark.parametrize("N,K", [(128, 64), (300, 200), (520, 136)])
def test_experts(counts, identity, N, K):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq
    r, pick = _routing(counts, identity)
    g = torch.Generator(device=DEV).manual_seed(N + K)
    a = torch.randn(r.T, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(len(counts), N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    rows = ops_seq.moe_gather_rows(a, r)
    n = sum(counts)
    rows[n:] = float("nan")     # rows that no expert has: read beside the last ones, never part of a result
    starts = torch.tensor([0] + counts).cumsum(0).tolist()
    for act, dtype in ((ops_seq.ACT_NONE, torch.bfloat16), (ops_seq.ACT_NONE, torch.float32), (ops_seq.ACT_RELU2, torch.bfloat16)):
        y = ops_seq.experts_linear(rows, w, r, dtype, act=act)
        for e, c in enumerate(counts):
            x = rows[starts[e]:starts[e + 1]]
            ref = x.double() @ w[e].double().t()
            tol = _bound(ref, x, w[e], 0.0 if dtype == torch.float32 else 2.0 ** -8)
            if act == ops_seq.ACT_RELU2:
                tol = 2.0 ** -8 * ref.square() + 2 * ref.abs() * _bound(ref, x, w[e], 0.0) + 1e-7
                ref = ref.clamp(min=0).square()
            assert bool(((y[starts[e]:starts[e + 1]].double() - ref).abs() <= tol).all()), (e, c, act, dtype)
