"""The SiLU of every fp16 value (silu_of_half, csrc/common.cuh): the bits of x / (1 + e^-x) in fp32 rounded to fp16, NaN where that is NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_every_fp16_value():
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    x = torch.arange(-32768, 32768, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.float16).view(64, 1024)
    got, f = ops.silu_mul(torch.cat([x, torch.ones_like(x)], 1).contiguous()), x.float()
    ref = (f / (1 + torch.exp(-f))).half()
    nan = torch.isnan(ref)
    assert torch.equal(torch.isnan(got), nan)
    assert bool(((got.view(torch.int16) == ref.view(torch.int16)) | nan).all())
