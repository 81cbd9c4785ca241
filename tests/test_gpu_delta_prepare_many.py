"""The delta rule's preparation over runs of tokens where its blocks are more than three an SM (csrc/seq_delta.cu, kRunBlocksMany), and just fewer, where another
build of the kernel takes over: the same bits on both sides for the same tokens.  Reference and tolerance: test_gpu_delta_prompts.py's."""
import pytest
import torch
from .test_gpu_delta_prompts import DEV, _prepared, _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [True, False])
@pytest.mark.parametrize("taps", [2, 4])
def test_both_sides_of_the_line(channels, taps):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops_seq as ops
    H, G, d = 16, 8, 128
    g = torch.Generator(device=DEV).manual_seed(taps + 10 * channels)
    C, n_dec = (2 * G + H) * d, H * d if channels else H
    conv_w, A_log, dt_bias = (torch.randn(*s, generator=g, device=DEV) * 0.5 for s in ((taps, C), (H,), (n_dec,)))

    def rows(lens):
        x = torch.cat(wide[:len(lens)])
        state = torch.zeros(len(lens), taps - 1, C, device=DEV)
        return ops.delta_prepare(x, 0, conv_w, state, x, C + n_dec, x, C, A_log, dt_bias, d ** -0.5, _step([(0, n) for n in lens], list(range(len(lens)))), H, G, d, d, channels)

    lens = [500, 385, 17, 1200]   # 902 tokens stay below 444 blocks, 2102 lie above
    wide = [torch.randn(n, C + n_dec + H, generator=g, device=DEV) for n in lens]
    few, many = rows(lens[:3]), rows(lens)
    assert torch.equal(few[:, :C + n_dec + H], many[:few.shape[0], :C + n_dec + H])
    at = 0
    for n, w in zip(lens, wide):
        want = _prepared(w[:, :C], w[:, C + n_dec:], w[:, C:C + n_dec], conv_w, A_log, dt_bias, H, G, d, channels)
        y = many[at:at + n, :want.shape[1]].double()
        assert bool(((y - want).abs() <= 2e-5 * want.abs() + 4e-6).all()), float((y - want).abs().max())
        at += n
