"""What follows when a bounded wait inside a kernel runs out (csrc/runtime.cu, b200_gave_up): the entry points of such kernels refuse further work
instead of returning success, and a step of generate_token raises instead of handing out tokens.  The word that kernels report in is set by hand:
no GPU."""
import ctypes
import types

import pytest
import torch

from tests.test_host_logic import _req, mods  # noqa: F401


@pytest.fixture(params=["load", "load_seq"])
def lib(request, mods):  # noqa: F811
    from tgis_b200 import _lib
    handle = getattr(_lib, request.param)()
    assert handle.b200_gave_up() == 0
    yield handle
    handle.b200_debug_set_gave_up(0)
    assert handle.b200_gave_up() == 0


def _entries(lib):
    """one call of every entry point whose kernels can give up, over 16-byte aligned buffers that are never touched"""
    buf = ctypes.create_string_buffer(4096)
    p = (ctypes.addressof(buf) + 15) // 16 * 16
    calls = {"fp16 linear": lambda: lib.b200_gemm_bf16(p, p, None, p, 0, 700, 256, 256, None, None)}
    if hasattr(lib, "b200_gemm_w4a16") and not lib._name.endswith("libb200_seq.so"):
        calls["int4 linear"] = lambda: lib.b200_gemm_w4a16(p, p, None, p, 700, 256, 256, 128, None, None)
        calls["prompt attention"] = lambda: lib.b200_attn_prefill_paged(p, 512, 700, p, p, 64, p, 64, p, p, p, 512, 1, 700, 4, 2, 128, 0.1, None)
    else:
        calls["hybrid attention"] = lambda: lib.b200_seq_talk_attn(p, p, 0, 512, 0, 256, p, 64, p, p, 1, p, None, p, 700, 4, 2, 128, 128, 0, 0, 0.1, 16, None, 1, None, None)
        calls["experts, few rows"] = lambda: lib.b200_seq_experts_gemm(p, p, p, 0, p, 64, 8, 256, 256, 0, None)
        calls["experts, many rows"] = lambda: lib.b200_seq_experts_gemm(p, p, p, 0, p, 4096, 8, 256, 256, 0, None)
        calls["heads"] = lambda: lib.b200_seq_heads_gemm(p, 512, 256, p, p, 0, 512, 256, 64, 2, 256, 256, None)
    return calls


def test_entry_points_refuse(lib):
    from tgis_b200 import _lib
    lib.b200_debug_set_gave_up(1)
    assert lib.b200_gave_up() == 1
    for name, call in _entries(lib).items():
        assert call() != 0 and b"a wait inside an earlier kernel ran out" in lib.b200_last_error(), name
    with pytest.raises(_lib.B200Error, match="ran out"):
        _lib.raise_if_gave_up()
    lib.b200_debug_set_gave_up(0)
    _lib.raise_if_gave_up()


@pytest.mark.parametrize("params", [{}, {"want_logprobs": True}])
def test_a_step_raises(lib, mods, params):  # noqa: F811
    """prefill, then a decoding step during which the report comes in"""
    from tgis_b200 import _lib
    from tgis_b200.models.flash_causal_lm import FlashCausalLM
    pb, Batch, tok, Mgr = mods["pb"], mods["Batch"], mods["tok"], mods["Mgr"]
    steps = []

    class FakeModel:
        def forward(self, input_ids, position_ids, cu_seqlens, cu_seqlens_q, max_s, inputs_embeds, past_key_values, prealloc, lm_head_indices=None):
            steps.append(len(steps))
            lib.b200_debug_set_gave_up(len(steps) == 2)
            lg = torch.zeros(len(input_ids), 64, dtype=torch.float16)
            return (lg if lm_head_indices is None else lg[lm_head_indices]), past_key_values

    class HostOnlyLM(FlashCausalLM):
        def __init__(self):
            self.model, self.device, self.tokenizer = FakeModel(), torch.device("cpu"), tok
            self.engine = types.SimpleNamespace(world_size=1)
            self.kv_cache_manager = Mgr(num_layers=1, num_heads=1, emb_dim=64, kv_heads=1, device="cpu", total_num_gpu_blocks=32)

        def _can_fuse_greedy(self, batch):
            return False

        def _decode_advance(self, batch):
            pass

    requests = [_req(pb, i, "test " * n, n, 4) for i, n in enumerate((3, 5))]
    if params:
        for r in requests:
            r.details.logprobs = True
    lm = HostOnlyLM()
    batch, errs = Batch.from_pb(pb.Batch(id=0, requests=requests), tok, torch.float16, torch.device("cpu"), None, None, True)
    assert not errs
    lm.generate_token(batch, first=True)
    with pytest.raises(_lib.B200Error, match="ran out"):
        lm.generate_token(batch)
