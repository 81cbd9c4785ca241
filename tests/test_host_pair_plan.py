"""Host-side plan of the linears on SM pairs (csrc/gemm_pair.cuh pair_plan) and the choice between them and the weight-streaming kernels
(csrc/gemm_f16.cu), no GPU needed."""
import ctypes

import pytest

from tests.test_host_gemm_plan import FAMILIES, SMS, _linears, lib  # noqa: F401

RING = {0: 6, 1: 5, 2: 6}   # full-size k-blocks that the ring has room for


def _plan(lib, kind, T, N, K, sms=SMS):  # noqa: F811
    out = (ctypes.c_int32 * 8)()
    assert lib.b200_debug_pair_plan(kind, T, N, K, sms, out) == 0, lib.b200_last_error()
    return dict(zip(("taken", "tn", "n_tt", "n_m", "pairs", "per_stage", "pieces", "piece_stages"), out))


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("family", list(FAMILIES))
def test_plans_cover_the_output_and_fit(lib, kind, family):  # noqa: F811
    for world in (1, 2, 4, 8):
        for which, N, K in _linears(family, world):
            if kind == 1 and (which == "head" or N % 32 or K % 32):
                continue
            for T in (65, 96, 127, 128, 129, 191, 200, 256, 257, 300, 1000, 4099, 70000):
                p = _plan(lib, kind, T, N, K)
                what = f"{family} tp{world} {which} N={N} K={K} T={T}: {p}"
                assert p["tn"] % 32 == 0 and 32 <= p["tn"] <= 256, what
                assert p["tn"] * p["n_tt"] >= T > p["tn"] * (p["n_tt"] - 1) and p["n_m"] * 256 >= N > (p["n_m"] - 1) * 256, what
                assert 1 <= p["pairs"] <= SMS // 2 and p["pairs"] <= p["n_tt"] * p["n_m"], what
                block = 128 * 64 * 2 + p["tn"] // 2 * 64 * 2
                stages = min(RING[kind] * (128 * 64 * 2 + 128 * 64 * 2) // (p["per_stage"] * block), 10)
                assert stages * p["per_stage"] >= 4, what       # int4: the four de-quantising teams take turns round the ring
                n_kb = -(-K // 64) if kind != 1 else 2 * -(-K // 128)
                n_stages = -(-n_kb // p["per_stage"])
                assert (p["pieces"] - 1) * p["piece_stages"] < n_stages <= p["pieces"] * p["piece_stages"], what
                if p["pieces"] > 1:                             # an accumulator per piece in 512 columns
                    assert kind != 1 and T <= 256, what
                    assert p["pieces"] * (64 if p["tn"] <= 64 else 128 if p["tn"] <= 128 else 256) <= 512, what


def test_which_kernel_takes_a_call(lib):  # noqa: F811
    """int4 up to 128 tokens, fp16 up to 64 and fp32 results up to 256 stay with the kernels that stream weights; between 65 and 256 tokens fp16 goes
    where it takes less, by times measured on B200"""
    for T in (1, 64, 128):
        assert not _plan(lib, 1, T, 4096, 4096)["taken"] and not _plan(lib, 2, T, 4096, 4096)["taken"]
    assert _plan(lib, 1, 129, 4096, 4096)["taken"] and not _plan(lib, 2, 256, 4096, 4096)["taken"] and _plan(lib, 2, 257, 4096, 4096)["taken"]
    for K, N in ((2048, 2560), (28672, 2048), (4096, 128256)):
        assert not _plan(lib, 0, 64, N, K)["taken"] and _plan(lib, 0, 257, N, K)["taken"]
    faster_streamed = [(65, 11008, 4096), (96, 11008, 4096), (65, 16384, 2048), (128, 16384, 2048), (65, 28672, 2048), (192, 28672, 2048), (65, 14336, 4096),
                       (128, 14336, 4096), (65, 24576, 6144), (128, 24576, 6144), (65, 28672, 8192), (128, 28672, 8192), (65, 11008, 2048), (65, 8192, 1024)]
    faster_on_pairs = [(65, 2048, 2560), (256, 2048, 2560), (65, 4096, 4096), (256, 4096, 4096), (65, 5632, 2048), (256, 11008, 4096), (256, 16384, 2048), (192, 20480, 5120),
                       (65, 20480, 5120), (128, 4096, 22016), (65, 2048, 32000), (192, 28672, 8192), (192, 24576, 6144), (128, 8192, 4096), (192, 8192, 1024)]
    for want, calls in ((0, faster_streamed), (1, faster_on_pairs)):
        for T, K, N in calls:
            assert _plan(lib, 0, T, N, K)["taken"] == want, (T, K, N)


def test_bad_arguments(lib):  # noqa: F811
    out = (ctypes.c_int32 * 8)()
    assert lib.b200_debug_pair_plan(3, 65, 128, 128, SMS, out) != 0
    assert lib.b200_debug_pair_plan(0, 0, 128, 128, SMS, out) != 0
