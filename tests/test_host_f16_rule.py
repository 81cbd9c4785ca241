"""Which kernel an fp16 linear of 65 to 256 tokens goes to where clusters can share its feature tiles (csrc/gemm_f16.cu, f16_cluster_us), no GPU needed: on the
side that took less when both were measured on B200, which holds these clusters of 2 .. 8 CTAs; where none shares a tile, the choice is b200_debug_pair_plan's."""
import ctypes

import pytest

HELD = (0, 0, 74, 45, 33, 26, 22, 15, 15)


@pytest.fixture(scope="module")
def on_pairs():
    import tgis_b200  # noqa: F401
    from tgis_b200 import _lib
    lib = _lib.load()
    return lambda T, K, N, held=HELD: lib.b200_debug_f16_on_pairs(T, N, K, 148, (ctypes.c_int32 * 9)(*held))


@pytest.mark.parametrize("T,K,N", [(65, 4096, 4096), (65, 5632, 2048), (65, 11008, 4096), (65, 16384, 2048), (65, 28672, 2048), (65, 20480, 5120), (128, 4096, 4096),
                                   (128, 5632, 2048), (128, 11008, 4096), (128, 16384, 2048), (128, 28672, 2048), (128, 20480, 5120), (256, 11008, 4096),
                                   (256, 16384, 2048), (256, 28672, 2048), (256, 20480, 5120), (65, 28672, 8192), (128, 28672, 8192), (256, 28672, 8192), (65, 5632, 9216),
                                   (128, 8192, 9216)])
def test_streamed(on_pairs, T, K, N):
    assert on_pairs(T, K, N) == 0


@pytest.mark.parametrize("T,K,N", [(128, 2048, 2560), (256, 2048, 2560), (256, 4096, 4096), (128, 4096, 22016), (256, 4096, 22016), (257, 11008, 4096), (200, 2048, 2048), (224, 24576, 6144), (192, 16384, 8192),
                                   (224, 8192, 8192)])
def test_on_pairs(on_pairs, T, K, N):
    assert on_pairs(T, K, N) == 1


def test_without_clusters(on_pairs):
    from tgis_b200 import _lib
    out = (ctypes.c_int32 * 8)()
    for T in (1, 64, 65, 128, 192, 256, 257):
        for K, N in ((2048, 2560), (4096, 4096), (5632, 2048), (20480, 5120), (28672, 2048), (4096, 22016)):
            assert _lib.load().b200_debug_pair_plan(0, T, N, K, 148, out) == 0
            if T > 64:
                assert on_pairs(T, K, N, (0,) * 9) == out[0], (T, K, N)


@pytest.mark.parametrize("T", [17, 64])
def test_up_to_64_tokens_by_the_table_given(on_pairs, T):
    """wide outputs go to the pairs unless clusters hold their feature tiles, whatever device there is"""
    assert on_pairs(T, 2048, 11264) == 1 and on_pairs(T, 2048, 11264, (0, 0, 88) + (0,) * 6) == 0 and on_pairs(T, 2048, 11264, (0,) * 9) == 1
    assert on_pairs(16, 2048, 11264) == 0
