"""An int4 linear over the same inputs gives the same bits every time.  Records of packed weights pass through rings that bulk copies refill while other
warps still load from them; where a slot was given back before the loads had ended, some columns took 32 k from another record, once in 2000 calls of 4099
tokens and once in 10000 of 129.  So the calls are many; nothing is compared with a tolerance."""
import pytest
import torch
from .test_gpu_gemm_w4_few import DEV, _weights

pytestmark = pytest.mark.gpu


# both kernels: warp pairs of SMs above 128 tokens, tensor-memory operands below; group sizes put one or several rows of scales into a record
@pytest.mark.parametrize("T,K,N,gs,gate_up,calls", [(4099, 14336, 4096, 128, False, 6000), (129, 14336, 4096, 128, False, 20000), (1000, 4096, 28672, 32, True, 3000),
                                                    (64, 4096, 28672, 128, True, 10000), (16, 14336, 4096, 64, False, 10000)])
def test_same_bits(T, K, N, gs, gate_up, calls):
    import tgis_b200  # noqa: F401
    from tgis_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    qweight, qzeros, scales, _ = _weights(g, N, K, gs)
    layout = ops.W4_LAYOUT_GATE_UP if gate_up else ops.W4_LAYOUT_PLAIN
    packed = ops.gptq_pack(qweight, qzeros, scales, gs, layout)
    xs = [torch.randn(T, K, generator=g, device=DEV).half() for _ in range(3)]   # (neighbouring calls differ, and so do the records' neighbours)
    call = lambda i: ops.gemm_w4a16(xs[i % 3], packed, N, gs, layout=layout, silu_mul=gate_up).view(torch.int16)  # noqa: E731
    first = [call(i) for i in range(3)]
    differ = torch.zeros((), dtype=torch.int64, device=DEV)
    for i in range(calls):
        differ += (call(i) != first[i % 3]).any()
    assert differ.item() == 0
