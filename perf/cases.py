"""The work whose speed this framework answers for: single layers of a served model over the sizes that serving brings (one user's token,
a decoding batch, ragged prompts), and two whole calls of a decoder.  Every case goes through the entry points that a program calls -
the modules of `utils`, the operators of `ops` and `ops_seq`, `FlashLlamaForCausalLM.forward`.

A case is a dict of plain values.  Sequence lengths of a batch are spread evenly over [lo, hi] by the case alone; values come from the seed.
"""
import math
import types

import torch

import tgis_b200  # noqa: F401
from tgis_b200 import ops, ops_seq
from tgis_b200.models.custom_modeling.flash_llama_modeling import FlashLlamaForCausalLM
from tgis_b200.utils.dist import FakeGroup
from tgis_b200.utils.gptq.exllamav2 import Ex4bitLinearV2
from tgis_b200.utils.layers import FastLinear
from tgis_b200.utils.mixers import RoutedExperts
from tgis_b200.utils.paged import PagedKVCacheManager, PagedKVState
from tgis_b200.utils.synthetic import SyntheticWeights, llama_config

DEV = "cuda:0"
PAGE = 16


# ------------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one user's next token: the fused q / k / v projection of Llama-3-8B, GPTQ int4 (groups of 128)
        dict(name="int4_qkv_one_token", kind="int4", T=1, K=4096, N=6144, group=128, gate_up=False),
        # a full decoding batch through Llama-3-8B's gate and up projections with SiLU(gate) * up
        dict(name="int4_gate_up_batch", kind="int4", T=64, K=4096, N=28672, group=128, gate_up=True),
        # an add-on prefill's prompts through Llama-3-8B's down projection
        dict(name="int4_down_prompts", kind="int4", T=4099, K=14336, N=4096, group=128, gate_up=False),
        # the head of TinyLlama-1.1B for a decoding batch of 32
        dict(name="f16_head_batch", kind="linear", dtype="float16", T=32, K=2048, N=32000, bias=False),
        # prompts through the widest projection of Pythia-12B, with its bias
        dict(name="f16_fc_prompts", kind="linear", dtype="float16", T=3001, K=5120, N=20480, bias=True),
        # decode attention of Llama-3-8B (32 heads over 8 key heads), 64 sequences between 1k and 2k
        dict(name="decode_attention_batch", kind="decode_attention", B=64, lo=1024, hi=2048, heads=32, kv_heads=8, dim=128),
        # prefill attention of Llama-3-8B over ragged prompts
        dict(name="prompt_attention", kind="prompt_attention", B=13, lo=300, hi=2048, past=0, heads=32, kv_heads=8, dim=128),
        # chunked attention of the hybrid families (bfloat16 pages, width 2048), prompts that cross a chunk border
        dict(name="hybrid_attention_prompts", kind="hybrid_attention", B=2, lo=1500, hi=2500, past=0, heads=16, kv_heads=4, dim=128, chunk=2048, window=0,
             sink=False),
        # 16 routed squared-ReLU experts beside 4 identity outputs (width 2048), prompts
        dict(name="hybrid_experts_prompts", kind="experts", T=2048, W=2048, ff=2112, E=16, identity=4, top=2),
        # delta rule with a decay per key channel (width 2048), prompts
        dict(name="hybrid_delta_prompts", kind="delta", B=4, lo=256, hi=768, heads=16, kv_heads=8, dim=128),
        # a whole decoding step of the first four layers of Llama-3-8B int4 and its head, 64 sequences
        dict(name="llama_int4_decode_step", kind="llama", arch="llama-3-8b", quantize="gptq", layers=4, B=64, lo=1024, hi=2000, decode=True),
        # a whole prefill of TinyLlama-1.1B, logits of every prompt's last token
        dict(name="llama_f16_prefill", kind="llama", arch="tinyllama-1.1b", quantize="", layers=22, B=8, lo=100, hi=1000, decode=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["int4", "int4", "int4", "linear", "linear", "linear", "decode_attention", "decode_attention", "prompt_attention", "prompt_attention",
                       "hybrid_attention", "experts", "delta", "llama"])
    if kind == "int4":
        K, N, gate_up = rng.choice([(4096, 6144, False), (4096, 4096, False), (4096, 28672, True), (14336, 4096, False), (4096, 12288, False), (4096, 22016, True),
                                    (11008, 4096, False), (2048, 2560, False), (5632, 2048, False)])
        return dict(kind=kind, T=_log_int(rng, 1, 4096 if not gate_up else 2048), K=K, N=N, group=rng.choice([32, 64, 128, 128, 128]), gate_up=gate_up)
    if kind == "linear":
        dtype = rng.choice(["float16", "float16", "bfloat16"])
        K, N = rng.choice([(2048, 2560), (2048, 2048), (2048, 11264), (5632, 2048), (2048, 32000), (4096, 4096), (4096, 12288), (4096, 22016), (11008, 4096),
                           (5120, 15360), (20480, 5120), (2048, 4096)])
        return dict(kind=kind, dtype=dtype, T=_log_int(rng, 1, 3500), K=K, N=N, bias=rng.random() < 0.5)
    if kind == "decode_attention":
        heads, kv_heads, dim = rng.choice([(32, 8, 128), (32, 32, 128), (32, 4, 64), (40, 40, 128)])
        B = _log_int(rng, 1, 64 if kv_heads <= 8 else 16)
        lo = _log_int(rng, 16, 2048)
        return dict(kind=kind, B=B, lo=lo, hi=rng.randint(lo, 2 * lo), heads=heads, kv_heads=kv_heads, dim=dim)
    if kind == "prompt_attention":
        heads, kv_heads, dim = rng.choice([(32, 8, 128), (32, 32, 128), (32, 4, 64), (40, 40, 128)])
        lo = _log_int(rng, 8, 1024)
        return dict(kind=kind, B=rng.randint(1, 10), lo=lo, hi=rng.randint(lo, 2 * lo), past=rng.choice([0, 0, rng.randint(1, 1500)]), heads=heads,
                    kv_heads=kv_heads, dim=dim)
    if kind == "hybrid_attention":
        heads, kv_heads = rng.choice([(16, 4), (32, 8)])
        lo = _log_int(rng, 1, 1200)
        chunk, window = rng.choice([(2048, 0), (2048, 0), (0, 2048), (0, 0)])
        return dict(kind=kind, B=rng.randint(1, 4), lo=lo, hi=rng.randint(lo, 2 * lo), past=rng.choice([0, 0, rng.randint(1, 2000)]), heads=heads, kv_heads=kv_heads,
                    dim=128, chunk=chunk, window=window, sink=rng.random() < 0.4)
    if kind == "experts":
        W = rng.choice([2048, 4096])
        return dict(kind=kind, T=_log_int(rng, 1, 2048), W=W, ff=W * 33 // 32, E=16, identity=4, top=2)
    if kind == "delta":
        heads = rng.choice([16, 32])
        lo = _log_int(rng, 1, 400)
        return dict(kind=kind, B=rng.randint(1, 6), lo=lo, hi=rng.randint(lo, 2 * lo), heads=heads, kv_heads=heads // 2, dim=128)
    arch, quantize, layers = rng.choice([("llama-3-8b", "gptq", 2), ("llama-2-7b", "gptq", 2), ("llama-2-7b", "", 2), ("tinyllama-1.1b", "", 12)])
    decode = rng.random() < 0.5
    if decode:
        lo = _log_int(rng, 16, 1000)
        return dict(kind=kind, arch=arch, quantize=quantize, layers=layers, B=_log_int(rng, 1, 64), lo=lo, hi=rng.randint(lo, 2 * lo), decode=True)
    lo = _log_int(rng, 8, 500)
    return dict(kind=kind, arch=arch, quantize=quantize, layers=layers, B=rng.randint(1, 6), lo=lo, hi=rng.randint(lo, 2 * lo), decode=False)


# ------------------------------------------------------------------------------------------------------------------ inputs
def _lengths(case):
    """the case's B lengths, spread over [lo, hi] in an order that looks random"""
    lo, hi = case["lo"], case["hi"]
    return [lo + int((hi - lo) * ((0.5 + 0.6180339887 * i) % 1.0) + 0.5) for i in range(case["B"])]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed * 7919 + 17)


def _normal(g, *shape, std=1.0, dtype=torch.float16):
    return torch.empty(*shape, dtype=torch.float32, device=DEV).normal_(0.0, std, generator=g).to(dtype)


def _int4_tensors(g, K, N, group):
    """checkpoint tensors of a GPTQ linear: dense codes, zeros around the middle, scales that give weights of std near 0.02"""
    qweight = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    zeros = torch.randint(5, 10, (K // group, N // 8, 8), generator=g, device=DEV, dtype=torch.int64)
    packed = (zeros << (4 * torch.arange(8, device=DEV))).sum(-1)
    qzeros = torch.where(packed >= 2 ** 31, packed - 2 ** 32, packed).to(torch.int32)
    scales = (torch.rand(K // group, N, generator=g, device=DEV) * 0.004 + 0.002).to(torch.float16)
    return qweight, qzeros, scales


def _block_table(g, lens):
    """pages of every sequence, scattered over the pool as after some hours of serving"""
    pages = [(n + PAGE - 1) // PAGE for n in lens]
    perm = torch.randperm(sum(pages) + 1, generator=g, device=DEV).to(torch.int32)
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    return table, sum(pages) + 1


def _slots(table, starts, ends):
    """cache row of every token starts[b] .. ends[b] - 1"""
    out = []
    for b, (s, e) in enumerate(zip(starts, ends)):
        pos = torch.arange(s, e, device=DEV)
        out.append(table[b, pos // PAGE].long() * PAGE + pos % PAGE)
    return torch.cat(out)


def _cumulative(lens):
    return torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)


def _inputs(case, seed):
    """the case's values, in plain tensors"""
    g, k = _gen(seed), case["kind"]
    x = types.SimpleNamespace()
    if k == "int4":
        x.qweight, x.qzeros, x.scales = _int4_tensors(g, case["K"], case["N"], case["group"])
        x.x = _normal(g, case["T"], case["K"])
    elif k == "linear":
        dtype = getattr(torch, case["dtype"])
        x.w = _normal(g, case["N"], case["K"], std=0.02, dtype=dtype)
        x.x = _normal(g, case["T"], case["K"], dtype=dtype)
        x.bias = _normal(g, case["N"], std=0.1, dtype=dtype) if case["bias"] else None
    elif k in ("decode_attention", "prompt_attention"):
        new = [1] * case["B"] if k == "decode_attention" else _lengths(case)
        x.lens = _lengths(case) if k == "decode_attention" else [case["past"] + n for n in new]
        x.new = new
        H, G, d = case["heads"], case["kv_heads"], case["dim"]
        x.table, blocks = _block_table(g, x.lens)
        x.k_pool, x.v_pool = _normal(g, blocks, G, PAGE, d), _normal(g, blocks, G, PAGE, d)
        x.qkv = _normal(g, sum(new), (H + 2 * G) * d)   # queries are the first columns of the fused projection
        x.context = torch.tensor(x.lens, dtype=torch.int32, device=DEV)
        x.cu = _cumulative(new)
    elif k == "hybrid_attention":
        x.new = _lengths(case)
        x.lens = [case["past"] + n for n in x.new]
        H, G, d = case["heads"], case["kv_heads"], case["dim"]
        x.table, blocks = _block_table(g, x.lens)
        x.cache = _normal(g, blocks, PAGE, 2 * G * d, dtype=torch.bfloat16)
        x.q = _normal(g, sum(x.new), H, d, dtype=torch.float32)
        x.sink = _normal(g, H, dtype=torch.float32) if case["sink"] else None
    elif k == "experts":
        T, W, ff, E = case["T"], case["W"], case["ff"], case["E"]
        x.up = _normal(g, E, ff, W, std=W ** -0.5, dtype=torch.bfloat16)
        x.down = _normal(g, E, W, ff, std=ff ** -0.5, dtype=torch.bfloat16)
        x.h = _normal(g, T, W, dtype=torch.bfloat16)
        x.logits = _normal(g, T, E + case["identity"], dtype=torch.float32)
        x.stream = _normal(g, T, W, dtype=torch.float32)
    elif k == "delta":
        H, G, d = case["heads"], case["kv_heads"], case["dim"]
        x.new = _lengths(case)
        T, C = sum(x.new), (2 * G + H) * d
        x.u = _normal(g, T, C, dtype=torch.float32)
        x.conv_w = _normal(g, 4, C, std=0.5, dtype=torch.bfloat16)
        x.beta = _normal(g, T, H, dtype=torch.float32)
        x.decay = _normal(g, T, H * d, dtype=torch.float32)
        x.A_log = (torch.rand(H, generator=g, device=DEV) * 2 - 2).to(torch.bfloat16)
        x.dt_bias = (torch.rand(H * d, generator=g, device=DEV) * 2 - 2).to(torch.bfloat16)
    else:
        x.config = llama_config(case["arch"], quantize=case["quantize"] or None, max_position_embeddings=4096, num_layers=case["layers"])
        x.weights = SyntheticWeights(x.config, DEV, torch.float16, FakeGroup(0, 1), quantize=x.config.quantize, seed=seed)
        c = x.config
        x.new = [1] * case["B"] if case["decode"] else _lengths(case)
        x.lens = _lengths(case) if case["decode"] else x.new
        x.table, blocks = _block_table(g, x.lens)
        x.ids = torch.randint(0, c.vocab_size, (sum(x.new),), generator=g, device=DEV)
        x.pool = _normal(g, c.num_hidden_layers, 2, blocks, c.num_key_value_heads, PAGE, c.hidden_size // c.num_attention_heads)
    return x


class _Named:
    """the `get_tensor` side of a checkpoint, over tensors that are there already"""

    process_group = FakeGroup(0, 1)

    def __init__(self, tensors):
        self.tensors = tensors

    def get_tensor(self, name):
        return self.tensors[name]


def _ragged_step(new, starts, table):
    T = sum(new)
    position = torch.cat([torch.arange(s, s + n, device=DEV) for s, n in zip(starts, new)])
    seq = torch.repeat_interleave(torch.arange(len(new), device=DEV, dtype=torch.int32), torch.tensor(new, device=DEV))
    if table is None:
        slots, table = torch.zeros(T, dtype=torch.int64, device=DEV), torch.zeros(len(new), 1, dtype=torch.int32, device=DEV)
    else:
        slots = _slots(table, starts, [s + n for s, n in zip(starts, new)])
    return ops_seq.RaggedStep(T=T, B=len(new), position_ids=position, cu_q=_cumulative(new), seq_of_token=seq, slot_mapping=slots, block_table=table,
                              state_slots=torch.arange(len(new), dtype=torch.int32, device=DEV))


def prepare(case, seed):
    """what a program holds before the call: packed weights, modules, caches, index tensors of the step"""
    x, k = _inputs(case, seed), case["kind"]
    s = types.SimpleNamespace(case=case, x=x)
    if k == "int4":
        s.linear = Ex4bitLinearV2(x.qweight, x.qzeros, x.scales, None, None, 4, case["group"])
        s.linear.post_init(layout=ops.W4_LAYOUT_GATE_UP if case["gate_up"] else ops.W4_LAYOUT_PLAIN)
        x.qweight = x.qzeros = x.scales = None
    elif k == "linear":
        if case["dtype"] == "float16":
            s.linear = FastLinear(x.w, x.bias)
    elif k in ("decode_attention", "prompt_attention"):
        s.q = x.qkv[:, :case["heads"] * case["dim"]].unflatten(1, (case["heads"], case["dim"]))
    elif k == "hybrid_attention":
        s.step = _ragged_step(x.new, [case["past"]] * case["B"], x.table)
    elif k == "experts":
        tensors = {"router": _normal(_gen(seed + 1), case["E"] + case["identity"], case["W"], dtype=torch.bfloat16)}
        tensors["correction"] = torch.zeros(case["E"] + case["identity"], dtype=torch.bfloat16, device=DEV)
        for e in range(case["E"]):
            tensors[f"e{e}.up"], tensors[f"e{e}.down"] = x.up[e], x.down[e]
        s.experts = RoutedExperts("mlp", _Named({f"mlp.{n}": t for n, t in tensors.items()}), experts=case["E"], identity=case["identity"], top=case["top"],
                                  limit=None, softmax_scores=True, correction=True, plain="relu2")
        x.up = x.down = None
        s.out = torch.empty_like(x.stream)
    elif k == "delta":
        H, d = case["heads"], case["dim"]
        s.step = _ragged_step(x.new, [0] * case["B"], None)
        s.S = torch.zeros(case["B"], H, d, d, dtype=torch.float32, device=DEV)
        s.conv = torch.zeros(case["B"], 3, x.u.shape[1], dtype=torch.float32, device=DEV)
    else:
        c = x.config
        s.model = FlashLlamaForCausalLM(c, x.weights)
        s.model.kv_cache_manager = PagedKVCacheManager(c.num_hidden_layers, c.num_attention_heads, c.hidden_size, kv_heads=c.num_key_value_heads, device=DEV,
                                                       total_num_gpu_blocks=x.pool.shape[2])
        s.model.kv_cache_manager.pool.copy_(x.pool)
        x.pool = None
        starts = [n - m for n, m in zip(x.lens, x.new)]
        s.kv = PagedKVState(sequence_ids=list(range(case["B"])), block_table=x.table, context_lens=torch.tensor(x.lens, dtype=torch.int32, device=DEV),
                            slot_mapping=_slots(x.table, starts, x.lens), max_blocks=x.table.shape[1])
        s.position = torch.cat([torch.arange(a, b, device=DEV) for a, b in zip(starts, x.lens)])
        s.cu = _cumulative(x.new)
        s.cu_q = s.cu if case["decode"] else None
        s.last = None if case["decode"] else (s.cu[1:] - 1).long()
    return s


# ------------------------------------------------------------------------------------------------------------------ one pass
def run(s):
    case, x = s.case, s.x
    k = case["kind"]
    if k == "int4":
        if case["gate_up"]:
            return ops.gemm_w4a16(x.x, s.linear.q_handle, case["N"], case["group"], layout=s.linear.pack_layout, silu_mul=True)
        return s.linear(x.x)
    if k == "linear":
        return s.linear(x.x) if case["dtype"] == "float16" else ops_seq.linear(x.x, x.w, x.bias, out_dtype=torch.float32)
    if k == "decode_attention":
        return ops.attn_decode_paged(s.q, x.k_pool, x.v_pool, x.table, x.context, max(x.lens), case["dim"] ** -0.5, case["kv_heads"])
    if k == "prompt_attention":
        return ops.attn_prefill_paged(s.q, x.k_pool, x.v_pool, x.table, x.context, x.cu, max(x.new), case["dim"] ** -0.5)
    if k == "hybrid_attention":
        d, G = case["dim"], case["kv_heads"]
        return ops_seq.talk_attn(x.q, x.cache, s.step, kv_heads=G, vdim=d, k_off=0, v_off=G * d, scale=d ** -0.5, chunk=case["chunk"], window=case["window"],
                                 sink=x.sink)
    if k == "experts":
        routing = ops_seq.moe_route(x.logits, case["top"], softmax_scores=True, identity=case["identity"])
        ops_seq.halves_step(s.out, init=x.stream, rows=s.experts.experts(x.h, routing), routing=routing, passed=x.h, dtype=torch.bfloat16)
        return s.out
    if k == "delta":
        H, G, d = case["heads"], case["kv_heads"], case["dim"]
        rows = ops_seq.delta_prepare(x.u, 0, x.conv_w, s.conv, x.beta, 0, x.decay, 0, x.A_log, x.dt_bias, d ** -0.5, s.step, H, G, d, d, channels=True)
        return ops_seq.delta_rows_scan(rows, s.S, s.step, H, G, d, d, channels=True), s.S, s.conv
    logits, _ = s.model.forward(x.ids, s.position, s.cu, s.cu_q, max(x.lens), None, s.kv, None, s.last)
    return logits


# ------------------------------------------------------------------------------------------------------------------ what a pass cannot do without
def _visible(case, new, lens, chunk=0, window=0):
    """(query, key) pairs of a step, and the keys that some query of it sees"""
    pairs = keys = 0
    for n, L in zip(new, lens):
        first = L
        for p in range(L - n, L):
            lo = max(p // chunk * chunk if chunk else 0, p - window + 1 if window else 0)
            pairs += p - lo + 1
            first = min(first, lo)
        keys += L - first
    return pairs, keys


def work(case):
    k = case["kind"]
    if k == "int4":
        T, K, N = case["T"], case["K"], case["N"]
        out = N // 2 if case["gate_up"] else N
        return {"bytes": K * N // 2 + K // case["group"] * N * 5 // 2 + 2 * T * (K + out), "flops": 2 * T * K * N}
    if k == "linear":
        T, K, N = case["T"], case["K"], case["N"]
        return {"bytes": 2 * K * N + 2 * T * K + T * N * (2 if case["dtype"] == "float16" else 4), "flops": 2 * T * K * N}
    if k in ("decode_attention", "prompt_attention"):
        H, G, d = case["heads"], case["kv_heads"], case["dim"]
        new = [1] * case["B"] if k == "decode_attention" else _lengths(case)
        lens = _lengths(case) if k == "decode_attention" else [case["past"] + n for n in new]
        pairs, keys = _visible(case, new, lens)
        return {"bytes": 2 * (2 * keys * G * d + 2 * sum(new) * H * d), "flops": 4 * pairs * H * d}
    if k == "hybrid_attention":
        H, G, d = case["heads"], case["kv_heads"], case["dim"]
        new = _lengths(case)
        pairs, keys = _visible(case, new, [case["past"] + n for n in new], case["chunk"], case["window"])
        return {"bytes": 2 * 2 * keys * G * d + 2 * 4 * sum(new) * H * d, "flops": 4 * pairs * H * d}
    if k == "experts":
        T, W, ff, E, I = case["T"], case["W"], case["ff"], case["E"], case["identity"]
        rows = T * case["top"] * E // (E + I)
        used = E * (1 - (1 - case["top"] / (E + I)) ** T)
        return {"bytes": int(2 * 2 * used * W * ff + T * W * (2 + 4 + 4) + T * (E + I) * 4), "flops": 4 * rows * W * ff}
    if k == "delta":
        H, G, d = case["heads"], case["kv_heads"], case["dim"]
        T = sum(_lengths(case))
        return {"bytes": 4 * T * ((2 * G + H) * d + H + H * d + H * d) + 4 * case["B"] * H * d * d, "flops": 7 * T * H * d * d}
    c = llama_config(case["arch"], num_layers=case["layers"])
    H, I, V, d = c.hidden_size, c.intermediate_size, c.vocab_size, c.hidden_size // c.num_attention_heads
    per_layer = H * (2 * H + 2 * c.num_key_value_heads * d) + 3 * H * I
    new = [1] * case["B"] if case["decode"] else _lengths(case)
    lens = _lengths(case)
    pairs, keys = _visible(case, new, lens)
    T = sum(new)
    weights = c.num_hidden_layers * per_layer * (0.5 + 2.5 / 128 if case["quantize"] else 2)
    return {"bytes": int(weights + 2 * V * H + 2 * case["B"] * V + 4 * c.num_hidden_layers * keys * c.num_key_value_heads * d + 2 * T * H),
            "flops": 2 * T * c.num_hidden_layers * per_layer + 2 * case["B"] * V * H + 4 * pairs * c.num_hidden_layers * c.num_attention_heads * d}


def tolerance(case):
    # about four times what two correct paths differ by: fp16 and bf16 results round to 2^-11 and 2^-8; a bf16 value between two products,
    # fp16 probabilities and, in a whole model, the roundings of all its layers come on top
    k = case["kind"]
    if k == "linear" and case["dtype"] == "bfloat16":
        return {"rel": 1e-5, "max": 4e-5}      # bfloat16 operands, 32-bit sums and results
    if k in ("int4", "linear"):
        return {"rel": 1e-3, "max": 2e-3} if not case.get("gate_up") else {"rel": 2e-3, "max": 8e-3}
    if k in ("decode_attention", "prompt_attention"):
        return {"rel": 1e-3, "max": 1.5e-2}
    if k == "hybrid_attention":
        return {"rel": 8e-3, "max": 2e-1}
    if k == "experts":
        return {"rel": 4e-3, "max": 2.5e-2}
    if k == "delta":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 1.25e-2, "max": 6.5e-2}


# ------------------------------------------------------------------------------------------------------------------ the same in 64 bits
def _dequantized(qweight, qzeros, scales, group):
    """W [K, N] of a GPTQ checkpoint: fp16 scale * (code - (zero + 1)), rounded to fp16 as the format defines its weights"""
    shift = 4 * torch.arange(8, device=DEV, dtype=torch.int32)
    q = ((qweight[:, None, :] >> shift[None, :, None]) & 15).reshape(-1, qweight.shape[1])
    z = ((qzeros[:, :, None] >> shift) & 15).reshape(qzeros.shape[0], -1) + 1
    w = q.half() - z.half().repeat_interleave(group, 0)
    return (scales.repeat_interleave(group, 0).double() * w.double()).half().double()


def _unswizzled(pool):
    """[..., 16, d] pages whose 16-byte chunks sit at chunk ^ (token & 7) -> the plain order"""
    chunks = pool.unflatten(-1, (-1, 8))
    t, c = torch.arange(PAGE, device=DEV)[:, None], torch.arange(chunks.shape[-2], device=DEV)[None, :]
    return chunks[..., t, c ^ (t & 7), :].flatten(-2)


def _attend(q, K, V, scale, pos0, chunk=0, window=0, sink=None):
    """q [n, H, d] at positions pos0 .., K / V [L, G, d], all float64 -> [n, H, d]"""
    n, H, _ = q.shape
    r = H // K.shape[1]
    p = pos0 + torch.arange(n, device=DEV)[:, None]
    j = torch.arange(K.shape[0], device=DEV)[None, :]
    ok = j <= p
    if chunk:
        ok = ok & (j // chunk == p // chunk)
    if window:
        ok = ok & (j > p - window)
    out = torch.empty(n, H, V.shape[-1], dtype=torch.float64, device=DEV)
    for h in range(H):
        s = (q[:, h] @ K[:, h // r].T * scale).masked_fill(~ok, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(n, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :K.shape[0]] @ V[:, h // r]
    return out


def _paged_rows(pool, table_row, L):
    """[blocks, G, 16, d] in the plain order -> [L, G, d] of one sequence"""
    return pool[table_row[:(L + PAGE - 1) // PAGE].long()].transpose(1, 2).flatten(0, 1)[:L]


def _exact_llama(case, x):
    c, w = x.config, x.weights
    d, H, G = c.hidden_size // c.num_attention_heads, c.num_attention_heads, c.num_key_value_heads

    def linear(h, *names):
        out = []
        for n in names:
            if c.quantize:
                W = _dequantized(w.get_tensor(n + ".qweight"), w.get_tensor(n + ".qzeros"), w.get_tensor(n + ".scales"), w.gptq_groupsize)
            else:
                W = w.get_tensor(n + ".weight").double().T
            out.append(h @ W)
        return out

    def norm(h):
        return h * torch.rsqrt(h.square().mean(1, keepdim=True) + c.rms_norm_eps)   # the synthetic norm weights are ones

    starts = [L - n for L, n in zip(x.lens, x.new)]
    pos = torch.cat([torch.arange(a, b, device=DEV) for a, b in zip(starts, x.lens)]).double()
    angle = pos[:, None] * c.rope_theta ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float64) / d)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(t):
        a, b = t[..., :d // 2], t[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    h = w.get_tensor("model.embed_tokens.weight")[x.ids].double()
    for i in range(c.num_hidden_layers):
        at = f"model.layers.{i}."
        q, k, v = (t.unflatten(1, (-1, d)) for t in linear(norm(h), *(f"{at}self_attn.{n}_proj" for n in "qkv")))
        q, k = turn(q), turn(k)
        o, row = torch.empty(q.shape, dtype=torch.float64, device=DEV), 0
        for b, (n, L) in enumerate(zip(x.new, x.lens)):
            K, V = k[row:row + n], v[row:row + n]
            if L > n:
                kept = [_paged_rows(_unswizzled(x.pool[i, j]), x.table[b], L - n).double() for j in range(2)]
                K, V = torch.cat([kept[0], K]), torch.cat([kept[1], V])
            o[row:row + n] = _attend(q[row:row + n], K, V, d ** -0.5, L - n)
            row += n
        h = h + linear(o.flatten(1), at + "self_attn.o_proj")[0]
        gate, up = linear(norm(h), at + "mlp.gate_proj", at + "mlp.up_proj")
        h = h + linear(gate * torch.sigmoid(gate) * up, at + "mlp.down_proj")[0]
    if not case["decode"]:
        h = h[(_cumulative(x.new)[1:] - 1).long()]
    return norm(h) @ w.get_tensor("lm_head.weight").double().T


def _exact_delta(case, x):
    B, H, G, d = case["B"], case["heads"], case["kv_heads"], case["dim"]
    L, C = max(x.new), x.u.shape[1]
    u = torch.zeros(B, L + 3, C, dtype=torch.float64, device=DEV)
    beta = torch.zeros(B, L, H, dtype=torch.float64, device=DEV)       # rows past a sequence's end: no write, no decay
    g = torch.ones(B, L, H, d, dtype=torch.float64, device=DEV)
    decay = torch.exp(-x.A_log.double().exp()[:, None] * torch.nn.functional.softplus(x.decay.double() + x.dt_bias.double()).unflatten(1, (H, d)))
    row = 0
    for b, n in enumerate(x.new):
        u[b, 3:3 + n], beta[b, :n], g[b, :n] = x.u[row:row + n].double(), torch.sigmoid(x.beta[row:row + n].double()), decay[row:row + n]
        row += n
    c = sum(u[:, j:j + L] * x.conv_w[j].double() for j in range(4))
    c = c * torch.sigmoid(c)

    def unit(t):
        t = t.unflatten(2, (G, d))
        return (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)

    q, k, v = unit(c[..., :G * d]) * d ** -0.5, unit(c[..., G * d:2 * G * d]), c[..., 2 * G * d:].unflatten(2, (H, d))
    S = torch.zeros(B, H, d, d, dtype=torch.float64, device=DEV)
    y = torch.empty(B, L, H, d, dtype=torch.float64, device=DEV)
    for t in range(L):
        S = g[:, t, :, :, None] * S
        write = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
        S = S + k[:, t, :, :, None] * write[:, :, None]
        y[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    conv = torch.stack([u[b, n:n + 3] for b, n in enumerate(x.new)])
    return torch.cat([y[b, :n].flatten(1) for b, n in enumerate(x.new)]), S, conv


def exact(case, seed):
    x, k = _inputs(case, seed), case["kind"]
    if k == "int4":
        y = x.x.double() @ _dequantized(x.qweight, x.qzeros, x.scales, case["group"])
        if case["gate_up"]:
            gate, up = y.chunk(2, 1)
            y = gate * torch.sigmoid(gate) * up
        return y
    if k == "linear":
        y = x.x.double() @ x.w.double().T
        return y if x.bias is None else y + x.bias.double()
    if k in ("decode_attention", "prompt_attention"):
        H, d = case["heads"], case["dim"]
        q = x.qkv[:, :H * d].unflatten(1, (H, d)).double()
        K, V = _unswizzled(x.k_pool), _unswizzled(x.v_pool)
        out, row = torch.empty_like(q), 0
        for b, (n, L) in enumerate(zip(x.new, x.lens)):
            out[row:row + n] = _attend(q[row:row + n], _paged_rows(K, x.table[b], L).double(), _paged_rows(V, x.table[b], L).double(), d ** -0.5, L - n)
            row += n
        return out
    if k == "hybrid_attention":
        G, d = case["kv_heads"], case["dim"]
        out, row = torch.empty(x.q.shape, dtype=torch.float64, device=DEV), 0
        for b, (n, L) in enumerate(zip(x.new, x.lens)):
            rows = x.cache[x.table[b, :(L + PAGE - 1) // PAGE].long()].flatten(0, 1)[:L].double().unflatten(1, (2, G, d))
            out[row:row + n] = _attend(x.q[row:row + n].double(), rows[:, 0], rows[:, 1], d ** -0.5, L - n, case["chunk"], case["window"], x.sink)
            row += n
        return out
    if k == "experts":
        score = torch.softmax(x.logits.double(), 1)
        value, pick = score.topk(case["top"], 1)
        weight = value / value.sum(1, keepdim=True)
        h, y = x.h.double(), x.stream.double()
        for e in range(case["E"] + case["identity"]):
            t, j = (pick == e).nonzero(as_tuple=True)
            if e < case["E"]:
                o = torch.relu(h[t] @ x.up[e].double().T).square() @ x.down[e].double().T
            else:
                o = h[t]
            y.index_add_(0, t, o * weight[t, j, None])
        return y
    if k == "delta":
        return _exact_delta(case, x)
    return _exact_llama(case, x)
