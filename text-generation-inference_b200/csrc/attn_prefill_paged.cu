// Prefill / chunked-prefill attention over the PAGED KV pool on the 5th-generation tensor cores.
//
// Replaces: utils/flash_attn.py:43-127 `attention(q, k, v, cu_seqlens, max_s, softmax_scale)` in its prefill form
// (flash_llama_modeling.py:271-278; flash_attn_2_cuda.varlen_fwd, causal) of server/text_generation_server, and
// the prefill half of the paged twin (paged_llama_modeling.py:253-264).  Unlike the reference's prefill it reads K and V from the
// block pool (the step's own tokens have just been appended by b200_rope_kv_write_paged), so the queries of a step may follow a
// CACHED context: query i of sequence b sits at absolute position context_lens[b] - n_q(b) + i and attends keys 0 .. that position.
// That is what an add-on prefill over a prompt prefix, a chunked prefill and a mixed prefill + decode step need.
//
// The kernel and its design: attn_prompt.cuh.
#include "attn_prompt.cuh"
#include "tmap.cuh"
#include "../../include/b200_tgis.h"

using namespace b200;

template <int D>
static int launch_prefill_paged(const void* q, int64_t q_stride, int64_t T_q, const void* k_pool, const void* v_pool, int64_t num_blocks,
                                const int32_t* block_table, int64_t bt_stride, const int32_t* context_lens, const int32_t* cu_q, void* out,
                                int64_t out_stride, int B, int max_q, int n_heads, int n_kv, float scale, cudaStream_t st) {
  using C = PfCfg<D>;
  unsigned* gave_up = b200_gave_up_word();
  if (!gave_up) return B200_ERR_CUDA;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_prompt_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) { b200_set_last_error(cudaGetErrorString(e)); return B200_ERR_CUDA; }
    configured = true;
  }
  const CUtensorMap* mq = get_tmap_2d(q, (uint64_t)T_q, (uint64_t)n_heads * D, (uint64_t)q_stride, kPfM, 64, TmapDtype::kF16, TmapSwizzle::k128B);
  const uint64_t pool_rows = (uint64_t)num_blocks * n_kv * kPageTokens;
  const CUtensorMap* mk = get_tmap_2d(k_pool, pool_rows, D, D, kPageTokens, 64, TmapDtype::kF16, TmapSwizzle::kNone);
  const CUtensorMap* mv = get_tmap_2d(v_pool, pool_rows, D, D, kPageTokens, 64, TmapDtype::kF16, TmapSwizzle::kNone);
  if (!mq || !mk || !mv) return B200_ERR_CUDA;
  PfParams p = {};
  p.gave_up = gave_up;
  p.block_table = block_table;
  p.bt_stride = bt_stride;
  p.context_lens = context_lens;
  p.cu_q = cu_q;
  p.out = out;
  p.out_stride = out_stride;
  p.n_heads = n_heads;
  p.n_kv = n_kv;
  p.B = B;
  // two heads of a key / value head are equally long and share their keys; neighbouring query tiles are not, and a short prompt has no second one
  const int tiles = (max_q + kPfM - 1) / kPfM;
  p.pair = (int64_t)B * tiles * n_heads <= b200_num_sms() ? kPfSingle : (n_heads / n_kv) % 2 == 0 ? kPfHeads : kPfTiles;
  p.n_units = p.pair == kPfHeads ? n_heads / 2 : n_heads;
  p.n_groups = p.pair == kPfTiles ? (tiles + 1) / 2 : tiles;
  p.scale_log2 = scale * 1.4426950408889634f;
  const int64_t items = (int64_t)p.n_units * p.n_groups * B;
  if (items > (1 << 30)) { b200_set_last_error("attn_prefill_paged: too many query tiles"); return B200_ERR_ARG; }
  p.more_blocks = items > b200_num_sms();
  B200_LAUNCH((attn_prompt_kernel<D, false>), dim3((unsigned)items), dim3(kPfThreads), (size_t)C::kSmemBytes, st, *mq, *mk, *mv, p);
  b200_count_launches(1);
  return B200_OK;
}

// q: this step's query tokens, head-major [n_heads][d] at q + t * q_token_stride (halves), T_q tokens in all, sequence b owning
// tokens cu_seqlens_q[b] .. cu_seqlens_q[b+1].  context_lens[b] = tokens of sequence b in the pool INCLUDING this step's
// (already written).  Causal over absolute positions.  max_q = the largest number of query tokens of a sequence.
extern "C" int b200_attn_prefill_paged(const void* q, int64_t q_token_stride, int64_t T_q, const void* k_pool, const void* v_pool,
                                       int64_t num_blocks, const int32_t* block_table, int64_t block_table_stride,
                                       const int32_t* context_lens, const int32_t* cu_seqlens_q, void* out, int64_t out_token_stride,
                                       int B, int max_q, int n_heads, int n_kv_heads, int head_dim, float softmax_scale, void* stream) {
  if (B == 0 || max_q == 0 || T_q == 0) return B200_OK;
  if (n_kv_heads <= 0 || n_heads % n_kv_heads != 0) { b200_set_last_error("attn_prefill_paged: bad head counts"); return B200_ERR_ARG; }
  if (((q_token_stride | out_token_stride) & 7) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15) || num_blocks <= 0) {
    b200_set_last_error("attn_prefill_paged: q / out must be 16-byte aligned with token strides that are multiples of 8 halves");
    return B200_ERR_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (head_dim == 128)
    return launch_prefill_paged<128>(q, q_token_stride, T_q, k_pool, v_pool, num_blocks, block_table, block_table_stride, context_lens,
                                     cu_seqlens_q, out, out_token_stride, B, max_q, n_heads, n_kv_heads, softmax_scale, st);
  if (head_dim == 64)
    return launch_prefill_paged<64>(q, q_token_stride, T_q, k_pool, v_pool, num_blocks, block_table, block_table_stride, context_lens,
                                    cu_seqlens_q, out, out_token_stride, B, max_q, n_heads, n_kv_heads, softmax_scale, st);
  b200_set_last_error("attn_prefill_paged: head_dim must be 64 or 128");
  return B200_ERR_UNSUPPORTED;
}
