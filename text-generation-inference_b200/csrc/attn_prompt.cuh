// The kernel of prompt-sized attention on the 5th-generation tensor cores, for two kinds of cache:
//   head-major pages of fp16 keys and values, queries and results fp16 (attn_prefill_paged.cu);
//   token-major pages of bfloat16 rows [... keys of all key heads ... | ... values ...], queries and results fp32, a chunked mask and / or a
//   sliding window, sink logits (seq_talk_attn.cu).
//
// Design (12 warps, one CTA per SM).  A block takes its own item and then those of blocks that have not started (cluster launch control): with items
// dealt out in turn the SMs were busy for 75 % of the time on ragged prompts.  Head-major items come longest first; token-major ones from the step's
// last tile backwards, which is longest first within a sequence (and within a chunk).  An item is TWO query tiles of 128 rows that meet the same keys, so that the tensor cores work for
// one while the other is in its soft-max: two query heads of a key / value head when their number is even, else two neighbouring query tiles
// of a head.  While every tile can have an SM to itself it does (the second tile of an item is empty): two soft-max warpgroups slow each
// other down.  Back to back, us, one query tile of one head per CTA / two / this:
// one prompt of 100 tokens, 32 / 8 heads, d = 128 6.8 / 8.0 / 6.8, of 300 11.2 / 12.3 / 10.7; 32 / 4 heads, d = 64, 129 tokens 7.1 / 8.2 / 6.8.
//   warp 0      TMA producer.  Q tiles [128 x d] through a 128B-swizzled tensor map; per 128-key tile 8 KV pages x (K, V) x d/64
//               slabs, each one cp.async.bulk.tensor box [16 tokens x 64 halves] of the pool: the pool stores every token row
//               with its 16-byte chunks XOR-swizzled by (token & 7), which IS the tcgen05 SWIZZLE_128B image, so
//               pages land in shared memory ready for the tensor core without any software swizzle.  2-stage rings of K and V.
//   warp 1      MMA issuer (one elected thread): P0 V, Q0 K of the next key tile, P1 V, Q1 K of the next key tile, and so on.
//               S = Q K^T: tcgen05.mma kind::f16, both operands K-major from shared memory, fp32 accumulator in TMEM.
//               O += P V: A = P from TMEM (fp16, written by the softmax warps over their S), B = V as an MN-major
//               shared-memory operand (keys are the MMA K dimension, d contiguous), accumulator O in TMEM.
//   warps 4..7, 8..11   softmax of the first and the second tile: thread = one query row = one TMEM lane (no shuffles).  tcgen05.ld S, causal
//               mask, fp32 online softmax in the log2 domain, P rounded to fp16 (flash-attn semantics) and stored back to TMEM, O
//               rescaled in TMEM when a row's maximum moves.  (The reference always is the maximum: one that lags until it is 2^8
//               behind saves rescaling, one prompt of 8192 tokens 472 us where this takes 544, but a largest weight that is not exactly 1 is rounded:
//               up to 7 % more error behind 1500 cached keys whose scores spread.)  The row's sum adds the rounded P, what the
//               products weigh.  S of tile j is complete only after P V of tile j - 1 (issue order), so O is quiescent whenever a
//               softmax warp runs.
// Causality over absolute positions prunes whole key tiles.  Bound: a row's chain.  Of the 3700 cycles between a warp's scores of one 128-key tile and of the next
// (d = 128, both tiles of an item at work) it waits 1100 for P V and Q K^T, takes 350 for the maximum, 490 to rescale O and 1750 for the exponentials (1024 if MUFU
// were its own); between items there is the pipeline's drain.  Measured on B200 (us back to back; before: one query tile of one head per CTA): 13 prompts of
// 300 to 2048 tokens, 32 / 8 heads, d = 128 570 -> 218; 16 x 1024 428 -> 184; 8192 1197 -> 482; d = 64, 32 / 4 heads, 16 x 1024 140; 300 tokens after 1500 cached ones x 4
// 110 -> 66; 64 tokens x 10 17.7 -> 12.8.  Forms that were no faster (that / this at the time): items dealt out in turn 294 / 219 at the first of these; four more warps for
// the results 258 / 218 (compiled for 128 registers); two threads a row 245 / 225; scores of 64 keys in two places by turns 276 / 220; O rescaled between the
// exponentials 241 / 227; a quarter of the exponentials as polynomials on the FMA units 244 / 236; at d = 64, P beside S and the next scores ahead of P V
// 144 / 140 (16 x 1024).
// Token-major caches differ in this: a tile is 128 / rep tokens x the rep query heads of a key head (all rows meet the same keys), an item two
// neighbouring tiles; the softmax warps bring their tile's fp32 queries as bfloat16 themselves; P is the sum of two bfloat16 values (one alone is 2^-9
// off, and a maximum taken over 128 keys leaves fewer weights at exactly 1 than the 16-key tiles of talk_attn_mma_kernel: prompts of 1618 and 2000 tokens,
// 16 / 4 heads, d = 128, against float64 1.91e-3 with one value, 1.88e-3 there, 1.47e-3 with two); key tiles start at the first
// visible key; a key or value page is a box [16 tokens x 64 columns] that the copy itself swizzles; and what lies in the cache beside the keys
// that an item's queries see (slots that were never written, another request's leavings) is zeros to the products: whole pages by copies from
// outside the cache's rows, the rest of the first and the last visible page by the issuing warp, at most 15 rows each.
#pragma once
#include "common.cuh"
#include "seq_common.cuh"

namespace b200 {

constexpr int kPfM = 128;        // queries per tile, two tiles per item
constexpr int kPfN = 128;        // keys per tile = 8 pages
constexpr int kPfThreads = 384;  // warp 0 TMA, warp 1 MMA, warps 4..11 softmax
constexpr int kPfSlabBytes = 128 * 128;  // 128 rows x 64 halves
constexpr int kPfPageSlabBytes = kPageTokens * 128;
constexpr int kPfCornerBytes = 32 * 128;  // a softmax warp's rows on their way out
constexpr int kPfStages = 2;
// Items that can be known ahead (of short ones the copies are up to two in front of the soft-max).  A block asks for the next one as the copies of its item
// come to its last kPfAskTiles key tiles: late, so that a long item is not left to a block that still has one while other SMs are idle, and early enough that
// the answer, and blocks without a tile among the answers, hide behind the products.  Blocks that asked as soon as there was room took three further items
// each as they started (us, that / this: hybrid prompts of 1618 and 2000 tokens, 16 / 4 heads, SMs busy for 60 % of the time 100 / 76; 6 prompts of 310 to 536, 32 / 32
// heads 44 / 38; 8 of 100 to 1000, 32 / 4 heads of 64, 64 / 53).
constexpr int kPfAhead = 2, kPfAskTiles = 2;
// Registers per thread: the launch has 384 x 168; the two softmax warpgroups take 200 each, the other one keeps 104.  216 and 72, with O rescaled in 64
// columns at a time instead of 16, spilled in both (us, flushed L2, that / this: 13 prompts of 300 to 2048 tokens, 32 / 8 heads, d = 128 246 / 225; hybrid
// prompts of 1618 and 2000 tokens, 16 / 4 heads 109 / 100; 6 portions of 300 to 600 behind 700 keys, 40 / 40 heads 115 / 101).
constexpr int kPfSoftmaxRegs = 200, kPfServeRegs = 104;

template <int D>
struct PfCfg {
  static constexpr int kSlabs = D / 64;
  static constexpr int kTileBytes = kSlabs * kPfSlabBytes;  // a Q, K or V tile
  static constexpr int kNumBars = 2 + 4 * kPfStages + 8 + 2 * kPfAhead + 2;    // q_full, q_empty | k_full, k_empty, v_full, v_empty | s_full[2], p_ready[2][2 halves], o_full[2]
  static constexpr int kSmemBytes = (2 + 2 * kPfStages) * kTileBytes + 8 * kPfCornerBytes + kNumBars * 8 + 16 + 1024;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
  static constexpr int kTmemCols = 512;  // S0 [0,128) | S1 [128,256) | O0 [256, 256 + D) | O1 behind it
};

// two tiles of an item: two query heads, two neighbouring query tiles, or the second one is empty
enum PfPair { kPfHeads, kPfTiles, kPfSingle };

struct PfParams {
  const int32_t* block_table;
  int64_t bt_stride;
  const int32_t* context_lens;
  const int32_t* cu_q;
  void* out;
  int64_t out_stride;
  int n_heads, n_kv, B;
  int pair;              // what an item's two tiles are (PfPair)
  int n_units, n_groups; // head (pair)s, query tile (pair)s of the longest sequence
  int more_blocks;       // the grid is larger than the GPU: blocks take more items
  float scale_log2;
  unsigned* gave_up;     // b200_gave_up_word
  // token-major caches only
  const float* q;        // [tokens][heads][D]
  const int64_t* position_ids;
  const float* sink;     // [heads] or NULL
  int k_off, v_off, chunk, window;
  int rep, log2_rep, tokens;  // query heads of a key head that share a tile, tokens of a tile: rep * tokens == 128 (rows / rep as divisions: 18 us of 76)
};

// one item: the rows and key tiles of its two query tiles
struct PfItem {
  int b, q_begin, past, last_page, kv_head;
  int q0[2], rows[2], head[2], k0[2], n_kt[2], j0, n;  // key tiles k0 .. n_kt - 1 of each, j0 .. n - 1 of both
  int lo, hi;  // token-major: first and last key that a query of the item sees
};

// first key that the query at position p sees
__device__ __forceinline__ int pf_first_visible(int p, int chunk, int window) {
  int lo = chunk > 0 ? (p / chunk) * chunk : 0;
  if (window > 0) lo = max(lo, p - window + 1);
  return lo;
}

// item i; n = 0: there is no such tile.  The whole warp calls it.
template <bool TOKEN_MAJOR>
__device__ __forceinline__ PfItem pf_item(const PfParams& p, int i) {
  PfItem it;
  if constexpr (TOKEN_MAJOR) {
    // two neighbouring tiles of `tokens` tokens x `rep` heads of a key head; last tiles of the step first
    int tile = p.n_groups - 1 - i / p.n_units;
    const int span = p.pair == kPfSingle ? p.tokens : 2 * p.tokens;  // tokens of an item
    it.kv_head = i % p.n_units;
    seq::find_ragged_tile(p.cu_q, p.B, 1, span, it.b, tile);
    it.n = it.j0 = 0;
    it.n_kt[0] = it.n_kt[1] = it.k0[0] = it.k0[1] = 0;
    if (it.b >= p.B) return it;
    it.q_begin = p.cu_q[it.b];
    const int n_q = p.cu_q[it.b + 1] - it.q_begin;
    it.past = (int)p.position_ids[it.q_begin];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      it.head[u] = it.kv_head * p.rep;
      it.q0[u] = tile * span + u * p.tokens;
      it.rows[u] = min(min(p.tokens, span - u * p.tokens), n_q - it.q0[u]) * p.rep;
      if (it.rows[u] > 0) {
        it.k0[u] = pf_first_visible(it.past + it.q0[u], p.chunk, p.window) / kPfN;
        it.n_kt[u] = (it.past + it.q0[u] + (it.rows[u] >> p.log2_rep) - 1) / kPfN + 1;
      }
    }
    it.j0 = it.n_kt[1] > 0 ? min(it.k0[0], it.k0[1]) : it.k0[0];
    it.n = max(it.n_kt[0], it.n_kt[1]);
    it.lo = pf_first_visible(it.past + it.q0[0], p.chunk, p.window);
    it.hi = it.past + min(n_q, it.q0[0] + span) - 1;
    return it;
  }
  // longest query tiles first
  const int per = p.B * p.n_units, group = p.n_groups - 1 - i / per, r = i % per, unit = r % p.n_units;
  it.b = r / p.n_units;
  it.q_begin = p.cu_q[it.b];
  const int n_q = p.cu_q[it.b + 1] - it.q_begin, L = p.context_lens[it.b];
  it.past = max(L - n_q, 0);  // cached tokens in front of this step's first query
  it.last_page = (L - 1) / kPageTokens;
  it.lo = it.hi = 0;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    it.head[u] = p.pair == kPfHeads ? 2 * unit + u : unit;
    it.q0[u] = (p.pair == kPfTiles ? 2 * group + u : group) * kPfM;
    it.rows[u] = u == 1 && p.pair == kPfSingle ? 0 : min(kPfM, n_q - it.q0[u]);
    it.k0[u] = 0;
    it.n_kt[u] = it.rows[u] > 0 ? (it.past + it.q0[u] + it.rows[u] - 1) / kPfN + 1 : 0;  // key tiles the last row reaches
  }
  it.kv_head = it.head[0] / (p.n_heads / p.n_kv);
  it.j0 = 0;
  it.n = max(it.n_kt[0], it.n_kt[1]);
  return it;
}

// Asks for a block of the grid that has not started: its index in x, or -1 when there is none left (no further request may follow then).
// One thread; `resp` 16 bytes of shared memory, `bar` an mbarrier of one arrival.
__device__ __forceinline__ int take_block(uint32_t* resp, uint64_t* bar, uint32_t parity, bool& ok) {
  fence_proxy_async_smem();  // the previous answer has been read
  mbar_arrive_expect_tx(bar, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(resp)), "r"(smem_u32(bar)) : "memory");
  mbar_wait_soft(bar, parity, ok);
  if (!ok) return -1;
  uint32_t taken, x;
  asm volatile(
      "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t"
      "ld.shared.b128 h, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
      : "=r"(taken), "=r"(x)
      : "r"(smem_u32(resp))
      : "memory");
  fence_proxy_async_smem();  // the next request writes the answer's place through the async proxy
  return taken ? (int)x : -1;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f32x2_split(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float add_f32_f16(float a, uint16_t h) {
  float r;
  asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(r) : "h"(h), "f"(a));
  return r;
}

// MN-major shared-memory operand, 128-byte swizzle: rows along K (here: keys) of 128 bytes = 64 MN elements, 8-row swizzle atoms
// `sbo` bytes apart, blocks of 64 MN elements `lbo` bytes apart.  Bit layout as umma_desc_kmajor_sw128 (common.cuh).
__device__ __forceinline__ uint64_t umma_desc_mnmajor_sw128(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// rows from .. to - 1 (if any) of a K or V tile become zeros; the whole warp calls it, and fences before the tensor cores read them
template <int SLABS>
__device__ __forceinline__ void pf_zero_rows(unsigned char* tile, int from, int to, int lane) {
  for (int i = from * 8 + lane; i < to * 8; i += 32)
#pragma unroll
    for (int s = 0; s < SLABS; ++s) *reinterpret_cast<uint4*>(tile + s * kPfSlabBytes + i * 16) = make_uint4(0u, 0u, 0u, 0u);
}

template <int D, bool TOKEN_MAJOR>
__global__ void __launch_bounds__(kPfThreads, 1)
attn_prompt_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                          const __grid_constant__ CUtensorMap tmap_v, const PfParams p) {
  using C = PfCfg<D>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* sQ = smem;
  unsigned char* sK = sQ + 2 * C::kTileBytes;
  unsigned char* sV = sK + kPfStages * C::kTileBytes;
  unsigned char* sOut = sV + kPfStages * C::kTileBytes;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sOut + 8 * kPfCornerBytes);
  uint64_t* q_empty = q_full + 1;
  uint64_t* k_full = q_empty + 1;
  uint64_t* k_empty = k_full + kPfStages;
  uint64_t* v_full = k_empty + kPfStages;
  uint64_t* v_empty = v_full + kPfStages;
  uint64_t* s_full = v_empty + kPfStages;
  uint64_t* p_ready = s_full + 2;
  uint64_t* o_full = p_ready + 4;
  uint64_t* next_full = o_full + 2;
  uint64_t* next_empty = next_full + kPfAhead;
  uint64_t* taken = next_empty + kPfAhead;
  uint64_t* ask = taken + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ask + 1);
  __shared__ __align__(16) uint32_t s_resp[4];
  __shared__ int s_next[kPfAhead];

  pdl_launch_dependents();
  const int warp = warp_id(), lane = lane_id();
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    mbar_init(q_full, TOKEN_MAJOR ? 4 : 1);
    mbar_init(q_empty, TOKEN_MAJOR ? 4 : 1);  // token-major: the second tile's q_full
    for (int s = 0; s < kPfStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(&s_full[u], 1);
      mbar_init(&p_ready[2 * u], 4);
      mbar_init(&p_ready[2 * u + 1], 4);
      mbar_init(&o_full[u], 1);
    }
    for (int s = 0; s < kPfAhead; ++s) {
      mbar_init(&next_full[s], 1);
      mbar_init(&next_empty[s], 10);  // producer, issuer, eight softmax warps
    }
    mbar_init(taken, 1);
    mbar_init(ask, 1);
    mbar_fence_init();
  }
  if (warp == 2) tmem_alloc<C::kTmemCols>(tmem_slot);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  // the next item of this CTA, or -1
  int at = 0, at_ph = 0;
  auto next_item = [&]() {
    mbar_wait_soft(&next_full[at], at_ph, ok);
    const int i = ok ? s_next[at] : -1;
    __syncwarp();
    if (lane == 0) mbar_arrive(&next_empty[at]);
    if (++at == kPfAhead) { at = 0; at_ph ^= 1; }
    return __reduce_max_sync(0xffffffffu, i);  // a warp reduction: the compiler knows its result, and the loops' control, to be uniform
  };
  pdl_wait();  // q, the index tensors and the pool's newest tokens are the previous kernels' output

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPfServeRegs));
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      int st = 0, ph = 1, qph = 1;
      for (int i = blockIdx.x; i >= 0; i = next_item()) {
        const PfItem it = pf_item<TOKEN_MAJOR>(p, i);
        if (it.n == 0) {  // only the block's own item can be empty
          if (lane == 0) mbar_arrive(ask);
          continue;
        }
        if constexpr (!TOKEN_MAJOR) mbar_wait_soft(q_empty, qph, ok);  // the previous item's last Q K^T
        qph ^= 1;
        if (!TOKEN_MAJOR && lane == 0) {
          mbar_arrive_expect_tx(q_full, ((it.n_kt[0] > 0) + (it.n_kt[1] > 0)) * C::kTileBytes);
          for (int u = 0; u < 2; ++u)
            if (it.n_kt[u] > 0)
              for (int s = 0; s < C::kSlabs; ++s)
                tma_load_2d(sQ + u * C::kTileBytes + s * kPfSlabBytes, &tmap_q, it.head[u] * D + s * 64, it.q_begin + it.q0[u], q_full);
        }
        const int32_t* bt = p.block_table + (int64_t)it.b * p.bt_stride;
        for (int j = it.j0; j < it.n; ++j) {
          if (lane == 0 && j == max(it.j0, it.n - kPfAskTiles)) mbar_arrive(ask);
          // 8 pages of this key tile, a lane each
          int page = j * (kPfN / kPageTokens) + (lane & 7), row;
          if constexpr (TOKEN_MAJOR) {
            // row of the cache viewed as [blocks * 16, row width]; a page without a visible key is not looked up (its entry may be any value):
            // the copy then lies in front of the first row and brings zeros
            row = page >= it.lo / kPageTokens && page <= it.hi / kPageTokens ? bt[page] * kPageTokens : -kPageTokens;
          } else {
            // row of the pool viewed as [blocks * n_kv * 16, d]; pages past the sequence's last one repeat it (masked by the softmax warps)
            row = (bt[min(page, it.last_page)] * p.n_kv + it.kv_head) * kPageTokens;
          }
          const int k_col = TOKEN_MAJOR ? p.k_off + it.kv_head * D : 0, v_col = TOKEN_MAJOR ? p.v_off + it.kv_head * D : 0;
          mbar_wait_soft(&k_empty[st], ph, ok);
          if (lane == 0) mbar_arrive_expect_tx(&k_full[st], C::kTileBytes);
          __syncwarp();
          if (lane < 8)
            for (int s = 0; s < C::kSlabs; ++s)
              tma_load_2d(sK + st * C::kTileBytes + s * kPfSlabBytes + lane * kPfPageSlabBytes, &tmap_k, k_col + s * 64, row, &k_full[st]);
          __syncwarp();
          mbar_wait_soft(&v_empty[st], ph, ok);
          if (lane == 0) mbar_arrive_expect_tx(&v_full[st], C::kTileBytes);
          __syncwarp();
          if (lane < 8)
            for (int s = 0; s < C::kSlabs; ++s)
              tma_load_2d(sV + st * C::kTileBytes + s * kPfSlabBytes + lane * kPfPageSlabBytes, &tmap_v, v_col + s * 64, row, &v_full[st]);
          __syncwarp();
          if (++st == kPfStages) { st = 0; ph ^= 1; }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      constexpr uint32_t fmt = TOKEN_MAJOR ? ((1u << 7) | (1u << 10)) : 0u;  // bfloat16 operands
      constexpr uint32_t idesc_qk = umma_idesc_f16_f32acc(kPfM, kPfN) | fmt;
      constexpr uint32_t idesc_pv = umma_idesc_f16_f32acc(kPfM, D) | (1u << 16) | fmt;  // B (= V) is MN-major
      const uint64_t qdesc = umma_desc_kmajor_sw128(smem_u32(sQ)), kdesc = umma_desc_kmajor_sw128(smem_u32(sK));
      const uint64_t vdesc = umma_desc_mnmajor_sw128(smem_u32(sV), kPfSlabBytes, 1024);
      int kst = 0, kph = 0, vst = 0, vph = 0, qph = 0, qph1 = 0, pph[2] = {0, 0};
      auto issue_qk = [&](int u) {
        if (elect_one()) {
          const uint64_t a = qdesc + (uint64_t)((u * C::kTileBytes) >> 4), b = kdesc + (uint64_t)((kst * C::kTileBytes) >> 4);
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint64_t off = (uint64_t)((k >> 2) * (kPfSlabBytes >> 4) + (k & 3) * 2);
            umma_f16_ss(tmem_base + u * kPfN, a + off, b + off, idesc_qk, k > 0 ? 1u : 0u);
          }
          umma_commit(&s_full[u]);
        }
        __syncwarp();
      };
      auto release = [&](uint64_t* bar) {
        if (elect_one()) umma_commit(bar);
        __syncwarp();
      };
      for (int i = blockIdx.x; i >= 0; i = next_item()) {
        PfItem it = pf_item<TOKEN_MAJOR>(p, i);
        it.n_kt[0] = __reduce_max_sync(0xffffffffu, it.n_kt[0]);
        it.n_kt[1] = __reduce_max_sync(0xffffffffu, it.n_kt[1]);
        it.n = max(it.n_kt[0], it.n_kt[1]);
        if (it.n == 0) continue;
        if constexpr (TOKEN_MAJOR) {
          it.k0[0] = __reduce_max_sync(0xffffffffu, it.k0[0]);
          it.k0[1] = __reduce_max_sync(0xffffffffu, it.k0[1]);
          it.j0 = __reduce_max_sync(0xffffffffu, it.j0);
          if (it.n_kt[0] > 0) {
            mbar_wait_soft(q_full, qph, ok);
            qph ^= 1;
          }
          if (it.n_kt[1] > 0) {
            mbar_wait_soft(q_empty, qph1, ok);
            qph1 ^= 1;
          }
          tcgen05_fence_after();
        } else {
          mbar_wait_soft(q_full, qph, ok);
          qph ^= 1;
        }
        for (int j = it.j0 - 1; j < it.n; ++j) {  // P V of key tile j, Q K^T of key tile j + 1
          const bool more = j + 1 < it.n;
          if (more) mbar_wait_soft(&k_full[kst], kph, ok);
          if (j >= it.j0) {
            mbar_wait_soft(&v_full[vst], vph, ok);
            if constexpr (TOKEN_MAJOR) {
              // value rows of the first and the last visible page that no query of the item sees: their weight is 0, but 0 x NaN is NaN
              const int key0 = j * kPfN;
              pf_zero_rows<C::kSlabs>(sV + vst * C::kTileBytes, max((it.lo & -kPageTokens) - key0, 0), min(it.lo - key0, kPfN), lane);
              pf_zero_rows<C::kSlabs>(sV + vst * C::kTileBytes, max(it.hi + 1 - key0, 0), min((it.hi | (kPageTokens - 1)) + 1 - key0, kPfN), lane);
              fence_proxy_async_smem();
              __syncwarp();
            }
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (j >= it.k0[u] && j < it.n_kt[u]) {
              const uint64_t b = vdesc + (uint64_t)((vst * C::kTileBytes) >> 4);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                mbar_wait_soft(&p_ready[2 * u + h], pph[u], ok);
                tcgen05_fence_after();
                if (elect_one()) {
#pragma unroll
                  for (int kk = h * 4; kk < h * 4 + 4; ++kk) {  // 16 keys = 2 swizzle atoms of 8 key rows = 2048 bytes per step
                    umma_f16_ts(tmem_base + 256 + u * D, tmem_base + u * kPfN + kk * 8, b + (uint64_t)((kk * 2048) >> 4), idesc_pv, (j > it.k0[u] || kk > 0) ? 1u : 0u);
                    if constexpr (TOKEN_MAJOR)  // the weights' second halves
                      umma_f16_ts(tmem_base + 256 + u * D, tmem_base + u * kPfN + kPfN / 2 + kk * 8, b + (uint64_t)((kk * 2048) >> 4), idesc_pv, 1u);
                  }
                  if (h == 1 && j == it.n_kt[u] - 1) umma_commit(&o_full[u]);
                }
                __syncwarp();
              }
              pph[u] ^= 1;
            } else {
              tcgen05_fence_after();
            }
            if (j + 1 >= it.k0[u] && j + 1 < it.n_kt[u]) issue_qk(u);
          }
          if (j >= it.j0) {
            release(&v_empty[vst]);
            if (++vst == kPfStages) { vst = 0; vph ^= 1; }
          }
          if (more) {
            release(&k_empty[kst]);
            if (++kst == kPfStages) { kst = 0; kph ^= 1; }
            if (!TOKEN_MAJOR && j + 2 == it.n) release(q_empty);
          }
        }
      }
    } else if (warp == 3) {
      // ------------------------------------------------------------------ scheduler: after the block's own item those of blocks that have not
      // started, as long as there are any; items without a tile are passed over here
      int slot = 0, ph = 1, tph = 0, aph = 0;
      auto publish = [&](int i) {
        mbar_wait_soft(&next_empty[slot], ph, ok);
        if (lane == 0) {
          s_next[slot] = i;
          mbar_arrive(&next_full[slot]);
        }
        if (++slot == kPfAhead) { slot = 0; ph ^= 1; }
      };
      for (int i = 0; p.more_blocks && i >= 0;) {
        mbar_wait_soft(ask, aph, ok);
        aph ^= 1;
        do {
          if (lane == 0) i = take_block(s_resp, taken, tph, ok);
          tph ^= 1;
          i = __shfl_sync(0xffffffffu, i, 0);
        } while (i >= 0 && pf_item<TOKEN_MAJOR>(p, i).n == 0);
        if (i >= 0) publish(i);
      }
      publish(-1);
    }
  } else {
    // ------------------------------------------------------------------ softmax warps: thread = query row = TMEM lane
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPfSoftmaxRegs));
    const int u = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tmem_s = tmem_base + lane_base + u * kPfN, tmem_o = tmem_base + lane_base + 256 + u * D;
    int sph = 0, oph = 0;
    for (int i = blockIdx.x; i >= 0; i = next_item()) {
      const PfItem it = pf_item<TOKEN_MAJOR>(p, i);
      const int n_kt = u ? it.n_kt[1] : it.n_kt[0], q0 = u ? it.q0[1] : it.q0[0];
      if (n_kt == 0) continue;
      // absolute positions of the warp's first query and of this row's; rows past the tile's last one are padding: computed, not stored
      const int rows = u ? it.rows[1] : it.rows[0], head = u ? it.head[1] : it.head[0], k0 = u ? it.k0[1] : it.k0[0];
      const int first = it.past + q0 + (TOKEN_MAJOR ? (quarter * 32 >> p.log2_rep) : quarter * 32);
      const int qpos = TOKEN_MAJOR ? it.past + q0 + (row >> p.log2_rep) : first + lane;
      int lo = 0, lo_last = 0;  // first key of this row, and of the warp's last row
      if constexpr (TOKEN_MAJOR) {
        lo = pf_first_visible(qpos, p.chunk, p.window);
        lo_last = __reduce_max_sync(0xffffffffu, lo);
        // the tile's queries, rounded to bfloat16, as a SWIZZLE_128B image; the last scores of the previous item are in: its Q is not read any more
        const float* src = p.q + ((int64_t)(it.q_begin + q0) * p.n_heads + head) * D;
        unsigned char* dst = sQ + u * C::kTileBytes;
#pragma unroll 1
        for (int r0 = 0; r0 < 32; r0 += 8) {
          float4 v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int r = quarter * 32 + r0 + k, tok = r >> p.log2_rep, hh = r - tok * p.rep;
            v[k] = r < rows && lane * 4 < D ? *reinterpret_cast<const float4*>(src + ((int64_t)tok * p.n_heads + hh) * D + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int r = quarter * 32 + r0 + k;
            if (lane * 4 < D) {
              const int slab = lane >> 4, ch = (lane & 15) >> 1;
              uint2 w;
              w.x = pack_bf16x2(v[k].x, v[k].y);
              w.y = pack_bf16x2(v[k].z, v[k].w);
              *reinterpret_cast<uint2*>(dst + slab * kPfSlabBytes + r * 128 + ((ch ^ (r & 7)) << 4) + (lane & 1) * 8) = w;
            }
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(u ? q_empty : q_full);
      }
      float m = 0.f;
      float sum[2] = {0.f, 0.f};  // two partial sums of the row
      for (int j = k0; j < n_kt; ++j) {
        mbar_wait_soft(&s_full[u], sph, ok);
        sph ^= 1;
        tcgen05_fence_after();
        float s[kPfN];
#pragma unroll
        for (int c = 0; c < kPfN / 32; ++c) tmem_ld_32x32b_x32(tmem_s + c * 32, reinterpret_cast<uint32_t(&)[32]>(s[c * 32]));
        tmem_ld_wait();
        const int key0 = j * kPfN;
        float scale = p.scale_log2;
        if (scale <= 0.f) {
#pragma unroll
          for (int c = 0; c < kPfN; ++c) s[c] *= scale;
          scale = 1.f;
        }
        // warp-uniform: some row of this warp has keys to mask in this tile.  Looked at 32 keys at a time, and the two ends by themselves: in one piece over all 128
        // it took 800 to 2000 cycles of the 3700 of a tile
        if (key0 + kPfN - 1 > first || key0 < lo_last) {
#pragma unroll
          for (int h = 0; h < kPfN / 32; ++h) {
            const int from = key0 + h * 32;
            if (from + 31 > first) {
#pragma unroll
              for (int c = 0; c < 32; ++c) s[h * 32 + c] = c <= qpos - from ? s[h * 32 + c] : -INFINITY;
            }
            if (TOKEN_MAJOR && from < lo_last) {
#pragma unroll
              for (int c = 0; c < 32; ++c) s[h * 32 + c] = c >= lo - from ? s[h * 32 + c] : -INFINITY;
            }
          }
        }
        float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int c = 4; c + 8 <= kPfN; c += 8) {
#pragma unroll
          for (int k = 0; k < 4; ++k) mx4[k] = max3(mx4[k], s[c + k], s[c + 4 + k]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) mx4[k] = fmaxf(mx4[k], s[kPfN - 4 + k]);
        const float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * scale;
        if (j == k0) {
          m = fmaxf(mx, -1.0e30f);  // finite: a row may meet its first visible key, or its first score above -infinity, in a later tile
          if (TOKEN_MAJOR && p.sink) {  // one more logit of the denominator
            const float sk = p.sink[head + (row & (p.rep - 1))] * 1.4426950408889634f;
            m = fmaxf(m, sk);
            sum[0] = fast_exp2(sk - m);
          }
        } else {
          const bool grew = mx > m;
          if (__any_sync(0xffffffffu, grew)) {
            const float alpha = grew ? fast_exp2(m - mx) : 1.f;
            if (grew) m = mx;
            sum[0] *= alpha;
            sum[1] *= alpha;
#pragma unroll
            for (int c = 0; c < D; c += 16) {  // few columns at once: the tile's scores hold 128 registers
              uint32_t o[16];
              tmem_ld_32x32b_x16(tmem_o + c, o);
              tmem_ld_wait();
#pragma unroll
              for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
#pragma unroll
              for (int k = 0; k < 16; k += 16) tmem_st_32x32b_x16(tmem_o + c + k, reinterpret_cast<const uint32_t(&)[16]>(o[k]));
            }
          }
        }
        const uint64_t scale2 = f32x2(scale, scale), neg_m = f32x2(-m, -m);
#pragma unroll
        for (int h = 0; h < kPfN / 32; ++h) {
          uint32_t pk[16], rest[TOKEN_MAJOR ? 16 : 1];
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float a, b;
            const uint64_t x = fma_f32x2(f32x2(s[h * 32 + c], s[h * 32 + c + 1]), scale2, neg_m);
            f32x2_split(x, a, b);
            a = fast_exp2(a);
            b = fast_exp2(b);
            if constexpr (TOKEN_MAJOR) {
              pk[c / 2] = pack_bf16x2(a, b);
              rest[c / 2] = pack_bf16x2(a - __uint_as_float(pk[c / 2] << 16), b - __uint_as_float(pk[c / 2] & 0xffff0000u));
              f32x2_split(add_f32x2(f32x2(sum[0], sum[1]), f32x2(a, b)), sum[0], sum[1]);
            } else {
              pk[c / 2] = pack_half2(a, b);
              sum[0] = add_f32_f16(sum[0], (uint16_t)pk[c / 2]);
              sum[1] = add_f32_f16(sum[1], (uint16_t)(pk[c / 2] >> 16));
            }
          }
          tmem_st_32x32b_x16(tmem_s + h * 16, pk);
          if constexpr (TOKEN_MAJOR) tmem_st_32x32b_x16(tmem_s + kPfN / 2 + h * 16, rest);
          if (h & 1) {  // half of P: its products run under the exponentials of the other half
            tmem_st_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[2 * u + (h >> 1)]);
          }
        }
      }
      mbar_wait_soft(&o_full[u], oph, ok);
      oph ^= 1;
      tcgen05_fence_after();
      const float l = sum[0] + sum[1], inv = l > 0.f ? 1.f / l : 0.f;
      // 64 columns at a time through the warp's corner of shared memory, so that a store covers whole lines (16-byte pieces of 32 rows at once cost
      // thirty-two passes of the store unit)
      unsigned char* corner = sOut + (warp - 4) * kPfCornerBytes;
      if constexpr (TOKEN_MAJOR) {
        float* op = reinterpret_cast<float*>(p.out) + ((int64_t)(it.q_begin + q0) * p.n_heads + head) * D;
#pragma unroll
        for (int c = 0; c < D; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(tmem_o + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 8; ++k)
            *reinterpret_cast<float4*>(corner + lane * 128 + ((k ^ (lane & 7)) << 4)) =
                make_float4(__uint_as_float(o[4 * k]) * inv, __uint_as_float(o[4 * k + 1]) * inv, __uint_as_float(o[4 * k + 2]) * inv, __uint_as_float(o[4 * k + 3]) * inv);
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int r = k * 4 + (lane >> 3), ch = lane & 7, rr = quarter * 32 + r, tok = rr >> p.log2_rep, hh = rr - tok * p.rep;
            if (rr < rows)
              *reinterpret_cast<float4*>(op + ((int64_t)tok * p.n_heads + hh) * D + c + ch * 4) = *reinterpret_cast<const float4*>(corner + r * 128 + ((ch ^ (r & 7)) << 4));
          }
          __syncwarp();
        }
      } else {
        __half* op = reinterpret_cast<__half*>(p.out) + (int64_t)(it.q_begin + q0 + quarter * 32) * p.out_stride + head * D;
#pragma unroll
        for (int c = 0; c < D; c += 64) {
          uint32_t o[64];
          tmem_ld_32x32b_x32(tmem_o + c, reinterpret_cast<uint32_t(&)[32]>(o[0]));
          tmem_ld_32x32b_x32(tmem_o + c + 32, reinterpret_cast<uint32_t(&)[32]>(o[32]));
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            uint4 w;
            w.x = pack_half2(__uint_as_float(o[8 * k]) * inv, __uint_as_float(o[8 * k + 1]) * inv);
            w.y = pack_half2(__uint_as_float(o[8 * k + 2]) * inv, __uint_as_float(o[8 * k + 3]) * inv);
            w.z = pack_half2(__uint_as_float(o[8 * k + 4]) * inv, __uint_as_float(o[8 * k + 5]) * inv);
            w.w = pack_half2(__uint_as_float(o[8 * k + 6]) * inv, __uint_as_float(o[8 * k + 7]) * inv);
            *reinterpret_cast<uint4*>(corner + lane * 128 + ((k ^ (lane & 7)) << 4)) = w;
          }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int r = k * 4 + (lane >> 3), ch = lane & 7;
            if (quarter * 32 + r < rows)
              *reinterpret_cast<uint4*>(op + (int64_t)r * p.out_stride + c + ch * 8) = *reinterpret_cast<const uint4*>(corner + r * 128 + ((ch ^ (r & 7)) << 4));
          }
          __syncwarp();
        }
      }
      tcgen05_fence_before();  // the next item's first P V overwrites O: it is issued after this warp's next arrival at p_ready
    }
  }

  if (!ok) gave_up(p.gave_up);
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc<C::kTmemCols>(tmem_base);
}

}  // namespace b200
