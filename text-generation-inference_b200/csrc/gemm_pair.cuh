// Prompt-sized linears  Y[T, N] = X[T, K] . W[N, K]^T  on PAIRS of SMs: `tcgen05.mma.cta_group::2`, 256 features x up to 256 tokens per
// accumulator tile, persistent over the tiles of the output.
//
// Used by gemm_f16.cu (fp16 / bfloat16 weights) and gemm_w4a16.cu (GPTQ int4 weights, de-quantised into shared memory) for calls of more
// tokens than their weight-streaming kernels are good at, and by seq_group_gemm.cu for routed experts with many rows each (row tiles of one expert,
// found from the plan's offsets).  Bound: the tensor pipe (an m256 n256 k16 product takes the pair 128 cycles) and,
// close behind it, the L2 -> shared-memory path.
//
//   * Swap-AB: features are the UMMA M dimension (each CTA of the pair holds 128 of the 256), tokens its N dimension.  A CTA stages its own
//     features and HALF of the tile's tokens: 32 KB per 64-wide k-block for 128 x 256 outputs, two thirds of what a single CTA needs.
//   * The token tile is any multiple of 32 up to 256, chosen per call so that the tiles fill the pairs (pair_plan), and the last one is cut
//     to the rows that are left: N is a run-time field of the instruction descriptor.
//   * Two accumulators in TMEM (2 x 256 columns): the epilogue of one tile runs under the products of the next.  Calls of up to 256 tokens cut k into
//     as many pieces as the weight-streaming kernel would, with an accumulator each (512 columns hold 2 of up to 256 tokens, 4 of 128, 8 of 64; more than
//     256 columns of them leave no second tile's room), and the epilogue adds them in fp32: one sum of all k in the tensor core is further off (fp16
//     results, k = 20480, 100 tokens: 2.084e-4 against float64, 2.073e-4 in that kernel's cuts and in pieces).
//   * int4: four teams of four warps turn 64 k of a record each into the SWIZZLE_128B image of an fp16 A tile (thread = feature row, eight
//     conflict-free 16-byte stores).  One de-quantised tile serves up to 256 tokens, twice as many as the weight-streaming kernel's, and shared
//     memory as the operand's place leaves TMEM to the accumulators.
//   * Gate|up weights with SiLU(gate) * up: a CTA takes 64 gate features and the 64 up features that belong to them, sixteen of each per epilogue
//     warp, so that both factors of an output sit in one warp, sixteen lanes apart.
//   * Lane = feature in the epilogue, transposed through shared memory into 16-byte stores; rows that those do not fit are stored by value.
//
// Measured on B200 (us, launches back to back over weights larger than L2; before = one CTA per tile): fp16 4099 x 4096 x 4096 133 -> 98, 300 x 4096 x
// 4096 31.2 -> 16.0, 3001 x 5120 x 20480 668 -> 425 (1.48 PFLOP/s; cuBLAS 442; a call by itself with flushed L2 785 -> 501); int4 4099 x 14336 x 4096 451
// -> 365 (1.32 PFLOP/s; by itself 514 -> 428), gate|up 1000 x 4096 x 28672 295 -> 199.
//
// Warp roles: 0..3 epilogue | (int4: 4..19 de-quantisation) | then W producer / TMEM allocation, x producer, MMA issuer (leader CTA), idle.
// Barriers: `full` and `tmem_empty` live in the leader (the pair's even CTA) and count both CTAs' work, `empty` and `tmem_full` live in
// each and are arrived at by multicast commits of the leader's products.  Every wait is bounded (mbar_wait_soft): a thread that gives up goes through
// the rest without waiting; the block then lets copies in flight land, tells the host, frees its TMEM and ends.  No role waits for what the previous
// kernel has still to deliver: what can be done ahead of it (the first round of the rings of records and stages) is done, then comes pdl_wait.
// A team skips phases of `empty` (the teams take turns): products complete in order, so having seen the stage of its last turn freed implies
// that every earlier one was, and no phase is mistaken for another while the ring is at least as deep as there are teams per stage count
// (four stages, or two when a stage holds two k-blocks).
#pragma once
#include "common.cuh"
#include "tmap.cuh"
#include "w4_format.cuh"
#include "../../include/b200_tgis.h"

#include <cuda_bf16.h>

namespace b200 {

constexpr int kPairM = 256;          // features per tile, 128 per CTA
constexpr int kPairMaxN = 256;       // tokens per tile
constexpr int kPairK = 64;           // k per block: one 128-byte swizzle row
constexpr int kPairABytes = 128 * kPairK * 2;
constexpr int kPairMaxStages = 10;
// a k-block: the CTA's features, and its half of the token tile
__host__ __device__ constexpr int pair_block_bytes(int tn) { return kPairABytes + (tn / 2) * kPairK * 2; }

// what the weights are, and what happens to the result (the first four as FMT of gemm_f16.cu)
enum PairKind { kPairF16 = 0, kPairBf16 = 1, kPairBf16F32 = 2, kPairBf16Relu2 = 3, kPairW4 = 4, kPairW4Silu = 5,
  // grouped: rows of X are compact, those of one expert side by side, W is one matrix per expert
  kPairExpBf16 = 6, kPairExpBf16F32 = 7, kPairExpRelu2 = 8,
  kPairF16Silu = 9 };

template <int KIND>
struct PairCfg {
  static constexpr bool kInt4 = KIND == kPairW4 || KIND == kPairW4Silu;
  static constexpr bool kExperts = KIND >= kPairExpBf16 && KIND <= kPairExpRelu2;
  static constexpr bool kOut32 = KIND == kPairBf16F32 || KIND == kPairExpBf16F32;
  static constexpr bool kAct = KIND == kPairW4Silu;
  static constexpr bool kHalves = KIND == kPairF16Silu;  // a CTA's features: 64 of the gate, then the 64 up features that belong to them
  static constexpr bool kPieces = !kInt4 && !kExperts && !kHalves;
  static constexpr int kThreads = kInt4 ? 768 : 256;
  static constexpr int kRingBytes = (kInt4 ? 5 : 6) * pair_block_bytes(kPairMaxN);
  static constexpr int kRecs = kInt4 ? 4 : 0;  // ring of int4 records (128 k each)
  static constexpr int kOutBytes = 4 * 32 * 32 * (kOut32 || kHalves ? 4 : 2);  // 32 tokens of an epilogue warp's features, four warps; kHalves: twice
  static constexpr int kNumBars = 2 * kPairMaxStages + 2 * kRecs + 4;
  static constexpr int kSmemBytes = kRingBytes + kRecs * kW4RecMaxBytes + kOutBytes + kNumBars * 8 + 16 + 1024;
  static constexpr int kDqWarp = 4, kServeWarp = kInt4 ? 20 : 4;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
};

struct PairParams {
  void* y;
  const void* bias;
  const unsigned char* packed;  // int4 records
  int T, N, ldy;
  int half;                     // SiLU: weight rows between a gate feature and its up feature; N is the number of outputs then
  int n_kb;                     // 64-wide k-blocks per tile (int4: two per record)
  int rec_per_tile, rec_bytes, group_rows, half_tiles;
  int tn, n_tt, n_m;            // token tile, token tiles, feature tiles
  int per_stage, n_stages;      // k-blocks per stage of the ring, stages per tile
  int stages, stage_bytes;      // depth of the ring
  int pieces, piece_stages, piece_cols;  // pieces of k with an accumulator each, stages and TMEM columns of a piece; one piece: two tiles' accumulators
  const int32_t* offsets;       // experts: first row of each, [E + 1]
  int E;
  int vec;                      // rows of y can be written in 16-byte pieces
  unsigned* gave_up;            // b200_gave_up_word
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Arrive at a barrier of either CTA.  Default (release.cta) semantics: all that the arrival has to order are this thread's own shared-memory
// writes, already handed to the async proxy by fence.proxy.async, or its TMEM reads (tcgen05.fence).  A cluster-scope release and
// acquire also order global memory - a fence through L2 on every hand-over: 735 us instead of 425 at 4099 x 14336 x 4096 int4.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// tensor copy into this CTA's shared memory whose bytes count in a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, int c0, int c1, uint32_t cluster_bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;"
      ::"r"(smem_u32(smem_dst)), "l"(m), "r"(c0), "r"(c1), "r"(cluster_bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void umma_pair_f16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive at the barrier of both CTAs when the products issued so far have completed
__device__ __forceinline__ void umma_pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void sts_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

template <int KIND>
__device__ __forceinline__ auto pair_value(float v) {
  if constexpr (KIND == kPairBf16 || KIND == kPairExpBf16) return __float2bfloat16_rn(v);
  else if constexpr (KIND == kPairBf16Relu2 || KIND == kPairExpRelu2) return __float2bfloat16_rn(v < 0.f ? 0.f : v * v);
  else if constexpr (KIND == kPairBf16F32 || KIND == kPairExpBf16F32) return v;
  else return __float2half_rn(v);
}
// SiLU(gate) * up of two tokens' accumulators: lanes 0..15 hold gate features and finish the first token, lanes 16..31 hold the up features
// of the same outputs and finish the second.  Both factors are rounded to fp16 first, as the separate linear would.
__device__ __forceinline__ __half act_pair(uint32_t first, uint32_t second, float bv, int lane) {
  const __half a = __float2half_rn(__uint_as_float(first) + bv), b = __float2half_rn(__uint_as_float(second) + bv);
  const bool up = lane >= 16;
  const __half other = __ushort_as_half((unsigned short)__shfl_xor_sync(0xffffffffu, (int)__half_as_ushort(up ? a : b), 16));
  const float g = __half2float(up ? other : a);
  return __hmul(__float2half_rn(silu_of_half(g)), up ? b : other);
}
template <int KIND>
__device__ __forceinline__ float pair_bias(const void* bias, int n) {
  if constexpr (KIND != kPairF16 && KIND < kPairW4) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[n]);
  else return __half2float(reinterpret_cast<const __half*>(bias)[n]);
}

struct PairTile {
  int m, t0, nn, row_end;  // feature tile; first row, padded rows and end of the rows of its token tile
  int expert;
};
// the tile a role is at, and (experts) where its rows lie: `before` row tiles belong to experts ahead of `e`
struct PairCursor {
  int e = 0, before = 0;
};

// Tile i in the order in which the pairs take them; false: there is none.  Sixteen token tiles share a weight tile before the next one, so that the
// weights come from HBM once per sixteen token tiles and the activations stay in L2.  Experts: all feature tiles of a row tile side by side; how many
// row tiles there are is only known here, from the plan's offsets (i ascends, so the cursor only moves on).
template <int KIND>
__device__ __forceinline__ bool pair_tile(const PairParams& p, int i, PairCursor& cur, PairTile& t) {
  if constexpr (PairCfg<KIND>::kExperts) {
    const int rt = i / p.n_m;
    t.m = i - rt * p.n_m;
    for (; cur.e < p.E; ++cur.e) {
      const int first = p.offsets[cur.e], end = p.offsets[cur.e + 1], n = (end - first + kPairMaxN - 1) / kPairMaxN;
      if (rt < cur.before + n) {
        t.expert = cur.e;
        t.t0 = first + (rt - cur.before) * kPairMaxN;
        t.nn = min(kPairMaxN, (end - t.t0 + 31) & ~31);
        t.row_end = end;
        return true;
      }
      cur.before += n;
    }
    return false;
  } else {
    if (i >= p.n_tt * p.n_m) return false;
    const int per = 16 * p.n_m, g = i / per, r = i - g * per, width = min(16, p.n_tt - g * 16);
    t.m = r / width;
    t.t0 = (g * 16 + r % width) * p.tn;
    t.nn = min(p.tn, (p.T - t.t0 + 31) & ~31);
    t.row_end = p.T;
    t.expert = 0;
    return true;
  }
}

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<KIND>::kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const PairParams p) {
  using C = PairCfg<KIND>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* recs = smem + C::kRingBytes;
  unsigned char* stage_out = recs + C::kRecs * kW4RecMaxBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(stage_out + C::kOutBytes);
  uint64_t* empty = full + kPairMaxStages;
  uint64_t* rec_full = empty + kPairMaxStages;
  uint64_t* rec_empty = rec_full + C::kRecs;
  uint64_t* tmem_full = rec_empty + C::kRecs;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  pdl_launch_dependents();
  const int warp = warp_id(), lane = lane_id();
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1, n_tiles = p.n_tt * p.n_m;

  if (threadIdx.x == 0) {
    if constexpr (!C::kInt4) tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], C::kInt4 ? 1 + 8 * p.per_stage : 1);  // the leader's x producer, and a team's four warps per k-block in each CTA
      mbar_init(&empty[s], 1);
    }
    for (int r = 0; r < C::kRecs; ++r) {
      mbar_init(&rec_full[r], 1);
      mbar_init(&rec_empty[r], 8);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 8);  // four epilogue warps in each CTA
    }
    mbar_fence_init();
  }
  if (warp == C::kServeWarp) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync();  // the pair's barriers and TMEM exist before anything signals across
  tcgen05_fence_after();
  const uint32_t tmem_d = *tmem_slot;
  bool ok = true;
  if constexpr (C::kExperts) pdl_wait();  // every role reads the plan's offsets

  if (warp == C::kServeWarp + 1) {
    // ------------------------------------------------------------------ TMA: half of the tile's tokens (and fp16 / bf16 features)
    if (elect_one()) {
      const uint64_t pol = policy_evict_last();
      int s = 0, ph = 1;
      pdl_wait();  // x is the previous kernel's output
      PairCursor cur;
      PairTile tl;
      for (int i = pair; pair_tile<KIND>(p, i, cur, tl); i += n_pairs) {
        const int m = tl.m, row_x = tl.t0 + (int)rank * (tl.nn >> 1), row_w = tl.expert * p.N + m * kPairM + (int)rank * 128;
        for (int kb = 0; kb < p.n_stages; ++kb) {
          mbar_wait_soft(&empty[s], ph, ok);
          unsigned char* st = smem + s * p.stage_bytes;
          const uint32_t bar = cluster_map(smem_u32(&full[s]), 0);
          if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * p.per_stage * ((C::kInt4 ? 0 : kPairABytes) + p.tn * kPairK));
          for (int j = 0; j < p.per_stage; ++j) {
            const int k0 = (kb * p.per_stage + j) * kPairK;
            if constexpr (C::kHalves) {
              const int gate = m * 128 + (int)rank * 64;
              tma_load_2d_pair(st + j * kPairABytes, &tmap_w, k0, gate, bar, pol);
              tma_load_2d_pair(st + j * kPairABytes + kPairABytes / 2, &tmap_w, k0, p.half + gate, bar, pol);
            } else if constexpr (!C::kInt4) {
              tma_load_2d_pair(st + j * kPairABytes, &tmap_w, k0, row_w, bar, pol);
            }
            tma_load_2d_pair(st + p.per_stage * kPairABytes + j * p.tn * kPairK, &tmap_x, k0, row_x, bar, pol);
          }
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == C::kServeWarp + 2) {
    // ------------------------------------------------------------------ products, issued by the leader for both CTAs
    pdl_wait();
    if (rank == 0) {
      constexpr uint32_t fmt = C::kInt4 || KIND == kPairF16 || C::kHalves ? 0u : ((1u << 7) | (1u << 10));
      const uint64_t desc0 = umma_desc_kmajor_sw128(smem_u32(smem));
      int s = 0, ph = 0, it = 0;
      PairCursor cur;
      PairTile tl;
      for (int i = pair;; i += n_pairs, ++it) {
        bool more = pair_tile<KIND>(p, i, cur, tl);
        if constexpr (C::kExperts) {  // values from memory: through a reduction, whose result the compiler knows to be warp-uniform
          more = __reduce_max_sync(0xffffffffu, (unsigned)more) != 0;
          tl.nn = __reduce_max_sync(0xffffffffu, tl.nn);
        }
        if (!more) break;
        const int nn = tl.nn;
        const bool one = C::kPieces && p.pieces * p.piece_cols > kPairMaxN;  // accumulators for one tile only
        const int buf = one ? 0 : it & 1, buf_ph = one ? it & 1 : (it >> 1) & 1;
        const uint32_t idesc = umma_idesc_f16_f32acc(kPairM, nn) | fmt;
        uint32_t d = tmem_d + buf * kPairMaxN;
        mbar_wait_soft(&tmem_empty[buf], buf_ph ^ 1, ok);
        int left = p.piece_stages;
        for (int kb = 0; kb < p.n_stages; ++kb) {
          if constexpr (C::kPieces) {
            if (left == 0) {
              left = p.piece_stages;
              d += p.piece_cols;
            }
          }
          const bool first = C::kPieces ? left == p.piece_stages : kb == 0;
          --left;
          mbar_wait_soft(&full[s], ph, ok);
          tcgen05_fence_after();
          const uint64_t da = desc0 + (uint64_t)((s * p.stage_bytes) >> 4), db = da + (uint64_t)((p.per_stage * kPairABytes) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kPairK / 16; ++k) umma_pair_f16_ss(d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (!first || k > 0) ? 1u : 0u);
            if (p.per_stage == 2) {
              const uint64_t da1 = da + (uint64_t)(kPairABytes >> 4), db1 = db + (uint64_t)((p.tn * kPairK) >> 4);
#pragma unroll
              for (int k = 0; k < kPairK / 16; ++k) umma_pair_f16_ss(d, da1 + (uint64_t)(k * 2), db1 + (uint64_t)(k * 2), idesc, 1u);
            }
            umma_pair_commit(&empty[s]);
            if (kb == p.n_stages - 1) umma_pair_commit(&tmem_full[buf]);
          }
          __syncwarp();
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (C::kInt4 && warp == C::kServeWarp) {
    // ------------------------------------------------------------------ TMA: int4 records (settled when they were packed: no wait for the previous kernel)
    if (elect_one()) {
      int r = 0, ph = 1;
      PairCursor cur;
      PairTile tl;
      for (int i = pair; pair_tile<KIND>(p, i, cur, tl); i += n_pairs) {
        const int m = tl.m;
        for (int kb = 0; kb < p.n_kb / 2; ++kb) {
          if (ph == 0) pdl_wait();
          mbar_wait_soft(&rec_empty[r], ph, ok);
          mbar_arrive_expect_tx(&rec_full[r], p.rec_bytes);
          unsigned char* dst = recs + r * kW4RecMaxBytes;
          const unsigned char* two = p.packed + ((size_t)m * p.rec_per_tile + kb) * 2 * p.rec_bytes;
          if constexpr (!C::kAct) {
            tma_bulk_g2s(dst, two + rank * p.rec_bytes, p.rec_bytes, &rec_full[r]);
          } else {
            // 64 rows of the gate record, then the same 64 of the up record, chunk by chunk
            for (int t = 0; t < 2; ++t) {
              const unsigned char* src = two + t * p.rec_bytes;
              for (int c = 0; c < 4; ++c)
                tma_bulk_g2s(dst + c * 2048 + t * 1024, src + c * 2048 + rank * 1024, 1024, &rec_full[r]);
              for (int q = 0; q < p.group_rows; ++q)
                tma_bulk_g2s(dst + kW4WordBytes + q * kW4MetaRowBytes + t * 256, src + kW4WordBytes + q * kW4MetaRowBytes + rank * 256, 256, &rec_full[r]);
            }
          }
          if (++r == C::kRecs) { r = 0; ph ^= 1; }
        }
      }
    }
  } else if (C::kInt4 && warp >= C::kDqWarp && warp < C::kServeWarp) {
    // ------------------------------------------------------------------ de-quantisation: k-blocks go round the four teams
    const int team = (warp - C::kDqWarp) >> 2, quarter = warp & 3, h = team & 1;                             // h: half of a record
    const int row = quarter * 32 + lane;                                                                     // row of the A tile
    const int src = C::kAct ? (lane >> 4) * 64 + quarter * 16 + (lane & 15) : row;                           // row of the record ring's image
    const uint32_t words = smem_u32(recs) + h * 4096 + src * 16, meta = smem_u32(recs) + kW4WordBytes + src * 4;
    const uint32_t dst_row = smem_u32(smem) + row * 128 + (p.per_stage == 2 ? h * kPairABytes : 0), swz = (uint32_t)(row & 7) << 4;
    const int n_recs = ((n_tiles - pair + n_pairs - 1) / n_pairs) * (p.n_kb / 2);
    const int ring_step = 4 / p.per_stage;  // stages between two of this team's
    int r = team >> 1, rph = 0, s = team / p.per_stage, ph = 1;
    uint32_t wq[8], mrec[2];
    auto fetch = [&]() {
      if (rph == 1) pdl_wait();
      mbar_wait_soft(&rec_full[r], rph, ok);
      lds_v4(words + r * kW4RecMaxBytes, &wq[0]);
      lds_v4(words + r * kW4RecMaxBytes + 2048, &wq[4]);
      // the 64 k of a half lie in one group row, or in two when a group is 32 wide
      mrec[0] = lds_u32(meta + r * kW4RecMaxBytes + (h * p.group_rows / 2) * kW4MetaRowBytes);
      mrec[1] = p.group_rows == 4 ? lds_u32(meta + r * kW4RecMaxBytes + (h * 2 + 1) * kW4MetaRowBytes) : mrec[0];
      fence_proxy_async_smem();  // the words are in registers before a bulk copy may take their place
      __syncwarp();
      if (lane == 0) mbar_arrive(&rec_empty[r]);
      r += 2;
      if (r >= C::kRecs) { r -= C::kRecs; rph ^= 1; }
    };
    if ((team >> 1) < n_recs) fetch();
    for (int i = team >> 1; i < n_recs; i += 2) {
      uint32_t v[32];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint32_t scale2, nz1024, nz64;
        dequant_consts(mrec[c >> 2], scale2, nz1024, nz64);
        dequant_word(wq[c], nz1024, nz64, scale2, &v[c * 4]);
      }
      if (ph == 0) pdl_wait();
      mbar_wait_soft(&empty[s], ph, ok);
      const uint32_t dst = dst_row + s * p.stage_bytes;
#pragma unroll
      for (int c = 0; c < 8; ++c) sts_v4(dst + ((uint32_t)(c << 4) ^ swz), v[c * 4], v[c * 4 + 1], v[c * 4 + 2], v[c * 4 + 3]);
      fence_proxy_async_smem();  // the products read the tile through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_map(smem_u32(&full[s]), 0));
      s += ring_step;
      if (s >= p.stages) { s -= p.stages; ph ^= 1; }
      if (i + 2 < n_recs) fetch();
    }
  } else if (warp < 4) {
    // ------------------------------------------------------------------ epilogue: lane = feature
    using Out = decltype(pair_value<KIND>(0.f));
    constexpr int kRow = C::kAct ? 16 : 32;  // features of a token per warp
    Out* out = reinterpret_cast<Out*>(stage_out) + warp * 32 * kRow;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    int it = 0, place = 0;
    pdl_wait();  // y and the bias belong to the stream order
    PairCursor cur;
    PairTile tl;
    for (int i = pair; pair_tile<KIND>(p, i, cur, tl); i += n_pairs, ++it) {
      const int m = tl.m, t0 = tl.t0, nn = tl.nn, row_end = tl.row_end;
      // act: lanes 0..15 hold gate features, lanes 16..31 the up features of the same outputs
      const int tile = p.half_tiles ? m + (int)rank * p.half_tiles : 2 * m + (int)rank;  // 128-feature tile of this CTA
      const int n = C::kAct ? m * 128 + (int)rank * 64 + warp * 16 + (lane & 15) : C::kHalves ? m * 128 + (int)rank * 64 + (warp & 1) * 32 + lane : tile * 128 + warp * 32 + lane;
      const int n0 = n - lane % kRow;                                       // the warp's first output feature
      const int n_w = C::kAct ? n + (lane >> 4) * p.half : C::kHalves ? n + (warp >> 1) * p.half : n;  // the weight row behind this lane
      const bool n_ok = n < p.N;
      const float bv = p.bias && n_ok ? pair_bias<KIND>(p.bias, n_w) : 0.f;
      const bool one = C::kPieces && p.pieces * p.piece_cols > kPairMaxN;
      const int buf = one ? 0 : it & 1, buf_ph = one ? it & 1 : (it >> 1) & 1;
      mbar_wait_soft(&tmem_full[buf], buf_ph, ok);
      tcgen05_fence_after();
      for (int c = 0; c < nn; c += 32) {
        uint32_t v[32];
        const uint32_t acc = tmem_d + lane_base + buf * kPairMaxN;
        tmem_ld_32x32b_x32(acc + c, v);
        tmem_ld_wait();
        if constexpr (C::kPieces) {
          for (int q = 1; q < p.pieces; q += 3) {  // up to three more pieces in flight at once
            uint32_t w[3][32];
#pragma unroll
            for (int k = 0; k < 3; ++k)
              if (q + k < p.pieces) tmem_ld_32x32b_x32(acc + (q + k) * p.piece_cols + c, w[k]);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 3; ++k)
              if (q + k < p.pieces)
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[k][j]));
          }
        }
        if (c + 32 >= nn) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(cluster_map(smem_u32(&tmem_empty[buf]), 0));
        }
        if constexpr (C::kHalves) {
          // both factors of an output meet in shared memory, [token][64 gate | 64 up], in two places by turns; a warp finishes eight tokens.  (Sixteen rows of
          // each to a warp, as the int4 kind has them, take eight copies a stage instead of two: 200 us where the product alone took 181.)
          __half* both = reinterpret_cast<__half*>(stage_out) + place * (32 * 128);
          place ^= 1;
#pragma unroll
          for (int j = 0; j < 32; ++j) both[j * 128 + warp * 32 + lane] = __float2half_rn(__uint_as_float(v[j]) + bv);
          asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int t = warp * 8 + e * 4 + (lane >> 3), f = (lane & 7) * 8, o = m * 128 + (int)rank * 64 + f;
            const uint4 gq = *reinterpret_cast<const uint4*>(both + t * 128 + f), uq = *reinterpret_cast<const uint4*>(both + t * 128 + 64 + f);
            const __half *g = reinterpret_cast<const __half*>(&gq), *up = reinterpret_cast<const __half*>(&uq);
            uint4 r;
            __half* rh = reinterpret_cast<__half*>(&r);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              rh[k] = __hmul(__float2half_rn(silu_of_half(__half2float(g[k]))), up[k]);
            }
            if (t0 + c + t < row_end && o < p.N) *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.y) + (size_t)(t0 + c + t) * p.ldy + o) = r;
          }
        } else if (p.vec) {
          // transpose 32 tokens x the warp's features through shared memory: rows of a token's features, written out in 16-byte pieces (one
          // 2-byte store per value and lane takes 9 us for a tile of 256 tokens, this way 1)
          __syncwarp();
          if constexpr (C::kAct) {
#pragma unroll
            for (int j = 0; j < 32; j += 2) out[(j + (lane >> 4)) * kRow + (lane & 15)] = act_pair(v[j], v[j + 1], bv, lane);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) out[j * kRow + lane] = pair_value<KIND>(__uint_as_float(v[j]) + bv);
          }
          __syncwarp();
          constexpr int kPieces = kRow * sizeof(Out) / 16, kTokens = 32 / kPieces;  // pieces of a row, tokens per pass of the warp
          const int f = lane % kPieces * (16 / (int)sizeof(Out));
          if (n0 + f < p.N) {
#pragma unroll
            for (int j = 0; j < 32; j += kTokens) {
              const int t = j + lane / kPieces;
              if (t0 + c + t < row_end)
                *reinterpret_cast<uint4*>(reinterpret_cast<Out*>(p.y) + (size_t)(t0 + c + t) * p.ldy + n0 + f) = *reinterpret_cast<const uint4*>(out + t * kRow + f);
            }
          }
        } else if constexpr (C::kAct) {
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const Out o = act_pair(v[j], v[j + 1], bv, lane);
            const int t = t0 + c + j + (lane >> 4);
            if (t < row_end && n_ok) reinterpret_cast<Out*>(p.y)[(size_t)t * p.ldy + n] = o;
          }
        } else if (n_ok) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (t0 + c + j < row_end) reinterpret_cast<Out*>(p.y)[(size_t)(t0 + c + j) * p.ldy + n] = pair_value<KIND>(__uint_as_float(v[j]) + bv);
        }
      }
    }
  }

  if (!ok) gave_up(p.gave_up);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync();  // the leader's products read the other CTA's shared memory and write its TMEM until the epilogues are done
  if (warp == C::kServeWarp) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_d) : "memory");
}

struct PairPlan {
  int tn, n_tt, n_m, n_pairs, per_stage;
  float us;  // estimate
  int pieces, piece_stages, piece_cols;
};

// Token tile of a call: of all cuts of T into equal tiles of 32-row steps, the one whose waves over the SM pairs cost least.  What a 64-wide
// k-block costs was measured on B200 (cold weights, tiles x k-blocks of 4096 x 4096 products, microseconds per wave): fp16 0.13 at 32 tokens,
// 0.15 at 64, 0.19 at 128, 0.26 at 192, 0.35 at 256; int4 0.22 at 32, 0.25 at 128, 0.29 at 192, 0.37 at 256 (below that, de-quantisation).
// Small tiles take two k-blocks per stage of the ring: a hand-over costs more than their products (16.2 us instead of 19.6 at 300 x 4096 x
// 4096 fp16, 21.3 instead of 23.3 int4); large ones need the depth more (97 instead of 98 and 30.3 instead of 31.5 at 4099 and 1000 tokens).
// `pieces`: how many pieces of k should have an accumulator of their own, as far as the tensor memory holds them.
static PairPlan pair_plan(int64_t T, int64_t N, int64_t n_kb, bool int4, int sms, int pieces = 1) {
  PairPlan best = {};
  const int pairs = sms / 2, n_m = (int)((N + kPairM - 1) / kPairM);
  for (int tn = 32; tn <= kPairMaxN; tn += 32) {
    const int n_tt = (int)((T + tn - 1) / tn), per_stage = tn <= (int4 ? 160 : 128) ? 2 : 1;
    const int64_t tiles = (int64_t)n_tt * n_m, waves = (tiles + pairs - 1) / pairs;
    const float kb = int4 ? (per_stage == 2 ? 0.21f + 0.0003f * tn : 0.13f + 0.00092f * tn) : (per_stage == 2 ? 0.105f + 0.00065f * tn : 0.09f + 0.001f * tn);
    const float us = waves * kb * n_kb + 0.013f * tn;  // the last tile's epilogue is not hidden
    if (best.tn == 0 || us < best.us) best = {tn, n_tt, n_m, (int)(tiles < pairs ? tiles : pairs), per_stage, us};
  }
  best.pieces = 1;
  best.piece_stages = (int)((n_kb + best.per_stage - 1) / best.per_stage);
  best.piece_cols = best.tn <= 64 ? 64 : best.tn <= 128 ? 128 : 256;
  if (pieces > 1) {
    const int n_stages = best.piece_stages, most = 512 / best.piece_cols, p = pieces < most ? pieces : most;
    best.piece_stages = (n_stages + p - 1) / p;
    best.pieces = (n_stages + best.piece_stages - 1) / best.piece_stages;
  }
  // what the cost above leaves out matters where another kernel is to be had: the launch, and the feature tiles' share of the memory's rate (B200,
  // one wave: 448 k-blocks of 8 tiles 62.6 us, 256 of 16 41.0, 320 of 20 52.6, 448 of 32 92.7)
  const int64_t tiles = (int64_t)best.n_tt * n_m, waves = (tiles + pairs - 1) / pairs;
  best.us += 3.f + 0.0016f * (n_m < pairs ? n_m : pairs) * waves * n_kb;
  return best;
}

// x [T, K], w: the fp16 / bf16 matrix [N, K], or NULL for int4 (pp holds the records)
template <int KIND>
static int launch_gemm_pair(const void* x, const void* w, int64_t K, PairParams pp, const PairPlan& pl, int time_id, cudaStream_t st) {
  using C = PairCfg<KIND>;
  pp.gave_up = b200_gave_up_word();
  if (!pp.gave_up) return B200_ERR_CUDA;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) { b200_set_last_error(cudaGetErrorString(e)); return B200_ERR_CUDA; }
    configured = true;
  }
  const CUtensorMap* mx = get_tmap_2d(x, pp.T, K, K, pl.tn / 2, kPairK, TmapDtype::kF16, TmapSwizzle::k128B);
  const uint64_t rows_w = (uint64_t)pp.N * (C::kExperts ? pp.E : C::kHalves ? 2 : 1);
  const CUtensorMap* mw = w ? get_tmap_2d(w, rows_w, K, K, C::kHalves ? 64 : 128, kPairK, TmapDtype::kF16, TmapSwizzle::k128B) : mx;
  if (!mx || !mw) return B200_ERR_CUDA;
  constexpr int kOut = C::kOut32 ? 4 : 2;
  pp.vec = ((uintptr_t)pp.y & 15) == 0 && (int64_t)pp.ldy * kOut % 16 == 0;
  pp.tn = pl.tn;
  pp.n_tt = pl.n_tt;
  pp.n_m = pl.n_m;
  pp.per_stage = pl.per_stage;
  pp.n_stages = (pp.n_kb + pl.per_stage - 1) / pl.per_stage;
  pp.pieces = pl.pieces > 1 ? pl.pieces : 1;
  pp.piece_stages = pl.pieces > 1 ? pl.piece_stages : pp.n_stages;
  pp.piece_cols = pl.piece_cols;
  pp.stage_bytes = pl.per_stage * pair_block_bytes(pl.tn);
  pp.stages = C::kRingBytes / pp.stage_bytes < kPairMaxStages ? C::kRingBytes / pp.stage_bytes : kPairMaxStages;
  b200_timing_mark(time_id, 0, st);
  B200_LAUNCH_AS("gemm_pair_kernel", gemm_pair_kernel<KIND>, dim3(2 * pl.n_pairs), dim3(C::kThreads), (size_t)C::kSmemBytes, st, *mw, *mx, pp);
  b200_timing_mark(time_id, 1, st);
  b200_count_launches(1);
  return B200_OK;
}

}  // namespace b200
