// GPTQ int4 linear  Y[T,N] = X[T,K] . dequant(Wq)[K,N]  on tcgen05 tensor cores, weights de-quantised in-kernel
// straight into TMEM (no fp16 scratch matrix, for any T).  This kernel takes calls of up to 128 tokens (kW4DecodeT) but for
// those of gemm_w4_few.cuh, gemm_pair.cuh larger ones.
//
// Replaces `exllamav2_kernels.make_q_matrix` / `gemm_half_q_half`
// (server/text_generation_server/utils/gptq/exllamav2.py:14-62,139-144), including its M > 50
// "dequantise everything to temp_dq, then cuBLAS" branch (:87), and follows the dequant formula of record
// utils/gptq/quant_linear.py:184-192:  W[k,n] = fp16( scales[g,n] * (q[k,n] - (qzeros[g,n] + 1)) ).
//
// Weight format.  `b200_gptq_pack` (the make_q_matrix analogue, once per linear at load time) turns the checkpoint
// tensors into a stream of self-contained UNIT RECORDS, one per (128-feature tile, 128-wide k-block):
//     words  [4 chunks][128 features][4 x u32]   8 KB   chunk c = k 32c..32c+31 of the block; inside a word the 8 nibbles
//                                                        are ordered k0 k2 k4 k6 | k1 k3 k5 k7 so one LOP3 yields a (k, k+1) pair
//     meta   [group_rows][128 features] u32      512 B per row: fp16 scale | (zero + 1) << 16, group_rows = max(1, 128 / groupsize)
// ordered (super-tile = pair of feature tiles, k-block, tile of the pair).  A CTA's work is a contiguous range of
// SUPER-UNITS (super-tile, k-block) == a contiguous byte range of HBM: one cp.async.bulk (TMA) per unit, no tensor map, and
// the shared-memory image is exactly what the dequant threads want (LDS.128, conflict free).  The two units of a
// super-unit share one activation tile (at T = 64 the activations are twice the weight bytes on the L2 -> SM path).
//
// Swap-AB like gemm_f16.cu: 128 output features = UMMA M, tokens = UMMA N (TN = 16..128), fp32 accumulators in TMEM.
// 24 warps, one CTA per SM.  The SM sub-partition arbiter favours high warp ids, so the pacing roles sit on top:
//   warp 22       TMA: unit records -> 12..16-deep (8 at TN = 128) weight ring; starts before the CTA set-up barrier.
//                 Only these bytes come from HBM.
//   warp 23       TMA: one activation tile [TN x 128] fp16 (two 128B-swizzled sub-tiles) per super-unit -> 6-deep ring
//                 (L2 hits); it lands on the super-unit's own barrier
//   warps 4..19   dequant: 4 teams x 4 warps; team = unit index mod 4, warp = TMEM lane quarter, thread = one feature row x
//                 all 128 k of the unit (16 words).  Per 8 weights: 4 LOP3 + SHF (magic-number fp16: 1024 + q / 64 + q),
//                 4 HADD2 (exact q - zero), 4 HMUL2 (x scale: bit-identical to the formula of record) -> tcgen05.st into a
//                 ring of A-operand tiles in TMEM (64 columns each), an arrival at the super-unit's barrier.  Teams run on their own clocks.
//   warps 20, 21  MMA issue, alternate super-units: wait for the super-unit's barrier (its activation tile and the 8 team-warp
//                 quarters of its two A tiles), then for the turn, 16 x tcgen05.mma.kind::f16 (A from TMEM, B from shared memory), a tcgen05.commit that frees both
//                 A stages (su_done) and one that frees the activation stage (x_empty)
//   warps 0..3    epilogue: tcgen05.ld of a finished super-tile, then fp16 store / fused SiLU(gate) * up store / fp32
//                 partial store when the super-tile is shared with other CTAs; they sleep while they wait
// Decode (T <= 128) is weight-streaming / HBM-bound: the (super-tile, k-block) space is cut into contiguous ranges, one
// per CTA, either equal shares of a super-tile or the balanced stream-K cut, whichever plan_w4's cost model prefers.
// Super-tiles shared by several CTAs are finished after the main loop by ALL their contributors: each sums one slice over
// the contributors' fp32 partials in contributor order (deterministic, unlike the reference kernel's fp16 atomicAdd across
// K slices; a reduce-scatter, so the tail costs one partial's worth of L2 reads per CTA however many CTAs share it).
// The contributors wait for one another: all CTAs of the grid are co-resident (grid <= #SMs, one CTA per SM).  Where that takes less,
// the CTAs of a cluster share a super-tile instead and add their parts through shared memory (launch_plan_w4).
//
// mbarrier rule used throughout: a thread that waits on a barrier observes every phase of it in order, or an earlier
// observation implies the skipped phase completed (see the ring-depth static_asserts).  Polls whose result is wanted
// later use test_wait: try_wait may suspend the thread until a time-out while the phase is pending.
#include "common.cuh"
#include "gemm_pair.cuh"
#include "gemm_w4_few.cuh"
#include "tmap.cuh"
#include "w4_format.cuh"
#include "../../include/b200_tgis.h"

#include <cstdlib>
#include <string>

namespace b200 {

// Warp roles.  The SM sub-partition arbiter favours the higher warp id, so the three single-thread roles that pace the
// pipeline (MMA issue, the two TMA producers) get the highest ids, the 16 issue-bound dequant warps sit in the middle and
// the mostly-waiting epilogue warps get the lowest (and sleep while they wait).
constexpr int kW4Teams = 4;
constexpr int kW4EpWarps = 4;                                   // warps 0..3
constexpr int kW4FirstDqWarp = kW4EpWarps;                      // warps 4..19
constexpr int kW4MmaWarp = kW4FirstDqWarp + 4 * kW4Teams;       // 20, 21: two MMA warps taking alternate super-units
constexpr int kW4WProdWarp = kW4MmaWarp + 2;                    // 22
constexpr int kW4XProdWarp = kW4MmaWarp + 3;                    // 23
constexpr int kW4Threads = (kW4XProdWarp + 1) * 32;             // 768
constexpr int kW4AColsPerStage = 64;  // 128 fp16 per row = 64 x 32-bit columns
constexpr int64_t kW4CounterBytes = 64 * 1024;

// kW4DecodeT (w4_format.cuh): most tokens of one token tile; more go to the SM pairs (gemm_pair.cuh).  At 128 tokens the pairs would win on wide outputs and short k only
// (us, this kernel / pairs: 2048 -> 2560 13.1 / 10.9, 4096 -> 28672 45.2 / 46.3, 4096 -> 4096 15.3 / 19.2, 14336 -> 4096 23.9 / 53.8); at 129 this
// kernel would need two token tiles (4096 -> 4096 40.1 / 19.6, 14336 -> 4096 107 / 58).
constexpr int kW4R = 2;  // feature tiles per super-tile: consecutive units (super-tile, k-block, r = 0..1) share one activation tile

// how a kernel ends: by its four epilogue warps; by all threads where a CTA has its last super-tile alone; super-tiles shared by clusters
enum W4End { kW4Plain, kW4Whole, kW4Cluster };
constexpr int kW4MostCluster = 8;   // CTAs that share a super-tile through shared memory
constexpr int kW4SumPitch = kW4R * kW4TileM + 4;  // floats of a token's sums in shared memory

template <int TN>
struct GemmW4Cfg {
  static constexpr int kSuRing = TN >= 128 ? 2 : 3;            // super-units whose A tiles fit in TMEM at once
  static constexpr int kAStages = kSuRing * kW4R;              // TMEM A-operand ring (per unit)
  static constexpr int kDBufs = TN >= 64 ? 1 : 2;              // accumulator sets (one set = kW4R tiles x TN columns)
  static constexpr int kDCols = kDBufs * kW4R * TN;
  static constexpr int kABase = kDCols < 64 ? 64 : kDCols;
  static constexpr int kTmemCols = 512;
  static constexpr int kXSubBytes = TN * 128;                  // one [TN x 64] fp16 sub-tile
  static constexpr int kXStageBytes = 2 * kXSubBytes;
  static constexpr int kXStages = TN >= 128 ? 4 : 6;           // activation ring (per super-unit = kW4R units)
  static constexpr int kWStages = TN >= 128 ? 8 : (TN == 64 ? 12 : 16);
  static constexpr int kNumBars = 2 * kWStages + 2 * kXStages + kSuRing + 6;
  static constexpr int kSmemBytes = kXStages * kXStageBytes + kWStages * kW4RecMaxBytes + kNumBars * 8 + 16 + 1024;
  static_assert(kABase + kAStages * kW4AColsPerStage <= kTmemCols, "TMEM budget");
  // a team observes every phase of the weight stages it uses only if a stage always belongs to the same team
  static_assert(kWStages % kW4Teams == 0, "weight ring depth must be a multiple of the team count");
  // a team at super-unit j has seen super-unit j - 2 - kSuRing complete, which implies j - 2 kSuRing did (no phase aliasing)
  static_assert(kSuRing >= 2, "A ring depth");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
  static_assert(TN * kW4SumPitch * 4 <= kXStages * kXStageBytes + kWStages * kW4RecMaxBytes, "the last super-tile's sums lie where the rings were");
};

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// wait of a warp that has nothing else to do for a long time: sleep between polls so it does not take issue slots
__device__ __forceinline__ void mbar_wait_relaxed(uint64_t* bar, uint32_t parity) {
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    __nanosleep(128);
    if (++spins > (1u << 23)) { __trap(); }
  }
}

struct W4Params {
  __half* y;
  float* partial;   // [super-tile][contributor][kW4R][TN][128] fp32
  unsigned* counters;  // [super-tile]: its n contributors count to n as their partials are written and to 2 n, which is 0 again, as they see n
  const __half* bias;
  const unsigned char* packed;  // unit records, (super-tile, k-block, r) order
  int T, N;
  int nkb;          // 128-wide k-blocks per tile
  int n_super;      // super-tiles (pairs of 128-feature tiles)
  int su_per_cta;   // contiguous (super-tile, k-block) super-units per CTA
  int total_su;
  int max_contrib;  // partial slots per super-tile
  int rec_bytes;    // 8192 + group_rows * 512
  int half_tiles;   // 0: super-tile s = feature tiles (2s, 2s+1); > 0 ("gate|up" layout): tiles (s, s + half_tiles)
  int act;          // 1: y[t, 128 s + m] = fp16(silu(fp16 gate)) * fp16 up  (needs the gate|up layout), row stride ldy
  int ldy;          // output row stride in halves
  int defer;        // 1: every super-tile segment is left as an fp32 partial in the workspace and the NEXT kernel of the stream sums
                    //    them (B200SplitK consumers: rmsnorm / rope / SiLU*up / all-reduce); no counters, no waiting on peer CTAs
  int cluster;      // > 0: a cluster of so many CTAs has one super-tile, each a part of k
  unsigned long long* trace;  // debug: per-CTA phase timestamps (globaltimer ns), NULL in production
};

// four features of a token at y; p.y may start off any four halves (rows are a multiple of 32 long, so the first address says it for all).  Single stores in a loop:
// unrolled in all three endings they lengthened the kernel for everybody (4096 -> 28672 with the SiLU at 64 tokens, replayed graph, 21.25 us, so 21.14)
__device__ __forceinline__ void w4_store(const W4Params& p, __half* y, uint2 o) {
  if ((reinterpret_cast<uintptr_t>(p.y) & 7) == 0) {
    *reinterpret_cast<uint2*>(y) = o;
  } else {
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      reinterpret_cast<unsigned short*>(y)[j] = (unsigned short)o.x;
      o.x = __funnelshift_r(o.x, o.y, 16);
      o.y >>= 16;
    }
  }
}

// The end of a CTA's last super-tile when nobody shares it: the epilogue warps leave its fp32 sums in shared memory ([token][kW4SumPitch]) and all 24 warps
// write the outputs, four features of a token each.  By the four epilogue warps alone, a feature per thread, the SiLU (then with divisions, a branch each, so one
// after the other) took 1.9 us at 16 tokens, 7.9 at 64 and 15 at 128 behind the last product (4096 -> 28672: 26.8 us of which 7.9 -> 21.5 with 2.4; 128 tokens 42.6 -> 32).
// kWhole: from 17 tokens on, and with the SiLU from 9 if no super-tile is shared; otherwise the outputs are too few to pay for the barrier, or for the code
// alone (14336 -> 4096 at one token 12.6 us without and 13.0 with it, 4096 -> 22016 with the SiLU at 16 tokens 18.0 and 18.2; 4096 -> 28672 with the SiLU 18.4 and
// 18.5 at one token, 19.7 and 18.7 at 16).
// four(at): sums of four features from `at` on, [token][kW4SumPitch]; items lo .. hi - 1 of T * per_tok are this CTA's
template <class Four>
__device__ __forceinline__ void w4_finish(const W4Params& p, int sup, int per_tok, int lo, int hi, Four four) {
  for (int i = lo + threadIdx.x; i < hi; i += kW4Threads) {
    const int tok = i / per_tok, f = (i % per_tok) * 4, r = f / kW4TileM, m = f % kW4TileM;
    float4 s = four(tok * kW4SumPitch + f);
    const int col = p.act ? sup * kW4TileM + f : (p.half_tiles ? sup + r * p.half_tiles : sup * kW4R + r) * kW4TileM + m;
    if (!p.act && col >= p.N) continue;   // N % 32 == 0: four columns never straddle it
    if (p.bias) {
      s.x += __half2float(p.bias[col]); s.y += __half2float(p.bias[col + 1]); s.z += __half2float(p.bias[col + 2]); s.w += __half2float(p.bias[col + 3]);
    }
    uint2 o;
    if (p.act) {
      float4 u = four(tok * kW4SumPitch + kW4TileM + f);
      if (p.bias) {
        const __half* b = p.bias + col + p.half_tiles * kW4TileM;
        u.x += __half2float(b[0]); u.y += __half2float(b[1]); u.z += __half2float(b[2]); u.w += __half2float(b[3]);
      }
      const __half h[4] = {silu_mul_f16(s.x, u.x), silu_mul_f16(s.y, u.y), silu_mul_f16(s.z, u.z), silu_mul_f16(s.w, u.w)};
      o = *reinterpret_cast<const uint2*>(h);
    } else {
      o = make_uint2(pack_half2(s.x, s.y), pack_half2(s.z, s.w));
    }
    w4_store(p, &p.y[(size_t)tok * p.ldy + col], o);
  }
}

// kGR = meta rows per unit record (1, 2 or 4 = 128 / groupsize, 1 for groupsize >= 128).
template <int TN, int kGR, int kEnd>
__global__ void __launch_bounds__(kW4Threads, 1)
gemm_w4a16_kernel(const __grid_constant__ CUtensorMap tmap_x, const W4Params p) {
  using C = GemmW4Cfg<TN>;
  constexpr bool kWhole = kEnd == kW4Whole, kCluster = kEnd == kW4Cluster;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* x_ring = smem;                                 // 1024-aligned stages (128B swizzle)
  unsigned char* w_ring = smem + C::kXStages * C::kXStageBytes; // 1024-aligned stages
  uint64_t* full_w = reinterpret_cast<uint64_t*>(w_ring + C::kWStages * kW4RecMaxBytes);
  uint64_t* empty_w = full_w + C::kWStages;
  uint64_t* su_full = empty_w + C::kWStages;    // [kXStages] super-unit j's inputs are there, its activation tile and the 8 team-warp quarters of its two A tiles
  uint64_t* x_empty = su_full + C::kXStages;    // [kXStages] the MMAs that read the stage's activation tile have completed
  uint64_t* su_done = x_empty + C::kXStages;    // [kSuRing] MMA commit of super-unit j -> barrier j % kSuRing: its A stages are free
  uint64_t* tmem_full = su_done + C::kSuRing;   // [2]
  uint64_t* tmem_empty = tmem_full + 2;         // [2]
  uint64_t* turn = tmem_empty + 2;              // [2] hand-over between the two MMA warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(turn + 2);
  __shared__ int s_fix[2][3];  // super-tiles this CTA shares with others: {super-tile, contributors, my index}
  __shared__ int s_nfix;
  __shared__ int s_whole;      // the last super-tile if this CTA has it alone: all threads finish it; -1: none

  pdl_launch_dependents();
  const int warp = warp_id(), lane = lane_id();
  // a contiguous range of super-units of the (super-tile, k-block) space
  const int c_sup = kCluster ? (int)blockIdx.x / p.cluster : 0, c_rank = kCluster ? (int)blockIdx.x % p.cluster : 0;
  const int su0 = kCluster ? c_sup * p.nkb + c_rank * p.nkb / p.cluster : blockIdx.x * p.su_per_cta;
  const int su1 = kCluster ? c_sup * p.nkb + (c_rank + 1) * p.nkb / p.cluster : min(p.total_su, su0 + p.su_per_cta);
  const int n_su = su1 - su0;
  const int n_units = n_su * kW4R;
  const int kb0 = su0 % p.nkb;
  auto unit_src = [&](int i) -> const unsigned char* {  // HBM address of this CTA's i-th unit record
    return p.packed + ((size_t)su0 * kW4R + i) * p.rec_bytes;
  };
#define W4_TRACE(id, who)                                                                              \
  do {                                                                                                 \
    if (p.trace && threadIdx.x == (who)) {                                                             \
      unsigned long long _t;                                                                           \
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(_t));                                           \
      p.trace[blockIdx.x * 64 + (id)] = _t;                                                            \
    }                                                                                                  \
  } while (0)
  W4_TRACE(0, 0);

  // The weights were settled when they were packed: the W producer initialises its own barriers and issues the first ring
  // of unit records before the CTA-wide set-up barrier (TMEM allocation, the other barriers), so HBM latency overlaps it.  (Brought to L2 only, and copied
  // after the wait for the kernel before, as gemm_f16.cu does: 16 to 128 tokens 0.5 to 1.3 us more, 4096 -> 6144 at 64 tokens 11.6 -> 12.6.)
  int w_issued = 0;
  if (warp == kW4WProdWarp) {
    if (elect_one()) {
      for (int s = 0; s < C::kWStages; ++s) {
        mbar_init(&full_w[s], 1);
        mbar_init(&empty_w[s], 4);  // the 4 warps of the team that owns the stage
      }
      mbar_fence_init();
      const uint64_t pol_w = policy_evict_first();
      const int n0 = min(n_units, C::kWStages);
      for (int i = 0; i < n0; ++i) {
        mbar_arrive_expect_tx(&full_w[i], p.rec_bytes);
        tma_bulk_g2s_hint(w_ring + i * kW4RecMaxBytes, unit_src(i), p.rec_bytes, &full_w[i], pol_w);
      }
    }
    w_issued = min(n_units, C::kWStages);
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < C::kXStages; ++s) {
      mbar_init(&su_full[s], 1 + 8);
      mbar_init(&x_empty[s], 1);
    }
    for (int b = 0; b < C::kSuRing; ++b) mbar_init(&su_done[b], 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], kW4EpWarps);
      mbar_init(&turn[b], 1);
    }
    s_nfix = 0;
    s_whole = -1;
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc<C::kTmemCols>(tmem_slot);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_d = tmem_base;               // accumulator sets
  const uint32_t tmem_a = tmem_base + C::kABase;   // A-operand ring
  W4_TRACE(1, 0);

  if (warp == kW4WProdWarp) {
    // ------------------------------------------------------------------ TMA producer: unit records (HBM stream); the first
    // ring was issued above
    if (elect_one()) {
      const uint64_t pol_w = policy_evict_first();
      int s = 0, ph = 0;  // stage 0 again: wait for its first release
      for (int i = w_issued; i < n_units; ++i) {
        mbar_wait(&empty_w[s], ph);
        mbar_arrive_expect_tx(&full_w[s], p.rec_bytes);
        tma_bulk_g2s_hint(w_ring + s * kW4RecMaxBytes, unit_src(i), p.rec_bytes, &full_w[s], pol_w);
        if (++s == C::kWStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == kW4XProdWarp) {
    // ------------------------------------------------------------------ TMA producer: activations (L2 resident),
    // one [TN x 128] tile per super-unit; the stage of super-unit j takes the tile of super-unit j + kXStages once the MMAs of j have completed
    if (elect_one()) {
      const uint64_t pol_x = policy_evict_last();
      int kb = kb0, s = 0, ph = 1;
      pdl_wait();  // x is the previous kernel's output; the weight ring is already streaming
      for (int j = 0; j < n_su; ++j) {
        mbar_wait(&x_empty[s], ph);
        mbar_arrive_expect_tx(&su_full[s], C::kXStageBytes);
        unsigned char* st = x_ring + s * C::kXStageBytes;
        tma_load_2d_hint(st, &tmap_x, kb * kW4BlockK, 0, &su_full[s], pol_x);
        tma_load_2d_hint(st + C::kXSubBytes, &tmap_x, kb * kW4BlockK + 64, 0, &su_full[s], pol_x);
        if (++kb == p.nkb) kb = 0;
        if (++s == C::kXStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == kW4MmaWarp || warp == kW4MmaWarp + 1) {
    // ------------------------------------------------------------------ MMA issuers.  tcgen05.mma issue is in order and the
    // queue is shallow, so a warp that has just issued 16 MMAs cannot hide its own bookkeeping (barrier polls, commit)
    // behind them: the tensor pipe would idle ~40 % of the time.  Two warps take alternate
    // super-units; while one is blocked issuing, the other has already found its inputs ready and only waits for its turn
    // (a barrier; words in shared memory that both polled took issue slots from the teams: 4096 -> 28672 at 9 tokens 19.7 us, 18.8 so, at 128 tokens 32.6 / 31.0,
    // 14336 -> 4096 at 64 15.3 / 14.8), so MMAs reach the pipe back to back and in super-unit order (summation order stays fixed).
    // Warp-uniform loops, one elected thread issues: keeps the tcgen05 operands in uniform registers.
    const int me = warp - kW4MmaWarp;
    constexpr uint32_t idesc = umma_idesc_f16_f32acc(kW4TileM, TN);
    const uint64_t bdesc0 = umma_desc_kmajor_sw128(smem_u32(x_ring));
    for (int j = me; j < n_su; j += 2) {
      const int kbj = kb0 + j;            // k-block index counted from the CTA's first super-tile
      const int kb = kbj % p.nkb, seg = kbj / p.nkb;
      const bool seg_first = (j == 0) || kb == 0;
      const bool seg_last = (j == n_su - 1) || kb == p.nkb - 1;
      const int buf = C::kDBufs == 2 ? (seg & 1) : 0;
      const int sx = j % C::kXStages, sj = j % C::kSuRing;
      mbar_wait(&su_full[sx], (j / C::kXStages) & 1);
      if (seg_first) {  // the epilogue drained this accumulator set's previous super-tile
        if (C::kDBufs == 2) mbar_wait(&tmem_empty[buf], ((seg >> 1) & 1) ^ 1);
        else mbar_wait(&tmem_empty[0], (seg & 1) ^ 1);
      }
      if (j > 0) mbar_wait(&turn[me], ((j - 1) >> 1) & 1);  // my turn
      tcgen05_fence_after();
      if (elect_one()) {
        const uint64_t bdesc = bdesc0 + (uint64_t)((sx * C::kXStageBytes) >> 4);
#pragma unroll
        for (int r = 0; r < kW4R; ++r) {
          const uint32_t d = tmem_d + (buf * kW4R + r) * TN, a = tmem_a + (sj * kW4R + r) * kW4AColsPerStage;
#pragma unroll
          for (int k = 0; k < kW4BlockK / 16; ++k)
            umma_f16_ts(d, a + k * 8, bdesc + (uint64_t)((k >> 2) * (C::kXSubBytes >> 4) + (k & 3) * 2), idesc, (!seg_first || k > 0) ? 1u : 0u);
        }
        mbar_arrive(&turn[me ^ 1]);
        umma_commit(&su_done[sj]);
        umma_commit(&x_empty[sx]);
        if (seg_last) umma_commit(&tmem_full[buf]);
      }
      __syncwarp();
    }
    W4_TRACE(6, kW4MmaWarp * 32);
  } else if (warp >= kW4FirstDqWarp) {
    // ------------------------------------------------------------------ dequant teams
    const int team = (warp - kW4FirstDqWarp) >> 2;  // unit index mod 4
    const int quarter = warp & 3;                   // TMEM lane quarter this warp may access
    const int m = quarter * 32 + lane;              // feature row within the tile
    const uint32_t a_row = tmem_a + ((uint32_t)(quarter * 32) << 16);
    const uint32_t w_thread = smem_u32(w_ring) + m * 16;
    const uint32_t meta_thread = smem_u32(w_ring) + kW4WordBytes + m * 4;
    uint32_t wq[16], mrec[kGR];
    int ws = team, wph = 0;   // weight-ring stage / parity of the unit being loaded
    int held = 0;             // stage whose words are on their way to registers: given back behind fence_proxy_async_smem
    // unit i (super-unit j = i / 2) lives in A stage i % kAStages and may be written once the MMAs of super-unit
    // j - kSuRing have completed: barrier su_done[j % kSuRing], phase j / kSuRing - 1
    auto load_unit = [&](bool landed) {
      if (!landed) mbar_wait(&full_w[ws], wph);
      const uint32_t st = ws * kW4RecMaxBytes;
#pragma unroll
      for (int c = 0; c < 4; ++c) lds_v4(w_thread + st + c * (kW4TileM * 16), &wq[c * 4]);
#pragma unroll
      for (int r = 0; r < kGR; ++r) mrec[r] = lds_u32(meta_thread + st + r * kW4MetaRowBytes);
      held = ws;
      ws += kW4Teams;
      if (ws >= C::kWStages) { ws -= C::kWStages; wph ^= 1; }
    };
    if (team < n_units) {
      load_unit(false);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_w[held]);
    }
    if (team == 0) W4_TRACE(2, kW4FirstDqWarp * 32);
    // the team's super-units j are two apart: places in the rings of A tiles and of activation tiles, parity of the A place's last use
    int jr = (team >> 1) % C::kSuRing, jx = team >> 1;
    uint32_t done_par = 1;
    for (int i = team; i < n_units; i += kW4Teams) {
      const bool more = i + kW4Teams < n_units;
      // barrier polls are issued well before their result is needed
      const int j = i >> 1;
      const uint32_t a_dst = a_row + (jr * kW4R + (team & 1)) * kW4AColsPerStage;
      const bool a_free = j < C::kSuRing || mbar_test_wait(&su_done[jr], done_par);  // looked at after chunk 0
      const bool w_landed = more && mbar_test_wait(&full_w[ws], wph);                // looked at after chunk 3
      uint32_t scale2, nz1024, nz64;
      dequant_consts(mrec[0], scale2, nz1024, nz64);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // chunk c = k 32c..32c+31 of the block; its meta row is c * kGR / 4
        if (c > 0 && (c * kGR) % 4 == 0) dequant_consts(mrec[c * kGR / 4], scale2, nz1024, nz64);
        uint32_t v[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) dequant_word(wq[c * 4 + j], nz1024, nz64, scale2, &v[j * 4]);
        if (c == 0) {
          if (!a_free) mbar_wait(&su_done[jr], done_par);  // the MMAs that read this A stage have completed
          tcgen05_fence_after();
        }
        tmem_st_32x32b_x16(a_dst + c * 16, v);
      }
      if (more) load_unit(w_landed);  // next unit's words: the shared-memory reads overlap the TMEM store latency
      tmem_st_wait();
      tcgen05_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&su_full[jx]);
        if (more) mbar_arrive(&empty_w[held]);
      }
      if ((jr += 2) >= C::kSuRing) { jr -= C::kSuRing; done_par ^= 1; }
      if ((jx += 2) >= C::kXStages) jx -= C::kXStages;
    }
    if (team == 0) W4_TRACE(4, kW4FirstDqWarp * 32);
  } else {
    // ------------------------------------------------------------------ epilogue warps: one pass per super-tile segment
    const int quarter = warp & 3;
    const int m = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    int seg = 0, nfix = 0;
    pdl_wait();  // outputs / bias / stream-K workspace belong to the stream order
    for (int u = su0; u < su1; ++seg) {
      const int sup = u / p.nkb;
      const int seg_end = min(su1, (sup + 1) * p.nkb);
      const int buf = C::kDBufs == 2 ? (seg & 1) : 0;
      // contributors of this super-tile: CTAs whose range intersects [sup*nkb, (sup+1)*nkb)
      const int c_first = (sup * p.nkb) / p.su_per_cta;
      const int c_last = ((sup + 1) * p.nkb - 1) / p.su_per_cta;
      const int n_contrib = kCluster ? 1 : c_last - c_first + 1;
      const int my_contrib = (int)blockIdx.x - c_first;
      float* part = p.partial + ((size_t)sup * p.max_contrib + my_contrib) * (kW4R * TN * kW4TileM);
      mbar_wait_relaxed(&tmem_full[buf], C::kDBufs == 2 ? ((seg >> 1) & 1) : (seg & 1));
      tcgen05_fence_after();
      W4_TRACE(8 + (seg & 3) * 2, 0);
      {
        // both tiles of the super-tile, kCh token columns at a time
        const int n0 = (p.half_tiles ? sup : sup * kW4R) * kW4TileM + m;
        const int n1 = (p.half_tiles ? sup + p.half_tiles : sup * kW4R + 1) * kW4TileM + m;
        const bool ok0 = n0 < p.N, ok1 = n1 < p.N;
        const bool direct = n_contrib == 1 && !p.defer, whole = kCluster || (kWhole && direct && seg_end == su1);
        const float bv0 = (p.bias && ok0 && direct) ? __half2float(p.bias[n0]) : 0.f;
        const float bv1 = (p.bias && ok1 && direct) ? __half2float(p.bias[n1]) : 0.f;
        constexpr int kCh = 16;  // columns fetched per tcgen05.wait::ld (32 spill)
#pragma unroll 1
        for (int c = 0; c < TN; c += kCh) {
          uint32_t d0[kCh], d1[kCh];
#pragma unroll
          for (int q = 0; q < kCh / 16; ++q) {
            tmem_ld_32x32b_x16(tmem_d + lane_base + (buf * kW4R + 0) * TN + c + q * 16, reinterpret_cast<uint32_t(&)[16]>(d0[q * 16]));
            tmem_ld_32x32b_x16(tmem_d + lane_base + (buf * kW4R + 1) * TN + c + q * 16, reinterpret_cast<uint32_t(&)[16]>(d1[q * 16]));
          }
          tmem_ld_wait();
          if (whole) {   // the rings have been used up: every product is done
            float* sums = reinterpret_cast<float*>(smem);
#pragma unroll
            for (int j = 0; j < kCh; ++j) {
              sums[(c + j) * kW4SumPitch + m] = __uint_as_float(d0[j]);
              sums[(c + j) * kW4SumPitch + kW4TileM + m] = __uint_as_float(d1[j]);
            }
          } else if (!direct) {
#pragma unroll
            for (int j = 0; j < kCh; ++j) {
              if (c + j < p.T) {
                part[(c + j) * kW4TileM + m] = __uint_as_float(d0[j]);
                part[(TN + c + j) * kW4TileM + m] = __uint_as_float(d1[j]);
              }
            }
          } else if (p.act) {
            if (ok0) {
#pragma unroll
              for (int j = 0; j < kCh; ++j) {
                const int t = c + j;
                if (t < p.T) p.y[(size_t)t * p.ldy + n0] = silu_mul_f16(__uint_as_float(d0[j]) + bv0, __uint_as_float(d1[j]) + bv1);
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < kCh; ++j) {
              const int t = c + j;
              if (t < p.T) {
                if (ok0) p.y[(size_t)t * p.ldy + n0] = __float2half_rn(__uint_as_float(d0[j]) + bv0);
                if (ok1) p.y[(size_t)t * p.ldy + n1] = __float2half_rn(__uint_as_float(d1[j]) + bv1);
              }
            }
          }
        }
      }
      if (kWhole && threadIdx.x == 0 && n_contrib == 1 && !p.defer && seg_end == su1) s_whole = sup;
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[buf]);
      W4_TRACE(9 + (seg & 3) * 2, 0);
      if (n_contrib > 1 && !p.defer) {
        // release: the epilogue barrier orders every thread's partial stores before thread 0's gpu-scope fence + count
        asm volatile("bar.sync 1, %0;" ::"n"(kW4EpWarps * 32) : "memory");
        if (threadIdx.x == 0) {
          __threadfence();
          atomicInc(&p.counters[sup], 2 * n_contrib - 1);
          s_fix[nfix][0] = sup;
          s_fix[nfix][1] = n_contrib;
          s_fix[nfix][2] = my_contrib;
        }
        ++nfix;
      }
      u = seg_end;
    }
    if (threadIdx.x == 0) s_nfix = nfix;
    W4_TRACE(5, 0);
  }

  // -------------------------------------------------------------------- shared super-tiles: every contributor reduces a slice
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc<C::kTmemCols>(tmem_base);
  const int nfix = s_nfix;
  if (nfix > 0) pdl_wait();
  W4_TRACE(40, 0);
  for (int f = 0; f < nfix; ++f) {
    const int sup = s_fix[f][0], n_contrib = s_fix[f][1], my_contrib = s_fix[f][2];
    if (threadIdx.x == 0) {
      // (one counter that wraps: with a second one for those who had finished, whose last owner re-armed both, a CTA ended 1 us later, behind an answer from L2;
      // us: 4096 -> 6144 at 9 tokens 9.2 -> 8.7, 4096 -> 22016 at 64 22.6 -> 21.7, 2048 -> 2560 at 16 5.9 -> 5.6)
      uint32_t spins = 0;
      while (ld_acquire_gpu(&p.counters[sup]) < (unsigned)n_contrib) {  // all contributors are co-resident (grid <= #SMs, 1 CTA/SM)
        __nanosleep(64);
        if (++spins > (1u << 24)) __trap();
      }
      atomicInc(&p.counters[sup], 2 * n_contrib - 1);
    }
    __syncthreads();
    W4_TRACE(41 + f * 3, 0);
    const float* base = p.partial + (size_t)sup * p.max_contrib * (kW4R * TN * kW4TileM);
    const int rows = min(p.T, TN);
    const int n_vec = kW4R * rows * (kW4TileM / 4);  // float4 elements: [r][row][32]
    const int per = (n_vec + n_contrib - 1) / n_contrib;
    const int hi = min(n_vec, (my_contrib + 1) * per);
    constexpr size_t kPartStride = (size_t)kW4R * TN * kW4TileM;
    if (!p.act) {
      for (int idx = my_contrib * per + (int)threadIdx.x; idx < hi; idx += kW4Threads) {
        const int r = idx / (rows * (kW4TileM / 4));
        const int rem = idx - r * rows * (kW4TileM / 4);
        const int tt = rem / (kW4TileM / 4), mm = (rem % (kW4TileM / 4)) * 4;
        const size_t off = (size_t)(r * TN + tt) * kW4TileM + mm;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int c0 = 0; c0 < n_contrib; c0 += 4) {  // contributor order: deterministic
          float4 ld[4];
#pragma unroll
          for (int cc = 0; cc < 4; ++cc)
            ld[cc] = (c0 + cc < n_contrib) ? __ldcg(reinterpret_cast<const float4*>(&base[(size_t)(c0 + cc) * kPartStride + off]))
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) { acc.x += ld[cc].x; acc.y += ld[cc].y; acc.z += ld[cc].z; acc.w += ld[cc].w; }
        }
        const int nn = (p.half_tiles ? sup + r * p.half_tiles : sup * kW4R + r) * kW4TileM + mm;
        if (nn < p.N) {  // N % 32 == 0: a float4 never straddles N
          if (p.bias) {
            acc.x += __half2float(p.bias[nn]); acc.y += __half2float(p.bias[nn + 1]);
            acc.z += __half2float(p.bias[nn + 2]); acc.w += __half2float(p.bias[nn + 3]);
          }
          uint2 o;
          o.x = pack_half2(acc.x, acc.y);
          o.y = pack_half2(acc.z, acc.w);
          w4_store(p, &p.y[(size_t)tt * p.ldy + nn], o);
        }
      }
    } else {
      // fused SiLU(gate) * up: an element needs both tiles of the super-tile; slices over [row][32 float4]
      const int n_vec_a = rows * (kW4TileM / 4);
      const int per_a = (n_vec_a + n_contrib - 1) / n_contrib;
      const int hi_a = min(n_vec_a, (my_contrib + 1) * per_a);
      for (int idx = my_contrib * per_a + (int)threadIdx.x; idx < hi_a; idx += kW4Threads) {
        const int tt = idx / (kW4TileM / 4), mm = (idx % (kW4TileM / 4)) * 4;
        const size_t off = (size_t)tt * kW4TileM + mm;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f), u = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int c0 = 0; c0 < n_contrib; c0 += 2) {  // contributor order: deterministic
          float4 lg[2], lu[2];
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            const bool in = c0 + cc < n_contrib;
            lg[cc] = in ? __ldcg(reinterpret_cast<const float4*>(&base[(size_t)(c0 + cc) * kPartStride + off])) : make_float4(0.f, 0.f, 0.f, 0.f);
            lu[cc] = in ? __ldcg(reinterpret_cast<const float4*>(&base[(size_t)(c0 + cc) * kPartStride + (size_t)TN * kW4TileM + off]))
                        : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            g.x += lg[cc].x; g.y += lg[cc].y; g.z += lg[cc].z; g.w += lg[cc].w;
            u.x += lu[cc].x; u.y += lu[cc].y; u.z += lu[cc].z; u.w += lu[cc].w;
          }
        }
        const int nn = sup * kW4TileM + mm;  // column of the [T, N / 2] output
        const int ng = nn, nu = nn + p.half_tiles * kW4TileM;
        if (p.bias) {
          g.x += __half2float(p.bias[ng]); g.y += __half2float(p.bias[ng + 1]); g.z += __half2float(p.bias[ng + 2]); g.w += __half2float(p.bias[ng + 3]);
          u.x += __half2float(p.bias[nu]); u.y += __half2float(p.bias[nu + 1]); u.z += __half2float(p.bias[nu + 2]); u.w += __half2float(p.bias[nu + 3]);
        }
        __half o[4] = {silu_mul_f16(g.x, u.x), silu_mul_f16(g.y, u.y), silu_mul_f16(g.z, u.z), silu_mul_f16(g.w, u.w)};
        w4_store(p, &p.y[(size_t)tt * p.ldy + nn], *reinterpret_cast<uint2*>(o));
      }
    }
    W4_TRACE(42 + f * 3, 0);
  }
  if (kWhole && s_whole >= 0) {
    if (nfix == 0) pdl_wait();
    const float* sums = reinterpret_cast<const float*>(smem);
    const int per_tok = p.act ? kW4TileM / 4 : kW4R * kW4TileM / 4;
    w4_finish(p, s_whole, per_tok, 0, p.T * per_tok, [&](int at) { return *reinterpret_cast<const float4*>(sums + at); });
  }
  if constexpr (kCluster) {
    // the cluster's CTAs add their parts of k through one another's shared memory, CTA r its share of the outputs, always in the order of the ranks
    pdl_wait();
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    W4_TRACE(41, 0);
    const uint32_t base = smem_u32(smem);
    const int d = p.cluster, per_tok = p.act ? kW4TileM / 4 : kW4R * kW4TileM / 4, items = p.T * per_tok, share = (items + d - 1) / d;
    w4_finish(p, c_sup, per_tok, c_rank * share, min(items, (c_rank + 1) * share), [&](int at) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 v[kW4MostCluster];
#pragma unroll
      for (int i = 0; i < kW4MostCluster; ++i) v[i] = i < d ? ld_cluster_v4(base + at * 4, i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kW4MostCluster; ++i) { acc.x += v[i].x; acc.y += v[i].y; acc.z += v[i].z; acc.w += v[i].w; }
      return acc;
    });
    W4_TRACE(42, 0);
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // nobody leaves while its sums are read
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  W4_TRACE(63, 0);
}

// checkpoint tensors -> unit records.  One thread per output u32.
__global__ void gptq_pack_kernel(const uint32_t* __restrict__ qweight, const uint32_t* __restrict__ qzeros,
                                 const __half* __restrict__ scales, uint32_t* __restrict__ packed, int64_t K, int64_t N, int groupsize,
                                 int group_rows, int nkb, int64_t n_words_total, int half_tiles, const int32_t* __restrict__ row_perm) {
  const int rec_words = (kW4WordBytes + group_rows * kW4MetaRowBytes) / 4;
  const int64_t G = (K + groupsize - 1) / groupsize;
  for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < n_words_total; o += (int64_t)gridDim.x * blockDim.x) {
    const int64_t rec = o / rec_words;          // record index in (super-tile, k-block, r) order
    const int r = (int)(o - rec * rec_words);
    const int64_t sup = rec / ((int64_t)nkb * kW4R);
    const int kb = (int)((rec / kW4R) % nkb);
    const int64_t tile = half_tiles ? sup + (rec % kW4R) * half_tiles : sup * kW4R + rec % kW4R;
    uint32_t out = 0;
    if (r < kW4WordBytes / 4) {
      const int c = r / (kW4TileM * 4), m = (r / 4) % kW4TileM, j = r % 4;
      const int64_t n = tile * kW4TileM + m;
      const int64_t kw = (int64_t)kb * (kW4BlockK / 8) + c * 4 + j;  // checkpoint word row: k = 8 kw .. 8 kw + 7
      if (n < N && kw * 8 < K) {
        if (!row_perm) {
          const uint32_t w = qweight[kw * N + n];
#pragma unroll
          for (int k = 0; k < 8; ++k) out |= ((w >> (4 * k)) & 15u) << (4 * ((k & 1) * 4 + (k >> 1)));
        } else {
          // act-order: packed row k' holds checkpoint row row_perm[k'] (rows sorted by group)
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int64_t src = row_perm[kw * 8 + k];
            const uint32_t q = (qweight[(src >> 3) * N + n] >> (4 * (src & 7))) & 15u;
            out |= q << (4 * ((k & 1) * 4 + (k >> 1)));
          }
        }
      }
    } else {
      const int mr = r - kW4WordBytes / 4;
      const int row = mr / kW4TileM, m = mr % kW4TileM;
      const int64_t n = tile * kW4TileM + m;
      const int64_t k0 = (int64_t)kb * kW4BlockK + (int64_t)row * (kW4BlockK / group_rows);
      out = 1u << 16;  // padding: scale 0, zero 1
      if (n < N && k0 < K) {
        const int64_t g = min(k0 / groupsize, G - 1);
        const uint32_t z = ((qzeros[g * (N / 8) + n / 8] >> (4 * (n % 8))) & 15u) + 1u;  // the +1 of quant_linear.py:185
        out = (uint32_t)__half_as_ushort(scales[g * N + n]) | (z << 16);
      }
    }
    packed[o] = out;
  }
}

static unsigned long long* g_w4_trace = nullptr;

// k-blocks per tile.  Rounded up to a multiple of 8 (empty records; the activation TMA zero-fills past K) when that adds
// at most 5 % of traffic: it lets a super-tile be cut into 2 / 4 / 8 equal CTA shares (Llama-2 down_proj: 86 -> 88).
static int w4_nkb(int64_t K) {
  const int nkb = (int)((K + kW4BlockK - 1) / kW4BlockK);
  const int up = (nkb + 7) / 8 * 8;
  return (up - nkb) * 20 <= nkb ? up : nkb;
}

struct W4Plan {
  int TN, nkb, n_super, su_per_cta, n_ctas, max_contrib;
  int cluster;   // > 0: so many CTAs share a super-tile and add their sums through shared memory; nothing goes to a workspace
  bool forced;   // B200_W4_SU's cut
};

constexpr float kW4SuUs = 0.35f * kW4R;   // us that a CTA takes for a super-unit
static float w4_whole_us(int nkb) { return kW4SuUs * nkb + 1.f; }   // ... for a super-tile that it has alone

// One token tile (T <= kW4DecodeT): how many super-units per CTA.  Candidates are the balanced stream-K cut (every SM the same
// number of units, but most CTAs then straddle two super-tiles: two fix-ups at the tail) and the aligned cuts nkb / d
// (a CTA = 1/d of one super-tile: one fix-up with d contributors, or none for d = 1, at the price of idle SMs when
// n_super * d is not close to a multiple of the SM count).  Costs in microseconds fitted to a sweep of the cut on B200
// (cold weights): 0.35 per unit in the main loop, ~1 for a direct epilogue, 4.5-6 for one split-K fix-up (partial store,
// gpu-scope fence, waiting for the slowest contributor, L2-latency-bound slice reduction), ~10 when CTAs straddle.
static W4Plan plan_w4(int64_t T, int64_t N, int64_t K, int sms, bool defer = false, float* cost_of = nullptr) {
  W4Plan pl;
  pl.cluster = 0;
  pl.TN = T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : 128;
  pl.nkb = w4_nkb(K);
  pl.n_super = (int)((N + kW4R * kW4TileM - 1) / (kW4R * kW4TileM));
  const int total = pl.n_super * pl.nkb;
  const int ctas = total < sms ? total : sms;
  int best = (total + ctas - 1) / ctas;
  if (best < 2 && pl.nkb >= 2) best = 2;  // one unit per team at least
  // deferred reduction (the consumer kernel sums the partials): no in-kernel fix-up, a CTA that straddles two super-tiles only
  // pays a mid-loop accumulator drain (~1 us)
  auto cost = [&](int su, bool aligned, int d) {
    if (!defer && aligned && d == 1) return w4_whole_us(su);
    const float fix = defer ? (aligned ? 0.f : 1.0f) : (aligned ? 4.5f + 0.2f * d : 10.0f);
    return kW4SuUs * su + fix;
  };
  float best_cost = cost(best, pl.nkb % best == 0, pl.nkb / best);
  for (int d = 1; d <= 8; d *= 2) {
    if (pl.nkb % d != 0) break;
    const int su = pl.nkb / d;
    if ((int64_t)pl.n_super * d > sms || su < 2) continue;
    const float c = cost(su, true, d);
    if (c < best_cost) { best_cost = c; best = su; }
  }
  pl.su_per_cta = best;
  static int env_su = -1;  // experiments: B200_W4_SU forces the cut
  if (env_su < 0) {
    const char* e = getenv("B200_W4_SU");
    env_su = e ? atoi(e) : 0;
  }
  pl.forced = env_su > 0 && (total + env_su - 1) / env_su <= sms;
  if (pl.forced) pl.su_per_cta = env_su;
  pl.n_ctas = (total + pl.su_per_cta - 1) / pl.su_per_cta;
  pl.max_contrib = (pl.nkb + pl.su_per_cta - 1) / pl.su_per_cta + 1;
  if (pl.su_per_cta % pl.nkb == 0) pl.max_contrib = 1;
  if (cost_of) *cost_of = best_cost;
  return pl;
}

static int w4_group_rows(int64_t K, int* groupsize) {
  if (*groupsize <= 0) *groupsize = (int)((K + kW4BlockK - 1) / kW4BlockK * kW4BlockK);  // one group
  return *groupsize >= kW4BlockK ? 1 : kW4BlockK / *groupsize;
}

}  // namespace b200

using namespace b200;

// debug: device buffer of [n_ctas][64] uint64 receiving per-CTA phase timestamps of the next int4 GEMM launches
extern "C" void b200_debug_w4_trace(void* device_buffer) { g_w4_trace = (unsigned long long*)device_buffer; }
extern "C" void b200_debug_w4_flags(int) {}

static bool w4_check_shape(int64_t N, int64_t K, int groupsize, const char* who) {
  if (K % 32 != 0 || N % 32 != 0 || K <= 0 || N <= 0) {  // exllamav2.py:118-119 asserts the same
    b200_set_last_error((std::string(who) + ": need K % 32 == 0 and N % 32 == 0").c_str());
    return false;
  }
  if (groupsize > 0 && (groupsize % 32 != 0 || (groupsize > kW4BlockK && groupsize % kW4BlockK != 0) ||
                        (groupsize < kW4BlockK && kW4BlockK % groupsize != 0))) {
    b200_set_last_error((std::string(who) + ": groupsize must be 32, 64, a multiple of 128, or <= 0 (one group)").c_str());
    return false;
  }
  return true;
}

extern "C" int64_t b200_gptq_packed_bytes(int64_t K, int64_t N, int groupsize) {
  if (!w4_check_shape(N, K, groupsize, "gptq_packed_bytes")) return B200_ERR_ARG;
  const int gr = w4_group_rows(K, &groupsize);
  const int64_t nkb = w4_nkb(K), ns = (N + kW4R * kW4TileM - 1) / (kW4R * kW4TileM);
  return ns * kW4R * nkb * (kW4WordBytes + gr * kW4MetaRowBytes);  // the last super-tile is padded with empty tiles
}

// layout 0: super-tile s = feature tiles (2s, 2s+1).  layout 1 ("gate|up", for a fused [gate; up] projection with
// N = 2 I, I % 128 == 0): super-tile s = tiles (s, s + I/128), i.e. gate feature n sits next to up feature n, which is what
// lets the GEMM apply SiLU(gate) * up in its epilogue (b200_gemm_w4a16_ex act = 1).
static int w4_half_tiles(int64_t N, int layout, const char* who) {
  if (layout == 0) return 0;
  if (layout != 1 || N % (2 * kW4TileM) != 0) {
    b200_set_last_error((std::string(who) + ": the gate|up layout needs N % 256 == 0").c_str());
    return -1;
  }
  return (int)(N / (2 * kW4TileM));
}

// qweight int32 [K/8, N], qzeros int32 [ceil(K/g), N/8], scales fp16 [ceil(K/g), N] (checkpoint layout, left untouched)
// -> packed (b200_gptq_packed_bytes bytes, 16-byte aligned).  row_perm == NULL: groups are k // groupsize (trivial g_idx).
// Act-order checkpoints (g_idx not sorted; exllamav2.py:31-48 builds q_perm for them): row_perm[k'] = the checkpoint row
// stored at packed row k', a stable arg-sort of g_idx, so that packed rows k' // groupsize share a group again; the GEMM
// is then fed x[:, row_perm] (b200_permute_columns).
extern "C" int b200_gptq_pack_ex(const void* qweight, const void* qzeros, const void* scales, const int32_t* row_perm, void* packed,
                                 int64_t K, int64_t N, int groupsize, int layout, void* stream) {
  if (!w4_check_shape(N, K, groupsize, "gptq_pack")) return B200_ERR_ARG;
  if (((uintptr_t)packed & 15) != 0) { b200_set_last_error("gptq_pack: packed buffer must be 16-byte aligned"); return B200_ERR_ARG; }
  const int half_tiles = w4_half_tiles(N, layout, "gptq_pack");
  if (half_tiles < 0) return B200_ERR_ARG;
  const int gr = w4_group_rows(K, &groupsize);
  const int nkb = w4_nkb(K);
  const int64_t n_words = b200_gptq_packed_bytes(K, N, groupsize) / 4;
  int64_t blocks = (n_words + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  gptq_pack_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const uint32_t*)qweight, (const uint32_t*)qzeros,
                                                                        (const __half*)scales, (uint32_t*)packed, K, N, groupsize, gr,
                                                                        nkb, n_words, half_tiles, row_perm);
  B200_CHECK_LAUNCH();
  b200_count_launches(1);
  return b200_settle(stream);   // products read records ahead of the wait for the kernel before them
}
extern "C" int b200_gptq_pack(const void* qweight, const void* qzeros, const void* scales, void* packed, int64_t K, int64_t N,
                              int groupsize, void* stream) {
  return b200_gptq_pack_ex(qweight, qzeros, scales, nullptr, packed, K, N, groupsize, 0, stream);
}

// bytes of split-K partials the int4 GEMM may write for this shape (the tile counters sit in the first 64 KiB)
// The plan a launch uses: the stream-K cut needs the workspace (partials + one counter per super-tile) and every CTA
// resident at once (the fix-up spins on its peers); otherwise each CTA takes whole super-tiles.  Clusters are compared with whichever of the two would run.
// clusters[d]: clusters of d CTAs that the chip holds (NULL: none).  The largest cluster whose super-tiles all fit in one wave, where it takes less.  Against whole super-tiles
// and aligned cuts, in the units of plan_w4: adding up through shared memory takes 2.5 us and 0.8 for each CTA whose sums are read, about as much as an aligned cut's
// fix-up, which has 8 contributors where the chip holds 15 clusters of 8 or fewer of more CTAs.  Us, through global memory / clusters, at 9, 64 and 128 tokens: 4096 ->
// 12288 (of 2) 12.2 / 12.1, 15.9 / 15.2, 23.0 / 21.6; 5120 -> 5120 (of 7) 8.9 / 8.6, 11.5 / 11.6, 16.2 / 16.3; the other side: 4096 -> 4096 (of 6) 6.9 / 7.2, 9.1 / 10.4,
// 12.5 / 14.7; 4096 -> 6144 (of 5) 8.3 / 8.6, 11.0 / 11.7, 15.1 / 15.9.
// Against cuts that straddle super-tiles (w4_clusters_less): few tokens, whose fix-up is short, against the SMs that clusters leave idle.
// 5632 -> 2048 (of 8) 8.3 / 6.7, 11.3 / 9.9, 15.8 / 14.7; 28672 -> 8192 (of 4) 29.4 / 31.9, 38.0 / 37.7, 56.5 / 54.7; 14336 -> 10240 (of 3) 21.8 / 23.4, 27.2 / 26.5, 39.4 / 37.2.
// In 1133 measured calls with clusters to choose, what is taken is 0.5 % slower on average than the better of the two; 26 take 1 to 6 % more than
// without clusters, one 22 % (12544 -> 11392 at 32 tokens, 22.7 / 27.8: 45 clusters, as many as the chip holds, whose time varies from call to call).
// us by which clusters of d CTAs, su super-units each, differ from a cut that straddles super-tiles, below 0; fitted to 570 calls of 9 to 128 tokens on B200: a super-unit's
// time at the token tile, a share of the memory for each CTA, the end of a super-tile
static bool w4_clusters_less(int64_t T, const W4Plan& cut, int d, int su) {
  const float unit = cut.TN <= 32 ? 0.44f : cut.TN <= 64 ? 0.48f : 0.71f;
  return unit * (su - cut.su_per_cta) + 0.049f * (cut.n_super * d - cut.n_ctas) + 0.4f + (0.0067f * d - 0.06f) * T < 0.f;
}
static W4Plan launch_plan_w4(int64_t T, int64_t N, int64_t K, int sms, bool has_workspace, bool defer = false, const int* clusters = nullptr) {
  float cost;
  W4Plan pl = plan_w4(T, N, K, sms, defer, &cost);
  if (defer) return pl;  // the caller checked: one token tile, workspace present; no counters, no co-residency requirement
  if (pl.max_contrib > 1 && (!has_workspace || (int64_t)pl.n_super * (int64_t)sizeof(unsigned) > kW4CounterBytes || pl.n_ctas > sms)) {
    pl.su_per_cta = pl.nkb;
    pl.n_ctas = pl.n_super;
    pl.max_contrib = 1;
    cost = w4_whole_us(pl.nkb);
  }
  if (!clusters || pl.forced) return pl;
  int d = kW4MostCluster;
  while (d > 1 && (d > pl.nkb || clusters[d] < pl.n_super)) --d;
  const int su = (pl.nkb + d - 1) / d;
  const bool straddles = pl.su_per_cta < pl.nkb && pl.nkb % pl.su_per_cta != 0;
  if (d > 1 && (straddles ? w4_clusters_less(T, pl, d, su) : kW4SuUs * su + 2.5f + 0.8f * d < cost)) {
    pl.cluster = d;
    pl.su_per_cta = su;
    pl.n_ctas = pl.n_super * d;
    pl.max_contrib = 1;
  }
  return pl;
}

// tests (no GPU needed): the cut through a workspace that is taken where no cluster shares super-tiles; out = {TN, k-blocks, super-tiles, 1, super-units per CTA,
// CTAs, contributor slots, R}
void b200_w4_plan_debug(int64_t T, int64_t N, int64_t K, int sms, int32_t* out) {
  const W4Plan pl = launch_plan_w4(T, N, K, sms, true);
  const int32_t v[8] = {pl.TN, pl.nkb, pl.n_super, 1, pl.su_per_cta, pl.n_ctas, pl.max_contrib, kW4R};
  for (int i = 0; i < 8; ++i) out[i] = v[i];
}

int64_t b200_w4_partial_bytes(int64_t T, int64_t N, int64_t K) {
  if (T > kW4DecodeT) return 0;
  const W4Plan pl = plan_w4(T, N, K, b200_num_sms());
  const int64_t need = pl.max_contrib <= 1 ? 0 : (int64_t)pl.n_super * pl.max_contrib * kW4R * pl.TN * kW4TileM * 4;
  // deferred reduction: every super-tile has at least one partial slot
  const W4Plan pd = plan_w4(T, N, K, b200_num_sms(), true);
  const int64_t nd = (int64_t)pd.n_super * pd.max_contrib * kW4R * pd.TN * kW4TileM * 4;
  return nd > need ? nd : need;
}

template <int TN, int kGR, int kEnd>
static int launch_gemm_w4(const CUtensorMap* mx, const void* packed, void* y, void* workspace, const void* bias, int T, int N,
                          const W4Plan& pl, int half_tiles, int act, int defer, cudaStream_t st) {
  using C = GemmW4Cfg<TN>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_w4a16_kernel<TN, kGR, kEnd>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) { b200_set_last_error(cudaGetErrorString(e)); return B200_ERR_CUDA; }
    configured = true;
  }
  W4Params p;
  p.y = (__half*)y;
  p.counters = (unsigned*)workspace;
  p.partial = workspace ? (float*)((char*)workspace + kW4CounterBytes) : nullptr;
  p.bias = (const __half*)bias;
  p.packed = (const unsigned char*)packed;
  p.T = T;
  p.N = N;
  p.nkb = pl.nkb;
  p.n_super = pl.n_super;
  p.su_per_cta = pl.su_per_cta;
  p.total_su = pl.n_super * pl.nkb;
  p.max_contrib = pl.max_contrib;
  p.rec_bytes = kW4WordBytes + kGR * kW4MetaRowBytes;
  p.half_tiles = half_tiles;
  p.act = act;
  p.ldy = act ? N / 2 : N;
  p.defer = defer;
  p.cluster = pl.cluster;
  p.trace = g_w4_trace;
  const dim3 grid(pl.n_ctas);
  b200_timing_mark(B200_TIME_GEMM_W4A16, 0, st);
  constexpr auto kernel = gemm_w4a16_kernel<TN, kGR, kEnd>;
  const cudaError_t e = b200_launch_cluster(kernel, grid, dim3(kW4Threads), (size_t)C::kSmemBytes, st, (unsigned)pl.cluster, *mx, p);
  if (e != cudaSuccess) { b200_set_last_error(cudaGetErrorString(e)); return B200_ERR_CUDA; }
  b200_step_trace_stamp("gemm_w4a16_kernel", st);
  b200_timing_mark(B200_TIME_GEMM_W4A16, 1, st);
  b200_count_launches(1);
  return B200_OK;
}

static const int* w4_clusters() {
  static const struct Table {
    int n[kW4MostCluster + 1];
    Table() : n{} {
      n[0] = n[1] = b200_num_sms();
      cudaFuncSetAttribute(gemm_w4a16_kernel<64, 1, kW4Cluster>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmW4Cfg<64>::kSmemBytes);
      b200_count_clusters(gemm_w4a16_kernel<64, 1, kW4Cluster>, kW4Threads, (size_t)GemmW4Cfg<64>::kSmemBytes, n);
    }
  } table;
  return table.n;
}

// tests: how an int4 call of up to kW4DecodeT tokens is cut (those that gemm_w4_few.cuh takes too) on a chip that holds clusters[d] clusters of d = 2 .. 8 CTAs; NULL: the
// present device's
extern "C" int b200_debug_w4_plan(int64_t T, int64_t N, int64_t K, int sms, int workspace, const int32_t* clusters, int32_t* out) {
  if (!out || T <= 0 || T > kW4DecodeT || N <= 0 || K <= 0 || sms <= 0) {
    b200_set_last_error("debug_w4_plan: bad arguments");
    return B200_ERR_ARG;
  }
  const W4Plan pl = launch_plan_w4(T, N, K, sms, workspace != 0, false, clusters ? clusters : w4_clusters());
  const int32_t v[8] = {pl.TN, pl.nkb, pl.n_super, pl.cluster, pl.su_per_cta, pl.n_ctas, pl.max_contrib, kW4R};
  for (int i = 0; i < 8; ++i) out[i] = v[i];
  return B200_OK;
}

// packed: output of b200_gptq_pack[_ex] for the same (K, N, groupsize, layout).
// act = 1 (layout 1 only): y [T, N/2] = SiLU(x Wgate) * (x Wup), the LlamaMLP activation (flash_llama_modeling.py:332-335) fused
// into the projection.  workspace as for b200_gemm_f16 (b200_gemm_workspace_bytes); without it every CTA takes whole
// super-tiles (no stream-K).
// splitk != NULL: deferred reduction - nothing is written to y; *splitk describes the fp32 partials left in the workspace.
static int gemm_w4a16_impl(const void* x, const void* packed, const void* bias, void* y, int64_t T, int64_t N, int64_t K, int groupsize,
                           int layout, int act, void* workspace, B200SplitK* splitk, void* stream) {
  if (T == 0 || N == 0) return B200_OK;
  if (!w4_check_shape(N, K, groupsize, "gemm_w4a16")) return B200_ERR_ARG;
  const int half_tiles = w4_half_tiles(N, layout, "gemm_w4a16");
  if (half_tiles < 0) return B200_ERR_ARG;
  if (act != 0 && (act != 1 || layout != 1)) { b200_set_last_error("gemm_w4a16: act = 1 needs the gate|up layout"); return B200_ERR_ARG; }
  const bool defer = splitk != nullptr;
  if (defer && (!workspace || T > 128)) {
    b200_set_last_error("gemm_w4a16_deferred: needs a workspace and T <= 128 (one token tile)");
    return B200_ERR_UNSUPPORTED;
  }
  const int gr = w4_group_rows(K, &groupsize);
  if (!defer && T > kW4DecodeT) {
    PairParams pp = {};
    pp.y = y;
    pp.bias = bias;
    pp.packed = (const unsigned char*)packed;
    pp.T = (int)T;
    pp.N = pp.ldy = (int)(act ? N / 2 : N);
    pp.half = half_tiles * kW4TileM;
    pp.n_kb = 2 * (int)((K + kW4BlockK - 1) / kW4BlockK);
    pp.rec_per_tile = w4_nkb(K);
    pp.rec_bytes = kW4WordBytes + gr * kW4MetaRowBytes;
    pp.group_rows = gr;
    pp.half_tiles = half_tiles;
    const PairPlan pl = pair_plan(T, N, pp.n_kb, true, b200_num_sms());
    return act ? launch_gemm_pair<kPairW4Silu>(x, nullptr, K, pp, pl, B200_TIME_GEMM_W4A16, (cudaStream_t)stream)
               : launch_gemm_pair<kPairW4>(x, nullptr, K, pp, pl, B200_TIME_GEMM_W4A16, (cudaStream_t)stream);
  }
  // (A deferred result has no fix-up to save: the step of Llama-3-8B stays 1 % faster with its partials left in global memory.)
  const W4FewPlan few = T <= kFewMostT && !defer ? few_plan(N, K, few_clusters()) : W4FewPlan{0, 0};
  if (few.d && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(y) & 7) == 0) {
    W4FewParams fp = {};
    fp.x = (const __half*)x;
    fp.y = (__half*)y;
    fp.bias = (const __half*)bias;
    fp.packed = (const unsigned char*)packed;
    fp.T = (int)T;
    fp.N = (int)N;
    fp.K = (int)K;
    fp.nkb = (int)((K + kW4BlockK - 1) / kW4BlockK);
    fp.rec_per_tile = w4_nkb(K);
    fp.half_tiles = half_tiles;
    fp.act = act;
    fp.ldy = (int)(act ? N / 2 : N);
    fp.x_blocks = few.blocks;
    fp.gave_up = b200_gave_up_word();
    if (!fp.gave_up) return B200_ERR_CUDA;
    return launch_w4_few_plan(fp, gr, (int)((N + kW4R * kW4TileM - 1) / (kW4R * kW4TileM)), few, (cudaStream_t)stream);
  }
  const W4Plan pl = launch_plan_w4(T, N, K, b200_num_sms(), workspace != nullptr, defer, w4_clusters());
  const CUtensorMap* mx = get_tmap_2d(x, T, K, K, pl.TN, 64, TmapDtype::kF16, TmapSwizzle::k128B);
  if (!mx) return B200_ERR_CUDA;
  if (defer) {
    splitk->partial = (const float*)((const char*)workspace + kW4CounterBytes);
    splitk->bias = bias;
    splitk->tiles_per_unit = kW4R;
    splitk->tn = pl.TN;
    splitk->nkb = pl.nkb;
    splitk->units_per_cta = pl.su_per_cta;
    splitk->max_contrib = pl.max_contrib;
    splitk->half_tiles = half_tiles;
    splitk->N = (int32_t)N;
    splitk->T = (int32_t)T;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int df = defer ? 1 : 0;
#define W4_DISPATCH(TNV, W)                                                                                                  \
  (gr == 1   ? launch_gemm_w4<TNV, 1, W>(mx, packed, y, workspace, bias, (int)T, (int)N, pl, half_tiles, act, df, st)         \
   : gr == 2 ? launch_gemm_w4<TNV, 2, W>(mx, packed, y, workspace, bias, (int)T, (int)N, pl, half_tiles, act, df, st)         \
             : launch_gemm_w4<TNV, 4, W>(mx, packed, y, workspace, bias, (int)T, (int)N, pl, half_tiles, act, df, st))
  if (pl.cluster) {
    switch (pl.TN) {
      case 16: return W4_DISPATCH(16, kW4Cluster);
      case 32: return W4_DISPATCH(32, kW4Cluster);
      case 64: return W4_DISPATCH(64, kW4Cluster);
      default: return W4_DISPATCH(128, kW4Cluster);
    }
  }
  switch (pl.TN) {
    case 16: return act && T > 8 && pl.max_contrib == 1 ? W4_DISPATCH(16, kW4Whole) : W4_DISPATCH(16, kW4Plain);
    case 32: return W4_DISPATCH(32, kW4Whole);
    case 64: return W4_DISPATCH(64, kW4Whole);
    default: return W4_DISPATCH(128, kW4Whole);
  }
#undef W4_DISPATCH
}
extern "C" int b200_gemm_w4a16_ex(const void* x, const void* packed, const void* bias, void* y, int64_t T, int64_t N, int64_t K,
                                  int groupsize, int layout, int act, void* workspace, void* stream) {
  return gemm_w4a16_impl(x, packed, bias, y, T, N, K, groupsize, layout, act, workspace, nullptr, stream);
}
extern "C" int b200_gemm_w4a16(const void* x, const void* packed, const void* bias, void* y, int64_t T, int64_t N, int64_t K,
                               int groupsize, void* workspace, void* stream) {
  return gemm_w4a16_impl(x, packed, bias, y, T, N, K, groupsize, 0, 0, workspace, nullptr, stream);
}
// Deferred split-K reduction: the GEMM leaves fp32 partials in `workspace` and fills *splitk; the next kernel of the stream
// (b200_rmsnorm_residual_splitk, b200_rope_kv_write_paged_splitk, b200_splitk_silu_mul, b200_splitk_reduce, the fused all-reduce)
// sums them in contributor order, without the grid-wide wait of b200_gemm_w4a16_ex's own fix-up and equal to its result up to the order of the fp32 sums
// (up to eight tokens that has a kernel with other cuts of k).  The bias is applied by the consumer.  T <= 128.
extern "C" int b200_gemm_w4a16_deferred(const void* x, const void* packed, const void* bias, int64_t T, int64_t N, int64_t K,
                                        int groupsize, int layout, void* workspace, B200SplitK* splitk, void* stream) {
  if (!splitk) { b200_set_last_error("gemm_w4a16_deferred: splitk is NULL"); return B200_ERR_ARG; }
  return gemm_w4a16_impl(x, packed, bias, nullptr, T, N, K, groupsize, layout, 0, workspace, splitk, stream);
}
