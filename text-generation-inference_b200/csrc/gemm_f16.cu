// fp16 linear  Y[T,N] = X[T,K] . W[N,K]^T  (fp32 accumulate, fp16 out) on tcgen05 tensor cores.
//
// Replaces the cuBLAS HGEMM behind `FastLinear.forward` / `TensorParallelHead.forward`
// (server/text_generation_server/utils/layers.py:110-111, 257-262).
//
// Swap-AB: the 128 output features of a weight tile are the UMMA M dimension (A operand, K-major, streamed
// from HBM once by TMA with 128B swizzle), the step's tokens are the UMMA N dimension (B operand, TN = 16..256),
// the fp32 accumulator D[128 x TN] lives in TMEM.  One token tile (T <= 256; larger calls, and those of more than 64 tokens that are faster there, go to
// gemm_pair.cuh) is weight-streaming / HBM-bound: the flattened
// (feature tile, 64-wide k-block) unit space is cut into equal contiguous ranges, one per SM (stream-K), so all 148 SMs
// pull the same number of weight bytes; a tile that straddles CTAs gets its fp32 partials summed in contributor order by
// the last CTA to finish (deterministic).  PDL: the weight ring is filled before griddepcontrol.wait.
// Warp roles: 0 = TMA producer, 1 = MMA issuer (one elected thread), 2..5 = epilogue (TMEM -> registers -> HBM).
#include "common.cuh"
#include "gemm_pair.cuh"
#include "tmap.cuh"
#include "../../include/b200_tgis.h"

#include <cstdlib>
#include <cuda_bf16.h>

namespace b200 {

// Element formats of one instantiation: 0 = fp16 operands, fp16 output (the flash families); 1 = bfloat16 operands, bfloat16
// output; 2 = bfloat16 operands, fp32 output (hybrid families: projections whose results enter a recurrence, a norm or the
// soft-max stay in 32 bits); 3 = as 1 with the square of ReLU on the result.  Same pipeline; the instruction descriptor's operand formats and the epilogue's stores differ.
template <int FMT>
__device__ __forceinline__ float gemm_load_bias(const void* bias, int n) {
  if constexpr (FMT == 0) return __half2float(reinterpret_cast<const __half*>(bias)[n]);
  else return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[n]);
}
template <int FMT>
__device__ __forceinline__ void gemm_store(void* y, size_t i, float v) {
  if constexpr (FMT == 0) reinterpret_cast<__half*>(y)[i] = __float2half_rn(v);
  else if constexpr (FMT == 1) reinterpret_cast<__nv_bfloat16*>(y)[i] = __float2bfloat16_rn(v);
  else if constexpr (FMT == 3) reinterpret_cast<__nv_bfloat16*>(y)[i] = __float2bfloat16_rn(v < 0.f ? 0.f : v * v);
  else reinterpret_cast<float*>(y)[i] = v;
}

constexpr int kGemmThreads = 192;
constexpr int kTileM = 128;  // features per tile
constexpr int kTileK = 64;   // fp16 elements per k-block = one 128-byte swizzle row
// Calls of more than kF16DecodeT tokens may go to the SM pairs (gemm_pair.cuh), calls of more than kF16MostT all do; between the two f16_cluster_us, or
// f16_stream_us where no cluster shares a tile, says which kernel takes less.  Measured on B200 in replayed graphs (us, this kernel / pairs) at 65 tokens: 4096 ->
// 4096 11.7 / 13.2, 4096 -> 22016 38.8 / 38.8, 5632 -> 2048 10.7 / 15.4, 11008 -> 4096 20.3 / 28.4, 16384 -> 2048 18.6 / 38.0, 28672 -> 2048 27.1 / 63.2, 28672 ->
// 8192 79 / 93, 20480 -> 5120 38 / 52, 2048 -> 2560 8.2 / 7.8; at 128: 13.0 / 13.6, 45.0 / 41.3, 12.0 / 15.6, 21.3 / 28.7, 20.0 / 38.0, 28.6 / 63.5, 84 / 97, 40 /
// 61, 9.5 / 8.2; at 256: 16.8 / 15.8, 74 / 51, 16.2 / 16.2, 26.9 / 34.9, 26.6 / 38.5, 37.8 / 63.5, 114 / 117 (129 / 142 under the power cap), 54 / 66, 12.9 / 9.3.
// Up to 64 tokens the pairs take wide outputs only (feature tiles that no wave of clusters holds), from kF16PairT tokens on; us, this kernel / pairs, at 16
// and 64 tokens: 2048 -> 11264 10.9 / 10.6 and 13.0 / 11.7, 2048 -> 32000 24.1 / 22.8 and 29.0 / 24.3, 4096 -> 12288 18.9 / 18.9 and 21.1 / 20.4, 5120 ->
// 15360 25.8 / 26.6 and 28.4 / 28.4, 4096 -> 22016 (a wave and a sixth) 31.4 / 34.7 and 37.0 / 38.5.
constexpr int kF16PairT = 16, kF16DecodeT = 64, kF16MostT = 256;
// fp32 results show how long a sum ran in the tensor cores: cut into stream-K pieces that are added in fp32 it is off by 5e-7 (against float64,
// k = 2048), in one piece by 2e-6.  So they stay here for as long as this kernel cuts them (one token tile).
constexpr int64_t kCounterBytes = 64 * 1024;

template <int TN>
struct GemmF16Cfg {
  static constexpr int kABytes = kTileM * kTileK * 2;
  static constexpr int kBBytes = TN * kTileK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = TN <= 64 ? 8 : (TN == 128 ? 6 : 4);
  static constexpr int kTmemCols = 2 * TN;   // clusters: an accumulator for either half of a CTA's k
  static constexpr int kSmemBytes = kStages * kStageBytes + (2 * kStages + 2) * 8 + 16 + 1024;
  static_assert(TN * (kTileM + 4) * 4 <= kStages * kStageBytes, "a cluster's sums lie where the ring was");
};

struct F16Params {
  void* y;
  float* partial;  // [feature tile][contributor][TN][128] fp32
  int* counters;   // [feature tile]
  const void* bias;
  int T, N;
  int nkb;            // 64-wide k-blocks per tile
  int units_per_cta;  // contiguous (tile, k-block) units per CTA
  int total_units;
  int max_contrib;    // partial slots per tile
  int cluster;        // > 0: a cluster of so many CTAs has one feature tile, each a part of k
  int held;           // 1: w was settled (b200_settle) and has not been written since
  int defer;          // 1: leave every tile segment as an fp32 partial for the consumer kernel (B200SplitK), no fix-up
};

constexpr int kF16SumPitch = kTileM + 4;   // floats of a token's sums in shared memory

// The end of a feature tile that a cluster shares: every CTA has fp32 sums of its part of k in shared memory ([token][kF16SumPitch]); CTA r adds its share of
// the outputs over all of them in their order.  Against partial sums in global memory that the last CTA to arrive adds by itself (us in a replayed graph,
// 8 / 32 / 64 tokens): 2048 -> 2048 5.1 / 8.2 / 13.0 -> 5.3 / 5.8 / 6.9, 4096 -> 4096 9.0 / 11.5 / 14.5 -> 9.4 / 10.2 / 10.9, 11008 -> 4096 16.5 / 18.9 / 21.9 ->
// 17.0 / 17.8 / 18.6, 20480 -> 5120 42.3 / 44.9 / 49.5 -> 35.2 / 36.1 / 40.7 (three CTAs to a tile instead of tiles that straddle CTAs).
template <int FMT>
__device__ __forceinline__ void f16_cluster_sum(const F16Params& p, const float* sums, int tile, int rank) {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const uint32_t base = smem_u32(sums);
  const int d = p.cluster, items = p.T * (kTileM / 4), share = (items + d - 1) / d, hi = min(items, (rank + 1) * share);
  for (int i = rank * share + (int)threadIdx.x; i < hi; i += kGemmThreads) {
    const int tok = i / (kTileM / 4), m = (i % (kTileM / 4)) * 4, n = tile * kTileM + m;
    const uint32_t at = base + (tok * kF16SumPitch + m) * 4;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < d; c += 4) {
      float v[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (c + j < d) {
          const float4 four = ld_cluster_v4(at, c + j);
          v[j][0] = four.x; v[j][1] = four.y; v[j][2] = four.z; v[j][3] = four.w;
        } else {
          v[j][0] = v[j][1] = v[j][2] = v[j][3] = 0.f;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] += v[j][e];
    }
    if (p.bias)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] += n + e < p.N ? gemm_load_bias<FMT>(p.bias, n + e) : 0.f;
    const size_t o = (size_t)tok * p.N + n;
    if (FMT == 0 && n + 3 < p.N && (p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7) == 0) {
      *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p.y) + o) = make_uint2(pack_half2(s[0], s[1]), pack_half2(s[2], s[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n + e < p.N) gemm_store<FMT>(p.y, o + e, s[e]);
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // nobody leaves while its sums are read
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int TN, int FMT>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const F16Params p) {
  using C = GemmF16Cfg<TN>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStageBytes);
  uint64_t* empty_bar = full_bar + C::kStages;
  uint64_t* tmem_full = empty_bar + C::kStages;
  uint64_t* tmem_empty = tmem_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 1);
  __shared__ int s_is_last;

  pdl_launch_dependents();
  const int warp = warp_id(), lane = lane_id();
  const int c_tile = p.cluster ? (int)blockIdx.x / p.cluster : 0, c_rank = p.cluster ? (int)blockIdx.x - c_tile * p.cluster : 0;
  const int u0 = p.cluster ? c_tile * p.nkb + c_rank * p.nkb / p.cluster : blockIdx.x * p.units_per_cta;
  const int u1 = p.cluster ? c_tile * p.nkb + (c_rank + 1) * p.nkb / p.cluster : min(p.total_units, u0 + p.units_per_cta);
  const int n_units = u1 - u0;
  const int tile0 = u0 / p.nkb, kb0 = u0 - tile0 * p.nkb;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    mbar_init(tmem_empty, 4);
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc<C::kTmemCols>(tmem_slot);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_d = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      const uint64_t pol_w = policy_evict_first(), pol_x = policy_evict_last();
      // While the previous kernel ends, the first ring's weight tiles are on their way: held weights to shared memory; others to L2 only, since they
      // may be that kernel's result.  us in
      // a replayed graph, tiles read ahead / only after the wait / brought to L2 ahead: one token 2048 -> 2560 5.4 / 5.7 / 5.65, 4096 -> 4096 8.65 / 9.6 /
      // 8.95, 11008 -> 4096 17.3 / 18.7 / 16.7, 2048 -> 32000 23.1 / 24.4 / 22.1; 32 tokens 4096 -> 4096 9.6 / 10.3 / 9.7, 4096 -> 22016 33.0 / 33.5 / 31.8.
      int tile = tile0, kb = kb0;
      const int npre = min(n_units, C::kStages);
      for (int i = 0; i < npre; ++i) {
        if (p.held) {
          mbar_arrive_expect_tx(&full_bar[i], C::kStageBytes);
          tma_load_2d_hint(smem + i * C::kStageBytes, &tmap_w, kb * kTileK, tile * kTileM, &full_bar[i], pol_w);
        } else {
          tma_prefetch_2d_hint(&tmap_w, kb * kTileK, tile * kTileM, pol_w);
        }
        if (++kb == p.nkb) { kb = 0; ++tile; }
      }
      pdl_wait();
      int from = 0;
      if (p.held) {
        for (int kbx = kb0; from < npre; ++from) {
          tma_load_2d_hint(smem + from * C::kStageBytes + C::kABytes, &tmap_x, kbx * kTileK, 0, &full_bar[from], pol_x);
          if (++kbx == p.nkb) kbx = 0;
        }
      } else {
        tile = tile0;
        kb = kb0;
      }
      for (int i = from; i < n_units; ++i) {
        const int s = i % C::kStages;
        mbar_wait(&empty_bar[s], ((i / C::kStages) & 1) ^ 1);
        mbar_arrive_expect_tx(&full_bar[s], C::kStageBytes);
        unsigned char* a = smem + s * C::kStageBytes;
        tma_load_2d_hint(a, &tmap_w, kb * kTileK, tile * kTileM, &full_bar[s], pol_w);
        tma_load_2d_hint(a + C::kABytes, &tmap_x, kb * kTileK, 0, &full_bar[s], pol_x);
        if (++kb == p.nkb) { kb = 0; ++tile; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = umma_idesc_f16_f32acc(kTileM, TN) | (FMT != 0 ? ((1u << 7) | (1u << 10)) : 0u);  // a/b format 1 = bf16
    const int half = p.cluster ? (n_units + 1) / 2 : n_units;   // clusters: the second half of the part of k has an accumulator of its own
    uint32_t d = tmem_d;
    int seg = 0, kb = kb0;
    for (int i = 0; i < n_units; ++i) {
      if (i == half) d += TN;
      const bool seg_first = (i == 0) || kb == 0 || i == half;
      const bool seg_last = (i == n_units - 1) || kb == p.nkb - 1;
      const int s = i % C::kStages;
      if (seg_first && seg > 0) mbar_wait(tmem_empty, (seg - 1) & 1);  // epilogue drained the previous segment's D
      mbar_wait(&full_bar[s], (i / C::kStages) & 1);
      tcgen05_fence_after();
      if (elect_one()) {
        const uint32_t a_addr = smem_u32(smem + s * C::kStageBytes);
        const uint64_t adesc = umma_desc_kmajor_sw128(a_addr);
        const uint64_t bdesc = umma_desc_kmajor_sw128(a_addr + C::kABytes);
#pragma unroll
        for (int k = 0; k < kTileK / 16; ++k)
          umma_f16_ss(d, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (!seg_first || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[s]);
        if (seg_last) umma_commit(tmem_full);
      }
      __syncwarp();
      if (seg_last) ++seg;
      if (++kb == p.nkb) kb = 0;
    }
  } else {
    // ------------------------------------------------------------------ epilogue: thread = one output feature
    const int quarter = warp & 3;
    const int m = quarter * 32 + lane;
    const int etid = threadIdx.x - 64;  // 0..127
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    pdl_wait();  // outputs / bias / stream-K workspace belong to the stream order
    int tile = tile0, kb = kb0, seg = 0;
    for (int i = 0; i < n_units;) {
      const int seg_len = min(p.nkb - kb, n_units - i);
      const int n = tile * kTileM + m;
      const bool n_ok = n < p.N;
      const int c_first = (tile * p.nkb) / p.units_per_cta;
      const int c_last = ((tile + 1) * p.nkb - 1) / p.units_per_cta;
      const int n_contrib = c_last - c_first + 1;
      const int my_contrib = (int)blockIdx.x - c_first;
      mbar_wait(tmem_full, seg & 1);
      tcgen05_fence_after();
      if (p.cluster) {   // one segment; the ring has been used up: every product is done
        float* sums = reinterpret_cast<float*>(smem);
#pragma unroll 1
        for (int c = 0; c < TN; c += 16) {
          uint32_t d0[16], d1[16];
          tmem_ld_32x32b_x16(tmem_d + lane_base + c, d0);
          tmem_ld_32x32b_x16(tmem_d + lane_base + TN + c, d1);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) sums[(c + j) * kF16SumPitch + m] = n_units > 1 ? __uint_as_float(d0[j]) + __uint_as_float(d1[j]) : __uint_as_float(d0[j]);
        }
        break;
      }
      const float bv = (p.bias && n_ok) ? gemm_load_bias<FMT>(p.bias, n) : 0.f;
      float* part = p.partial + ((size_t)tile * p.max_contrib + my_contrib) * (TN * kTileM);
#pragma unroll 1
      for (int c = 0; c < TN; c += 16) {
        uint32_t d[16];
        tmem_ld_32x32b_x16(tmem_d + lane_base + c, d);
        tmem_ld_wait();
        if (n_contrib == 1 && !p.defer) {
          if (n_ok) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int t = c + j;
              if (t < p.T) gemm_store<FMT>(p.y, (size_t)t * p.N + n, __uint_as_float(d[j]) + bv);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) part[(c + j) * kTileM + m] = __uint_as_float(d[j]);
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty);
      if (n_contrib > 1 && !p.defer) {
        // last-arriving contributor sums the slots in contributor order (deterministic); release / acquire through
        // thread 0's gpu-scope fences around the counter, ordered with the other threads by the named barrier
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (etid == 0) {
          __threadfence();
          const int prev = atomicAdd(&p.counters[tile], 1);
          s_is_last = prev == n_contrib - 1;
          if (s_is_last) {
            p.counters[tile] = 0;  // re-armed for the next launch (graph replay safe)
            __threadfence();
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (s_is_last) {
          const float* base = p.partial + (size_t)tile * p.max_contrib * (TN * kTileM);
          const int n_vec = min(p.T, TN) * (kTileM / 4);
          const bool vec_ok = (p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7) == 0;
          for (int idx0 = etid; idx0 < n_vec; idx0 += 256) {
            float4 acc[2];
            float4 ld[2][4];
#pragma unroll
            for (int e = 0; e < 2; ++e) acc[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int c0 = 0; c0 < n_contrib; c0 += 4) {
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int idx = idx0 + e * 128;
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                  ld[e][cc] = (idx < n_vec && c0 + cc < n_contrib)
                                  ? __ldcg(reinterpret_cast<const float4*>(&base[(size_t)(c0 + cc) * (TN * kTileM) + idx * 4]))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
                }
              }
#pragma unroll
              for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                  acc[e].x += ld[e][cc].x; acc[e].y += ld[e][cc].y; acc[e].z += ld[e][cc].z; acc[e].w += ld[e][cc].w;
                }
              }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int idx = idx0 + e * 128;
              const int tt = idx / (kTileM / 4), mm = (idx % (kTileM / 4)) * 4;
              const int nn = tile * kTileM + mm;
              if (idx < n_vec) {
                const float a4[4] = {acc[e].x, acc[e].y, acc[e].z, acc[e].w};
                if (FMT == 0 && vec_ok && nn + 3 < p.N) {
                  float b4[4] = {0.f, 0.f, 0.f, 0.f};
                  if (p.bias) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) b4[q] = gemm_load_bias<FMT>(p.bias, nn + q);
                  }
                  uint2 o;
                  o.x = pack_half2(a4[0] + b4[0], a4[1] + b4[1]);
                  o.y = pack_half2(a4[2] + b4[2], a4[3] + b4[3]);
                  *reinterpret_cast<uint2*>(&reinterpret_cast<__half*>(p.y)[(size_t)tt * p.N + nn]) = o;
                } else {
#pragma unroll
                  for (int q = 0; q < 4; ++q)
                    if (nn + q < p.N)
                      gemm_store<FMT>(p.y, (size_t)tt * p.N + nn + q, a4[q] + (p.bias ? gemm_load_bias<FMT>(p.bias, nn + q) : 0.f));
                }
              }
            }
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");  // s_is_last is reused by the next segment
      }
      i += seg_len;
      kb = 0;
      ++tile;
      ++seg;
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc<C::kTmemCols>(tmem_d);
  if (p.cluster) {
    pdl_wait();
    f16_cluster_sum<FMT>(p, reinterpret_cast<const float*>(smem), c_tile, c_rank);
  }
}

struct F16Plan {
  int TN, nkb, n_tiles_n, units_per_cta, n_ctas, max_contrib;
};

// CTAs of a cluster -> clusters that the chip holds at one CTA per SM (148 SMs in GPCs of unlike size: 15 clusters of eight, 22 of six, 26 of five, 33 of
// four, 45 of three, 74 of two).  More would be a second wave, which takes a launch twice as long.
static const int* f16_clusters() {
  static const struct Table {
    int n[9];
    Table() : n{0, 0, 74, 45, 33, 26, 22, 15, 15} {   // (plans made without a device)
      constexpr auto kernel = gemm_f16_kernel<64, 0>;
      constexpr int smem = GemmF16Cfg<64>::kSmemBytes;
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      b200_count_clusters(kernel, kGemmThreads, smem, n);
    }
  } table;
  return table.n;
}
// CTAs per feature tile: the most that one wave of clusters allows, of at least four k-blocks; 0: not two
static int f16_cluster(int64_t N, int64_t K, const int* clusters) {
  const int64_t tiles = (N + kTileM - 1) / kTileM, nkb = (K + kTileK - 1) / kTileK;
  for (int d = 8; d >= 2; --d)
    if (clusters[d] >= tiles && nkb / d >= 4) return d;
  return 0;
}

// a call of up to kF16MostT tokens: one token tile
static F16Plan plan_f16(int64_t T, int64_t N, int64_t K, int sms, bool defer = false) {
  F16Plan pl;
  pl.TN = T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : T <= 128 ? 128 : 256;
  pl.nkb = (int)((K + kTileK - 1) / kTileK);
  pl.n_tiles_n = (int)((N + kTileM - 1) / kTileM);
  const int total = pl.n_tiles_n * pl.nkb;
  const int ctas = total < sms ? total : sms;
  pl.units_per_cta = (total + ctas - 1) / ctas;
  if (pl.units_per_cta < 4 && pl.nkb >= 4) pl.units_per_cta = 4;
  // prefer the largest aligned cut nkb / d (d = 8, 4, 2, 1) that fits the SM count: a CTA that straddles two tiles pays two
  // fix-ups (measured on B200: 17.4 -> 14.4 us at 64 x 4096 x 4096, 47.7 -> 33.9 us at T = 256)
  if (!defer) {
    for (int d = 8; d >= 1; d >>= 1) {
      if (pl.nkb % d == 0 && (int64_t)pl.n_tiles_n * d <= sms && pl.nkb / d >= 4) { pl.units_per_cta = pl.nkb / d; break; }
    }
  }
  pl.n_ctas = (total + pl.units_per_cta - 1) / pl.units_per_cta;
  pl.max_contrib = (pl.nkb + pl.units_per_cta - 1) / pl.units_per_cta + 1;
  if (pl.units_per_cta % pl.nkb == 0) pl.max_contrib = 1;
  return pl;
}

// Microseconds of a call of 65 to 256 tokens without clusters (the note on kF16DecodeT): a 64-wide k-block of a 128-feature tile takes a CTA its own
// time or the memory's, whichever is longer, and the fix-up of a tile reads a partial of every contributor.
static float f16_stream_us(const F16Plan& pl, int64_t T) {
  const int contrib = pl.units_per_cta % pl.nkb == 0 ? 1 : pl.nkb % pl.units_per_cta == 0 ? pl.nkb / pl.units_per_cta : pl.max_contrib;
  const float straddle = pl.units_per_cta % pl.nkb == 0 || pl.nkb % pl.units_per_cta == 0 ? 1.f : 2.f;
  const float unit = pl.TN == 128 ? fmaxf(0.29f, 0.0026f * pl.n_ctas) : fmaxf(0.35f, 0.0031f * pl.n_ctas);
  return unit * pl.units_per_cta + straddle * (4.f + (float)T * (0.0125f * contrib + 0.035f));
}

// The same where clusters of d CTAs share a tile: its own k-blocks, at the rate of a CTA or, above 128 tokens, of the memory, and the end of a tile, which grows with the
// tokens whose sums go through shared memory.  The line to pair_plan's time is what is fitted, not the time itself (that is off by more than 10 % at 200 of 790 shapes, by 40 % at
// the widest): of 792 calls of 1024 .. 28672 -> 512 .. 9216 at 65 to 256 tokens what is taken is 0.1 % slower on average than the better of the two kernels, of the 360 larger ones
// under the power cap 0.5 %; 7 are 1 to 4 % slower than by the model without clusters.  (By that model, too many went to the pairs; us, so / now: 5632 -> 2048 at 65
// and 200 tokens 15.5 / 10.7, 16.1 / 15.2; 11008 -> 4096 at 200 35.0 / 26.8; 8192 -> 4096 at 128 22.7 / 17.7; 20480 -> 5120 at 65 51.7 / 38.1.  With up to 0.0025 us for each
// CTA below 129 tokens still too many, 5632 -> 9216 at 65 24.1 / 22.0; with 0.0031 above too few, 24576 -> 6144 at 224 87.6 / 83.4, under the power cap 16384 -> 9216 at 256 95.4 / 88.7.)
static float f16_cluster_us(int64_t T, int64_t N, int64_t K, int d) {
  const int64_t nkb = (K + kTileK - 1) / kTileK, ctas = (N + kTileM - 1) / kTileM * d;
  const float unit = T <= 128 ? 0.25f : fmaxf(0.385f, 0.0033f * ctas);
  return unit * ((nkb + d - 1) / d) + 5.1f + 0.0212f * T;
}

}  // namespace b200

using namespace b200;

// gemm_w4a16.cu; weak: a library built without the int4 kernels (libb200_seq.so) resolves them to null
__attribute__((weak)) int64_t b200_w4_partial_bytes(int64_t T, int64_t N, int64_t K);  // stream-K partials
__attribute__((weak)) void b200_w4_plan_debug(int64_t T, int64_t N, int64_t K, int sms, int32_t* out);

// tests (no GPU needed): the stream-K plan of one GEMM launch.  kind 0 = fp16 weights, 1 = int4.
// out[8] = {token tile, k-blocks per tile, feature tiles (int4: super-tiles), 1, units per CTA, CTAs,
//           contributor slots per tile in the workspace, feature tiles per unit (int4: 2)}
// Calls of more than 256 (int4: 128) tokens have no such plan (b200_debug_pair_plan).
extern "C" int b200_debug_gemm_plan(int kind, int64_t T, int64_t N, int64_t K, int sms, int32_t* out) {
  if (!out || T <= 0 || T > (kind == 1 ? kW4DecodeT : kF16MostT) || N <= 0 || K <= 0 || sms <= 0 || (kind != 0 && kind != 1)) {
    b200_set_last_error("debug_gemm_plan: bad arguments");
    return B200_ERR_ARG;
  }
  if (kind == 1) {
    if (!b200_w4_plan_debug) { b200_set_last_error("debug_gemm_plan: this library has no int4 kernels"); return B200_ERR_UNSUPPORTED; }
    b200_w4_plan_debug(T, N, K, sms, out);
    return B200_OK;
  }
  const F16Plan pl = plan_f16(T, N, K, sms);
  const int32_t v[8] = {pl.TN, pl.nkb, pl.n_tiles_n, 1, pl.units_per_cta, pl.n_ctas, pl.max_contrib, 1};
  for (int i = 0; i < 8; ++i) out[i] = v[i];
  return B200_OK;
}

// tests (no GPU needed): out[8] = {1 if a launch (with a workspace) takes the SM pairs, token tile, token tiles, feature tiles, SM pairs, k-blocks per
// stage, pieces of k, stages of a piece}.  kind 0 = fp16 weights (and bfloat16 with results of 16 bits), 1 = int4, 2 = bfloat16 with fp32 results
static bool f16_takes_pairs(int fmt, int64_t T, int64_t N, int64_t K, bool workspace, int sms, const int* clusters);
static int f16_pieces(int64_t T, int64_t N, int64_t K, int sms);
extern "C" int b200_debug_pair_plan(int kind, int64_t T, int64_t N, int64_t K, int sms, int32_t* out) {
  if (!out || T <= 0 || N <= 0 || K <= 0 || sms <= 1 || kind < 0 || kind > 2) {
    b200_set_last_error("debug_pair_plan: bad arguments");
    return B200_ERR_ARG;
  }
  const int64_t n_kb = kind == 1 ? 2 * ((K + 127) / 128) : (K + kPairK - 1) / kPairK;
  const PairPlan pl = pair_plan(T, N, n_kb, kind == 1, sms, kind == 1 ? 1 : f16_pieces(T, N, K, sms));
  const int taken = kind == 1 ? T > kW4DecodeT : f16_takes_pairs(kind == 2 ? 2 : 0, T, N, K, true, sms, T <= kF16DecodeT ? f16_clusters() : nullptr);
  const int32_t v[8] = {taken, pl.tn, pl.n_tt, pl.n_m, pl.n_pairs, pl.per_stage, pl.pieces, pl.piece_stages};
  for (int i = 0; i < 8; ++i) out[i] = v[i];
  return B200_OK;
}

// tests: whether an fp16 call of T tokens with a workspace goes to the SM pairs on a chip that holds clusters[d] clusters of d = 2 .. 8 CTAs
extern "C" int b200_debug_f16_on_pairs(int64_t T, int64_t N, int64_t K, int sms, const int32_t* clusters) {
  if (!clusters || T <= 0 || N <= 0 || K <= 0 || sms <= 1) {
    b200_set_last_error("debug_f16_on_pairs: bad arguments");
    return B200_ERR_ARG;
  }
  return f16_takes_pairs(0, T, N, K, true, sms, clusters) ? 1 : 0;
}

extern "C" int64_t b200_gemm_workspace_bytes(int64_t T, int64_t N, int64_t K) {
  if (T > kF16MostT) return kCounterBytes;
  const F16Plan pl = plan_f16(T, N, K, 148);
  int64_t f16 = pl.max_contrib > 1 ? (int64_t)pl.n_tiles_n * pl.max_contrib * pl.TN * kTileM * 4 : 0;
  // deferred reduction leaves a partial for every tile, even un-split ones
  const F16Plan pd = plan_f16(T, N, K, 148, true);
  const int64_t fd = (int64_t)pd.n_tiles_n * pd.max_contrib * pd.TN * kTileM * 4;
  if (fd > f16) f16 = fd;
  const int64_t w4 = b200_w4_partial_bytes ? b200_w4_partial_bytes(T, N, K) : 0;
  return kCounterBytes + (f16 > w4 ? f16 : w4);
}

// upper bound of b200_gemm_workspace_bytes over every T (stream-K only happens while there is a single token tile)
extern "C" int64_t b200_gemm_workspace_bytes_max(int64_t N, int64_t K) {
  int64_t best = kCounterBytes;
  for (int64_t T : {1, 16, 17, 32, 33, 64, 65, 128, 129, 256}) {
    const int64_t b = b200_gemm_workspace_bytes(T, N, K);
    if (b > best) best = b;
  }
  return best;
}

// whether a call's kernel is that of gemm_pair.cuh; clusters: as f16_cluster (NULL: none)
static bool f16_takes_pairs(int fmt, int64_t T, int64_t N, int64_t K, bool workspace, int sms, const int* clusters) {
  if (T <= kF16PairT || (fmt == 2 && T <= kF16MostT)) return false;
  if (T > kF16MostT || (!workspace && T > kF16DecodeT)) return true;
  const F16Plan pl = plan_f16(T, N, K, sms);
  if (T <= kF16DecodeT) {
    // Wide outputs: both stream the weights at the memory's rate, the pairs without fix-ups; but the pairs' last wave has to be a full one, and over
    // three waves and more the fix-ups no longer show (4096 -> 128256 at 64 tokens 168 us, 96 % of the memory's rate).
    const int64_t n_m = (N + kPairM - 1) / kPairM, pairs = sms / 2, waves = (n_m + pairs - 1) / pairs;
    return (!clusters || f16_cluster(N, K, clusters) == 0) && workspace && waves <= 2 && (waves == 1 || n_m * 5 >= waves * pairs * 4);
  }
  if ((int64_t)pl.n_tiles_n * 4 > kCounterBytes) return true;
  const int d = clusters ? f16_cluster(N, K, clusters) : 0;
  return pair_plan(T, N, pl.nkb, false, sms).us <= (d ? f16_cluster_us(T, N, K, d) : f16_stream_us(pl, T));
}
// pieces of k on the pairs: as many as this file's kernel cuts a call of its size into
static int f16_pieces(int64_t T, int64_t N, int64_t K, int sms) {
  if (T > kF16MostT) return 1;
  const F16Plan pl = plan_f16(T, N, K, sms);
  return (pl.nkb + pl.units_per_cta - 1) / pl.units_per_cta;
}

template <int TN, int FMT>
static int launch_gemm_f16(const CUtensorMap* mw, const CUtensorMap* mx, void* y, void* workspace, const void* bias, int T, int N,
                           const F16Plan& pl, int cluster, int held, int defer, cudaStream_t st) {
  using C = GemmF16Cfg<TN>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_f16_kernel<TN, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) { b200_set_last_error(cudaGetErrorString(e)); return B200_ERR_CUDA; }
    configured = true;
  }
  F16Params p;
  p.y = y;
  p.counters = (int*)workspace;
  p.partial = workspace ? (float*)((char*)workspace + kCounterBytes) : nullptr;
  p.bias = bias;
  p.T = T;
  p.N = N;
  p.nkb = pl.nkb;
  p.units_per_cta = pl.units_per_cta;
  p.total_units = pl.n_tiles_n * pl.nkb;
  p.max_contrib = pl.max_contrib;
  p.cluster = cluster;
  p.held = held;
  p.defer = defer;
  const dim3 grid(cluster ? pl.n_tiles_n * cluster : pl.n_ctas);
  b200_timing_mark(B200_TIME_GEMM_F16, 0, st);
  constexpr auto kernel = gemm_f16_kernel<TN, FMT>;
  const cudaError_t le = b200_launch_cluster(kernel, grid, dim3(kGemmThreads), (size_t)C::kSmemBytes, st, (unsigned)cluster, *mw, *mx, p);
  if (le != cudaSuccess) { b200_set_last_error(cudaGetErrorString(le)); return B200_ERR_CUDA; }
  b200_step_trace_stamp("gemm_f16_kernel", st);
  b200_timing_mark(B200_TIME_GEMM_F16, 1, st);
  b200_count_launches(1);
  return B200_OK;
}

// workspace: >= b200_gemm_workspace_bytes(T, N, K) bytes whose first 64 KiB (tile counters) were zeroed once by the
// caller, or NULL (every CTA then takes whole tiles: no stream-K).
// splitk != NULL: deferred reduction (see b200_gemm_w4a16_deferred): y is not written.
template <int FMT>
static int gemm_f16_impl(const void* x, const void* w, const void* bias, void* y, int64_t T, int64_t N, int64_t K, void* workspace,
                         B200SplitK* splitk, bool held, void* stream) {
  if (T == 0 || N == 0) return B200_OK;
  if (K % 8 != 0 || K < 64) { b200_set_last_error("gemm_f16: need K % 8 == 0 and K >= 64"); return B200_ERR_ARG; }
  const bool defer = splitk != nullptr;
  if (defer && (!workspace || T > 256 || N % 8 != 0)) {
    b200_set_last_error("gemm_f16_deferred: needs a workspace, T <= 256 (one token tile) and N % 8 == 0");
    return B200_ERR_UNSUPPORTED;
  }
  if (!defer && f16_takes_pairs(FMT, T, N, K, workspace != nullptr, b200_num_sms(), f16_clusters())) {
    PairParams pp = {};
    pp.y = y;
    pp.bias = bias;
    pp.T = (int)T;
    pp.N = pp.ldy = (int)N;
    pp.n_kb = (int)((K + kPairK - 1) / kPairK);
    return launch_gemm_pair<FMT>(x, w, K, pp, pair_plan(T, N, pp.n_kb, false, b200_num_sms(), f16_pieces(T, N, K, b200_num_sms())), B200_TIME_GEMM_F16, (cudaStream_t)stream);
  }
  F16Plan pl = plan_f16(T, N, K, b200_num_sms(), defer);
  if (!defer && pl.max_contrib > 1 && (!workspace || (int64_t)pl.n_tiles_n * 4 > kCounterBytes)) {
    pl.units_per_cta = pl.nkb;
    pl.n_ctas = pl.n_tiles_n;
    pl.max_contrib = 1;
  }
  const CUtensorMap* mw = get_tmap_2d(w, N, K, K, kTileM, kTileK, TmapDtype::kF16, TmapSwizzle::k128B);
  const CUtensorMap* mx = get_tmap_2d(x, T, K, K, pl.TN, kTileK, TmapDtype::kF16, TmapSwizzle::k128B);
  if (!mw || !mx) return B200_ERR_CUDA;
  if (defer) {
    splitk->partial = (const float*)((const char*)workspace + kCounterBytes);
    splitk->bias = bias;
    splitk->tiles_per_unit = 1;
    splitk->tn = pl.TN;
    splitk->nkb = pl.nkb;
    splitk->units_per_cta = pl.units_per_cta;
    splitk->max_contrib = pl.max_contrib;
    splitk->half_tiles = 0;
    splitk->N = (int32_t)N;
    splitk->T = (int32_t)T;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int df = defer ? 1 : 0;
  int cluster = defer ? 0 : f16_cluster(N, K, f16_clusters());
  // Few tokens leave partial sums of a few KB, and equal parts of a tile may be more CTAs than clusters allow (us, this kernel without / with clusters,
  // eight tokens: 5632 -> 2048 6.9 / 7.5, 4096 -> 4096 9.0 / 9.3, 2048 -> 2048 5.1 / 5.2; fewer CTAs, 2048 -> 2560 5.6 / 5.5, 20480 -> 5120 42.3 / 35.2).
  if (T <= 8 && workspace && pl.nkb % pl.units_per_cta == 0 && pl.n_ctas >= pl.n_tiles_n * cluster) cluster = 0;
  switch (pl.TN) {
    case 16: return launch_gemm_f16<16, FMT>(mw, mx, y, workspace, bias, (int)T, (int)N, pl, cluster, held, df, st);
    case 32: return launch_gemm_f16<32, FMT>(mw, mx, y, workspace, bias, (int)T, (int)N, pl, cluster, held, df, st);
    case 64: return launch_gemm_f16<64, FMT>(mw, mx, y, workspace, bias, (int)T, (int)N, pl, cluster, held, df, st);
    case 128: return launch_gemm_f16<128, FMT>(mw, mx, y, workspace, bias, (int)T, (int)N, pl, cluster, held, df, st);
    default: return launch_gemm_f16<256, FMT>(mw, mx, y, workspace, bias, (int)T, (int)N, pl, cluster, held, df, st);
  }
}
extern "C" int b200_gemm_f16(const void* x, const void* w, const void* bias, void* y, int64_t T, int64_t N, int64_t K,
                             void* workspace, void* stream) {
  return gemm_f16_impl<0>(x, w, bias, y, T, N, K, workspace, nullptr, false, stream);
}
extern "C" int b200_gemm_f16_held(const void* x, const void* w, const void* bias, void* y, int64_t T, int64_t N, int64_t K,
                                  void* workspace, void* stream) {
  return gemm_f16_impl<0>(x, w, bias, y, T, N, K, workspace, nullptr, true, stream);
}
// y [T, I] = SiLU(x Wg^T) * (x Wu^T) for w = [Wg; Wu] [2 I, K] (bias [2 I] or NULL), both factors rounded to fp16 first as b200_gemm_f16 and
// b200_silu_mul do, with the same sums.  Prompts only (T > 256: SM pairs, gemm_pair.cuh): the [T, 2 I] between the two does not go through memory.
// Measured on B200 (us, b200_gemm_f16 and b200_silu_mul / this, back to back): 2048 -> 2 x 5632 at 300 tokens 23.9 / 17.5, 1000 44.5 / 36.6,
// 4674 180 / 152 (the product alone 150); 4096 -> 2 x 11008 at 1000 146 / 131, 4674 703 / 629 (582).
extern "C" int b200_gemm_f16_silu(const void* x, const void* w, const void* bias, void* y, int64_t T, int64_t I, int64_t K, void* stream) {
  if (I == 0) return B200_OK;
  if (T <= kF16MostT || K % 8 != 0 || K < 64 || I % 8 != 0 || ((uintptr_t)y & 15)) {
    b200_set_last_error("gemm_f16_silu: need more than 256 tokens, K % 8 == 0, K >= 64, I % 8 == 0 and a 16-byte aligned y");
    return B200_ERR_UNSUPPORTED;
  }
  PairParams pp = {};
  pp.y = y;
  pp.bias = bias;
  pp.T = (int)T;
  pp.N = pp.ldy = pp.half = (int)I;
  pp.n_kb = (int)((K + kPairK - 1) / kPairK);
  return launch_gemm_pair<kPairF16Silu>(x, w, K, pp, pair_plan(T, 2 * ((I + 127) / 128 * 128), pp.n_kb, false, b200_num_sms()), B200_TIME_GEMM_F16, (cudaStream_t)stream);
}
// bfloat16 x [T, K] and w [N, K] (bias bfloat16 or NULL) -> y [T, N]; out_kind 0: bfloat16, 1: fp32, 2: bfloat16 after the square of
// ReLU.  Same kernel, workspace and rules as b200_gemm_f16.
extern "C" int b200_gemm_bf16(const void* x, const void* w, const void* bias, void* y, int out_kind, int64_t T, int64_t N, int64_t K,
                              void* workspace, void* stream) {
  if (out_kind == 2) return gemm_f16_impl<3>(x, w, bias, y, T, N, K, workspace, nullptr, false, stream);
  if (out_kind == 1) return gemm_f16_impl<2>(x, w, bias, y, T, N, K, workspace, nullptr, false, stream);
  return gemm_f16_impl<1>(x, w, bias, y, T, N, K, workspace, nullptr, false, stream);
}
extern "C" int b200_gemm_f16_deferred(const void* x, const void* w, const void* bias, int64_t T, int64_t N, int64_t K, void* workspace,
                                      B200SplitK* splitk, void* stream) {
  if (!splitk) { b200_set_last_error("gemm_f16_deferred: splitk is NULL"); return B200_ERR_ARG; }
  return gemm_f16_impl<0>(x, w, bias, nullptr, T, N, K, workspace, splitk, false, stream);
}
extern "C" int b200_gemm_f16_deferred_held(const void* x, const void* w, const void* bias, int64_t T, int64_t N, int64_t K, void* workspace,
                                           B200SplitK* splitk, void* stream) {
  if (!splitk) { b200_set_last_error("gemm_f16_deferred_held: splitk is NULL"); return B200_ERR_ARG; }
  return gemm_f16_impl<0>(x, w, bias, nullptr, T, N, K, workspace, splitk, true, stream);
}
