// GPTQ int4 linears of up to eight tokens and few k-blocks per SM: Y[T, N] = X[T, K] . dequant(Wq), the weights going from HBM through registers straight
// into the fragments of warp-level products (mma.sync m16n8k16: 16 features x 8 tokens x 16 k).  Such a call is mostly what surrounds the products: the
// kernel of gemm_w4a16.cu pays for tensor memory, hand-overs from warp to warp and partial sums that cross global memory (more than half of its 9 us at 4096 -> 6144).
//
// A cluster of `d` CTAs has one super-tile (256 features; the format's pair of feature tiles), each CTA a part of k: unit records as gemm_w4a16.cu describes
// them, read in place.  16 warps: warp w has the features 16 (w & 7) .. + 15 of both tiles and every other k-block.  Lane (g, t) = (lane / 4, lane % 4) reads
// the 16-byte piece of features g and g + 8 that holds k 32 t .. 32 t + 31 of the block; a word's eight weights are its part of two products.  Which k
// stand in which place of a product does not matter as long as the activations are placed alike: lane (g, t) has token g's 16 bytes at k 32 t + 8 j for word j.
// Activations of the CTA's whole part of k are copied to shared memory at the start, block by block behind barriers of their own; 32-k pieces lie 80 bytes
// apart, so that a fragment's load touches every bank once.  At the end the warps leave fp32 sums in shared memory and the cluster adds them, CTA r its
// share of the outputs over all 2 d sums in their order, through distributed shared memory.
// Measured on B200 at one token, 4096 -> 6144 (us): launch, first weights and activations 3.3, products 3.4 (de-quantisation: 13 instructions per 8 weights,
// eight of them at half rate), sums 0.9.  us in a replayed graph, gemm_w4a16_kernel / here, 1 and 8 tokens: 4096 -> 6144 8.8 / 8.1 and 8.8 / 8.4, 4096 -> 4096
// 7.25 / 6.8 and 7.3 / 7.4, 2048 -> 2560 5.8 / 4.2 and 5.8 / 4.9; 12 tokens in two tiles of eight: 4096 -> 6144 9.0 / 9.5.  Many k-blocks per CTA (4096 -> 28672:
// 18.3 / 20.4) stay there: its de-quantisation runs as fast, and what surrounds it counts less.
#pragma once
#include "common.cuh"
#include "w4_format.cuh"
#include "../../include/b200_tgis.h"

namespace b200 {

constexpr int kFewThreads = 512, kFewPiece = 80, kFewRow = 4 * kFewPiece;   // bytes of a 32-k piece and of a token's 128 k in shared memory
constexpr int kFewPitch = 260;   // floats of a token's 256 features in a partial sum
constexpr int kFewMostT = 8, kFewMostBlocks = 8;   // tokens; k-blocks of a CTA

struct W4FewParams {
  const __half* x;
  __half* y;
  const __half* bias;
  const unsigned char* packed;
  int T, N, K, nkb, rec_per_tile, half_tiles, act, ldy, x_blocks;   // x_blocks: k-blocks a CTA has at most
  unsigned* gave_up;   // b200_gave_up_word
};

constexpr int few_smem(int x_blocks) {   // activations, later the sums
  const int a = x_blocks * 8 * kFewRow, b = 2 * 8 * kFewPitch * 4;
  return a > b ? a : b;
}

__device__ __forceinline__ void few_ld(uint4& v, const unsigned char* p, uint64_t policy) {
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p), "l"(policy));
}

// kGR: meta rows per unit record
template <int kGR>
__global__ void __launch_bounds__(kFewThreads, 1) gemm_w4_few_kernel(const W4FewParams p) {
  extern __shared__ __align__(16) unsigned char xs[];
  float* sums = reinterpret_cast<float*>(xs);                    // [k-blocks' parity][token][kFewPitch]
  __shared__ uint64_t landed[kFewMostBlocks];                    // [k-block]: its activations
  constexpr int kRec = kW4WordBytes + kGR * kW4MetaRowBytes;
  pdl_launch_dependents();
  uint32_t rank, d;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(d));
  const int sup = blockIdx.x / d, warp = warp_id(), lane = lane_id(), g = lane >> 2, t = lane & 3, odd = warp >> 3, f0 = (warp & 7) * 16 + g;
  const int kb0 = (int)(rank * p.nkb / d), n = (int)((rank + 1) * p.nkb / d) - kb0;

  // the CTA's records are on their way to L2 while the kernel before ends (as fast as reading them ahead of it: 4096 -> 6144 at one token 8.0 and 8.0 us)
  if (threadIdx.x < n) tma_bulk_prefetch(p.packed + ((size_t)sup * p.rec_per_tile + kb0 + threadIdx.x) * 2 * kRec, 2 * kRec);
  struct Block {
    uint4 w[2][2];       // [tile][feature f0, f0 + 8]
    uint32_t meta[2][2];
  } blk[2];
  const uint64_t policy = policy_evict_first();
  const unsigned char* src = p.packed + ((size_t)sup * p.rec_per_tile + kb0 + odd) * 2 * kRec + t * (kW4TileM * 16) + f0 * 16;
  const unsigned char* msrc = src - t * (kW4TileM * 16) - f0 * 12 + kW4WordBytes + (t * kGR / 4) * kW4MetaRowBytes;
  int next = odd;
  auto fetch = [&](Block& b) {   // the warp's next k-block
    if (next < n) {
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          few_ld(b.w[r][e], src + r * kRec + e * 128, policy);
          b.meta[r][e] = __ldg(reinterpret_cast<const uint32_t*>(msrc + r * kRec + e * 32));
        }
    }
    next += 2;
    src += 4 * kRec;
    msrc += 4 * kRec;
  };
  if (threadIdx.x < n) mbar_init(&landed[threadIdx.x], kFewThreads);
  mbar_fence_init();
  __syncthreads();
  pdl_wait();
  fetch(blk[0]);
  fetch(blk[1]);
  for (int i = 0; i < n; ++i) {
    if (threadIdx.x < p.T * 16) {   // 16-byte pieces of the block; what lies behind K is zero
      const int tok = threadIdx.x >> 4, o = threadIdx.x & 15, k = (kb0 + i) * kW4BlockK + o * 8;
      cp_async_16(xs + (i * 8 + tok) * kFewRow + (o >> 2) * kFewPiece + (o & 3) * 16, p.x + (size_t)tok * p.K + (k < p.K ? k : 0), k < p.K);
    }
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&landed[i])) : "memory");
  }

  float acc[2][4] = {};
  bool ok = true;
  auto use = [&](const Block& b, int i) {
    const uint32_t xa = smem_u32(xs) + (i * 8 + g) * kFewRow + t * kFewPiece;
    uint32_t c[2][2][3];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) dequant_consts(b.meta[r][e], c[r][e][0], c[r][e][1], c[r][e][2]);
    mbar_wait_soft(&landed[i], 0, ok);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t a[2][2][4];   // [tile][product][register]
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t lo[4], hi[4];
        const uint32_t wl = j == 0 ? b.w[r][0].x : j == 1 ? b.w[r][0].y : j == 2 ? b.w[r][0].z : b.w[r][0].w;
        const uint32_t wh = j == 0 ? b.w[r][1].x : j == 1 ? b.w[r][1].y : j == 2 ? b.w[r][1].z : b.w[r][1].w;
        dequant_word(wl, c[r][0][1], c[r][0][2], c[r][0][0], lo);
        dequant_word(wh, c[r][1][1], c[r][1][2], c[r][1][0], hi);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          a[r][q][0] = lo[2 * q];
          a[r][q][1] = hi[2 * q];
          a[r][q][2] = lo[2 * q + 1];
          a[r][q][3] = hi[2 * q + 1];
        }
      }
      uint32_t x[4];
      lds_v4(xa + j * 16, x);
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int r = 0; r < 2; ++r) mma_m16n8k16_f16f32(acc[r], a[r][q], x[2 * q], x[2 * q + 1]);
    }
  };
  for (int i = odd; i < n; i += 4) {
    use(blk[0], i);
    fetch(blk[0]);
    if (i + 2 < n) {
      use(blk[1], i + 2);
      fetch(blk[1]);
    }
  }

  // sums: lane (g, t) has features f0 and f0 + 8 of tokens 2 t and 2 t + 1
  __syncthreads();   // the activations are used up (and all copies have landed: each was waited for by somebody)
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int e = 0; e < 4; ++e) sums[(odd * 8 + 2 * t + (e & 1)) * kFewPitch + r * 128 + f0 + (e >> 1) * 8] = acc[r][e];
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const uint32_t base = smem_u32(sums);
  auto total = [&](int tok, int f) {   // four features, both parities of every CTA in order
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t c = 0; c < d; c += 4) {
      float4 v[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int o = 0; o < 2; ++o)
          v[i][o] = c + i < d ? ld_cluster_v4(base + ((o * 8 + tok) * kFewPitch + f) * 4, c + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          s.x += v[i][o].x;
          s.y += v[i][o].y;
          s.z += v[i][o].z;
          s.w += v[i][o].w;
        }
    }
    return s;
  };
  auto add_bias = [&](float4& s, int col) {
    if (!p.bias) return;
    s.x += __half2float(p.bias[col]);
    s.y += __half2float(p.bias[col + 1]);
    s.z += __half2float(p.bias[col + 2]);
    s.w += __half2float(p.bias[col + 3]);
  };
  const int per_tok = p.act ? 32 : 64, items = p.T * per_tok, share = (items + (int)d - 1) / (int)d, hi = min(items, ((int)rank + 1) * share);
  for (int i = (int)rank * share + (int)threadIdx.x; i < hi; i += kFewThreads) {
    const int tok = i / per_tok, f = (i % per_tok) * 4, r = f >> 7, m = f & 127;
    float4 s = total(tok, f);
    if (p.act) {   // SiLU(gate) * up: an output needs both tiles
      float4 u = total(tok, f + 128);
      const int col = sup * kW4TileM + f;
      add_bias(s, col);
      add_bias(u, col + p.half_tiles * kW4TileM);
      const __half o[4] = {silu_mul_f16(s.x, u.x), silu_mul_f16(s.y, u.y), silu_mul_f16(s.z, u.z), silu_mul_f16(s.w, u.w)};
      *reinterpret_cast<uint2*>(&p.y[(size_t)tok * p.ldy + col]) = *reinterpret_cast<const uint2*>(o);
    } else {
      const int col = (p.half_tiles ? sup + r * p.half_tiles : sup * 2 + r) * kW4TileM + m;
      if (col < p.N) {   // N % 32 == 0: four columns never straddle it
        add_bias(s, col);
        *reinterpret_cast<uint2*>(&p.y[(size_t)tok * p.ldy + col]) = make_uint2(pack_half2(s.x, s.y), pack_half2(s.z, s.w));
      }
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // nobody leaves while its sums are read
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (!ok) gave_up(p.gave_up);
}

// CTAs of a cluster -> clusters that the chip holds at one CTA per SM (GPCs of 16 to 20 SMs leave some over).  A second wave would double the launch.
static const int* few_clusters() {
  static const struct Table {
    int n[9];
    Table() : n{} {
      n[0] = n[1] = b200_num_sms();
      b200_count_clusters(gemm_w4_few_kernel<1>, kFewThreads, few_smem(kFewMostBlocks), n);
    }
  } table;
  return table.n;
}

// d == 0: the call does not go this way
struct W4FewPlan {
  int d, blocks;   // CTAs of a cluster, k-blocks of a CTA at most
};
static W4FewPlan few_plan(int64_t N, int64_t K, const int* clusters) {
  W4FewPlan pl = {0, 0};
  const int64_t n_super = (N + 2 * kW4TileM - 1) / (2 * kW4TileM), nkb = (K + kW4BlockK - 1) / kW4BlockK;
  int d = 8;
  while (d > 0 && (d > nkb || clusters[d] < n_super)) --d;
  if (d == 0) return pl;
  pl.blocks = (int)((nkb + d - 1) / d);
  if (pl.blocks <= kFewMostBlocks) pl.d = d;
  return pl;
}

template <int kGR>
static int launch_w4_few(const W4FewParams& p, int n_super, int d, cudaStream_t st) {
  b200_timing_mark(B200_TIME_GEMM_W4A16, 0, st);
  const cudaError_t e = b200_launch_cluster(gemm_w4_few_kernel<kGR>, dim3((unsigned)(n_super * d)), dim3(kFewThreads), (size_t)few_smem(p.x_blocks), st, (unsigned)d, p);
  if (e != cudaSuccess) { b200_set_last_error(cudaGetErrorString(e)); return B200_ERR_CUDA; }
  b200_step_trace_stamp("gemm_w4_few_kernel", st);
  b200_timing_mark(B200_TIME_GEMM_W4A16, 1, st);
  b200_count_launches(1);
  return B200_OK;
}

static int launch_w4_few_plan(const W4FewParams& p, int gr, int n_super, const W4FewPlan& pl, cudaStream_t st) {
  return gr == 1 ? launch_w4_few<1>(p, n_super, pl.d, st) : gr == 2 ? launch_w4_few<2>(p, n_super, pl.d, st) : launch_w4_few<4>(p, n_super, pl.d, st);
}

}  // namespace b200
