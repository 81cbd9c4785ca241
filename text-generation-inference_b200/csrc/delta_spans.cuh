// Gated delta rule over prompts, sixteen tokens (a span) at a time: what a span's tokens do to one another is solved once per (span, head), ahead of
// the memory and in parallel over the whole step; what is left in order is one pass over the memory per span.  With G_j = g_1 .. g_j (products per
// key channel over the span, never a quotient) and
//   A_ji = k_j^T (g_(i+1) .. g_j) k_i  (i < j),   B_ji = q_j^T (g_(i+1) .. g_j) k_i  (i <= j),   M = (I + diag(beta) A)^-1 diag(beta)
//   W = M (G_j k_j)_j,   Q = (G_j q_j)_j - B W,   U = M V,   Y = B U
// the memory S [dk, dv] that the span finds gives
//   u = U - W S,   y = Y + Q S,   S <- G_16 S + sum_i (g_(i+1) .. g_16 k_i) u_i^T.
// For unit keys and beta <= 1 row j of W is no longer than beta_j, so nothing grows on the way.  All of it is fp32.
//
//   delta_span_prepare_kernel  two warps per (span, head): the 256 sums A and B over key channels, M by forward substitution; leaves one record per
//                              (span, head) as the scan wants it in shared memory, U behind it, Y in the place of the results
//   delta_span_scan_kernel     a block per (sequence, head, 32 value columns), a warp per 8 of them, the memory in registers, records by bulk copies a
//                              span ahead
// What bounds it: fp32 products - 3 dk per token and value column, in packed pairs, two cycles of a scheduler each - and about as much the registers that shared
// memory fills (128 bytes a cycle: a loaded value meets four columns), and, on small grids, the latency of a warp's span.  A chain over four tokens
// (delta_chunk_kernel) leaves the units idle for two thirds of the time: its blocks meet twice per sixteen tokens, and four dependent sums over lanes stand
// between a token and the next.
#pragma once
#include "seq_common.cuh"

#include <utility>

namespace b200 {
namespace seq {

constexpr int kSpan = 16, kSpanCols = 32, kSpanPitch = 20;   // tokens; value columns of a block; row pitch of 16 x 16 matrices in floats
constexpr int kSpanPrepHeads = 2;                             // of a block of delta_span_prepare_kernel

// a record in floats: W, Q, decayed k_i: [pair of tokens][pair of channels][token of the pair][channel of the pair], then G_16; U [token][dv] follows
template <int DK>
struct SpanRecord {
  static constexpr int kW = 0, kQ = kSpan * DK, kD = 2 * kSpan * DK, kG = 3 * kSpan * DK, kFloats = kG + DK;
  static_assert(kFloats % 4 == 0, "bulk copies");
};
__host__ __device__ constexpr int span_record_floats(int dk, int dv) { return 3 * kSpan * dk + dk + kSpan * dv; }

// The spans of a step count from its first sequence on; a pair of launches covers those numbered from .. from + cap - 1.
__device__ __forceinline__ int spans_of(const int32_t* cu_q, int b) { return (cu_q[b + 1] - cu_q[b] + kSpan - 1) / kSpan; }

__device__ __forceinline__ uint64_t span_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t span_mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t span_pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 span_split(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// lane l is left with the sum over lanes of v[l]
__device__ __forceinline__ float fold32(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = upper ? v[i] : v[i + o], keep = upper ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// y = L x for a lower triangular L in shared memory; what stands behind a token does not reach it, finite or not
__device__ __forceinline__ void span_lower(const float (&Lm)[kSpan][kSpanPitch], const float (&x)[kSpan], float (&y)[kSpan]) {
#pragma unroll
  for (int j = 0; j < kSpan; ++j) {
#pragma unroll
    for (int i = 0; i <= j; i += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&Lm[j][i]);
      y[j] = i == 0 ? f.x * x[0] : fmaf(f.x, x[i], y[j]);
      if (i + 1 <= j) y[j] = fmaf(f.y, x[i + 1], y[j]);
      if (i + 2 <= j) y[j] = fmaf(f.z, x[i + 2], y[j]);
      if (i + 3 <= j) y[j] = fmaf(f.w, x[i + 3], y[j]);
    }
  }
}

// Two warps per (span, head).  Sums run over key channels: a lane adds the channels lane + 32 c, then 32 sums at a time are folded over the lanes.  Decays are
// products along four tokens and over whole fours, so that a sum of tokens j and i takes one product per channel: (k_j from its four's start) (fours between)
// (k_i to its four's end); pairs within four tokens are multiplied out.  Inputs are copied to shared memory first, all at once; loops stay loops, for the
// instruction cache (4 x 256 - 768 tokens, 16 heads: 56 us, 64 with all
// 256 sums in one run of instructions; what is left is latency at twelve warps an SM).  width and *_col: row width of `pre` and its columns of
// keys, values, decays and write strengths (queries: column 0).
template <int DK>
struct SpanPrep {
  // floats: q, k, g (then within every four tokens decayed from their start: q, k; to their end: k), the fours' whole decays; A, then M; B
  static constexpr int kIn = 3 * kSpan * DK + 4 * DK, kMat = kSpan * kSpanPitch, kHead = kIn + 2 * kMat, kBytes = kSpanPrepHeads * kHead * 4;
};
template <int DK>
__global__ void __launch_bounds__(kSpanPrepHeads * 64, 3) delta_span_prepare_kernel(const float* __restrict__ pre, int width, int k_col, int v_col, int g_col, int b_col,
                                                                                    const int32_t* __restrict__ cu_q, int B, int from, int H, int group, int channels,
                                                                                    int dv, float* __restrict__ out, float* __restrict__ y, int64_t ld_y) {
  using R = SpanRecord<DK>;
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  const int lane = lane_id(), part = warp_id() & 1, slot = warp_id() >> 1, h = blockIdx.y * kSpanPrepHeads + slot;
  // which sequence's which span
  int b = -1, tile = from + blockIdx.x;
  for (int b0 = 0; b0 < B && b < 0; b0 += 32) {
    const int nt = b0 + lane < B ? spans_of(cu_q, b0 + lane) : 0;
    int upto = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, tile < upto);
    if (hit) {
      const int at = __ffs(hit) - 1;
      b = b0 + at;
      tile -= __shfl_sync(0xffffffffu, upto - nt, at);
    } else {
      tile -= __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  if (b >= 0 && h < H) {
    auto sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(slot + 1) : "memory"); };   // the two warps
    const int t0 = cu_q[b] + tile * kSpan, n_tok = min(kSpan, cu_q[b + 1] - t0);
    const float* row = pre + (int64_t)t0 * width;
    float* rec = out + ((int64_t)blockIdx.x * H + h) * span_record_floats(DK, dv);
    float* in = sm + slot * SpanPrep<DK>::kHead;
    float(&A)[kSpan][kSpanPitch] = *reinterpret_cast<float(*)[kSpan][kSpanPitch]>(in + SpanPrep<DK>::kIn);
    float(&Bm)[kSpan][kSpanPitch] = *reinterpret_cast<float(*)[kSpan][kSpanPitch]>(in + SpanPrep<DK>::kIn + SpanPrep<DK>::kMat);
    // a token that the step does not have changes nothing: k = q = 0, g = 1
    for (int i = part * 32 + lane; i < 3 * kSpan * DK / 4; i += 64) {
      const int what = i / (kSpan * DK / 4), j = (i / (DK / 4)) % kSpan, c = (i % (DK / 4)) * 4;
      float* dst = in + (what * kSpan + j) * DK + c;
      const float* src = row + (int64_t)j * width + (what == 2 ? g_col + (channels ? h * DK + c : h) : what * k_col + (h / group) * DK + c);
      if (j < n_tok && (what < 2 || channels)) {
        cp_async_16(dst, src, true);
      } else {
        const float none = what < 2 ? 0.f : (j < n_tok ? *src : 1.f);
        *reinterpret_cast<float4*>(dst) = make_float4(none, none, none, none);
      }
    }
    cp_async_commit();
    const float strength = lane < n_tok ? row[(int64_t)lane * width + b_col + h] : 0.f;   // of token `lane`
    float *qs = in + lane, *ks = qs + kSpan * DK, *gs = ks + kSpan * DK, *fours = gs + kSpan * DK;
    const int odd = lane & 1, at = (lane >> 1) * 4 + odd * 2;
    auto put = [&](int plane, int tp, int c, float first, float second) {   // a channel's values of tokens 2 tp and 2 tp + 1, by lane pairs
      const float got = __shfl_xor_sync(0xffffffffu, odd ? first : second, 1);
      *reinterpret_cast<float2*>(rec + plane + tp * DK * 2 + c * 2 + at) = odd ? make_float2(got, second) : make_float2(first, got);
    };
    cp_async_wait<0>();
    sync();
    {   // two fours each
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
#pragma unroll 1
      for (int c = 0; c < DK; c += 32) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int at = (part * 2 + e) * 4 * DK + c;
          float k[4], q[4], g[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            k[j] = ks[at + j * DK];
            q[j] = qs[at + j * DK];
            g[j] = gs[at + j * DK];
          }
          float t[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int i = 0; i < j; ++i) t[i] *= g[j];
            t[j] = k[j];
#pragma unroll
            for (int i = 0; i < j; ++i) v[e * 16 + j * (j - 1) / 2 + i] = fmaf(k[j], t[i], v[e * 16 + j * (j - 1) / 2 + i]);
#pragma unroll
            for (int i = 0; i <= j; ++i) v[e * 16 + 6 + j * (j + 1) / 2 + i] = fmaf(q[j], t[i], v[e * 16 + 6 + j * (j + 1) / 2 + i]);
          }
          float G = 1.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            G *= g[j];
            ks[at + j * DK] = k[j] * G;
            qs[at + j * DK] = q[j] * G;
            gs[at + j * DK] = t[j];
          }
          fours[(part * 2 + e) * DK + c] = G;
        }
      }
      const float sum = fold32(v, lane);
      const int e = lane & 15, f = e - 6;
      const int j = e < 6 ? (e < 1 ? 1 : e < 3 ? 2 : 3) : (f < 1 ? 0 : f < 3 ? 1 : f < 6 ? 2 : 3), four = (part * 2 + (lane >> 4)) * 4;
      if (e < 6) A[four + j][four + e - j * (j - 1) / 2] = sum;
      else Bm[four + j][four + f - j * (j + 1) / 2] = sum;
    }
    sync();
#pragma unroll 1
    for (int m = 0; m < 3; ++m) {   // pairs of fours: 1 0, 2 1, 3 0 / 3 2, 2 0, 3 1
      const int J = part == 0 ? m + 1 : (m == 1 ? 2 : 3), I = part == 0 ? (m == 1 ? 1 : 0) : (m == 0 ? 2 : m - 1);
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
#pragma unroll 1
      for (int c = 0; c < DK; c += 32) {
        float between = 1.f, t[4];
        for (int f = I + 1; f < J; ++f) between *= fours[f * DK + c];
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = between * gs[(I * 4 + i) * DK + c];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float k = ks[(J * 4 + j) * DK + c], q = qs[(J * 4 + j) * DK + c];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            v[j * 4 + i] = fmaf(k, t[i], v[j * 4 + i]);
            v[16 + j * 4 + i] = fmaf(q, t[i], v[16 + j * 4 + i]);
          }
        }
      }
      const float sum = fold32(v, lane);
      (lane < 16 ? A : Bm)[J * 4 + ((lane >> 2) & 3)][I * 4 + (lane & 3)] = sum;
    }
    sync();
    {
      float x[kSpan];   // column `lane` of M (lanes 16 .. 31: nothing)
#pragma unroll
      for (int j = 0; j < kSpan; ++j) {
        float s0 = j == lane ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
        for (int i = 0; i < j; i += 2) {
          s0 = fmaf(-A[j][i], x[i], s0);
          if (i + 1 < j) s1 = fmaf(-A[j][i + 1], x[i + 1], s1);
        }
        const float beta = __shfl_sync(0xffffffffu, strength, j);
        x[j] = j < lane ? 0.f : beta * (s0 + s1);
      }
      sync();
      if (part == 0 && lane < kSpan)
#pragma unroll
        for (int j = 0; j < kSpan; ++j) A[j][lane] = x[j];
      sync();
    }
    // (below M and B are read anew for every channel and column: 272 registers of them would spill)
#pragma unroll 1
    for (int c = 32 * part; c < DK; c += 64) {
      float kg[kSpan], wv[kSpan], bw[kSpan], G = 1.f, behind = 1.f;
#pragma unroll
      for (int j = 0; j < kSpan; ++j) {
        kg[j] = G * ks[j * DK + c];
        if (j % 4 == 3) G *= fours[j / 4 * DK + c];
      }
      rec[R::kG + c + lane] = G;
      __syncwarp();
      span_lower(A, kg, wv);
      __syncwarp();
      span_lower(Bm, wv, bw);
      G = 1.f;
#pragma unroll
      for (int tp = 0; tp < kSpan / 2; ++tp) {
        put(R::kW, tp, c, wv[2 * tp], wv[2 * tp + 1]);
        put(R::kQ, tp, c, G * qs[2 * tp * DK + c] - bw[2 * tp], G * qs[(2 * tp + 1) * DK + c] - bw[2 * tp + 1]);
        if (tp % 2 == 1) G *= fours[tp / 2 * DK + c];
      }
#pragma unroll
      for (int tp = kSpan / 2 - 1; tp >= 0; --tp) {
        put(R::kD, tp, c, behind * gs[2 * tp * DK + c], behind * gs[(2 * tp + 1) * DK + c]);
        if (tp % 2 == 0) behind *= fours[tp / 2 * DK + c];
      }
    }
#pragma unroll 1
    for (int c = 32 * part; c < dv; c += 64) {
      float vv[kSpan], u[kSpan], yy[kSpan];
#pragma unroll
      for (int j = 0; j < kSpan; ++j) vv[j] = j < n_tok ? row[(int64_t)j * width + v_col + h * dv + c + lane] : 0.f;
      __syncwarp();
      span_lower(A, vv, u);
      __syncwarp();
      span_lower(Bm, u, yy);
#pragma unroll
      for (int j = 0; j < kSpan; ++j) {
        rec[R::kFloats + j * dv + c + lane] = u[j];
        if (j < n_tok) y[(int64_t)(t0 + j) * ld_y + h * dv + c + lane] = yy[j];
      }
    }
  }
  pdl_launch_dependents();   // only now: the scan's few long blocks shall find every SM empty, not crowd where the first of these have ended
}

template <int DK>
struct SpanScan {
  static constexpr int kWarps = kSpanCols / 8, kStage = SpanRecord<DK>::kFloats, kU = 2 * kStage, kUWarp = kSpan * 32, kBytes = (kU + kWarps * kUWarp) * 4;
};

// A lane holds the channels 32 i + 2 rl, + 1 (rl = lane & 15) of four columns, packed by channel pairs; entry x is column c0 + (x ^ perm), so that a sum over
// lanes always keeps the lower half of what it has.  After the folds a lane has the token lane & 3 of every four, of column c0 + perm.  (Eight columns a
// lane load a third less from shared memory, but leave half as many warps, each with twice as long a span: 143 -> 197 us, 4 x 256 - 768 tokens, 16 heads;
// the chain over four tokens took 257.)
template <int DK>
__global__ void __launch_bounds__(SpanScan<DK>::kWarps * 32, 3) delta_span_scan_kernel(const float* __restrict__ rec, float* __restrict__ S_state,
                                                                                       const int32_t* __restrict__ state_slots, const int32_t* __restrict__ cu_q,
                                                                                       const int64_t* __restrict__ position_ids, float* __restrict__ y, int64_t ld_y,
                                                                                       int from, int cap, int B, int H, int dv, unsigned* gave_up_word) {
  using R = SpanRecord<DK>;
  using L = SpanScan<DK>;
  constexpr int NP = DK / 32;   // pairs of channels
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  __shared__ uint64_t full[2];
  const int lane = lane_id(), w = warp_id(), rl = lane & 15, half = lane >> 4, perm = (lane >> 2) & 3, jq = lane & 3;
  const int parts = dv / kSpanCols, rest = (int)(blockIdx.x % (H * parts)), h = rest / parts;
  // blocks start in the order of their numbers: the longest sequences first, so that short ones fill what is left (up to 32 of them; more even out by themselves)
  int b = blockIdx.x / (H * parts);
  if (B <= 32) {
    const int nt = lane < B ? spans_of(cu_q, lane) : 0;
    int upto = nt, rank = 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    // spans inside the part; of as many, tokens decide
    const int inside = max(0, min(upto, from + cap) - max(upto - nt, from));
    const int mine = lane < B ? inside * kSpan - (inside > 0 && upto <= from + cap ? nt * kSpan - (cu_q[lane + 1] - cu_q[lane]) : 0) : -1;
    for (int i = 0; i < B; ++i) {
      const int other = __shfl_sync(0xffffffffu, mine, i);
      rank += other > mine || (other == mine && i < lane);
    }
    b = __ffs(__ballot_sync(0xffffffffu, lane < B && rank == b)) - 1;
  }
  int first = 0;   // spans of the sequences ahead
  for (int i = lane; i < b; i += 32) first += spans_of(cu_q, i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
  const int lo = max(0, from - first), spans = min(spans_of(cu_q, b), from + cap - first) - lo;   // the sequence's spans inside the part
  if (spans <= 0) return;
  const int t_begin = cu_q[b] + lo * kSpan, n_all = min(cu_q[b + 1] - t_begin, spans * kSpan), v0 = (rest % parts) * kSpanCols;
  const bool fresh = lo == 0 && position_ids[t_begin] == 0;
  const int64_t step = (int64_t)H * span_record_floats(DK, dv);
  const float* src = rec + ((int64_t)(first + lo - from) * H + h) * span_record_floats(DK, dv);
  if (threadIdx.x == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  auto load = [&](int s) {
    mbar_arrive_expect_tx(&full[s & 1], R::kFloats * 4);
    tma_bulk_g2s(sm + (s & 1) * L::kStage, src + s * step, R::kFloats * 4, &full[s & 1]);
  };
  if (threadIdx.x == 0) load(0);
  const int cw = (w * 2 + half) * 4;                            // a lane's columns
  float* Sp = S_state + (((int64_t)state_slots[b] * H + h) * DK + 2 * rl) * dv + v0 + cw;
  const float* up = src + R::kFloats + jq * dv + v0 + cw + perm;
  float* yp = y + (int64_t)(t_begin + jq) * ld_y + h * dv + v0 + cw + perm;
  float* Us = sm + L::kU + w * L::kUWarp + half * 16;           // [token][half][perm][entry]: u as the update wants it
  uint64_t S[NP][4];
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    float a[4] = {0.f, 0.f, 0.f, 0.f}, c[4] = {0.f, 0.f, 0.f, 0.f};
    if (!fresh) {
      permute4(*reinterpret_cast<const float4*>(Sp + (int64_t)(32 * i) * dv), perm & 1, perm & 2, a);
      permute4(*reinterpret_cast<const float4*>(Sp + (int64_t)(32 * i + 1) * dv), perm & 1, perm & 2, c);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) S[i][x] = span_pair(a[x], c[x]);
  }
  bool ok = true;
  float u[4], o[4];   // the span's U and Y, then u and y
  auto ahead = [&](int s) {
#pragma unroll
    for (int qd = 0; qd < 4; ++qd) {
      const bool live = s * kSpan + qd * 4 + jq < n_all;
      u[qd] = live ? up[s * step + qd * 4 * dv] : 0.f;
      o[qd] = live ? yp[(int64_t)(s * kSpan + qd * 4) * ld_y] : 0.f;
    }
  };
  ahead(0);

  // four tokens' products of one kind with the memory: this lane's token and column of them
  auto meet = [&](const float* vec, int qd) {
    uint64_t P[4][4];   // [column][token]
#pragma unroll
    for (int i = 0; i < NP; ++i) {
#pragma unroll
      for (int tp = 0; tp < 2; ++tp) {
        const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(vec + (qd * 2 + tp) * DK * 2 + 64 * i);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          P[c][2 * tp] = i == 0 ? span_mul2(k.x, S[i][c]) : span_fma2(k.x, S[i][c], P[c][2 * tp]);
          P[c][2 * tp + 1] = i == 0 ? span_mul2(k.y, S[i][c]) : span_fma2(k.y, S[i][c], P[c][2 * tp + 1]);
        }
      }
    }
    float p[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float2 a = span_split(P[e >> 2][e & 3]);
      p[e] = a.x + a.y;
    }
    fold<16>(p, 8);
    fold<8>(p, 4);
    halve<4>(p, 2, lane & 2);
    halve<2>(p, 1, lane & 1);
    return p[0];
  };
  auto span = [&](const float* st, int s, auto n_fours) {
    constexpr int Q = decltype(n_fours)::value;   // groups of four tokens
    const float* vec = st + rl * 4;
#pragma unroll
    for (int qd = 0; qd < Q; ++qd) u[qd] -= meet(vec + R::kW, qd);
#pragma unroll
    for (int qd = 0; qd < Q; ++qd)
#pragma unroll
      for (int e = 0; e < 4; ++e)   // for the lanes whose order is e: this column is their entry perm ^ e
        Us[(qd * 4 + jq) * 32 + e * 4 + (perm ^ e)] = u[qd];
#pragma unroll
    for (int qd = 0; qd < Q; ++qd) o[qd] += meet(vec + R::kQ, qd);
#pragma unroll
    for (int qd = 0; qd < Q; ++qd)
      if (s * kSpan + qd * 4 + jq < n_all) yp[(int64_t)(s * kSpan + qd * 4) * ld_y] = o[qd];
    ahead(s + 1);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const uint64_t G = *reinterpret_cast<const uint64_t*>(st + R::kG + 2 * rl + 32 * i);
#pragma unroll
      for (int c = 0; c < 4; ++c) S[i][c] = span_mul2(G, S[i][c]);
    }
#pragma unroll
    for (int tp = 0; tp < 2 * Q; ++tp) {
      const float4 ua = *reinterpret_cast<const float4*>(Us + (tp * 2) * 32 + perm * 4), ub = *reinterpret_cast<const float4*>(Us + (tp * 2 + 1) * 32 + perm * 4);
      const uint64_t a[4] = {span_pair(ua.x, ua.x), span_pair(ua.y, ua.y), span_pair(ua.z, ua.z), span_pair(ua.w, ua.w)};
      const uint64_t c[4] = {span_pair(ub.x, ub.x), span_pair(ub.y, ub.y), span_pair(ub.z, ub.z), span_pair(ub.w, ub.w)};
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(vec + R::kD + tp * DK * 2 + 64 * i);
#pragma unroll
        for (int e = 0; e < 4; ++e) S[i][e] = span_fma2(d.y, c[e], span_fma2(d.x, a[e], S[i][e]));
      }
    }
    __syncwarp();
  };
  for (int s = 0; s < spans; ++s) {
    if (s > 0) {   // the other stage is used up
      fence_proxy_async_smem();
      __syncthreads();
    }
    if (threadIdx.x == 0 && s + 1 < spans) load(s + 1);
    const float* st = sm + (s & 1) * L::kStage;
    mbar_wait_soft(&full[s & 1], (s >> 1) & 1, ok);
    const int n = n_all - s * kSpan;
    if (n > kSpan - 4) span(st, s, std::integral_constant<int, 4>{});
    else if (n > 4) span(st, s, std::integral_constant<int, 3>{});
    else span(st, s, std::integral_constant<int, 1>{});
  }
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    float2 f[4];
    float a[4], c[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) f[x] = span_split(S[i][x]);
    permute4(make_float4(f[0].x, f[1].x, f[2].x, f[3].x), perm & 1, perm & 2, a);
    permute4(make_float4(f[0].y, f[1].y, f[2].y, f[3].y), perm & 1, perm & 2, c);
    *reinterpret_cast<float4*>(Sp + (int64_t)(32 * i) * dv) = make_float4(a[0], a[1], a[2], a[3]);
    *reinterpret_cast<float4*>(Sp + (int64_t)(32 * i + 1) * dv) = make_float4(c[0], c[1], c[2], c[3]);
  }
  if (!ok) gave_up(gave_up_word);
}

}  // namespace seq
}  // namespace b200
