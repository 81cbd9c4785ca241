// Unit records of a packed GPTQ int4 weight and the arithmetic that turns their words into fp16 weights (gemm_w4a16.cu describes the
// format; the decode kernel there and the prompt kernel of gemm_pair.cuh read it).
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int kW4DecodeT = 128;  // calls of up to so many tokens stay with gemm_w4a16.cu's kernel
constexpr int kW4TileM = 128;
constexpr int kW4BlockK = 128;
constexpr int kW4WordBytes = (kW4BlockK / 8) * kW4TileM * 4;  // 8192
constexpr int kW4MetaRowBytes = kW4TileM * 4;                 // 512
constexpr int kW4MaxGroupRows = 4;                            // groupsize >= 32
constexpr int kW4RecMaxBytes = kW4WordBytes + kW4MaxGroupRows * kW4MetaRowBytes;  // 10240 = shared-memory stage stride

__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(b), "r"(c));  // (a & b) | c
  return r;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void lds_v4(uint32_t addr, uint32_t* v) {
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t hadd2_u(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t hmul2_u(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// one packed word (8 weights along k) -> 4 half2 (k, k+1) pairs, each fp16(scale * (q - zero)):
//   low nibbles:  0x6400 | q      = 1024 + q   (ulp 1);     + (-(1024 + zero)) is exact
//   high nibbles: 0x5400 | q << 4 = 64 + q     (ulp 1/16);  + (-(64 + zero))   is exact
// then one rounding in the multiplication by the scale, as in fp16(scale * (q - zero)).
__device__ __forceinline__ void dequant_word(uint32_t w, uint32_t nz1024, uint32_t nz64, uint32_t scale2, uint32_t* out) {
  const uint32_t w8 = w >> 8;
  const uint32_t q0 = lop3_and_or(w, 0x000f000fu, 0x64006400u);   // (k0, k1)
  const uint32_t q1 = lop3_and_or(w, 0x00f000f0u, 0x54005400u);   // (k2, k3)
  const uint32_t q2 = lop3_and_or(w8, 0x000f000fu, 0x64006400u);  // (k4, k5)
  const uint32_t q3 = lop3_and_or(w8, 0x00f000f0u, 0x54005400u);  // (k6, k7)
  out[0] = hmul2_u(hadd2_u(q0, nz1024), scale2);
  out[1] = hmul2_u(hadd2_u(q1, nz64), scale2);
  out[2] = hmul2_u(hadd2_u(q2, nz1024), scale2);
  out[3] = hmul2_u(hadd2_u(q3, nz64), scale2);
}
// meta word (fp16 scale | (zero + 1) << 16) -> the three half2 constants of dequant_word
__device__ __forceinline__ void dequant_consts(uint32_t rec, uint32_t& scale2, uint32_t& nz1024, uint32_t& nz64) {
  scale2 = prmt(rec, rec, 0x1010);             // fp16 scale in both halves
  const uint32_t z2 = prmt(rec, rec, 0x3232);  // zero + 1 (1..16) in both halves
  nz1024 = 0xE400E400u + z2;                   // -(1024 + zero), exact
  nz64 = 0xD400D400u + (z2 << 4);              // -(64 + zero), exact
}

// fp16(fp16(silu(fp16 g)) * fp16 u) from the two fp32 accumulators: exactly what the separate linear (fp16 output) followed
// by silu_mul_kernel (elementwise.cu; torch fp16 SiLU = fp32 x / (1 + exp(-x)), one rounding, then an fp16 multiply) gives
__device__ __forceinline__ __half silu_mul_f16(float gate_acc, float up_acc) {
  const float g = __half2float(__float2half_rn(gate_acc));
  const __half a = __float2half_rn(silu_of_half(g));
  return __hmul(a, __float2half_rn(up_acc));
}

}  // namespace b200
