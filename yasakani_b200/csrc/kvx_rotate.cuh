// The sign-Hadamard-256 rotation of Family B (kvx_rotate, src/kvx_codec.cuh:35-49) on rows held in registers: eight lanes per row, or a warp.
#pragma once
#include "kv4_common.cuh"

namespace kv4 {
namespace {

// Bit 0 of the reference's 32-bit multiply-xorshift hash of d + 1: set = the element's sign is flipped.
__host__ __device__ constexpr uint32_t kvx_sign_bit(int d) {
  uint32_t x = (uint32_t)d + 1u;
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x & 1u;
}
struct SignTable { uint32_t w[8]; };                       // 256 sign bits, bit d of the table = kvx_sign_bit(d)
constexpr SignTable make_signs() {
  SignTable t{};
  for (int d = 0; d < 256; ++d) t.w[d >> 5] |= kvx_sign_bit(d) << (d & 31);
  return t;
}
__constant__ SignTable c_signs = make_signs();
// Element layout of a row over 8 lanes: lane ll (0..7) holds v[4k + e] = element d = 32k + 4ll + e (k 0..7, e 0..3), so every
// load and store instruction of the 8 lanes covers one contiguous run of the row.  A warp holds 4 rows (lanes 8s .. 8s+7).
// Multiplying by +-1 is a sign-bit flip (exact, also for zeros and infinities).
__device__ __forceinline__ void apply_signs(float (&v)[32], int ll) {
  #pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t bits = c_signs.w[k] >> (4 * ll);
    #pragma unroll
    for (int e = 0; e < 4; ++e) v[4 * k + e] = __uint_as_float(__float_as_uint(v[4 * k + e]) ^ (((bits >> e) & 1u) << 31));
  }
}

// Butterflies + 1/16 in the reference's stage order h = 1, 2, ... 128.  Bits 0-1 of d are register bits (e), bits 2-4 the lane
// within the row (shuffles), bits 5-7 register bits again (k).  Lower index: a + b; upper: lower - upper.
__device__ __forceinline__ void hadamard256(float (&v)[32], int ll) {
  #pragma unroll
  for (int rb = 1; rb < 4; rb *= 2) {                      // h = 1, 2
    #pragma unroll
    for (int i = 0; i < 32; ++i)
      if (!(i & rb)) { const float lo = v[i], up = v[i + rb]; v[i] = __fadd_rn(lo, up); v[i + rb] = __fsub_rn(lo, up); }
  }
  #pragma unroll
  for (int m = 1; m < 8; m *= 2) {                         // h = 4, 8, 16
    const uint32_t flip = (ll & m) ? 0x80000000u : 0u;     // upper lane: other - self = other + (-self), exactly
    #pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float self = v[i], other = __shfl_xor_sync(0xffffffffu, self, m);
      v[i] = __fadd_rn(other, __uint_as_float(__float_as_uint(self) ^ flip));
    }
  }
  #pragma unroll
  for (int rb = 4; rb < 32; rb *= 2) {                     // h = 32, 64, 128
    #pragma unroll
    for (int i = 0; i < 32; ++i)
      if (!(i & rb)) { const float lo = v[i], up = v[i + rb]; v[i] = __fadd_rn(lo, up); v[i + rb] = __fsub_rn(lo, up); }
  }
  #pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __fmul_rn(v[i], 0.0625f);
}

// The same with a warp per row: lane l holds v[e] = element 4l + e and v[4 + e] = element 128 + 4l + e (e 0..3).  Sign bits of those eight: bit e of w[0] and w[1].
struct LaneSigns { uint32_t w[2]; };
__device__ __forceinline__ LaneSigns lane_signs(int lane) {
  return {{c_signs.w[lane >> 3] >> (4 * (lane & 7)), c_signs.w[4 + (lane >> 3)] >> (4 * (lane & 7))}};
}
// Stages h = 1, 2 in the registers, 4 ... 64 over the lanes, 128 in the registers, then each element times its factor(element's index in v).
template <class F> __device__ __forceinline__ void hadamard256_warp(float (&v)[8], int lane, F factor) {
  #pragma unroll
  for (int rb = 1; rb < 4; rb *= 2)
    #pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & rb)) { const float lo = v[i], up = v[i + rb]; v[i] = __fadd_rn(lo, up); v[i + rb] = __fsub_rn(lo, up); }
  #pragma unroll
  for (int m = 1; m < 32; m *= 2) {
    const float flip = (lane & m) ? -1.f : 1.f;            // the product is exact: one rounding, as of the sum
    #pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = fmaf(v[i], flip, __shfl_xor_sync(0xffffffffu, v[i], m));
  }
  #pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float lo = v[i], up = v[i + 4];
    v[i] = __fmul_rn(__fadd_rn(lo, up), factor(i)); v[i + 4] = __fmul_rn(__fsub_rn(lo, up), factor(i + 4));
  }
}

}  // namespace
}  // namespace kv4
