// Family-B cache codec, step 2 (sm_100a): trellis ("CDQ") re-quantisation of 256-value KV rows and their packed payload.
//
// Arithmetic and formats are the reference's, bit for bit: tb_fakequant (src/kvq_gpu.cuh:54-148) = tbf_pre / tbf_chain /
// tbf_sel (src/kvq_fast.cuh:96-232), blob fields "KVQP v1" (src/kvq_gpu.cuh:57-68, src/engine35.cpp:50-53).
//   row -> (- mean) -> up to two low-rank projections (fp16 coefficients) -> rms
//   for each of nm scale multipliers: s = fp16(rms * mult); x_i = clamp(rint(r / s * 256), +-2048); for each of the 4 chains
//   of 64 values a Viterbi search over 256 states (an 8-bit shift register that takes kk = 3 / 4 / 5 new bits per step;
//   cost (x_i - code[state])^2); the multiplier with the smallest squared error wins (first on ties)
//   payload: the kk new bits of every step, MSB first, 8*kk 32-bit words per row; side words: scale, two fp16 coefficients.
// Sums over a row follow the reference's order (a xor-butterfly over each run of 32 values, then the eight run sums in
// order), and every product that feeds a rounding decision is an explicit _rn operation, so no FMA contraction moves a bit.
#include "kv4_common.cuh"
#include <cstring>

namespace kv4 {
namespace {

__device__ __forceinline__ unsigned tb_u16(const uint8_t* p) { return (unsigned)p[0] | ((unsigned)p[1] << 8); }
__device__ __forceinline__ unsigned tb_u32(const uint8_t* p) { return tb_u16(p) | (tb_u16(p + 2) << 16); }
__device__ __forceinline__ float tb_f32(const uint8_t* p) { return __uint_as_float(tb_u32(p)); }
__device__ __forceinline__ float tb_f16r(float v) { return __half2float(__float2half_rn(v)); }

struct TbGroup { int ok, mode, kk, tix, guard, m, has_mu; unsigned go, off_m, off_t; };
__device__ __forceinline__ TbGroup tb_group(const uint8_t* b, int g) {
  TbGroup P;
  P.off_m = tb_u32(b + 32); P.off_t = tb_u32(b + 36);
  const unsigned off_g = tb_u32(b + 40), ngrp = tb_u32(b + 28);
  P.ok = (unsigned)g < ngrp;
  P.go = P.ok ? tb_u32(b + off_g + 4u * (unsigned)g) : 0u;
  P.mode = P.ok ? b[P.go] : 0; P.kk = P.ok ? b[P.go + 1] : 4; P.tix = P.ok ? b[P.go + 2] : 0; P.guard = P.ok ? b[P.go + 3] : 0;
  P.m = P.ok ? b[P.go + 4] : 0; P.has_mu = P.ok ? b[P.go + 5] : 0;
  return P;
}

// ---- encoder: one block of four warps per row, one warp per chain of 64 values.
//
// A step of the search takes new(d) = min over the 2^KK predecessors {j * UU + u}, u = d >> KK, of old(p), plus (x - code[d])^2: every
// state is a candidate of one group u only, so 256 candidates and 256 costs a step.  What bounds it is instruction issue
// (integer), so the whole step stays in registers: a lane holds eight states, four values of j for two values of u,
//   p = jhi << (SH+2) | jlo << SH | umid << 1 | ulo,     registers e = (jlo, ulo), lane = (jhi, umid)     (SH = 8 - KK, UU = 2^SH)
// the minimum over jlo is in the lane (one fused add-minimum per state), the first exchange over jhi halves the lane's two
// values of u (each lane of the pair keeps one), the other exchanges are plain; the new states of a lane need 4 (KK = 3, 4) or
// 1 (KK = 5) of the UU minima, one shuffle each: 6 / 7 / 4 shuffles and about 35 instructions a step, no shared memory on the path and no barrier.
// x^2 is left out of the costs: it adds the same number to every state of a step.  A cost travels as a key, cost << 5 | j, whose j is part
// of the state's own constant: the minimum over keys is the minimum cost with the first j on ties (the reference's rule,
// src/kvq_gpu.cuh:101-102) and carries its back pointer, one byte per group and step.
// Width of the keys: |f| = |c^2 - 2xc| <= F = C^2 + 4096 C with C = max |code| and |x| <= 2048, and f differs by at most D = 8192 C between
// two states; any state is reached from any other in three steps, so the costs of a step spread over at most 3 D.  They are
// brought back to one of them every four steps: |cost| <= 3 D + 4 F < 2^26 for C <= 1400, and a key fits 32 bits.  Profiles with larger codes
// take 64-bit keys (the same code, no bringing back).
// 4,096 rows, 5 multipliers, on a B200: 1,335 us (one warp per (row, multiplier, chain), costs in shared memory, every lane walking its
// group's predecessors; a second kernel for choice and packing) -> 448 (minima kept instead of back pointers, candidates recomputed on
// the way back: 76 instructions a step) -> 321 (55 a step; issue slots 77 % busy, integer ALU 65 %, the
// multiply pipe 53 %).
constexpr int TB_NM = 16;                                // multipliers at most (the blob's limit)
struct TbRowSmem {
  uint8_t bp[4][64 * 32];                                // back pointers of each chain: [t][u], the low five bits
  short code[256]; float red[8]; int cmax[4]; uint8_t fld[256];
  struct Mult { uint8_t st[256]; float err[8]; } mult[1];  // one per multiplier: its states and its error sums
  static size_t bytes(int nm) { return sizeof(TbRowSmem) + (nm - 1) * sizeof(Mult); }
};
struct TbP { const uint8_t* blob; int nm; const float* x; const int* grp; const int* pos; int rows; float* y; uint8_t* pay; int pay_stride; uint32_t* side; };

__device__ __forceinline__ int tb_addmin(int a, int b, int c) { return __viaddmin_s32(a, b, c); }
__device__ __forceinline__ long long tb_addmin(long long a, long long b, long long c) { return min(a + b, c); }

// States of the best path of this warp's chain for the scaled values xa (steps 0-31, a lane each) and xb (steps 32-63): returned
// as (state of step lane, state of step lane + 32).  K = int or long long, the type of the keys.
template <int KK, class K> __device__ __forceinline__ int2 tb_search(uint8_t* bp, const short* code, int xa, int xb, int lane) {
  constexpr int SH = 8 - KK, UU = 1 << SH, NQ = KK == 5 ? 1 : 4;
  constexpr bool NARROW = sizeof(K) == 4;
  const int umid = lane & ((1 << (SH - 1)) - 1), jhi = lane >> (SH - 1);
  K m2c[8], c2[8];
  int src[NQ];
  #pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int p = (jhi << (SH + 2)) | ((e >> 1) << SH) | (umid << 1) | (e & 1), c = code[p];
    m2c[e] = (K)(-2 * c) * 32; c2[e] = (K)c * c * 32 + (p >> SH);
  }
  #pragma unroll
  for (int q = 0; q < NQ; ++q) {                         // the lane that holds the minimum of group (new state >> KK)
    const int g = ((jhi << (SH + 2)) | (q << SH) | (umid << 1)) >> KK;
    src[q] = ((g & 1) << (SH - 1)) | (g >> 1);
  }
  const bool upper = (lane >> (SH - 1)) & 1;             // of a pair of lanes the upper one keeps the odd u
  const int my_u = (umid << 1) | (upper ? 1 : 0);
  // Only state 0 exists at first.  Every state is reachable after three steps, so the others have to stay behind by more than 6 F
  // (5e7 for C = 1400) until then, and within the width of a key.
  K keep = my_u == 0 ? (K)(-(1 << 25)) * 32 : (K)(NARROW ? (1 << 24) + (1 << 23) : 0x40000000) * 32;
  uint8_t* mine = bp + (lane < UU ? my_u : 0);           // lanes below UU hold every u once (the jhi bits above the first are zero)
  auto costs = [&](int x, K (&t)[8], K (&m)[NQ]) {
    keep &= ~(K)31;
    #pragma unroll
    for (int q = 0; q < NQ; ++q) m[q] = __shfl_sync(0xffffffffu, keep, src[q]);
    #pragma unroll
    for (int e = 0; e < 8; ++e) t[e] = x * m2c[e] + c2[e];
  };
  auto step = [&](int x, int t) {                        // the minima of step t + 1 from those of step t
    K ct[8], m[NQ];
    costs(x, ct, m);
    K a = ct[0] + m[0], b = ct[1] + m[0];
    #pragma unroll
    for (int q = 1; q < 4; ++q) {
      a = tb_addmin(ct[2 * q], m[NQ == 1 ? 0 : q], a);
      b = tb_addmin(ct[2 * q + 1], m[NQ == 1 ? 0 : q], b);
    }
    const K other = __shfl_xor_sync(0xffffffffu, upper ? a : b, 1 << (SH - 1));
    keep = min(upper ? b : a, other);
    #pragma unroll
    for (int k = SH; k < 5; ++k) keep = min(keep, __shfl_xor_sync(0xffffffffu, keep, 1 << k));
    if (lane < UU) mine[(t + 1) * UU] = (uint8_t)keep;
  };
  #pragma unroll 1
  for (int t = 0; t < 60; t += 4) {
    const int xs = t < 32 ? xa : xb;
    #pragma unroll
    for (int i = 0; i < 4; ++i) step(__shfl_sync(0xffffffffu, xs, (t + i) & 31), t + i);
    if (NARROW) keep -= __shfl_sync(0xffffffffu, keep, 0) & ~(K)31;
  }
  #pragma unroll
  for (int t = 60; t < 63; ++t) step(__shfl_sync(0xffffffffu, xb, t - 32), t);
  // best final state: smallest (cost, state)
  K ct[8], m[NQ];
  costs(__shfl_sync(0xffffffffu, xb, 31), ct, m);
  K best = 0; int bs = 0;
  #pragma unroll
  for (int e = 0; e < 8; ++e) {                          // a lane's states grow with jlo, then ulo
    const K c = (ct[e] + m[NQ == 1 ? 0 : e >> 1]) & ~(K)31;
    if (e == 0 || c < best) { best = c; bs = (jhi << (SH + 2)) | ((e >> 1) << SH) | (umid << 1) | (e & 1); }
  }
  #pragma unroll
  for (int o = 16; o; o >>= 1) {
    const K c = __shfl_xor_sync(0xffffffffu, best, o); const int b2 = __shfl_xor_sync(0xffffffffu, bs, o);
    if (c < best || (c == best && b2 < bs)) { best = c; bs = b2; }
  }
  __syncwarp();                                          // the back pointers are complete
  int2 out = make_int2(0, 0);
  int st = bs;
  #pragma unroll 1
  for (int half = 1; half >= 0; --half) {
    int keep_st = 0;
    #pragma unroll 8
    for (int i = 31; i >= 0; --i) {
      if (lane == i) keep_st = st;
      const int u = st >> KK;
      st = ((bp[(32 * half + i) * UU + u] & 31) << SH) | u;      // (the row of step 0 is read but never used)
    }
    if (half) out.y = keep_st; else out.x = keep_st;
  }
  __syncwarp();                                          // they may be overwritten
  return out;
}

__global__ void __launch_bounds__(128, 7) tb_encode_kernel(TbP A) {
  extern __shared__ __align__(16) unsigned char tbe_smem[];
  TbRowSmem& S = *reinterpret_cast<TbRowSmem*>(tbe_smem);
  const int row = blockIdx.x, c = threadIdx.x >> 5, lane = threadIdx.x & 31, d0 = 64 * c + lane, d1 = d0 + 32;     // this thread's two values
  const uint8_t* b = A.blob;
  const TbGroup P = tb_group(b, A.grp[row]);
  const int words = A.pay_stride / 4;
  unsigned* pay = A.pay ? reinterpret_cast<unsigned*>(A.pay + (size_t)row * A.pay_stride) : nullptr;
  float ra = A.x[(size_t)row * 256 + d0], rb = A.x[(size_t)row * 256 + d1];
  if (!P.ok || A.pos[row] < P.guard) {                   // stored as it is: the payload and the side words are zero
    if (A.y) { A.y[(size_t)row * 256 + d0] = ra; A.y[(size_t)row * 256 + d1] = rb; }
    if (pay) for (int w = threadIdx.x; w < words; w += 128) pay[w] = 0u;
    if (A.side && threadIdx.x < 2) A.side[2 * row + threadIdx.x] = 0u;
    return;
  }
  // the reference's row sum: a xor-butterfly over each run of 32 values, then the eight runs in order (src/kvq_fast.cuh:33-43)
  auto runs = [&](float va, float vb, float* out) {
    #pragma unroll
    for (int o = 16; o; o >>= 1) { va += __shfl_xor_sync(0xffffffffu, va, o); vb += __shfl_xor_sync(0xffffffffu, vb, o); }
    if (lane == 0) { out[2 * c] = va; out[2 * c + 1] = vb; }
  };
  auto rowsum = [&](float va, float vb) -> float {
    runs(va, vb, S.red);
    __syncthreads();
    float t = 0.f;
    #pragma unroll
    for (int w = 0; w < 8; ++w) t = __fadd_rn(t, S.red[w]);
    __syncthreads();
    return t;
  };
  const uint8_t* mup = b + P.go + 8;
  const uint8_t* Up = mup + (P.has_mu ? 512 : 0);
  auto f16at = [&](const uint8_t* p, int d) { return __half2float(__ushort_as_half((unsigned short)tb_u16(p + 2 * d))); };
  float mua = 0.f, mub = 0.f, u0a = 0.f, u0b = 0.f, u1a = 0.f, u1b = 0.f, c0 = 0.f, c1 = 0.f;
  if (P.has_mu) { mua = f16at(mup, d0); mub = f16at(mup, d1); ra = __fsub_rn(ra, mua); rb = __fsub_rn(rb, mub); }
  if (P.m > 0) {
    u0a = f16at(Up, d0); u0b = f16at(Up, d1);
    c0 = tb_f16r(rowsum(__fmul_rn(ra, u0a), __fmul_rn(rb, u0b)));
    ra = __fsub_rn(ra, __fmul_rn(c0, u0a)); rb = __fsub_rn(rb, __fmul_rn(c0, u0b));
  }
  if (P.m > 1) {
    u1a = f16at(Up + 512, d0); u1b = f16at(Up + 512, d1);
    c1 = tb_f16r(rowsum(__fmul_rn(ra, u1a), __fmul_rn(rb, u1b)));
    ra = __fsub_rn(ra, __fmul_rn(c1, u1a)); rb = __fsub_rn(rb, __fmul_rn(c1, u1b));
  }
  float xqa, xqb, psc; int fa, fb, kb;
  if (P.mode == 1) {                                     // flat 4-bit codes (src/kvq_fast.cuh:193-198)
    float am = fmaxf(fabsf(ra), fabsf(rb));
    #pragma unroll
    for (int o = 16; o; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if (lane == 0) S.red[c] = am;
    __syncthreads();
    am = fmaxf(fmaxf(S.red[0], S.red[1]), fmaxf(S.red[2], S.red[3]));
    float s7 = __fdiv_rn(am, 7.f); if (s7 == 0.f) s7 = 1.f;
    const float qa = fminf(fmaxf(rintf(__fdiv_rn(ra, s7)), -7.f), 7.f), qb = fminf(fmaxf(rintf(__fdiv_rn(rb, s7)), -7.f), 7.f);
    xqa = __fmul_rn(qa, s7); xqb = __fmul_rn(qb, s7); fa = (int)qa + 8; fb = (int)qb + 8; psc = s7; kb = 4;
  } else {
    const unsigned to = tb_u32(b + P.off_t + 4u * (unsigned)P.tix);
    const float gain = tb_f32(b + to + 4);
    int cm = 0;
    for (int i = threadIdx.x; i < 256; i += 128) { const int v = (short)tb_u16(b + to + 12 + 2 * i); S.code[i] = (short)v; cm = max(cm, abs(v)); }
    cm = __reduce_max_sync(0xffffffffu, cm);
    if (lane == 0) S.cmax[c] = cm;
    float rms = __fsqrt_rn(__fdiv_rn(rowsum(__fmul_rn(ra, ra), __fmul_rn(rb, rb)), 256.f));     // its barriers also publish the codes
    if (rms == 0.f) rms = 1.f;
    const bool narrow = max(max(S.cmax[0], S.cmax[1]), max(S.cmax[2], S.cmax[3])) <= 1400;
    auto scale = [&](int mi) { const float s = tb_f16r(__fmul_rn(rms, tb_f32(b + P.off_m + 4u * (unsigned)mi))); return s == 0.f ? 1.f : s; };
    auto value = [&](int st, float s) { return __fmul_rn(__fmul_rn(__fmul_rn((float)(int)S.code[st], 0.00390625f), gain), s); };
    #pragma unroll 1
    for (int mi = 0; mi < A.nm; ++mi) {
      const float s = scale(mi);
      const int xa = (int)fminf(fmaxf(rintf(__fmul_rn(__fdiv_rn(ra, s), 256.f)), -2048.f), 2048.f);
      const int xb = (int)fminf(fmaxf(rintf(__fmul_rn(__fdiv_rn(rb, s), 256.f)), -2048.f), 2048.f);
      int2 st = make_int2(0, 0);
      if (P.kk == 3) st = narrow ? tb_search<3, int>(S.bp[c], S.code, xa, xb, lane) : tb_search<3, long long>(S.bp[c], S.code, xa, xb, lane);
      else if (P.kk == 4) st = narrow ? tb_search<4, int>(S.bp[c], S.code, xa, xb, lane) : tb_search<4, long long>(S.bp[c], S.code, xa, xb, lane);
      else if (P.kk == 5) st = narrow ? tb_search<5, int>(S.bp[c], S.code, xa, xb, lane) : tb_search<5, long long>(S.bp[c], S.code, xa, xb, lane);
      const float da = __fsub_rn(ra, value(st.x, s)), db = __fsub_rn(rb, value(st.y, s));
      runs(__fmul_rn(da, da), __fmul_rn(db, db), S.mult[mi].err);
      S.mult[mi].st[d0] = (uint8_t)st.x; S.mult[mi].st[d1] = (uint8_t)st.y;
    }
    __syncthreads();
    float best_e = 0.f; int best = 0;
    for (int mi = 0; mi < A.nm; ++mi) {                  // the smallest squared error, the first on ties
      float e = 0.f;
      #pragma unroll
      for (int w = 0; w < 8; ++w) e = __fadd_rn(e, S.mult[mi].err[w]);
      if (mi == 0 || e < best_e) { best_e = e; best = mi; }
    }
    const float s = scale(best);
    const int sa = S.mult[best].st[d0], sb = S.mult[best].st[d1];
    xqa = value(sa, s); xqb = value(sb, s);
    fa = sa & ((1 << P.kk) - 1); fb = sb & ((1 << P.kk) - 1); psc = s; kb = P.kk;
  }
  if (A.y) {
    if (P.m > 0) { xqa = __fadd_rn(xqa, __fmul_rn(c0, u0a)); xqb = __fadd_rn(xqb, __fmul_rn(c0, u0b)); }
    if (P.m > 1) { xqa = __fadd_rn(xqa, __fmul_rn(c1, u1a)); xqb = __fadd_rn(xqb, __fmul_rn(c1, u1b)); }
    if (P.has_mu) { xqa = __fadd_rn(xqa, mua); xqb = __fadd_rn(xqb, mub); }
    A.y[(size_t)row * 256 + d0] = xqa; A.y[(size_t)row * 256 + d1] = xqb;
  }
  if (pay) {
    S.fld[d0] = (uint8_t)fa; S.fld[d1] = (uint8_t)fb;
    __syncthreads();
    for (int w = threadIdx.x; w < words; w += 128) {     // MSB-first bit stream, 32 bits per word (src/kvq_fast.cuh:228-232)
      unsigned v = 0u;
      if (w < 8 * kb) {
        const int e0 = 32 * w / kb;                      // the field that holds the word's first bit
        for (int e = e0; e * kb < 32 * w + 32; ++e) {
          const int sh = 32 - (e + 1) * kb + 32 * w;     // where the field's last bit sits in the word; negative: it runs into the next word
          v |= sh >= 0 ? (unsigned)S.fld[e] << sh : (unsigned)S.fld[e] >> -sh;
        }
      }
      pay[w] = v;
    }
    if (A.side && threadIdx.x == 0) {
      A.side[2 * row] = __float_as_uint(psc);
      A.side[2 * row + 1] = (unsigned)__half_as_ushort(__float2half_rn(c0)) | ((unsigned)__half_as_ushort(__float2half_rn(c1)) << 16);
    }
  }
}

// Packed rows back to values (the reference's tba_unpack_kernel, src/kvq_attn.cuh:39-72): one warp per row.  The state of a
// value is the 8-bit window of the row's bit stream that ends with its field (shorter at the start of a chain of 64), so
// every value decodes on its own: two payload words from the warp's shared-memory copy of the row, one funnel shift, one
// code lookup.  Lane owns values 32*w + lane, so the stores of a warp are contiguous.
struct TbDecP { const uint8_t* blob; const int* grp; const int* pos; const uint8_t* pay; int pay_stride; const uint32_t* side; const float* yin; float* y; int rows; };
__global__ void __launch_bounds__(256) tb_unpack_kernel(TbDecP A) {
  __shared__ unsigned s_w[8][44];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x * 8 + warp;
  if (row >= A.rows) return;
  const uint8_t* b = A.blob;
  const TbGroup P = tb_group(b, A.grp[row]);
  const bool packed = P.ok && A.pos[row] >= P.guard && P.mode <= 1;
  if (!packed) {
    #pragma unroll
    for (int w = 0; w < 8; ++w) A.y[(size_t)row * 256 + 32 * w + lane] = A.yin ? A.yin[(size_t)row * 256 + 32 * w + lane] : 0.f;
    return;
  }
  const int kb = P.mode == 1 ? 4 : P.kk, nw = 8 * kb;
  const unsigned* wp = reinterpret_cast<const unsigned*>(A.pay + (size_t)row * A.pay_stride);
  for (int i = lane; i < 44; i += 32) s_w[warp][i] = i < nw ? wp[i] : 0u;
  __syncwarp();
  const float s = __uint_as_float(A.side[2 * (size_t)row]);
  const unsigned pc = A.side[2 * (size_t)row + 1];
  const unsigned to = tb_u32(b + P.off_t + 4u * (unsigned)P.tix);
  const float gain = P.mode == 0 ? tb_f32(b + to + 4) : 1.f;
  const uint8_t* mup = b + P.go + 8;
  const uint8_t* Up = mup + (P.has_mu ? 512 : 0);
  const float c0 = __half2float(__ushort_as_half((unsigned short)(pc & 0xffffu))), c1 = __half2float(__ushort_as_half((unsigned short)(pc >> 16)));
  #pragma unroll
  for (int w = 0; w < 8; ++w) {
    const int d = 32 * w + lane, endb = kb * (d + 1), first = kb * (d & ~63);
    const int lo = P.mode == 1 ? endb - 4 : max(endb - 8, first), len = endb - lo;
    const unsigned hiw = s_w[warp][lo >> 5], low = s_w[warp][(lo >> 5) + 1];
    const unsigned v = __funnelshift_l(low, hiw, lo & 31) >> (32 - len);     // bits [lo, lo + len) of the MSB-first stream
    float xq;
    if (P.mode == 1) xq = __fmul_rn((float)((int)v - 8), s);
    else xq = __fmul_rn(__fmul_rn(__fmul_rn((float)(int)(short)tb_u16(b + to + 12 + 2 * v), 0.00390625f), gain), s);
    float x = xq;
    if (P.m > 0) x = __fadd_rn(x, __fmul_rn(c0, __half2float(__ushort_as_half((unsigned short)tb_u16(Up + 2 * d)))));
    if (P.m > 1) x = __fadd_rn(x, __fmul_rn(c1, __half2float(__ushort_as_half((unsigned short)tb_u16(Up + 2 * (256 + d))))));
    if (P.has_mu) x = __fadd_rn(x, __half2float(__ushort_as_half((unsigned short)tb_u16(mup + 2 * d))));
    A.y[(size_t)row * 256 + d] = x;
  }
}


// ---------------------------------------------------------------------------------------------------------------------
// Decode attention straight over packed rows: every key and value row is unpacked inside the kernel by tb_unpack_kernel's
// rule and consumed at once; nothing unpacked is written to memory.  The counterpart of the reference's attention over packed
// rows (launch_q35_atxpk, src/q35_atxpk3.cuh / q35_atxpk4.cuh) for passes of a few rows, on CUDA cores.  Row r at *d_pos + r
// sees keys 0 .. *d_pos + r; grid (splits, kvh, M); a warp takes every eighth run of 32 keys of the split.  Online softmax in
// the exp2 domain, one rescale per 32 keys.  Partials in the layout of yskn_kv8_attention.
constexpr int TBA_WARPS = 8;
struct TbAttnP { yskn_tb_attn_args a; int G; };
struct TbTab { float cg[256], mu[256], u0[256], u1[256]; };          // one group's code table (x gain / 256) and row terms

// per-group constants of the unpack rule
struct TbRule { int packed_ok, mode, kb, guard, m, has_mu; };
__device__ __forceinline__ TbRule tb_stage_group(const uint8_t* b, int g, TbTab& T) {   // all threads of the CTA
  const TbGroup P = tb_group(b, g);
  TbRule R{P.ok && P.mode <= 1, P.mode, P.mode == 1 ? 4 : P.kk, P.guard, P.m, P.has_mu};
  const unsigned to = tb_u32(b + P.off_t + 4u * (unsigned)P.tix);
  const float gain = P.mode == 0 ? tb_f32(b + to + 4) : 1.f;
  const uint8_t* mup = b + P.go + 8;
  const uint8_t* Up = mup + (P.has_mu ? 512 : 0);
  for (int i = threadIdx.x; i < 256; i += blockDim.x) {
    T.cg[i] = !R.packed_ok ? 0.f : (P.mode == 1 ? (float)(i - 8) : __fmul_rn(__fmul_rn((float)(int)(short)tb_u16(b + to + 12 + 2 * i), 0.00390625f), gain));
    T.mu[i] = R.packed_ok && P.has_mu ? __half2float(__ushort_as_half((unsigned short)tb_u16(mup + 2 * i))) : 0.f;
    T.u0[i] = R.packed_ok && P.m > 0 ? __half2float(__ushort_as_half((unsigned short)tb_u16(Up + 2 * i))) : 0.f;
    T.u1[i] = R.packed_ok && P.m > 1 ? __half2float(__ushort_as_half((unsigned short)tb_u16(Up + 2 * (256 + i)))) : 0.f;
  }
  return R;
}
// ---- 32 keys per warp step.  Scores: a lane takes one key and walks its 256 fields (the window offsets
// are then the same in every lane and known at compile time per code width); the row terms of the unpack rule leave the inner
// loop: q.x = s * sum_d q_d cg[v_d] + c0 (q.U0) + c1 (q.U1) + q.mu, with the three dot products formed once per CTA.  Values: a
// lane takes eight channels of every key, O = sum_t p_t s_t cg[v_td] + (sum p_t c0_t) U0 + (sum p_t c1_t) U1 + (sum p_t) mu.
// The unpacked values themselves are those of tb_unpack_kernel; only the order of the fp32 sums differs (tolerance parity).
constexpr int TBA_PW = 41;                                           // staged payload row: 40 words + 1 (conflict-free lane stride)
struct TbWarpSm { unsigned kp[2][32 * TBA_PW]; unsigned vp[2][32 * TBA_PW]; float pw[32][8]; int vplain[32]; };   // two staging buffers: the next 32 keys arrive while these are used
__device__ __forceinline__ void tb_cp4(unsigned* dst, const unsigned* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int KB, bool FLAT>
__device__ __forceinline__ void tb_scores32(const unsigned* row, const float* cg, const float (*q)[8], float (&dot)[8]) {
  #pragma unroll 1
  for (int c = 0; c < 4; ++c) {                                      // chains of 64 fields: same bit offsets, 2*KB words further
    const unsigned* wr = row + 2 * KB * c;
    #pragma unroll
    for (int i = 0; i < 64; ++i) {
      constexpr int dummy = 0; (void)dummy;
      const int endb = KB * (i + 1), lo = FLAT ? endb - 4 : (endb - 8 > 0 ? endb - 8 : 0), len = endb - lo;
      const unsigned v = __funnelshift_l(wr[(lo >> 5) + 1], wr[lo >> 5], lo & 31) >> (32 - len);
      const float cv = cg[v];
      const float4 qa = *reinterpret_cast<const float4*>(&q[64 * c + i][0]), qb = *reinterpret_cast<const float4*>(&q[64 * c + i][4]);
      dot[0] = fmaf(cv, qa.x, dot[0]); dot[1] = fmaf(cv, qa.y, dot[1]); dot[2] = fmaf(cv, qa.z, dot[2]); dot[3] = fmaf(cv, qa.w, dot[3]);
      dot[4] = fmaf(cv, qb.x, dot[4]); dot[5] = fmaf(cv, qb.y, dot[5]); dot[6] = fmaf(cv, qb.z, dot[6]); dot[7] = fmaf(cv, qb.w, dot[7]);
    }
  }
}

template <int KB, bool FLAT>
__device__ __forceinline__ void tb_values32(const TbWarpSm& W, const unsigned* vp, const float* cg, const float* plain, int lane, int nk, float (&acc)[8][8]) {
  int wi[8], sh[8], ln[8];
  #pragma unroll
  for (int w = 0; w < 8; ++w) {
    const int d = 32 * w + lane, endb = KB * (d + 1), first = KB * (d & ~63), lo = FLAT ? endb - 4 : max(endb - 8, first);
    wi[w] = lo >> 5; sh[w] = lo & 31; ln[w] = 32 - (endb - lo);
  }
  #pragma unroll 2
  for (int j = 0; j < nk; ++j) {
    const float4 pa = *reinterpret_cast<const float4*>(&W.pw[j][0]), pb = *reinterpret_cast<const float4*>(&W.pw[j][4]);
    const float pg[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
    const unsigned* row = vp + j * TBA_PW;
    const bool pl = W.vplain[j] != 0;                                // warp-uniform: a row the profile leaves unpacked
    #pragma unroll
    for (int w = 0; w < 8; ++w) {
      float x;
      if (pl) x = plain ? __ldg(plain + (size_t)j * 256 + 32 * w + lane) : 0.f;
      else x = cg[__funnelshift_l(row[wi[w] + 1], row[wi[w]], sh[w]) >> ln[w]];
      #pragma unroll
      for (int g = 0; g < 8; ++g) acc[g][w] = fmaf(pg[g], x, acc[g][w]);
    }
  }
}

template <int DT>
__global__ void __launch_bounds__(TBA_WARPS * 32) tb_attn32_kernel(TbAttnP P) {
  extern __shared__ __align__(16) unsigned char tba_smem[];
  const yskn_tb_attn_args& A = P.a;
  const int G = P.G, split = blockIdx.x, kvh = blockIdx.y, r = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  TbTab* tk = reinterpret_cast<TbTab*>(tba_smem); TbTab* tv = tk + 1;
  float (*q)[8] = reinterpret_cast<float (*)[8]>(tv + 1);            // [256][8]: q * qscale * log2(e), heads past G are zero
  float (*kq)[8] = q + 256;                                           // [3][8]: q.U0, q.U1, q.mu of the key group
  TbWarpSm* Wall = reinterpret_cast<TbWarpSm*>(kq + 4);
  TbWarpSm& W = Wall[warp];
  float* mbuf = reinterpret_cast<float*>(Wall);                       // [warp][8][258], takes the staging area's place after the loop
  const TbRule rk = tb_stage_group(A.blob, __ldg(A.grp_k + kvh), *tk), rv = tb_stage_group(A.blob, __ldg(A.grp_v + kvh), *tv);
  const float qs = A.qscale * 1.4426950408889634f;
  for (int e = threadIdx.x; e < 256 * 8; e += TBA_WARPS * 32) {
    const int d = e >> 3, g = e & 7;
    q[d][g] = g < G ? act_load<DT>(A.q16, ((size_t)r * A.nh + kvh * G + g) * 256 + d) * qs : 0.f;
  }
  __syncthreads();
  if (threadIdx.x < 24) {
    const int which = threadIdx.x >> 3, g = threadIdx.x & 7;
    const float* vec = which == 0 ? tk->u0 : (which == 1 ? tk->u1 : tk->mu);
    float a = 0.f;
    for (int d = 0; d < 256; ++d) a = fmaf(q[d][g], vec[d], a);
    kq[which][g] = a;
  }
  __syncthreads();
  const int pos = __ldg(A.d_pos) + r, len = max(0, min(pos + 1, A.max_ctx));
  const int per = (len + (int)gridDim.x - 1) / (int)gridDim.x, t0 = min(len, split * per), t1 = min(len, t0 + per);
  const size_t row0 = (size_t)kvh * A.max_ctx;
  const int psw = A.pay_stride / 4, nwk = 8 * rk.kb, nwv = 8 * rv.kb;
  float acc[8][8], m[8], l[8], a0[8], a1[8], am[8];
  #pragma unroll
  for (int g = 0; g < 8; ++g) {
    m[g] = -1e30f; l[g] = a0[g] = a1[g] = am[g] = 0.f;
    #pragma unroll
    for (int w = 0; w < 8; ++w) acc[g][w] = 0.f;
  }
  // payload rows of 32 keys into staging buffer `b`, asynchronously (4-byte copies: the padded row stride is not a multiple of 16)
  auto stage = [&](int tc, int b) {
    const int nk = min(32, t1 - tc);
    const unsigned* kw = reinterpret_cast<const unsigned*>(A.k_pay) + (row0 + tc) * psw;
    const unsigned* vw = reinterpret_cast<const unsigned*>(A.v_pay) + (row0 + tc) * psw;
    for (int idx = lane; idx < nk * 40; idx += 32) {
      const int rr = idx / 40, i = idx - 40 * rr;
      if (i < nwk) tb_cp4(&W.kp[b][rr * TBA_PW + i], kw + (size_t)rr * psw + i); else W.kp[b][rr * TBA_PW + i] = 0u;
      if (i < nwv) tb_cp4(&W.vp[b][rr * TBA_PW + i], vw + (size_t)rr * psw + i); else W.vp[b][rr * TBA_PW + i] = 0u;
    }
    if (lane < nk) { W.kp[b][lane * TBA_PW + 40] = 0u; W.vp[b][lane * TBA_PW + 40] = 0u; }
  };
  int buf = 0;
  if (t0 + 32 * warp < t1) stage(t0 + 32 * warp, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int tc = t0 + 32 * warp; tc < t1; tc += 32 * TBA_WARPS, buf ^= 1) {
    const int nk = min(32, t1 - tc);
    __syncwarp();                                                    // every lane is done with the other buffer
    if (tc + 32 * TBA_WARPS < t1) stage(tc + 32 * TBA_WARPS, buf ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");           // this step's rows have landed (this lane's copies)
    __syncwarp();                                                    // ... and every other lane's
    const int t = tc + lane;
    const bool live = lane < nk, kpk = rk.packed_ok && t >= rk.guard, vpk = rv.packed_ok && t >= rv.guard;
    float sk = 0.f, c0k = 0.f, c1k = 0.f, sv = 1.f, c0v = 0.f, c1v = 0.f;
    if (live && kpk) {
      sk = __uint_as_float(__ldg(A.k_side + 2 * (row0 + t))); const unsigned pc = __ldg(A.k_side + 2 * (row0 + t) + 1);
      c0k = rk.m > 0 ? __half2float(__ushort_as_half((unsigned short)(pc & 0xffffu))) : 0.f;
      c1k = rk.m > 1 ? __half2float(__ushort_as_half((unsigned short)(pc >> 16))) : 0.f;
    }
    if (live && vpk) {
      sv = __uint_as_float(__ldg(A.v_side + 2 * (row0 + t))); const unsigned pc = __ldg(A.v_side + 2 * (row0 + t) + 1);
      c0v = rv.m > 0 ? __half2float(__ushort_as_half((unsigned short)(pc & 0xffffu))) : 0.f;
      c1v = rv.m > 1 ? __half2float(__ushort_as_half((unsigned short)(pc >> 16))) : 0.f;
    }
    float dot[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const unsigned* myrow = W.kp[buf] + lane * TBA_PW;
    if (rk.mode == 1) tb_scores32<4, true>(myrow, tk->cg, q, dot);
    else if (rk.kb == 3) tb_scores32<3, false>(myrow, tk->cg, q, dot);
    else if (rk.kb == 4) tb_scores32<4, false>(myrow, tk->cg, q, dot);
    else tb_scores32<5, false>(myrow, tk->cg, q, dot);
    float sc[8];
    #pragma unroll
    for (int g = 0; g < 8; ++g) sc[g] = fmaf(sk, dot[g], fmaf(c0k, kq[0][g], fmaf(c1k, kq[1][g], kq[2][g])));
    if (live && !kpk) {                                              // a key row the profile leaves unpacked: the plain row
      #pragma unroll
      for (int g = 0; g < 8; ++g) sc[g] = 0.f;
      if (A.k_plain) {
        const float* pr = A.k_plain + (row0 + t) * 256;
        for (int d = 0; d < 256; ++d) {
          const float x = __ldg(pr + d);
          #pragma unroll
          for (int g = 0; g < 8; ++g) sc[g] = fmaf(q[d][g], x, sc[g]);
        }
      }
    }
    W.vplain[lane] = vpk ? 0 : 1;
    #pragma unroll
    for (int g = 0; g < 8; ++g) {
      if (g >= G) { W.pw[lane][g] = 0.f; continue; }
      float mx = live ? sc[g] : -1e30f;
      #pragma unroll
      for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[g], mx), al = exp2f(m[g] - mn), p = live ? exp2f(sc[g] - mn) : 0.f;
      float s0 = p, s1 = p * c0v, s2 = p * c1v, s3 = vpk ? p : 0.f;
      #pragma unroll
      for (int o = 16; o; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o); s3 += __shfl_xor_sync(0xffffffffu, s3, o);
      }
      l[g] = fmaf(l[g], al, s0); a0[g] = fmaf(a0[g], al, s1); a1[g] = fmaf(a1[g], al, s2); am[g] = fmaf(am[g], al, s3); m[g] = mn;
      #pragma unroll
      for (int w = 0; w < 8; ++w) acc[g][w] *= al;
      W.pw[lane][g] = p * sv;
    }
    __syncwarp();
    const float* vpl = A.v_plain ? A.v_plain + (row0 + tc) * 256 : nullptr;
    if (rv.mode == 1) tb_values32<4, true>(W, W.vp[buf], tv->cg, vpl, lane, nk, acc);
    else if (rv.kb == 3) tb_values32<3, false>(W, W.vp[buf], tv->cg, vpl, lane, nk, acc);
    else if (rv.kb == 4) tb_values32<4, false>(W, W.vp[buf], tv->cg, vpl, lane, nk, acc);
    else tb_values32<5, false>(W, W.vp[buf], tv->cg, vpl, lane, nk, acc);
  }
  // ---- the row terms of the value group, then the merge of the warps (natural-log m, as the merge kernel expects)
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                                   // the staging area becomes the merge buffer
  #pragma unroll
  for (int g = 0; g < 8; ++g) {
    if (g >= G) continue;
    float* wb = mbuf + ((size_t)warp * 8 + g) * 258;
    if (lane == 0) { wb[0] = m[g]; wb[1] = l[g]; }
    #pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int d = 32 * w + lane;
      wb[2 + d] = fmaf(a0[g], tv->u0[d], fmaf(a1[g], tv->u1[d], fmaf(am[g], tv->mu[d], acc[g][w])));
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < G * 256; e += TBA_WARPS * 32) {
    const int g = e >> 8, d = e & 255;
    float M2 = -1e30f;
    #pragma unroll
    for (int w = 0; w < TBA_WARPS; ++w) M2 = fmaxf(M2, mbuf[((size_t)w * 8 + g) * 258]);
    float L2 = 0.f, o = 0.f;
    #pragma unroll
    for (int w = 0; w < TBA_WARPS; ++w) {
      const float* wb = mbuf + ((size_t)w * 8 + g) * 258;
      const float f = wb[0] > -1e29f ? exp2f(wb[0] - M2) : 0.f;
      L2 += f * wb[1]; o += f * wb[2 + d];
    }
    const size_t pidx = ((size_t)r * A.splits + split) * A.nh + kvh * G + g;
    if (d == 0) { A.pm[pidx] = M2 > -1e29f ? M2 * 0.6931471805599453f : -1e30f; A.pl[pidx] = L2; }
    A.pacc[pidx * 256 + d] = o;
  }
}

}  // namespace

int launch_tb_decode(const uint8_t* blob, const int* grp, const int* pos, const uint8_t* pay, int pay_stride, const uint32_t* side, const float* yin,
                     float* y, int rows, cudaStream_t st) {
  if (!blob || !grp || !pos || !pay || !side || !y) KV4_REJECT("yskn_tb_decode: null buffer");
  if (rows <= 0 || pay_stride < 160 || pay_stride % 4 || ((uintptr_t)pay & 3)) KV4_REJECT("yskn_tb_decode: bad shape (rows %d, payload stride %d)", rows, pay_stride);
  TbDecP A{blob, grp, pos, pay, pay_stride, side, yin, y, rows};
  tb_unpack_kernel<<<(rows + 7) / 8, 256, 0, st>>>(A);
  return launch_status("tb_unpack_kernel");
}

size_t tb_scratch_bytes(int, int) { return 0; }              // the encoder keeps everything on chip

// Host-side check of a "KVQP v1" blob, the reference loader's (src/engine35.cpp:50-53) plus its table checks
// (src/kvq_fast.hpp:66-69); *nm = number of scale multipliers.
int tb_blob_info(const uint8_t* b, size_t n, int* nm) {
  auto u16 = [&](size_t o) { return (unsigned)b[o] | ((unsigned)b[o + 1] << 8); };
  auto u32 = [&](size_t o) { return u16(o) | (u16(o + 2) << 16); };
  if (!b || n < 100 || memcmp(b, "KVQP", 4) != 0 || u16(4) != 1 || u16(6) != 96 || u32(8) != n) KV4_REJECT("yskn_tb_blob_info: not a KVQP v1 blob");
  if (u16(16) != 256 || u16(18) != 16 || u16(20) != 4 || u32(28) != 128u) KV4_REJECT("yskn_tb_blob_info: needs D 256, 16 layers, 4 kv heads");
  const unsigned nt = u16(22), off_t = u32(36), off_g = u32(40), ngrp = u32(28);
  if ((size_t)off_t + 4 * (size_t)nt > n || (size_t)off_g + 4 * (size_t)ngrp > n || (size_t)u32(32) + 4 * (size_t)u16(24) > n) KV4_REJECT("yskn_tb_blob_info: offsets beyond the blob");
  for (unsigned t = 0; t < nt; ++t) {
    const size_t o = u32(off_t + 4 * t);
    if (o + 12 + 512 > n || b[o] != 8 || b[o + 2] != 64 || b[o + 3] != 8) KV4_REJECT("yskn_tb_blob_info: code tables must have L 8, chain 64, F 8");
  }
  for (unsigned g = 0; g < ngrp; ++g) {
    const size_t go = u32(off_g + 4 * g);
    if (go + 8 > n) KV4_REJECT("yskn_tb_blob_info: group record %u beyond the blob", g);
    const int mode = b[go], kk = b[go + 1], tix = b[go + 2], m = b[go + 4], mu = b[go + 5];
    if (mode > 1 || (mode == 0 && (kk < 3 || kk > 5 || (unsigned)tix >= nt)) || m > 2 || go + 8 + (mu ? 512 : 0) + 512 * (size_t)m > n)
      KV4_REJECT("yskn_tb_blob_info: group record %u has fields this codec does not have", g);
  }
  const int k = (int)u16(24);
  if (k < 1 || k > 16) KV4_REJECT("yskn_tb_blob_info: %d scale multipliers (1..16)", k);
  if (nm) *nm = k;
  return 0;
}

int launch_tb_encode(const uint8_t* blob, int nm, const float* x, const int* grp, const int* pos, int rows, float* y, uint8_t* pay, int pay_stride,
                     uint32_t* side, void* scratch, size_t scratch_bytes, cudaStream_t st) {
  (void)scratch; (void)scratch_bytes;
  if (!blob || !x || !grp || !pos) KV4_REJECT("yskn_tb_encode: null buffer");
  if (rows <= 0 || nm < 1 || nm > TB_NM) KV4_REJECT("yskn_tb_encode: bad shape (rows %d, multipliers %d)", rows, nm);
  if (pay && (pay_stride < 160 || pay_stride % 4 || ((uintptr_t)pay & 3))) KV4_REJECT("yskn_tb_encode: payload rows need a stride of at least 160 bytes, a multiple of 4");
  static std::atomic<unsigned long long> attr{0};
  if (first_use_on_device(attr)) KV4_CUDA(cudaFuncSetAttribute(tb_encode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TbRowSmem::bytes(TB_NM)));
  tb_encode_kernel<<<rows, 128, TbRowSmem::bytes(nm), st>>>(TbP{blob, nm, x, grp, pos, rows, y, pay, pay_stride, side});
  return launch_status("tb_encode_kernel");
}

int launch_tb_attention(const yskn_tb_attn_args& a, int act_dtype, cudaStream_t st) {
  if (!a.q16 || !a.blob || !a.k_pay || !a.v_pay || !a.k_side || !a.v_side || !a.grp_k || !a.grp_v || !a.d_pos || !a.pm || !a.pl || !a.pacc)
    KV4_REJECT("yskn_tb_attention: null buffer");
  if (a.kvh <= 0 || a.nh <= 0 || a.nh % a.kvh || a.nh / a.kvh > 8 || a.M <= 0 || a.M > 65535 || a.kvh > 65535 || a.splits <= 0 || a.max_ctx <= 0)
    KV4_REJECT("yskn_tb_attention: bad shape (kvh %d, nh %d, M %d, splits %d, max_ctx %d): at most 8 query heads per kv-head", a.kvh, a.nh, a.M, a.splits, a.max_ctx);
  if (a.pay_stride < 160 || a.pay_stride % 4 || (((uintptr_t)a.k_pay | (uintptr_t)a.v_pay) & 3)) KV4_REJECT("yskn_tb_attention: bad payload stride %d or alignment", a.pay_stride);
  const size_t stage = sizeof(TbWarpSm) * TBA_WARPS, merge = (size_t)TBA_WARPS * 8 * 258 * 4;
  const size_t smem = 2 * sizeof(TbTab) + (256 + 4) * 8 * 4 + (stage > merge ? stage : merge);
  TbAttnP P{a, a.nh / a.kvh};
  const dim3 grid(a.splits, a.kvh, a.M);
  if (act_dtype == YSKN_KV4_BF16) {
    static std::atomic<unsigned long long> attr{0};
    if (first_use_on_device(attr)) KV4_CUDA(cudaFuncSetAttribute(tb_attn32_kernel<YSKN_KV4_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    tb_attn32_kernel<YSKN_KV4_BF16><<<grid, TBA_WARPS * 32, smem, st>>>(P);
  } else if (act_dtype == YSKN_KV4_F16) {
    static std::atomic<unsigned long long> attr{0};
    if (first_use_on_device(attr)) KV4_CUDA(cudaFuncSetAttribute(tb_attn32_kernel<YSKN_KV4_F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    tb_attn32_kernel<YSKN_KV4_F16><<<grid, TBA_WARPS * 32, smem, st>>>(P);
  } else KV4_REJECT("yskn_tb_attention: q16 is bf16 or fp16 (act_dtype %d)", act_dtype);
  return launch_status("tb_attn32_kernel");
}

}  // namespace kv4
