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
#include <type_traits>

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

// Offset of a trellis group's code table.  A flat group has none: its table index is not checked by the loader and may lie beyond the blob, so
// nothing is read through it (0: the header, which every blob has).
__device__ __forceinline__ unsigned tb_table(const uint8_t* b, const TbGroup& P) { return P.ok && P.mode == 0 ? tb_u32(b + P.off_t + 4u * (unsigned)P.tix) : 0u; }

// ---- encoder: one block per row, one warp per multiplier and pair of chains, sixteen lanes per chain of 64 values.
//
// A step of the search takes new(d) = min over the 2^KK predecessors {j * UU + u}, u = d >> KK, of old(p), plus (x - code[d])^2: every
// state is a candidate of one group u only, so 256 candidates and 256 costs a step.  What bounds it is instruction issue
// (integer), so the whole step stays in registers: a lane holds sixteen states p = j << SH | u (SH = 8 - KK, UU = 2^SH), one multiply-add for each cost and
// one fused add-minimum for each candidate, and both chains of a warp go through the same instructions, the few that hand minima on among them:
//   KK   lane (4 bits)          registers                 minima handed on            exchanged
//   3    u4 u3 u1 u0            j (8), u2                 8 shuffles                  none (a lane has every j of its two u)
//   4    top bit of j, u3 .. u1 the other bits of j, u0   8 shuffles                  1 (each lane of a pair keeps one u)
//   5    top bit of j, u        the other bits of j (16)  4 shuffles                  1
// (The new states of a lane need the minima of the groups p >> KK.  For KK = 3 the bit of u in the registers is u2: the lane's states of both values need the
// same eight, and which of its two values a lane hands on follows from j alone.)  About 48 instructions a step of two chains; the form before it,
// a warp per chain with eight states a lane, takes 55 a step of one, of which 39 are exchanges, masks and stores (tb_search_chain).
// x^2 is left out of the costs: it adds the same number to every state of a step.  A cost travels as a key, cost << 5 | j, whose j is part
// of the state's own constant: the minimum over keys is the minimum cost with the first j on ties (the reference's rule,
// src/kvq_gpu.cuh:101-102) and carries its back pointer, one byte per group and step.
// Width of the keys: |f| = |c^2 - 2xc| <= F = C^2 + 4096 C with C = max |code| and |x| <= 2048, and f differs by at most D = 8192 C between
// two states; any state is reached from any other in three steps, so the costs of a step spread over at most 3 D.  They are
// brought back to one of them every four steps: |cost| <= 3 D + 4 F < 2^26 for C <= 1400, and a key fits 32 bits.  Profiles with larger codes
// take 64-bit keys (no bringing back).
// 4,096 rows, 5 multipliers, on a B200: 1,335 us (one warp per (row, multiplier, chain), costs in shared memory, every lane walking its group's predecessors; a
// second kernel for choice and packing) -> 448 (minima kept instead of back pointers, candidates recomputed on the way back) -> 321 (eight states a
// lane, a warp per chain that walks the multipliers) -> 238.  Issue slots 64 % busy, integer ALU 49 %, shuffles and shared memory 49 %; 25 warps
// an SM at 72 registers instead of 20 at 96 are slower (262), 15 at 128 too (273).
// Where a warp per chain stays: with one multiplier, whose two pairs of chains would leave two of the block's four warps idle (28 warps an SM; 4,096 rows 83 us
// by pairs, 75 by chains; 64-bit keys 318 and 178), and with 64-bit keys and many rows, where sixteen states a lane do not fit the registers and the codes are read again
// every step (4,096 rows of 2 / 5 / 16 multipliers 362 / 972 / 3,237 us by pairs, 327 / 838 / 2,625 by chains; 8 rows, bound by the dependent steps, 23.5 / 40 / 122
// and 31.7 / 46 / 136).
// Blocks of ten warps (every multiplier and pair of chains at once) for a few rows, which are bound by the chains of 64 dependent steps; of five, twice as
// many an SM, for more rows than two rounds of the former: with unpacking 100 rows 28.0 / 33.9 us, 600 53.5 / 55.6, 1,000 84.8 / 80.9, 4,096 270 / 250 (ten / five).
constexpr int TB_NM = 16;                                // multipliers at most (the blob's limit)
constexpr int TB_WIDE = 10, TB_NARROW = 5, TB_ONE = 4, TB_WIDE_ROWS = 2 * 2 * 148;     // warps of a block at most, three forms; rows that the wide one takes
struct TbRowSmem {
  short code[256]; float res[256]; float red[8]; int cmax[16]; uint8_t fld[256];
  TbGroup grp; float coef[2];                              // what the search does not need waits here, not in registers
  struct Warp { int xs[128]; uint8_t bp[2][64 * 32]; };    // scaled values; back pointers of each chain: [t][u], the low five bits
  struct Mult { uint8_t st[256]; float err[8]; };          // one per multiplier: its states and its error sums
  static int warps(int nm, int most) { return 2 * nm < 4 ? 4 : 2 * nm < most ? 2 * nm : most; }      // four at least: they hold the row
  static size_t bytes(int nm, int most) { return sizeof(TbRowSmem) + warps(nm, most) * sizeof(Warp) + nm * sizeof(Mult); }
};
static_assert(sizeof(TbRowSmem) % 16 == 0 && sizeof(TbRowSmem::Warp) % 16 == 0, "xs is read sixteen bytes at a time");
struct TbP { const uint8_t* blob; int nm; const float* x; const int* grp; const int* pos; int rows; float* y; uint8_t* pay; int pay_stride; uint32_t* side; int whole; };

__device__ __forceinline__ int tb_addmin(int a, int b, int c) { return __viaddmin_s32(a, b, c); }
__device__ __forceinline__ long long tb_addmin(long long a, long long b, long long c) { return min(a + b, c); }

// Only state 0 exists at first.  Every state is reachable after three steps, so the others have to stay behind by more than 6 F
// (5e7 for C = 1400) until then, and within the width of a key.
template <class K> constexpr K TB_START = (K)(-(1 << 25)) * 32;
template <class K> constexpr K TB_FAR = (K)(sizeof(K) == 4 ? (1 << 24) + (1 << 23) : 0x40000000) * 32;

// The best final state of a chain, smallest (cost, state) over 2 O lanes, and the way back from it; `first` is 0 in the lane that stores.
template <int KK, int O, class K> __device__ __forceinline__ void tb_walk(const uint8_t* bp, K best, int st, uint8_t* states, int first) {
  constexpr int SH = 8 - KK, UU = 1 << SH;
  #pragma unroll
  for (int o = O; o; o >>= 1) {
    const K c = __shfl_xor_sync(0xffffffffu, best, o); const int b2 = __shfl_xor_sync(0xffffffffu, st, o);
    if (c < best || (c == best && b2 < st)) { best = c; st = b2; }
  }
  __syncwarp();                                          // the back pointers are complete
  #pragma unroll 8
  for (int t = 63; t >= 0; --t) {
    if (first == 0) states[t] = (uint8_t)st;
    const int u = st >> KK;
    st = ((bp[t * UU + u] & 31) << SH) + u;              // (the row of step 0 is read but never used)
  }
  __syncwarp();                                          // they may be overwritten, and the states are complete
}

// States of the best path of this half warp's chain of scaled values xs (bp, xs and states are the chain's own).  K = int or long long, the type of the keys.
template <int KK, class K> __device__ __forceinline__ void tb_search(uint8_t* bp, const short* code, const int* xs, uint8_t* states, int lane) {
  constexpr int SH = 8 - KK, UU = 1 << SH, NQ = KK == 5 ? 4 : 8;
  constexpr bool NARROW = sizeof(K) == 4;
  const int l = lane & 15, half = lane & 16;
  auto state = [&](int e) {
    return KK == 3 ? ((e >> 1) << 5) | ((l >> 2) << 3) | ((e & 1) << 2) | (l & 3) : KK == 4 ? ((l >> 3) << 7) | ((e >> 1) << 4) | ((l & 7) << 1) | (e & 1)
                                                                                           : ((l >> 3) << 7) | (e << 3) | (l & 7);
  };
  int m2c[16], c2[16];                                   // 32-bit keys: a cost is x * m2c + c2; 64-bit ones read the code again (c (c - 2x) fits 32 bits)
  if (NARROW)
    #pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int p = state(e), c = code[p];
      m2c[e] = -2 * c * 32; c2[e] = c * c * 32 + (p >> SH);
    }
  int src[NQ];                                           // the lane that holds the minimum of group (new state >> KK)
  #pragma unroll
  for (int q = 0; q < NQ; ++q)
    src[q] = half | (KK == 3 ? ((q >> 1) << 2) | (l >> 2) : KK == 4 ? ((q & 1) << 3) | ((l >> 3) << 2) | (q >> 1) : ((l >> 3) << 2) | q);
  const bool upper = l >> 3;                             // KK = 4: of a pair of lanes the upper one keeps the odd u
  const int my_u = KK == 3 ? ((l >> 2) << 3) | (l & 3) : KK == 4 ? ((l & 7) << 1) | (upper ? 1 : 0) : l & 7;
  K ka = my_u == 0 ? TB_START<K> : TB_FAR<K>, kb = TB_FAR<K>;          // minima of the lane's groups (kb: KK = 3, the one with u2 = 1)
  uint8_t* mine = bp + my_u;
  auto costs = [&](int x, K (&t)[16], K (&m)[NQ]) {
    ka &= ~(K)31;
    if (KK == 3) kb &= ~(K)31;
    #pragma unroll
    for (int q = 0; q < NQ; ++q) m[q] = __shfl_sync(0xffffffffu, KK == 3 && (q & 1) ? kb : ka, src[q]);
    #pragma unroll
    for (int e = 0; e < 16; ++e)
      if (NARROW) t[e] = x * m2c[e] + c2[e];
      else { const int p = state(e), c = code[p]; t[e] = (K)(c * (c - 2 * x)) * 32 + (p >> SH); }
  };
  auto mi = [](int e) { return KK == 5 ? e >> 2 : e >> 1; };
  auto step = [&](int x, int t) {                        // the minima of step t + 1 from those of step t
    K ct[16], m[NQ];
    costs(x, ct, m);
    K a = ct[0] + m[0], b = ct[1] + m[mi(1)];
    #pragma unroll
    for (int e = 2; e < 16; e += 2) {
      a = tb_addmin(ct[e], m[mi(e)], a);
      b = tb_addmin(ct[e + 1], m[mi(e + 1)], b);
    }
    if (KK == 3) {
      ka = a; kb = b;
      mine[(t + 1) * UU] = (uint8_t)a; mine[(t + 1) * UU + 4] = (uint8_t)b;
    } else {
      if (KK == 4) ka = min(upper ? b : a, __shfl_xor_sync(0xffffffffu, upper ? a : b, 8));
      else { ka = min(a, b); ka = min(ka, __shfl_xor_sync(0xffffffffu, ka, 8)); }
      if (KK == 4 || l < UU) mine[(t + 1) * UU] = (uint8_t)ka;
    }
  };
  #pragma unroll 1
  for (int t = 0; t < 60; t += 4) {
    const int4 x = *reinterpret_cast<const int4*>(xs + t);
    step(x.x, t); step(x.y, t + 1); step(x.z, t + 2); step(x.w, t + 3);
    if (NARROW) { const K b0 = __shfl_sync(0xffffffffu, ka, half) & ~(K)31; ka -= b0; if (KK == 3) kb -= b0; }
  }
  const int4 x = *reinterpret_cast<const int4*>(xs + 60);
  step(x.x, 60); step(x.y, 61); step(x.z, 62);
  // best final state: smallest (cost, state)
  K ct[16], m[NQ];
  costs(x.w, ct, m);
  K best = 0; int bs = 0;
  #pragma unroll
  for (int e = 0; e < 16; ++e) {
    const K c = (ct[e] + m[mi(e)]) & ~(K)31;
    const int p = state(e);
    if (e == 0 || c < best || (c == best && p < bs)) { best = c; bs = p; }
  }
  tb_walk<KK, 8>(bp, best, bs, states, l);
}

// The same with the whole warp on one chain, eight states a lane,
//   p = jhi << (SH+2) | jlo << SH | umid << 1 | ulo,     registers e = (jlo, ulo), lane = (jhi, umid):
// the minimum over jlo is in the lane, the first exchange over jhi halves the lane's two values of u (each lane of the pair keeps one), the others are plain;
// the new states need 4 (KK = 3, 4) or 1 (KK = 5) of the UU minima.
template <int KK, class K> __device__ __forceinline__ void tb_search_chain(uint8_t* bp, const short* code, const int* xs, uint8_t* states, int lane) {
  constexpr int SH = 8 - KK, UU = 1 << SH, NQ = KK == 5 ? 1 : 4;
  constexpr bool NARROW = sizeof(K) == 4;
  const int umid = lane & ((1 << (SH - 1)) - 1), jhi = lane >> (SH - 1);
  auto state = [&](int e) { return (jhi << (SH + 2)) | ((e >> 1) << SH) | (umid << 1) | (e & 1); };    // a lane's states grow with e
  int m2c[8];                                            // a cost is one multiply-add, a wide one for 64-bit keys
  K c2[8];
  int src[NQ];
  #pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int p = state(e), c = code[p];
    m2c[e] = -2 * c * 32; c2[e] = (K)c * c * 32 + (p >> SH);
  }
  #pragma unroll
  for (int q = 0; q < NQ; ++q) {                         // the lane that holds the minimum of group (new state >> KK)
    const int g = ((jhi << (SH + 2)) | (q << SH) | (umid << 1)) >> KK;
    src[q] = ((g & 1) << (SH - 1)) | (g >> 1);
  }
  const bool upper = (lane >> (SH - 1)) & 1;             // of a pair of lanes the upper one keeps the odd u
  const int my_u = (umid << 1) | (upper ? 1 : 0);
  K keep = my_u == 0 ? TB_START<K> : TB_FAR<K>;
  uint8_t* mine = bp + (lane < UU ? my_u : 0);           // lanes below UU hold every u once (the jhi bits above the first are zero)
  auto costs = [&](int x, K (&t)[8], K (&m)[NQ]) {
    keep &= ~(K)31;
    #pragma unroll
    for (int q = 0; q < NQ; ++q) m[q] = __shfl_sync(0xffffffffu, keep, src[q]);
    #pragma unroll
    for (int e = 0; e < 8; ++e) t[e] = (K)x * m2c[e] + c2[e];
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
    keep = min(upper ? b : a, __shfl_xor_sync(0xffffffffu, upper ? a : b, 1 << (SH - 1)));
    #pragma unroll
    for (int k = SH; k < 5; ++k) keep = min(keep, __shfl_xor_sync(0xffffffffu, keep, 1 << k));
    if (lane < UU) mine[(t + 1) * UU] = (uint8_t)keep;
  };
  #pragma unroll 1
  for (int t = 0; t < 60; t += 4) {
    const int4 x = *reinterpret_cast<const int4*>(xs + t);
    step(x.x, t); step(x.y, t + 1); step(x.z, t + 2); step(x.w, t + 3);
    if (NARROW) keep -= __shfl_sync(0xffffffffu, keep, 0) & ~(K)31;
  }
  const int4 x = *reinterpret_cast<const int4*>(xs + 60);
  step(x.x, 60); step(x.y, 61); step(x.z, 62);
  K ct[8], m[NQ];
  costs(x.w, ct, m);
  K best = 0; int bs = 0;
  #pragma unroll
  for (int e = 0; e < 8; ++e) {
    const K c = (ct[e] + m[NQ == 1 ? 0 : e >> 1]) & ~(K)31;
    if (e == 0 || c < best) { best = c; bs = state(e); }
  }
  tb_walk<KK, 16>(bp, best, bs, states, lane);
}

template <int W>
__global__ void __launch_bounds__(W * 32, W == TB_ONE ? 7 : 20 / W) tb_encode_kernel(TbP A) {
  extern __shared__ __align__(16) unsigned char tbe_smem[];
  TbRowSmem& S = *reinterpret_cast<TbRowSmem*>(tbe_smem);
  const int nt = blockDim.x, nwarps = nt >> 5;
  TbRowSmem::Warp* const warps = reinterpret_cast<TbRowSmem::Warp*>(tbe_smem + sizeof(TbRowSmem));
  TbRowSmem::Mult* const mult = reinterpret_cast<TbRowSmem::Mult*>(warps + nwarps);
  const int row = blockIdx.x, c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool own = c < 4;                                // the first four warps hold the row, two values a thread
  const int d0 = 64 * (c & 3) + lane, d1 = d0 + 32;
  const uint8_t* b = A.blob;
  TbGroup P = tb_group(b, A.grp[row]);
  const int words = A.pay_stride / 4;
  unsigned* pay = A.pay ? reinterpret_cast<unsigned*>(A.pay + (size_t)row * A.pay_stride) : nullptr;
  float ra = A.x[(size_t)row * 256 + d0], rb = A.x[(size_t)row * 256 + d1];
  if (!P.ok || A.pos[row] < P.guard) {                   // stored as it is
    if (A.y && own) { A.y[(size_t)row * 256 + d0] = ra; A.y[(size_t)row * 256 + d1] = rb; }
    if (A.whole) {
      for (int w = threadIdx.x; w < words; w += nt) pay[w] = 0u;
      if (threadIdx.x < 2) A.side[2 * row + threadIdx.x] = 0u;
    }
    return;
  }
  // the reference's row sum: a xor-butterfly over each run of 32 values, then the eight runs in order (src/kvq_fast.cuh:33-43)
  auto run_sum = [&](float v) {
    #pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  auto rowsum = [&](float va, float vb) -> float {
    va = run_sum(va); vb = run_sum(vb);
    if (own && lane == 0) { S.red[2 * c] = va; S.red[2 * c + 1] = vb; }
    __syncthreads();
    float t = 0.f;
    #pragma unroll
    for (int w = 0; w < 8; ++w) t = __fadd_rn(t, S.red[w]);
    __syncthreads();
    return t;
  };
  auto f16at = [&](const uint8_t* p, int d) { return __half2float(__ushort_as_half((unsigned short)tb_u16(p + 2 * d))); };
  float c0 = 0.f, c1 = 0.f;
  {
    const uint8_t* mup = b + P.go + 8;
    const uint8_t* Up = mup + (P.has_mu ? 512 : 0);
    if (P.has_mu) { ra = __fsub_rn(ra, f16at(mup, d0)); rb = __fsub_rn(rb, f16at(mup, d1)); }
    if (P.m > 0) {
      const float ua = f16at(Up, d0), ub = f16at(Up, d1);
      c0 = tb_f16r(rowsum(__fmul_rn(ra, ua), __fmul_rn(rb, ub)));
      ra = __fsub_rn(ra, __fmul_rn(c0, ua)); rb = __fsub_rn(rb, __fmul_rn(c0, ub));
    }
    if (P.m > 1) {
      const float ua = f16at(Up + 512, d0), ub = f16at(Up + 512, d1);
      c1 = tb_f16r(rowsum(__fmul_rn(ra, ua), __fmul_rn(rb, ub)));
      ra = __fsub_rn(ra, __fmul_rn(c1, ua)); rb = __fsub_rn(rb, __fmul_rn(c1, ub));
    }
  }
  float xqa, xqb, psc; int fa, fb, kb;
  if (P.mode == 1) {                                     // flat 4-bit codes (src/kvq_fast.cuh:193-198)
    float am = fmaxf(fabsf(ra), fabsf(rb));
    #pragma unroll
    for (int o = 16; o; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if (own && lane == 0) S.red[c] = am;
    __syncthreads();
    am = fmaxf(fmaxf(S.red[0], S.red[1]), fmaxf(S.red[2], S.red[3]));
    float s7 = __fdiv_rn(am, 7.f); if (s7 == 0.f) s7 = 1.f;
    const float qa = fminf(fmaxf(rintf(__fdiv_rn(ra, s7)), -7.f), 7.f), qb = fminf(fmaxf(rintf(__fdiv_rn(rb, s7)), -7.f), 7.f);
    xqa = __fmul_rn(qa, s7); xqb = __fmul_rn(qb, s7); fa = (int)qa + 8; fb = (int)qb + 8; psc = s7; kb = 4;
  } else {
    const unsigned to = tb_table(b, P);
    const float gain = tb_f32(b + to + 4);
    int cm = 0;
    for (int i = threadIdx.x; i < 256; i += nt) { const int v = (short)tb_u16(b + to + 12 + 2 * i); S.code[i] = (short)v; cm = max(cm, abs(v)); }
    cm = __reduce_max_sync(0xffffffffu, cm);
    if (lane == 0) S.cmax[c] = cm;
    if (own) { S.res[d0] = ra; S.res[d1] = rb; }
    if (threadIdx.x == 0) { S.grp = P; S.coef[0] = c0; S.coef[1] = c1; }
    float rms = __fsqrt_rn(__fdiv_rn(rowsum(__fmul_rn(ra, ra), __fmul_rn(rb, rb)), 256.f));     // its barriers also publish the codes and the row
    if (rms == 0.f) rms = 1.f;
    for (int w = 0; w < nwarps; ++w) cm = max(cm, S.cmax[w]);
    const bool narrow = cm <= 1400;
    auto scale = [&](int mi) { const float s = tb_f16r(__fmul_rn(rms, tb_f32(b + P.off_m + 4u * (unsigned)mi))); return s == 0.f ? 1.f : s; };
    auto value = [&](int st, float s) { return __fmul_rn(__fmul_rn(__fmul_rn((float)(int)S.code[st], 0.00390625f), gain), s); };
    // a unit: a multiplier and the N = 128 or 64 values from e0 on that this warp searches
    auto unit_of = [&](int mi, int e0, auto n, auto search) {
      constexpr int R = decltype(n)::value / 32;
      const float s = scale(mi);
      TbRowSmem::Warp& B = warps[c];
      #pragma unroll
      for (int r = 0; r < R; ++r)
        B.xs[32 * r + lane] = (int)fminf(fmaxf(rintf(__fmul_rn(__fdiv_rn(S.res[e0 + 32 * r + lane], s), 256.f)), -2048.f), 2048.f);
      __syncwarp();
      uint8_t* const st = mult[mi].st + e0;
      if (P.kk == 3) search(std::integral_constant<int, 3>{}, B, st);
      else if (P.kk == 4) search(std::integral_constant<int, 4>{}, B, st);
      else if (P.kk == 5) search(std::integral_constant<int, 5>{}, B, st);
      else { for (int r = 0; r < R; ++r) st[32 * r + lane] = 0; __syncwarp(); }
      #pragma unroll
      for (int r = 0; r < R; ++r) {
        const float d = __fsub_rn(S.res[e0 + 32 * r + lane], value(st[32 * r + lane], s)), e = run_sum(__fmul_rn(d, d));
        if (lane == 0) mult[mi].err[e0 / 32 + r] = e;
      }
    };
    auto pairs = [&](auto key) {
      #pragma unroll 1
      for (int unit = c; unit < 2 * A.nm; unit += nwarps)
        unit_of(unit >> 1, 128 * (unit & 1), std::integral_constant<int, 128>{}, [&](auto kk, TbRowSmem::Warp& B, uint8_t* st) {
          const int h = lane >> 4;
          tb_search<decltype(kk)::value, decltype(key)>(B.bp[h], S.code, B.xs + 64 * h, st + 64 * h, lane);
        });
    };
    auto chains = [&](auto key) {
      #pragma unroll 1
      for (int unit = c; unit < 4 * A.nm; unit += nwarps)
        unit_of(unit >> 2, 64 * (unit & 3), std::integral_constant<int, 64>{}, [&](auto kk, TbRowSmem::Warp& B, uint8_t* st) {
          tb_search_chain<decltype(kk)::value, decltype(key)>(B.bp[0], S.code, B.xs, st, lane);
        });
    };
    if constexpr (W == TB_ONE) { if (narrow) chains(int{}); else chains((long long)0); }
    else if (narrow) pairs(int{});
    else if constexpr (W == TB_WIDE) pairs((long long)0);
    else chains((long long)0);
    __syncthreads();
    float best_e = 0.f; int best = 0;
    for (int mi = 0; mi < A.nm; ++mi) {                  // the smallest squared error, the first on ties
      float e = 0.f;
      #pragma unroll
      for (int w = 0; w < 8; ++w) e = __fadd_rn(e, mult[mi].err[w]);
      if (mi == 0 || e < best_e) { best_e = e; best = mi; }
    }
    P = S.grp; c0 = S.coef[0]; c1 = S.coef[1];
    const float s = scale(best);
    const int sa = mult[best].st[d0], sb = mult[best].st[d1];
    xqa = value(sa, s); xqb = value(sb, s);
    fa = sa & ((1 << P.kk) - 1); fb = sb & ((1 << P.kk) - 1); psc = s; kb = P.kk;
  }
  if (A.y && own) {
    const uint8_t* mup = b + P.go + 8;
    const uint8_t* Up = mup + (P.has_mu ? 512 : 0);
    if (P.m > 0) { xqa = __fadd_rn(xqa, __fmul_rn(c0, f16at(Up, d0))); xqb = __fadd_rn(xqb, __fmul_rn(c0, f16at(Up, d1))); }
    if (P.m > 1) { xqa = __fadd_rn(xqa, __fmul_rn(c1, f16at(Up + 512, d0))); xqb = __fadd_rn(xqb, __fmul_rn(c1, f16at(Up + 512, d1))); }
    if (P.has_mu) { xqa = __fadd_rn(xqa, f16at(mup, d0)); xqb = __fadd_rn(xqb, f16at(mup, d1)); }
    A.y[(size_t)row * 256 + d0] = xqa; A.y[(size_t)row * 256 + d1] = xqb;
  }
  if (pay) {
    if (own) { S.fld[d0] = (uint8_t)fa; S.fld[d1] = (uint8_t)fb; }
    __syncthreads();
    for (int w = threadIdx.x; w < (A.whole ? words : 8 * kb); w += nt) {      // MSB-first bit stream, 32 bits per word (src/kvq_fast.cuh:228-232)
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
  const unsigned to = tb_table(b, P);
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
// rows (launch_q35_atxpk, src/q35_atxpk3.cuh / q35_atxpk4.cuh) for passes of a few rows.  Row r at *d_pos + r sees keys
// 0 .. *d_pos + r; grid (splits, kvh, M).  Partials in the layout of yskn_kv8_attention.
//
// A packed token is 264 bytes for its key and value together (4 bits), but 512 table look-ups: shared-memory wavefronts and issue
// slots bound this kernel, not HBM.  So
//   * the code table is replicated per lane (256 x 32 words, 32 KB for keys and 32 KB for values, at addresses that are a multiple of their
//     size): a look-up is one funnel shift, one AND-OR that yields the address, one conflict-free load; the words carry the code as
//     an fp16 in both halves, so two of them become an operand register by one byte permute.  Codes are integers up to 2,048 in
//     size, exact in fp16 (a table with larger ones takes the row path below); the gain and the row's scale stay outside in fp32;
//   * products run on mma.sync m16n8k16, tokens x heads for the scores, channels x heads for the values.  The contraction order
//     of the scores is free, so lane (g, j) reads chain j of tokens g and g + 8, and for the values half a chain of four tokens: every
//     window offset is a compile-time constant per code width;
//   * a query row is bf16 or fp16: brought to a maximum of 2^13 .. 2^14 by a power of two it is exact in fp16 (what lies 2^38 below that maximum
//     apart), and power, qscale and log2(e) are put on the fp32 score;
//   * a weight (probability x row scale x gain) enters as two fp16 numbers (two MMAs), an integer of up to 2^11 and the rest, after a power of two
//     of its head (and warp) that keeps the largest weight of the sum between 2^9 and 2^11; an error of at most 2^-13 of that unit.  The power moves with
//     the running maximum, and when a weight outgrows it, and leaves the sums in the merge entry.  Without it small values (row scale 0.01: 4e-3
//     of the result) sat among fp16's subnormals and large flat ones overflowed;
//   * the tensor core's accumulators truncate: a tile's products are summed on their own and added in rounded fp32, and the integer part of the weights makes its
//     sum exact (below 2^24).  Carried from tile to tile the error grew with their number (2.3e-6 of a row at 30,011 tokens in 37 splits, 1e-4 in
//     one), with a rounded fp16 in the place of the integer a bias of half a unit was left.  Error of a row against 64 bits, rms over 500 .. 32,768
//     tokens in 37 splits: 2.9e-7 .. 4.6e-7, of a scalar fp32 loop over the same rows 4.9e-7 .. 7.1e-7;
//   * the row terms of the unpack rule leave the loops: q.x = s * gain / 256 * sum_d q_d code_d + c0 (q.U0) + c1 (q.U1) + q.mu, and
//     O = sum_t p_t s_t code_t + (sum p_t c0_t) U0 + (sum p_t c1_t) U1 + (sum p_t) mu.
// Rows that the profile leaves unpacked (positions below the guard, at most 255; a group without packed rows) take the row path, a warp
// per token in fp32.  32,768 tokens of 4 kv-heads on a B200: 152 us (32 keys per warp step in scalar fp32, tables in shared memory with
// bank conflicts) -> 33.9 us, of which 14 are set-up, merge and the launch.
constexpr int TBA_WARPS = 12;                                        // 3 per scheduler at up to 168 registers
struct TbAttnP { yskn_tb_attn_args a; int G; };
constexpr uint32_t TBA_TAB = 32768;                                  // bytes of a replicated table, and the alignment of its shared-memory address
struct TbAttnSm {                                                    // in front of the tables
  uint2 qf[16][32];                                                  // Q x its head's power of two as B fragments of k-step s, lane
  float q[8][260];                                                   // q in fp32 (row path, row terms)
  float cg[2][256];                                                  // codes of the key and of the value group (row path: x gain)
  float term[2][3][256];                                             // row terms U0, U1, mu of both groups, channel d at tba_slot(d)
  float kq[4][8];                                                    // q.U0, q.U1, q.mu of the key group, x qscale * log2(e); that over the power of two in qf
  int qmax[8];                                                       // largest |q| of a head, as bits
  int big;                                                           // some code does not fit fp16 exactly
};
constexpr int TBA_MS = 260;                                          // merge entry of a (warp, head): m, l, -, -, then channel d at tba_slot(d)
constexpr uint32_t TBA_MERGE = TBA_WARPS * 8 * TBA_MS * 4;           // merge area: takes the tables' place after the loop
constexpr uint32_t TBA_SMEM = sizeof(TbAttnSm) + TBA_TAB + (TBA_MERGE > 2 * TBA_TAB ? TBA_MERGE : 2 * TBA_TAB);     // one TBA_TAB for the alignment

struct TbRule { int packed_ok, mode, kb, guard, m, has_mu; float gain; };     // per-group constants of the unpack rule

__device__ __forceinline__ uint32_t tba_lds(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t tba_pack(float lo, float hi) { uint32_t d; asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo)); return d; }
__device__ __forceinline__ void tba_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Powers of two from 2^-120 to 2^120 by exponent; the exponent of a number (zero and subnormals: -127, infinities: 128).
constexpr int TBA_EXP = 120;
__device__ __forceinline__ int tba_exponent(float x) { return (int)((__float_as_uint(x) >> 23) & 255u) - 127; }
__device__ __forceinline__ float tba_pow2(int e) { return __uint_as_float((unsigned)(min(max(e, -TBA_EXP), TBA_EXP) + 127) << 23); }
__device__ __forceinline__ float tba_inverse(float pow2) { return __uint_as_float((254u << 23) - __float_as_uint(pow2)); }
__device__ __forceinline__ uint32_t tba_transpose(uint32_t a) { uint32_t d; asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a)); return d; }

// Where channel d sits in a merge entry and in the row terms: the eight lanes g of an access (channels 32g + c) fall into eight banks, the
// four lanes j of a merge store (heads 2j, 520 words apart) into four groups of eight.  (Channels in order: 8-way conflicts, 10 us.)
__device__ __forceinline__ int tba_slot(int d) { return (d & 31) * 8 + (d >> 5); }

// The window of value i of a run of fields that starts at word 0 (`prev` = the word in front, zero at the start of a chain), at bits
// 7 .. 14: the byte offset of its table row.
template <int KB, int NWORD> __device__ __forceinline__ uint32_t tba_window(const uint32_t (&w)[NWORD], uint32_t prev, int i) {
  const int lo = KB * (i + 1) - 8;                                   // first bit of the window in the MSB-first stream; negative: in `prev`
  const int k = lo >> 5, o = lo & 31;                                // floor
  const uint32_t hi = k < 0 ? prev : w[k < 0 ? 0 : k];
  if (o > 24) return __funnelshift_r(w[k + 1 < NWORD ? k + 1 : NWORD - 1], hi, 49 - o);
  return o <= 17 ? hi >> (17 - o) : hi << (o - 17);
}

// Words of a run of fields: NWORD consecutive 32-bit words.  v16: rows are 16-byte aligned (then so are the runs of 4-bit codes).
template <int NWORD> __device__ __forceinline__ void tba_words(const uint32_t* p, bool v16, uint32_t (&w)[NWORD]) {
  if (NWORD % 4 == 0 && v16) {
    #pragma unroll
    for (int k = 0; k < NWORD / 4; ++k) {
      const uint4 u = reinterpret_cast<const uint4*>(p)[k];
      w[(4 * k) % NWORD] = u.x; w[(4 * k + 1) % NWORD] = u.y; w[(4 * k + 2) % NWORD] = u.z; w[(4 * k + 3) % NWORD] = u.w;
    }
  } else {
    #pragma unroll
    for (int k = 0; k < NWORD; ++k) w[k] = p[k];
  }
}

// Raw scores of a tile's 16 tokens: rows g and g + 8 of the tile, heads 2j and 2j + 1 (c[0] c[1] | c[2] c[3]).
template <int KB>
__device__ __forceinline__ void tba_scores(const uint32_t* ra, const uint32_t* rb, bool v16, uint32_t tab, const uint2* qf, float (&s)[4]) {
  uint32_t wa[2 * KB], wb[2 * KB];
  tba_words(ra, v16, wa); tba_words(rb, v16, wb);
  float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};      // two chains
  #pragma unroll
  for (int k = 0; k < 16; ++k) {                                     // k-step: values 4k .. 4k+3 of the chain
    uint32_t a[4], b[4];
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
      a[e] = tba_lds((tba_window<KB>(wa, 0u, 4 * k + e) & 0x7F80u) | tab);
      b[e] = tba_lds((tba_window<KB>(wb, 0u, 4 * k + e) & 0x7F80u) | tab);
    }
    const uint2 q = qf[k * 32];
    tba_mma(c[k & 1], __byte_perm(a[0], a[1], 0x5410), __byte_perm(b[0], b[1], 0x5410), __byte_perm(a[2], a[3], 0x5410), __byte_perm(b[2], b[3], 0x5410),
            q.x, q.y);
  }
  #pragma unroll
  for (int e = 0; e < 4; ++e) s[e] = c[0][e] + c[1][e];
}

// O^T += V^T P^T over a tile: this lane's 32 channels (half a chain) of tokens 2j, 2j+1, 2j+8, 2j+9 (rows r[0..3]).
template <int KB>
__device__ __forceinline__ void tba_values(const uint32_t* const (&r)[4], bool odd, bool v16, uint32_t tab, const uint32_t (&ph)[2], const uint32_t (&pl)[2],
                                           float (&acc)[16][4]) {
  uint32_t w[4][KB], prev[4];
  #pragma unroll
  for (int t = 0; t < 4; ++t) { tba_words(r[t], v16, w[t]); prev[t] = odd ? r[t][-1] : 0u; }
  #pragma unroll
  for (int mt = 0; mt < 16; ++mt) {                                  // m-tile: channels 2 mt and 2 mt + 1 of the run as rows g and g + 8
    uint32_t x[2][4];
    #pragma unroll
    for (int c = 0; c < 2; ++c)
      #pragma unroll
      for (int t = 0; t < 4; ++t) x[c][t] = tba_lds((tba_window<KB>(w[t], prev[t], 2 * mt + c) & 0x7F80u) | tab);
    const uint32_t a0 = __byte_perm(x[0][0], x[0][1], 0x5410), a1 = __byte_perm(x[1][0], x[1][1], 0x5410), a2 = __byte_perm(x[0][2], x[0][3], 0x5410),
                   a3 = __byte_perm(x[1][2], x[1][3], 0x5410);
    float ch[4] = {0.f, 0.f, 0.f, 0.f}, cl[4] = {0.f, 0.f, 0.f, 0.f};
    tba_mma(ch, a0, a1, a2, a3, ph[0], ph[1]);
    tba_mma(cl, a0, a1, a2, a3, pl[0], pl[1]);
    #pragma unroll
    for (int e = 0; e < 4; ++e) acc[mt][e] += ch[e] + cl[e];
  }
}

// Value d of a row on its own (tb_unpack_kernel's rule), as its code.
__device__ __forceinline__ float tba_value(const uint32_t* row, const float* cg, int kb, int d) {
  const int endb = kb * (d + 1), lo = max(endb - 8, kb * (d & ~63));
  const uint32_t w0 = row[lo >> 5], w1 = (lo & 31) + (endb - lo) > 32 ? row[(lo >> 5) + 1] : 0u;
  return cg[__funnelshift_l(w1, w0, lo & 31) >> (32 - (endb - lo))];
}

template <int DT>
__global__ void __launch_bounds__(TBA_WARPS * 32, 1) tb_attn_kernel(TbAttnP P) {
  extern __shared__ __align__(16) unsigned char tba_smem[];
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(tba_smem);
  const uint32_t TK = (base + (uint32_t)sizeof(TbAttnSm) + TBA_TAB - 1) & ~(TBA_TAB - 1), TV = TK + TBA_TAB;
  const yskn_tb_attn_args& A = P.a;
  const int G = P.G, split = blockIdx.x, kvh = blockIdx.y, r = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  TbAttnSm& S = *reinterpret_cast<TbAttnSm*>(tba_smem);
  float* mbuf = reinterpret_cast<float*>(tba_smem + (TK - base));          // [warp][8][TBA_MS]
  asm volatile("griddepcontrol.wait;" ::: "memory");                 // programmatic dependent launch, both directions
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const float qs = A.qscale * 1.4426950408889634f;
  const int pos = *A.d_pos + r, len = max(0, min(pos + 1, A.max_ctx));
  const int per = (len + (int)gridDim.x - 1) / (int)gridDim.x, t0 = min(len, split * per), t1 = min(len, t0 + per);
  const size_t row0 = (size_t)kvh * A.max_ctx;
  const int psw = A.pay_stride / 4;
  const uint32_t *kpay = reinterpret_cast<const uint32_t*>(A.k_pay) + row0 * psw, *vpay = reinterpret_cast<const uint32_t*>(A.v_pay) + row0 * psw;
  auto prefetch = [&](int tc) {                                      // the rows of a tile into L2: a row per lane, keys 0-15, values 16-31
    const int t = tc + (lane & 15);
    if (t >= t1) return;
    const uint32_t* p = (lane < 16 ? kpay : vpay) + (size_t)t * psw;
    asm volatile("prefetch.global.L2 [%0];\n prefetch.global.L2 [%1];" ::"l"(p), "l"(p + 31));
    if (!(lane & 15)) asm volatile("prefetch.global.L2 [%0];" ::"l"((lane < 16 ? A.k_side : A.v_side) + 2 * (row0 + t)));
  };
  // ---- set-up.  The profile is a chain of five dependent reads (header, group offset, record, table offset, table); both groups walk it side by
  //      side and everything at its end is requested at once (one group after the other, entry by entry, took 20 us).
  constexpr int NQ = (256 * 8 + TBA_WARPS * 32 - 1) / (TBA_WARPS * 32);
  float qv[NQ];                                                      // on their way while the chain is walked
  #pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const int e = threadIdx.x + k * TBA_WARPS * 32, h = e >> 8, d = e & 255;
    qv[k] = h < G ? act_load<DT>(A.q16, ((size_t)r * A.nh + kvh * G + h) * 256 + d) : 0.f;
  }
  const int gk = A.grp_k[kvh], gv = A.grp_v[kvh];
  prefetch(t0 + 16 * warp);                                          // (waits for the position: behind the first loads of the chain)
  if (threadIdx.x == 0) S.big = 0;
  if (threadIdx.x < 8) S.qmax[threadIdx.x] = 0;
  TbRule rk, rv;
  {
    const TbGroup Pg[2] = {tb_group(A.blob, gk), tb_group(A.blob, gv)};
    unsigned to[2];
    #pragma unroll
    for (int w = 0; w < 2; ++w) to[w] = tb_table(A.blob, Pg[w]);
    float gain[2];
    #pragma unroll
    for (int w = 0; w < 2; ++w) gain[w] = tb_f32(A.blob + to[w] + 4);        // (no table: not used)
    const int i = threadIdx.x;
    float x[2][4];                                                   // code, U0, U1, mu of entry / channel i
    #pragma unroll
    for (int w = 0; w < 2; ++w) {
      const TbGroup& R = Pg[w];
      const uint8_t* mup = A.blob + R.go + 8;
      const uint8_t* Up = mup + (R.has_mu ? 512 : 0);
      const bool pk = R.ok && R.mode <= 1 && i < 256;
      auto f16at = [&](const uint8_t* p) { return __half2float(__ushort_as_half((unsigned short)tb_u16(p))); };
      // a flat code of 4 bits is the low half of the 8-bit window: flat groups use the same windows with a periodic table
      x[w][0] = !pk ? 0.f : R.mode == 1 ? (float)((i & 15) - 8) : (float)(short)tb_u16(A.blob + to[w] + 12 + 2 * i);
      x[w][1] = pk && R.m > 0 ? f16at(Up + 2 * i) : 0.f;
      x[w][2] = pk && R.m > 1 ? f16at(Up + 512 + 2 * i) : 0.f;
      x[w][3] = pk && R.has_mu ? f16at(mup + 2 * i) : 0.f;
    }
    #pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int e = threadIdx.x + k * TBA_WARPS * 32;
      if (e < 256 * 8) S.q[e >> 8][e & 255] = qv[k];
    }
    __syncthreads();                                                 // S.big and S.qmax are cleared
    #pragma unroll
    for (int k = 0; k < NQ; ++k) {                                   // a warp's 32 entries are of one head
      const int h = (threadIdx.x + k * TBA_WARPS * 32) >> 8, top = __reduce_max_sync(0xffffffffu, __float_as_int(qv[k]) & 0x7fffffff);
      if (h < 8 && lane == 0) atomicMax(&S.qmax[h], top);
    }
    if (i < 256)
      #pragma unroll
      for (int w = 0; w < 2; ++w) {
        S.cg[w][i] = x[w][0];
        #pragma unroll
        for (int k = 0; k < 3; ++k) S.term[w][k][tba_slot(i)] = x[w][1 + k];
        if (fabsf(x[w][0]) > 2048.f) S.big = 1;
      }
    rk = TbRule{Pg[0].ok && Pg[0].mode <= 1, Pg[0].mode, Pg[0].mode == 1 ? 4 : Pg[0].kk, Pg[0].guard, Pg[0].m, Pg[0].has_mu, Pg[0].mode == 0 ? gain[0] * 0.00390625f : 1.f};
    rv = TbRule{Pg[1].ok && Pg[1].mode <= 1, Pg[1].mode, Pg[1].mode == 1 ? 4 : Pg[1].kk, Pg[1].guard, Pg[1].m, Pg[1].has_mu, Pg[1].mode == 0 ? gain[1] * 0.00390625f : 1.f};
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * 256 * 8; e += TBA_WARPS * 32) {  // thread = (table, state, four lanes)
    const int w = e >> 11, st = (e >> 3) & 255, l4 = (e & 7) * 4;
    const uint32_t h = __half_as_ushort(__float2half_rn(S.cg[w][st])), v = h | (h << 16);
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"((w ? TV : TK) + st * 128 + l4 * 4), "r"(v) : "memory");
  }
  if (threadIdx.x < 8) S.kq[3][threadIdx.x] = qs * tba_inverse(tba_pow2(13 - tba_exponent(__int_as_float(S.qmax[threadIdx.x]))));
  for (int i = warp; i < 24; i += TBA_WARPS) {                       // q.U0, q.U1, q.mu of each head, a warp per product
    const int which = i >> 3, h = i & 7;
    float a = 0.f;
    #pragma unroll
    for (int k = 0; k < 8; ++k) a = fmaf(S.q[h][32 * k + lane], S.term[0][which][tba_slot(32 * k + lane)], a);
    #pragma unroll
    for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) S.kq[which][h] = a * qs;
  }
  for (int e = threadIdx.x; e < 16 * 32; e += TBA_WARPS * 32) {      // k-slots (2j, 2j+1, 2j+8, 2j+9) of step s = channels 64j + 4s .. + 3
    const int s = e >> 5, ln = e & 31, h = ln >> 2, c = 64 * (ln & 3) + 4 * s;
    const float f = tba_pow2(13 - tba_exponent(__int_as_float(S.qmax[h])));
    S.qf[s][ln] = make_uint2(tba_pack(S.q[h][c] * f, S.q[h][c + 1] * f), tba_pack(S.q[h][c + 2] * f, S.q[h][c + 3] * f));
  }
  __syncthreads();
  // tokens below tf take the row path: either side unpacked there, or codes that fp16 does not hold
  const int tf = rk.packed_ok && rv.packed_ok && !S.big ? min(t1, max(t0, max(rk.guard, rv.guard))) : t1;
  // Rows that stay unpacked (the first tokens of a sequence) come from fp32 rows nobody has touched: asked into L2 here, read behind the tiles.
  if (t0 + warp < min(tf, t0 + TBA_WARPS) && lane < 16) {
    const float* const plain = lane < 8 ? A.k_plain : A.v_plain;
    if (plain) asm volatile("prefetch.global.L2 [%0];" ::"l"(plain + (row0 + t0 + warp) * 256 + 32 * (lane & 7)));
  }
  const bool v16 = !((A.pay_stride | (int)((uintptr_t)A.k_pay | (uintptr_t)A.v_pay)) & 15);
  const uint2* qf = &S.qf[0][lane];
  const uint32_t tabk = TK | (lane * 4), tabv = TV | (lane * 4);

  float acc[16][4];                                                  // O^T: [m-tile][(channel 32g + 2 mt | + 1) x (head 2j | 2j + 1)]
  #pragma unroll
  for (int mt = 0; mt < 16; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f;
  // heads 2j, 2j+1 (log2 domain); l (of packed values: the mean row's weight too) and the sums of p c0, p c1 are this lane's share of the tokens
  float m[2] = {-1e30f, -1e30f}, l[2] = {0.f, 0.f}, a0[2] = {0.f, 0.f}, a1[2] = {0.f, 0.f};
  float u[2] = {tba_pow2(TBA_EXP), tba_pow2(TBA_EXP)};               // acc holds sum x u
  auto side = [&](const uint32_t* sd, int t, int mm, float& s, float& c0, float& c1) {
    s = __uint_as_float(sd[2 * (row0 + t)]);
    const uint32_t pc = sd[2 * (row0 + t) + 1];
    c0 = mm > 0 ? __half2float(__ushort_as_half((unsigned short)(pc & 0xffffu))) : 0.f;
    c1 = mm > 1 ? __half2float(__ushort_as_half((unsigned short)(pc >> 16))) : 0.f;
  };
  for (int tc = tf + 16 * warp; tc < t1; tc += 16 * TBA_WARPS) {
    prefetch(tc + 16 * TBA_WARPS);
    const bool live0 = tc + g < t1, live1 = tc + g + 8 < t1;
    const int ta = min(tc + g, t1 - 1), tb = min(tc + g + 8, t1 - 1);  // tokens past the end repeat the last one with weight zero
    float ks[2], kc0[2], kc1[2], vs[2], vc0[2], vc1[2];
    side(A.k_side, ta, rk.m, ks[0], kc0[0], kc1[0]); side(A.k_side, tb, rk.m, ks[1], kc0[1], kc1[1]);
    side(A.v_side, ta, rv.m, vs[0], vc0[0], vc1[0]); side(A.v_side, tb, rv.m, vs[1], vc0[1], vc1[1]);
    if (!live0) vs[0] = vc0[0] = vc1[0] = 0.f;
    if (!live1) vs[1] = vc0[1] = vc1[1] = 0.f;
    float s[4];
    {
      const uint32_t *pa = kpay + (size_t)ta * psw + j * 2 * rk.kb, *pb = kpay + (size_t)tb * psw + j * 2 * rk.kb;
      if (rk.kb == 4) tba_scores<4>(pa, pb, v16, tabk, qf, s);
      else if (rk.kb == 5) tba_scores<5>(pa, pb, v16, tabk, qf, s);
      else tba_scores<3>(pa, pb, v16, tabk, qf, s);
    }
    float p[2][2];                                                   // [row g | g + 8][head]
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
      const volatile float* kq = &S.kq[0][2 * j + h];                // read per tile: the registers are needed for the sums
      const float kq0 = kq[0], kq1 = kq[8], kqm = kq[16], qu = kq[24];
      const float sa = fmaf(ks[0] * rk.gain, s[h] * qu, fmaf(kc0[0], kq0, fmaf(kc1[0], kq1, kqm)));
      const float sb = fmaf(ks[1] * rk.gain, s[2 + h] * qu, fmaf(kc0[1], kq0, fmaf(kc1[1], kq1, kqm)));
      p[0][h] = live0 ? sa : -INFINITY; p[1][h] = live1 ? sb : -INFINITY;
    }
    float x0 = fmaxf(p[0][0], p[1][0]), x1 = fmaxf(p[0][1], p[1][1]), f0 = 1.f, f1 = 1.f;
    const bool bump = __any_sync(0xffffffffu, x0 > m[0] + 8.f || x1 > m[1] + 8.f);     // lazy rescale: the running max may lag by 2^8
    if (bump) {
      #pragma unroll
      for (int o = 4; o <= 16; o <<= 1) { x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, o)); x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o)); }
      const float n0 = fmaxf(m[0], x0), n1 = fmaxf(m[1], x1);
      f0 = exp2f(m[0] - n0); f1 = exp2f(m[1] - n1);
      m[0] = n0; m[1] = n1;
      l[0] *= f0; a0[0] *= f0; a1[0] *= f0; l[1] *= f1; a0[1] *= f1; a1[1] *= f1;
    }
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
      p[0][h] = exp2f(p[0][h] - m[h]); p[1][h] = exp2f(p[1][h] - m[h]);
      l[h] += p[0][h] + p[1][h];
      a0[h] = fmaf(p[0][h], vc0[0], fmaf(p[1][h], vc0[1], a0[h])); a1[h] = fmaf(p[0][h], vc1[0], fmaf(p[1][h], vc1[1], a1[h]));
    }
    float w[2][2];                                                   // weights
    #pragma unroll
    for (int h = 0; h < 2; ++h) { w[0][h] = p[0][h] * (vs[0] * rv.gain); w[1][h] = p[1][h] * (vs[1] * rv.gain); }
    float w0 = fmaxf(fabsf(w[0][0]), fabsf(w[1][0])), w1 = fmaxf(fabsf(w[0][1]), fabsf(w[1][1]));
    if (bump || __any_sync(0xffffffffu, w0 * u[0] > 2048.f || w1 * u[1] > 2048.f)) {       // the powers of two follow the largest weight of the sum
      #pragma unroll
      for (int o = 4; o <= 16; o <<= 1) { w0 = fmaxf(w0, __shfl_xor_sync(0xffffffffu, w0, o)); w1 = fmaxf(w1, __shfl_xor_sync(0xffffffffu, w1, o)); }
      const float b0 = 512.f * tba_inverse(u[0]) * f0, b1 = 512.f * tba_inverse(u[1]) * f1;  // the weight u was made for, under the new maximum
      const float n0 = tba_pow2(9 - tba_exponent(fmaxf(w0, b0))), n1 = tba_pow2(9 - tba_exponent(fmaxf(w1, b1)));
      f0 *= tba_inverse(u[0]); f1 *= tba_inverse(u[1]);
      u[0] = n0; u[1] = n1;
      #pragma unroll
      for (int mt = 0; mt < 16; ++mt) {                              // two factors: their product may leave the range of a float
        acc[mt][0] = acc[mt][0] * f0 * n0; acc[mt][1] = acc[mt][1] * f1 * n1; acc[mt][2] = acc[mt][2] * f0 * n0; acc[mt][3] = acc[mt][3] * f1 * n1;
      }
    }
    uint32_t ph[2], pl[2];                                           // weights x u, whole part and rest, transposed into B registers
    #pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float y0 = w[q][0] * u[0], y1 = w[q][1] * u[1];
      const float h0 = rintf(y0), h1 = rintf(y1);
      ph[q] = tba_transpose(tba_pack(h0, h1));
      pl[q] = tba_transpose(tba_pack(isinf(h0) ? 0.f : y0 - h0, isinf(h1) ? 0.f : y1 - h1));      // an infinite row scale stays infinite
    }
    const int tv[4] = {min(tc + 2 * j, t1 - 1), min(tc + 2 * j + 1, t1 - 1), min(tc + 2 * j + 8, t1 - 1), min(tc + 2 * j + 9, t1 - 1)};
    const uint32_t* vr[4];
    #pragma unroll
    for (int q = 0; q < 4; ++q) vr[q] = vpay + (size_t)tv[q] * psw + g * rv.kb;
    if (rv.kb == 4) tba_values<4>(vr, g & 1, v16, tabv, ph, pl, acc);
    else if (rv.kb == 5) tba_values<5>(vr, g & 1, v16, tabv, ph, pl, acc);
    else tba_values<3>(vr, g & 1, v16, tabv, ph, pl, acc);
  }
  // ---- this warp's (m, l, O) per head into the merge area (the tables' place); the row terms of the value group added
  #pragma unroll
  for (int o = 4; o <= 16; o <<= 1)
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], o); a0[h] += __shfl_xor_sync(0xffffffffu, a0[h], o);
      a1[h] += __shfl_xor_sync(0xffffffffu, a1[h], o);
    }
  __syncthreads();
  float* wb = mbuf + (size_t)warp * 8 * TBA_MS;
  #pragma unroll
  for (int mt = 0; mt < 16; ++mt)
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int h = e & 1, d = 32 * g + 2 * mt + (e >> 1);
      wb[(2 * j + h) * TBA_MS + 4 + tba_slot(d)] =
          fmaf(a0[h], S.term[1][0][tba_slot(d)], fmaf(a1[h], S.term[1][1][tba_slot(d)], fmaf(l[h], S.term[1][2][tba_slot(d)], acc[mt][e] * tba_inverse(u[h]))));
    }
  if (g == 0) {
    #pragma unroll
    for (int h = 0; h < 2; ++h) { wb[(2 * j + h) * TBA_MS] = m[h]; wb[(2 * j + h) * TBA_MS + 1] = l[h]; }
  }
  __syncwarp();
  // ---- the row path: a token per warp step, lane = channels 32 k + lane, fp32 throughout, straight into the warp's merge entry.  Only the first split has
  //      such tokens as a rule (those below the guard), and the pass waits for it: with its two rows read one after the other from memory and a barrier a
  //      head it took 5 us of a pass of 39.6 over 30,011 tokens; asked into L2 ahead and read together 37.9 (2,000 tokens 19.0 -> 17.4).
  for (int t = t0 + warp; t < tf; t += TBA_WARPS) {
    const bool kpk = rk.packed_ok && t >= rk.guard, vpk = rv.packed_ok && t >= rv.guard;
    float s0, c0, c1, x[8], y[8];                                    // key and value row, both on their way before either is used
    #pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int d = 32 * k + lane;
      if (!kpk) x[k] = A.k_plain ? A.k_plain[(row0 + t) * 256 + d] : 0.f;
      if (!vpk) y[k] = A.v_plain ? A.v_plain[(row0 + t) * 256 + d] : 0.f;
    }
    if (vpk) {
      side(A.v_side, t, rv.m, s0, c0, c1);
      #pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int d = 32 * k + lane, i = tba_slot(d);
        y[k] = fmaf(c0, S.term[1][0][i], fmaf(c1, S.term[1][1][i], fmaf(tba_value(vpay + (size_t)t * psw, S.cg[1], rv.kb, d) * rv.gain, s0, S.term[1][2][i])));
      }
    }
    if (kpk) {
      side(A.k_side, t, rk.m, s0, c0, c1);
      #pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = tba_value(kpay + (size_t)t * psw, S.cg[0], rk.kb, 32 * k + lane) * rk.gain * s0;
    }
    float sc[8], mo[8], lo[8];
    #pragma unroll
    for (int h = 0; h < 8; ++h) {
      float a = 0.f;
      #pragma unroll
      for (int k = 0; k < 8; ++k) a = fmaf(S.q[h][32 * k + lane], x[k], a);
      #pragma unroll
      for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      a *= qs;
      sc[h] = kpk ? a + fmaf(c0, S.kq[0][h], fmaf(c1, S.kq[1][h], S.kq[2][h])) : a;
      mo[h] = wb[h * TBA_MS]; lo[h] = wb[h * TBA_MS + 1];
    }
    __syncwarp();                                                    // every lane has read m and l
    #pragma unroll
    for (int h = 0; h < 8; ++h) {
      if (h >= G) break;
      float* e = wb + h * TBA_MS;
      const float mn = fmaxf(mo[h], sc[h]), f = exp2f(mo[h] - mn), pw = exp2f(sc[h] - mn);
      if (lane == 0) { e[0] = mn; e[1] = fmaf(lo[h], f, pw); }
      #pragma unroll
      for (int k = 0; k < 8; ++k) e[4 + tba_slot(32 * k + lane)] = fmaf(e[4 + tba_slot(32 * k + lane)], f, pw * y[k]);   // a lane's own eight entries
    }
    __syncwarp();
  }
  // ---- the merge of the warps (natural-log m, as the merge kernel expects)
  __syncthreads();
  if (threadIdx.x < 8 * TBA_WARPS) {                                 // the warps' weights, and the row's m and l
    const int h = threadIdx.x / TBA_WARPS, w = threadIdx.x % TBA_WARPS;
    float M2 = -1e30f;
    #pragma unroll
    for (int k = 0; k < TBA_WARPS; ++k) M2 = fmaxf(M2, mbuf[((size_t)k * 8 + h) * TBA_MS]);
    const float mw = mbuf[((size_t)w * 8 + h) * TBA_MS];
    S.q[h][w] = mw > -1e29f ? exp2f(mw - M2) : 0.f;                  // the queries are done with
    if (w == 0) S.q[h][TBA_WARPS] = M2;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < G * 256; e += TBA_WARPS * 32) {
    const int h = e >> 8, i = e & 255, d = (i & 7) * 32 + (i >> 3);  // entries in their order: tba_slot(d) = i
    float L2 = 0.f, o = 0.f;
    #pragma unroll
    for (int w = 0; w < TBA_WARPS; ++w) {
      const float* src = mbuf + ((size_t)w * 8 + h) * TBA_MS;
      const float f = S.q[h][w];
      L2 += f * src[1]; o += f * src[4 + i];
    }
    const size_t pidx = ((size_t)r * A.splits + split) * A.nh + kvh * G + h;
    const float M2 = S.q[h][TBA_WARPS];
    if (i == 0) { A.pm[pidx] = M2 > -1e29f ? M2 * 0.6931471805599453f : -1e30f; A.pl[pidx] = L2; }
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
                     uint32_t* side, int whole, cudaStream_t st) {
  if (!blob || !x || !grp || !pos) KV4_REJECT("yskn_tb_encode: null buffer");
  if (rows <= 0 || nm < 1 || nm > TB_NM) KV4_REJECT("yskn_tb_encode: bad shape (rows %d, multipliers %d)", rows, nm);
  if (pay && (pay_stride < 160 || pay_stride % 4 || ((uintptr_t)pay & 3))) KV4_REJECT("yskn_tb_encode: payload rows need a stride of at least 160 bytes, a multiple of 4");
  static std::atomic<unsigned long long> attr{0};
  if (first_use_on_device(attr)) {
    KV4_CUDA(cudaFuncSetAttribute(tb_encode_kernel<TB_WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TbRowSmem::bytes(TB_NM, TB_WIDE)));
    KV4_CUDA(cudaFuncSetAttribute(tb_encode_kernel<TB_NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TbRowSmem::bytes(TB_NM, TB_NARROW)));
    KV4_CUDA(cudaFuncSetAttribute(tb_encode_kernel<TB_ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TbRowSmem::bytes(1, TB_ONE)));
  }
  const TbP P{blob, nm, x, grp, pos, rows, y, pay, pay_stride, side, whole};
  const int most = nm == 1 ? TB_ONE : rows <= TB_WIDE_ROWS ? TB_WIDE : TB_NARROW;
  auto kern = most == TB_ONE ? tb_encode_kernel<TB_ONE> : most == TB_WIDE ? tb_encode_kernel<TB_WIDE> : tb_encode_kernel<TB_NARROW>;
  kern<<<rows, 32 * TbRowSmem::warps(nm, most), TbRowSmem::bytes(nm, most), st>>>(P);
  return launch_status("tb_encode_kernel");
}

int launch_tb_attention(const yskn_tb_attn_args& a, int act_dtype, cudaStream_t st) {
  if (!a.q16 || !a.blob || !a.k_pay || !a.v_pay || !a.k_side || !a.v_side || !a.grp_k || !a.grp_v || !a.d_pos || !a.pm || !a.pl || !a.pacc)
    KV4_REJECT("yskn_tb_attention: null buffer");
  if (a.kvh <= 0 || a.nh <= 0 || a.nh % a.kvh || a.nh / a.kvh > 8 || a.M <= 0 || a.M > 65535 || a.kvh > 65535 || a.splits <= 0 || a.max_ctx <= 0)
    KV4_REJECT("yskn_tb_attention: bad shape (kvh %d, nh %d, M %d, splits %d, max_ctx %d): at most 8 query heads per kv-head", a.kvh, a.nh, a.M, a.splits, a.max_ctx);
  if (a.pay_stride < 160 || a.pay_stride % 4 || (((uintptr_t)a.k_pay | (uintptr_t)a.v_pay) & 3)) KV4_REJECT("yskn_tb_attention: bad payload stride %d or alignment", a.pay_stride);
  const int smem = (int)TBA_SMEM;
  TbAttnP P{a, a.nh / a.kvh};
  const dim3 grid(a.splits, a.kvh, a.M);
  if (act_dtype == YSKN_KV4_BF16) {
    static std::atomic<unsigned long long> attr{0};
    if (first_use_on_device(attr)) KV4_CUDA(cudaFuncSetAttribute(tb_attn_kernel<YSKN_KV4_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return launch_pdl("tb_attn_kernel", tb_attn_kernel<YSKN_KV4_BF16>, grid, TBA_WARPS * 32, smem, st, P);
  }
  if (act_dtype == YSKN_KV4_F16) {
    static std::atomic<unsigned long long> attr{0};
    if (first_use_on_device(attr)) KV4_CUDA(cudaFuncSetAttribute(tb_attn_kernel<YSKN_KV4_F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return launch_pdl("tb_attn_kernel", tb_attn_kernel<YSKN_KV4_F16>, grid, TBA_WARPS * 32, smem, st, P);
  }
  KV4_REJECT("yskn_tb_attention: q16 is bf16 or fp16 (act_dtype %d)", act_dtype);
}

}  // namespace kv4
