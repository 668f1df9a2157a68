// KV4 GQA flash-decode for sm_100a: TMA-staged packed cache, int4 -> fp16 in registers, warp-level
// tensor-core tiles, online softmax by warp shuffles, split-K partials.
//
// Semantics: the reference's attention_gqa_kernel (src/attention_gqa.cu:17-118) -- row r at *d_pos + r sees keys
// 0..pos; 32-token groups before the row's own group are read as int4 (k = nib*scale + zero), the own group from
// the fp16 shadow; K is rotated at read time; V is int4 per token; output = (m, l, un-normalised O) per split.
// Results agree with the reference to the attention tolerance, not bit for bit: the split boundaries are whole
// 32-token groups and the products run on tensor cores with fp16 operands.
//
// Why tensor cores for an HBM-bound kernel: one cached token costs 292 bytes but 2*G*HD = 3072 multiply-adds
// (G 6, HD 256); at 75 % of HBM bandwidth that is ~50 T multiply-adds/s, more than the fp32 pipes deliver.
//
// Work split.  grid (splits, Hkv, M), one CTA per SM when splits*Hkv*M = 148.  A CTA owns a run of 128-token units
// (four 32-token groups) of one kv-head.  One producer warp streams each unit into an mbarrier ring with seven
// copies: K 128 x HD/2 bytes and V 128 x HD/2 bytes by tiled TMA (128-byte swizzle), four K scale rows, four K zero
// rows, 128 V scales, 128 V zeros (tiles; bulk copies in a multi-request pass) and the four rope rows of the groups' first
// positions (one strided TMA tile).  Few, large copies matter: the number of copies in flight per SM is limited, not only their bytes.
// Seven consumer warps take the groups round-robin and keep their own (m, l, O) state.  A group is two 16-token
// MMA tiles:
//   S^T[16 tok x 8 heads]  = K[16 tok x HD] . Q^T[HD x 8 heads]          (m16n8k16, HD/16 steps)
//   O^T[HD x 8 heads]     += V^T[HD x 16 tok] . P^T[16 tok x 8 heads]    (HD/16 m-tiles)
// so one K/V tile serves all G <= 8 query heads of the group, and the packed bytes go from shared memory straight
// into A-fragment registers:
//   * a 32-bit word holds 8 nibbles; one AND reads nibbles (x, x+4) in place as two fp16 subnormals, n * 2^-24 at bits 0..3 of a
//     half, n * 2^-20 at bits 4..7: exactly one A register, because the contraction order over channels is free.  The tensor core
//     forms products with subnormals exactly, so the factor is taken out of the fp32 sum (one accumulator per factor); it aligns them
//     for the sum by the exponent 2^-14 of a subnormal, though, not by their leading bit, see V.  K's per-channel scale is folded into Q
//     once per group (q' = q*scale); the zero points become a per-head bias, sum q*zero, formed by two more MMA rows.
//   * for V the contraction runs over tokens: a transposed 8x8 shared-memory load (ldmatrix.trans) hands a lane the same
//     four channels of two consecutive tokens in one register, which is the pairing an A register wants.  V's per-token
//     scale is folded into P and its zero point into a per-head scalar.  No offset may ride along in these sums: the tensor
//     core's fp32 accumulators truncate, and one that carried 1024 * sum(p) lost about 2e-3 of the output at 262,144 tokens.
//     A warp's sum of O runs over up to 1,000 tokens, so the truncation at the alignment above counts here, and the nibbles are read
//     at bits 3..6 (n * 2^-21) and 7..10 (n * 2^-17; bit 10 is the exponent's last, under which the format is still linear), for
//     one shift more per word.  Error of the rows against double precision at 262,144 / 65,536 / 32,768 tokens, mean of six caches,
//     even channels and odd ones: 1.59e-3 1.58e-3 / 1.15e-3 1.14e-3 / 1.18e-3 1.18e-3.  At bits 0..3 and 4..7: 2.29e-3 1.59e-3 /
//     1.34e-3 1.15e-3 / 1.29e-3 1.18e-3.  With offsets (1024 + n taken out by a subtraction, 64 + n by MMA rows of ones): 1.54e-3 6.70e-3 /
//     1.14e-3 1.26e-3 / 1.16e-3 1.19e-3.  For K, whose sums run over a head's channels only, the position changes nothing (0.1 %).
//     Time with offsets, and now: 262,144 tokens 85.7 -> 82.0 us, eight sequences 124.2 -> 115.7 us (both tiles of a group in
//     step, see below, included).
//   * RoPE: Q is rotated back by the group's first position (one table row per group), the remaining angle
//     (0..31 tokens) is applied to the rotary channels of K with the table's first 32 rows.  cos/sin of
//     (t0 + dt) are thereby formed by angle addition from the caller's table entries for t0 and dt.  The table's own
//     angle at t is the fp32 product t*freq, which differs from the sum of the two entries' angles by up to one ulp of
//     t*freq (0.03 rad at t = 262,144 for the highest frequency): a per-token perturbation of the score of about 1e-3,
//     random in sign, that changed no digit of the measured error at 262,144 tokens (a build that read the table row of
//     every token for the eight highest frequencies gave the same error and ran 16 % slower).
// Lane (g = lane/4, j = lane%4) owns words w = 4i + j of a packed K row, so a rotary pair (c, c + RD/2) stays
// in one lane.
//
// Every wait is bounded: a wait that runs out sets a device status word and the CTA drains and returns.
#include "kv4_common.cuh"
#include <cuda.h>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <cstring>
#include <vector>

namespace kv4 {

__device__ int g_decode_status = 0;          // 0 ok; 1 = a consumer wait ran out; 2 = a producer wait ran out

namespace {

#ifndef KV4_DECODE_NCW
#define KV4_DECODE_NCW 7                     // consumer warps per CTA
#endif
// 8 warps = 2 per SM sub-partition, one CTA per SM, up to 255 registers a thread.  Measured at 262,144 tokens, with the offsets' arithmetic:
// 4 / 6 / 8 / 12 / 16 warps (255 / 255 / 255 / 168 / 128 registers) = 127 / 111 / 83.5 / 90.2 / 107 us per step
constexpr int NCW = KV4_DECODE_NCW;
constexpr int NTHREADS = (NCW + 1) * 32;
constexpr uint32_t WAIT_LIMIT = 1u << 22;    // polls of try_wait before giving up (each poll suspends up to ~us)
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

constexpr int NSTAGE = 5;                    // ring depth (128-token units in flight per CTA); with four, rows of a batch took 15-20 % longer
template <int HD, int RD, bool Q> struct Lay {
  static constexpr int UG = 4;                             // groups per unit (one ring stage)
  static constexpr int ROWB = HD / 2;                      // bytes of one packed row
  static constexpr int KB = 32 * ROWB;                     // packed K (or V) bytes of one group
  static constexpr int SCB = HD * 2;                       // one fp16 scale row
  static constexpr int ROPEB = RD / 2 * 8;                 // one rope row
  static constexpr int SHADOW = 32 * HD * 2;               // fp16 rows of the open group (= UG*KB: it takes K's place)
  static constexpr int OFF_K = 0, OFF_V = UG * KB, OFF_KS = 2 * UG * KB, OFF_KZ = OFF_KS + UG * SCB, OFF_VS = OFF_KZ + UG * SCB,
                       OFF_VZ = OFF_VS + UG * 64, OFF_ROPE = OFF_VZ + UG * 64;
  static constexpr int STAGE = (OFF_ROPE + UG * ROPEB + 1023) / 1024 * 1024;
  static constexpr int NW = HD / 32;                       // packed words per lane per row
  static constexpr int NR = RD / 32;                       // of which rotary (first NR); pairs (i, i + NR/2)
  static constexpr int NP = NR / 2;
  static constexpr int QFRAG = NW * 32 * 16;               // Q as B fragments: [i][lane] x 16 bytes
  static constexpr int RELT = 4 * (NP ? NP : 1) * 2 * 32 * 16;   // relative rotation: [tile][half][i][xpair][lane] x 16 B
  static constexpr int OFF_STAGES = 0;
  static constexpr int OFF_QFRAG = NSTAGE * STAGE;
  static constexpr int OFF_RELT = OFF_QFRAG + QFRAG;
  static constexpr int OFF_BARS = OFF_RELT + RELT;         // full[NSTAGE], empty[NSTAGE]
  static constexpr int OFF_MISC = OFF_BARS + 2 * NSTAGE * 8;   // abort flag
  static constexpr int OFF_TAG = OFF_MISC + 4;             // [NSTAGE] the unit last issued into each stage
  static constexpr int OFF_RESP = (OFF_TAG + 4 * NSTAGE + 15) / 16 * 16, OFF_CLC = OFF_RESP + 32;   // queue: two cancel responses, their full / empty barriers
  static constexpr int OFF_ORDER = OFF_CLC + 32, OFF_POS = OFF_ORDER + 64;                   // queue: rows by length; their positions
  static constexpr int OFF_ML = (OFF_POS + 256 + 15) / 16 * 16;                              // (m, l) of heads 2j, 2j+1 per (warp, j)
  static constexpr int NH = HD / 32;                       // m-tiles of one half
  // O of all warps, half of the m-tiles at a time: [warp][m-tile][lane] x 16 bytes.  Without the queue it aliases the ring, which is empty by
  // then: the block then leaves room on its SM for a block of the merge kernel, which starts ahead of its end.
  static constexpr int OFF_MERGE = Q ? OFF_ML + NCW * 4 * 16 : 0, MERGE = NCW * NH * 512;
  static constexpr int TOTAL = Q ? OFF_MERGE + MERGE : OFF_ML + NCW * 4 * 16;
  static_assert(Q || MERGE <= NSTAGE * STAGE, "merge buffer must fit in the ring");
  static_assert(SHADOW == UG * KB, "the open group's fp16 rows take the place of the unit's packed K");
  static_assert(NR % 2 == 0 && NR <= NW, "rotary width must be a multiple of 64 and at most head_dim");
  static_assert(TOTAL <= 227 * 1024, "shared memory budget of one CTA");
};

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Ask the hardware for a block of this grid that has not started: its index (or "none left") arrives in 16 bytes of shared memory.
__device__ __forceinline__ void cancel_next(uint32_t resp, uint32_t bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(resp), "r"(bar) : "memory");
}
__device__ __forceinline__ bool cancel_result(uint32_t resp, int& x, int& y, int& z) {
  uint32_t ok;
  asm volatile("{\n .reg .b128 h;\n .reg .pred p;\n .reg .b32 w;\n ld.shared.b128 h, [%4];\n"
               " clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n selp.u32 %0, 1, 0, p;\n"
               " mov.u32 %1, 0;\n mov.u32 %2, 0;\n mov.u32 %3, 0;\n"
               " @p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, w}, h;\n}"
               : "=r"(ok), "=r"(x), "=r"(y), "=r"(z) : "r"(resp) : "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the next response into these bytes is ordered behind this read
  return ok != 0;
}
// Bounded wait; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v; asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4_t(uint32_t a, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ uint32_t movmatrix_t(uint32_t a) { uint32_t d; asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a)); return d; }
__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) { uint32_t d; asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo)); return d; }
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) { uint32_t d; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) { uint32_t d; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d; }
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) { uint32_t d; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t hneg2(uint32_t a) { uint32_t d; asm("neg.f16x2 %0, %1;" : "=r"(d) : "r"(a)); return d; }
// A 32-bit word of a packed row holds nibbles 0..7.  One AND pairs nibbles (X, X+4) as the two halves of a register
// WITHOUT moving them (one shift, w >> 8, serves X = 2, 3), and the halves are fp16 subnormals: a nibble at bits 0..3 reads as n * 2^-24, at
// bits 4..7 as n * 2^-20.  The tensor core multiplies subnormals exactly, so the factor leaves behind the fp32 sum, and nothing is added to the
// operands.  V's words are first shifted by 3 (w << 3 for X = 0, 1 and w >> 5 for X = 2, 3): n * 2^-21 and n * 2^-17.  Rotary words need the value itself: under exponent 2^10 (0x6400) or 2^6 (0x5400) the halves read as 1024 + n or 64 + n, and the
// constant leaves by an exact subtraction.
constexpr uint32_t NIB_E = 0x000F000Fu, NIB_O = 0x00F000F0u;
constexpr float NIB_E_INV = 16777216.f, NIB_O_INV = 1048576.f;     // 2^24, 2^20
constexpr float VNIB_E_INV = 2097152.f, VNIB_O_INV = 131072.f;     // 2^21, 2^17
constexpr uint32_t NEG_E = 0xE400E400u, NEG_O = 0xD400D400u;       // -(1024, 1024), -(64, 64)
// (a & m) | c as ONE LOP3.  LOP3 takes a single immediate, so with two literal constants the compiler emits AND then OR
// (measured: 562 LOP3 per group instead of ~280); the masks and offsets are therefore kept in registers that the
// compiler cannot fold (NibK).
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t m, uint32_t c) {
  uint32_t d; asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(m), "r"(c)); return d;
}
struct NibK { uint32_t m0, m1, e, o; };                          // the masks; (1024, 1024), (64, 64)
__device__ __forceinline__ NibK nib_consts() {
  NibK k;
  asm volatile("mov.u32 %0, 0x000F000F;\n mov.u32 %1, 0x00F000F0;\n mov.u32 %2, 0x64006400;\n mov.u32 %3, 0x54005400;"
               : "=r"(k.m0), "=r"(k.m1), "=r"(k.e), "=r"(k.o));
  return k;
}
__device__ __forceinline__ void nib_off_regs(uint32_t w, uint32_t (&o)[4], const NibK& c) {
  const uint32_t w8 = w >> 8;
  o[0] = and_or(w, c.m0, c.e); o[1] = and_or(w, c.m1, c.o);
  o[2] = and_or(w8, c.m0, c.e); o[3] = and_or(w8, c.m1, c.o);
}
// eight consecutive fp16 (r.x = (e0,e1) .. r.w = (e6,e7)) -> register X pairing elements (X, X+4)
__device__ __forceinline__ void pair_regs(const uint4& r, uint32_t (&o)[4]) {
  o[0] = __byte_perm(r.x, r.z, 0x5410); o[1] = __byte_perm(r.x, r.z, 0x7632);
  o[2] = __byte_perm(r.y, r.w, 0x5410); o[3] = __byte_perm(r.y, r.w, 0x7632);
}
__device__ __forceinline__ float lds_h(uint32_t a) {
  unsigned short v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a)); return __half2float(__ushort_as_half(v));
}

// ---------------------------------------------------------------- kernel
// Tensor maps of one cache.  The scales and zeros come as tiles too: as bulk copies of 2 KB and 256 bytes the same step took 82.2 instead of
// 81.1 us at 262,144 tokens.  In a multi-request pass they are bulk copies all the same, because its table in device memory holds the maps of K and V
// only (yskn_kv4_ms_rows): eight sequences 116.3 us, with a table of six maps 115.8.
struct Maps { CUtensorMap k, v, ks, kz, vs, vz; };
static_assert(sizeof(Maps) == 6 * 128, "yskn_kv4_ms_maps_bytes and the header give 128 bytes a map");
struct DecodeP {
  yskn_attn_g_args A;
  Shard sh;
  int g;
  int early;          // the caller's promise (yskn_kv4_attn_ext): *d_pos and every cache row below it are final before the
                      // preceding kernel of the stream ends, so they may be read ahead of griddepcontrol.wait
  yskn_kv4_ms_rows ms;  // rows of several sequences (ms.pos != nullptr): row r reads the cache ms.layers[ms.slot[r]] at position ms.pos[r]
};

// Q ("queue"): for grids of more blocks than the GPU holds at once (several rows, or several sequences).  A CTA that has
// issued the last copy of its item cancels a block that has not started (clusterlaunchcontrol) and takes over its indexes, so
// the ring fills with the next item's keys while the consumers finish, merge and store this one.  Rows of several
// sequences are taken longest first: the last blocks to start are then the shortest.  What each (split, kv-head, row) computes, and so every
// bit of it, does not depend on Q.  Before, each item paid its launch, set-up, first-copy latency and merge by itself, and the longest
// rows of a batch came last: eight sequences of 2,048 .. 131,072 tokens 171 -> 124 us with their merge, five rows over 20,011 tokens 67.6 ->
// 55.6 us with their append and merge, eight rows over 172 tokens 48.8 -> 38 us.
template <int HD, int RD, int DT, bool Q, bool multi>
__global__ void __launch_bounds__(NTHREADS, 1)
kv4_decode_mma_kernel(const __grid_constant__ Maps maps, const __grid_constant__ CUtensorMap mapR, const DecodeP P) {
  using L = Lay<HD, RD, Q>;
  constexpr int NW = L::NW, NR = L::NR, NP = L::NP, NRd = NR > 0 ? NR : 1;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const yskn_attn_g_args& A = P.A;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  const int G = P.g;
  // Programmatic dependent launch in both directions (src/pdl.cuh:15-30 is the reference's form of this): this grid may be
  // scheduled while the previous kernel of the stream drains and waits here before it reads anything that kernel wrote
  // (position, query, appended rows); the merge kernel that follows may be scheduled early in turn and waits for this grid
  // to finish before it reads the partials.
  // With `early` (the reference's Q35AttnArgs.early, src/q35_kernels.cu:1195-1206) the position is read and the producer
  // fills the ring with rows below the base position BEFORE the wait: those rows were final before the predecessor started.
  const bool early = P.early != 0;
  if (!early) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }

  // ---- which groups an item (split, kv-head, row) covers (local token indices of this shard)
  struct Item { int split, kvh, r, base_local, len, nq, nu4, u0, nu; bool has_tail; };
  auto item_at = [&](int x, int y, int z) {
    Item t;
    t.split = x; t.kvh = y;
    t.r = Q && multi ? smem[L::OFF_ORDER + z] : z;              // Q: rows by length
    t.base_local = multi ? P.ms.pos[t.r] : *A.d_pos - P.sh.start;   // row 0's local position: rows below it are never written again
    const int pos = multi ? t.base_local : t.base_local + t.r;
    t.len = max(0, min(pos + 1, P.sh.len));
    const int cg = pos >= 0 ? pos / 32 : 0;                     // first group that is not read as int4
    t.nq = min(cg, t.len / 32);                                 // int4 groups, all fully visible
    t.has_tail = t.len > t.nq * 32;                             // the open group lives in this shard
    t.nu4 = (t.nq + L::UG - 1) / L::UG;                         // int4 units of four groups (the last may hold fewer)
    const int units = t.nu4 + (t.has_tail ? 1 : 0);             // the open group is a unit of its own, the last one
    const int per = (units + (int)gridDim.x - 1) / (int)gridDim.x;
    t.u0 = min(units, x * per); t.nu = min(units, t.u0 + per) - t.u0;
    return t;
  };

  const uint32_t bar_full = sbase + L::OFF_BARS, bar_empty = bar_full + NSTAGE * 8;
  const uint32_t bar_clc = sbase + L::OFF_CLC, resp = sbase + L::OFF_RESP;       // Q: full[2], empty[2]; two responses
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + L::OFF_MISC);
  volatile int* s_tag = reinterpret_cast<volatile int*>(smem + L::OFF_TAG);
  if (sbase & 1023u) { if (threadIdx.x == 0) atomicExch(&g_decode_status, 3); return; }   // the swizzled tiles need a 1 KB base
  if (threadIdx.x == 0) {
    // a stage is free again once the consumers of its four groups have arrived (without Q units with fewer groups are never reused)
    for (int s = 0; s < NSTAGE; ++s) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, L::UG); }
    if (Q) for (int s = 0; s < 2; ++s) { mbar_init(bar_clc + 8 * s, 1); mbar_init(bar_clc + 16 + 8 * s, NCW); }
    for (int s = 0; s < NSTAGE; ++s) s_tag[s] = -1;
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (Q && multi) {                                             // rows by falling length, ties by index (at most 64 rows)
    int* s_pos = reinterpret_cast<int*>(smem + L::OFF_POS);
    if (threadIdx.x < A.M) s_pos[threadIdx.x] = P.ms.pos[threadIdx.x];
    __syncthreads();
    if (threadIdx.x < A.M) {
      const int mine = s_pos[threadIdx.x];
      int rank = 0;
      for (int i = 0; i < A.M; ++i) rank += s_pos[i] > mine || (s_pos[i] == mine && i < (int)threadIdx.x);
      smem[L::OFF_ORDER + rank] = (uint8_t)threadIdx.x;
    }
  }
  __syncthreads();

  Item it = item_at(blockIdx.x, blockIdx.y, blockIdx.z);

  if (warp == NCW) {
    // =========================================================== producer warp
    int k = 0;                                                  // units issued by this CTA so far
    bool waited = !early, go = true, asked = false;
    // The next item is claimed when a ring's worth of this one's units is still to be issued.  Claimed always at the start of this one,
    // every second item was bound to a CTA at once and the lengths no longer evened out (five sequences of 1,204 .. 57,119 tokens:
    // 58 -> 70 us); claimed after the last unit, the answer came too late for short items (five rows over 20,011 tokens: 57.5 -> 61 us).
    auto claim = [&](int n) {
      if (lane != 0 || *s_abort) return;
      if (n >= 2 && !mbar_wait(bar_clc + 16 + 8 * (n & 1), ((n >> 1) - 1) & 1)) { atomicExch(&g_decode_status, 2); *s_abort = 1; return; }
      mbar_expect_tx(bar_clc + 8 * (n & 1), 16);
      cancel_next(resp + 16 * (n & 1), bar_clc + 8 * (n & 1));
      asked = true;
    };
    for (int n = 0; ; ++n) {                                    // items
      const int nq = it.nq, nu4 = it.nu4, kvh = it.kvh;
      const bool has_tail = it.has_tail;
      const size_t row0 = (size_t)kvh * A.max_ctx;              // first row of this kv-head in the [Hkv*max_ctx] arrays
      const int slot = multi ? P.ms.slot[it.r] : 0;
      const yskn_kv_layer kvl = multi ? P.ms.layers[slot] : A.kv;
      const CUtensorMap* const mk = multi ? static_cast<const CUtensorMap*>(P.ms.maps) + 2 * slot : &maps.k;   // K, V; of one cache all six
      for (int u = it.u0; u < it.u0 + it.nu; ++u) {
        const int s = k % NSTAGE;
        // an early unit: one of the first ring fills, int4 only, every token below the base position
        if (!waited && (k >= NSTAGE || (has_tail && u == nu4) || min(nq, (u + 1) * L::UG) * 32 > max(0, min(it.base_local, P.sh.len)))) {
          asm volatile("griddepcontrol.wait;" ::: "memory");
          asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
          waited = true;
        }
        if (Q && u == max(it.u0, it.u0 + it.nu - NSTAGE)) claim(n);
        int ok = 1;
        if (lane == 0) {
          if (k >= NSTAGE && !mbar_wait(bar_empty + 8 * s, ((k / NSTAGE) - 1) & 1)) { atomicExch(&g_decode_status, 2); *s_abort = 1; }
          if (*s_abort) ok = 0;
        }
        go = __shfl_sync(0xffffffffu, ok, 0) != 0;
        if (!go) break;
        const bool tail = has_tail && u == nu4;
        const int g0 = tail ? nq : u * L::UG;                    // its first group (local index)
        const uint32_t st = sbase + L::OFF_STAGES + s * L::STAGE, bar = bar_full + 8 * s;
        // Tiles are whole units always: what lies behind the last group of a unit, or of the array, is unused.  Bulk copies (the table of a
        // multi-request pass holds the maps of K and V only) end with the unit's last group, which may be the array's.
        const int ngr = !multi ? L::UG : tail ? 1 : min(L::UG, nq - u * L::UG);
        if (lane == 0) s_tag[s] = k;
        if (lane == 0) mbar_expect_tx(bar, 2 * L::UG * L::KB + 2 * ngr * ((tail ? 0 : L::SCB) + 64) + L::UG * L::ROPEB);   // SHADOW == UG*KB
        __syncwarp();                                            // the barrier is armed before any copy is issued
        const int tok0 = (int)row0 + g0 * 32, grp0 = kvh * (A.max_ctx / 32) + g0;
        // One copy per lane: seven issue slots in parallel
        switch (lane) {
          case 0: if (tail) bulk_1d(st + L::OFF_K, kvl.kshadow + (size_t)tok0 * HD, L::SHADOW, bar);
                  else tma_2d(st + L::OFF_K, mk, 0, tok0, bar); break;
          case 1: tma_2d(st + L::OFF_V, mk + 1, 0, tok0, bar); break;
          case 2: if (!tail) { if (multi) bulk_1d(st + L::OFF_KS, kvl.kscale + (size_t)grp0 * HD, ngr * L::SCB, bar); else tma_2d(st + L::OFF_KS, mk + 2, 0, grp0, bar); } break;
          case 3: if (!tail) { if (multi) bulk_1d(st + L::OFF_KZ, kvl.kzero + (size_t)grp0 * HD, ngr * L::SCB, bar); else tma_2d(st + L::OFF_KZ, mk + 3, 0, grp0, bar); } break;
          case 4: if (multi) bulk_1d(st + L::OFF_VS, kvl.vscale + tok0, ngr * 64, bar); else tma_2d(st + L::OFF_VS, mk + 4, g0 * 32, kvh, bar); break;
          case 5: if (multi) bulk_1d(st + L::OFF_VZ, kvl.vzero + tok0, ngr * 64, bar); else tma_2d(st + L::OFF_VZ, mk + 5, g0 * 32, kvh, bar); break;
          case 6: if (RD > 0) tma_2d(st + L::OFF_ROPE, &mapR, 0, g0 + P.sh.start / 32, bar); break;   // rows 32*(g0..g0+3) of the table
          default: break;
        }
        ++k;
      }
      if (!Q) break;
      if (!waited) { asm volatile("griddepcontrol.wait;" ::: "memory"); asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); waited = true; }
      if (it.nu == 0) claim(n);
      int x = 0, y = 0, z = 0, more = 0;
      if (lane == 0 && asked) {                                  // also after an abort: the answer has landed before the CTA ends
        if (!mbar_wait(bar_clc + 8 * (n & 1), (n >> 1) & 1)) { atomicExch(&g_decode_status, 2); *s_abort = 1; }
        else more = cancel_result(resp + 16 * (n & 1), x, y, z) ? 1 : 0;
        if (*s_abort) more = 0;
        asked = false;
      }
      more = __shfl_sync(0xffffffffu, more, 0);
      if (!more) break;
      it = item_at(__shfl_sync(0xffffffffu, x, 0), __shfl_sync(0xffffffffu, y, 0), __shfl_sync(0xffffffffu, z, 0));
    }
    if (!waited) { asm volatile("griddepcontrol.wait;" ::: "memory"); asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
    // After an abort nobody may have consumed the last copies: wait (bounded) until they have landed before the CTA ends.
    if (lane == 0 && *s_abort)
      for (int i = max(0, k - NSTAGE); i < k; ++i) mbar_wait(bar_full + 8 * (i % NSTAGE), (i / NSTAGE) & 1);
  } else {
    // =========================================================== consumer warps
    if (early) {                                                // q16 and the partial buffers belong to the predecessor until here
      asm volatile("griddepcontrol.wait;" ::: "memory");
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    // ---- one-time set-up, spread over the consumer threads
    const int ct = threadIdx.x;                                 // 0..NCW*32-1
    constexpr int NQE = (NW * 32 * 4 + NCW * 32 - 1) / (NCW * 32);   // Q entries per thread
    // Q as B fragments, pre-scaled by qscale*log2(e): entry [i][lane'] = 4 regs x, w = 4i+j': reg x = (q[g'][8w+x], q[g'][8w+x+4]) of a
    // rotary word, (q[g'][8w+2x], q[g'][8w+2x+1]) of a plain one (its scale and zero rows lie so, and only the product is put in nibble order)
    const float qs = A.qscale * LOG2E;
    auto q_entry = [&](int e, const Item& t) -> uint32_t {
      const int x = e & 3, ln = (e >> 2) & 31, i = e >> 7, gg = ln >> 2, jj = ln & 3;
      const int c = 8 * (4 * i + jj) + (i < NR ? x : 2 * x), d = i < NR ? 4 : 1;
      float lo = 0.f, hi = 0.f;
      if (gg < G) {
        const size_t qb = ((size_t)t.r * A.nh + t.kvh * G + gg) * HD;
        lo = act_load<DT>(A.q16, qb + c) * qs; hi = act_load<DT>(A.q16, qb + c + d) * qs;
      }
      return pack_h2(lo, hi);
    };
    {
      #pragma unroll
      for (int n = 0; n < NQE; ++n) { const int e = ct + n * NCW * 32; if (e < NW * 32 * 4) reinterpret_cast<uint32_t*>(smem + L::OFF_QFRAG)[e] = q_entry(e, it); }
      // relative rotation by dt = 0..31 tokens, from the table's rows 0..31: entry [tile][half][i][xp][lane'] =
      // {cd_{2xp}, sd_{2xp}, cd_{2xp+1}, sd_{2xp+1}}, each a half2 over frequencies (8w+x, 8w+x+4), w = 4i+j'
      if (RD > 0) {
        constexpr int NPd = NP > 0 ? NP : 1;
        for (int e = ct; e < 4 * NP * 2 * 32; e += NCW * 32) {
          const int ln = e & 31, xp = (e >> 5) & 1, i = (e >> 6) % NPd, th = (e >> 6) / NPd;   // th = tile*2 + half
          const int gg = ln >> 2, jj = ln & 3, dt = 8 * th + gg, w = 4 * i + jj;
          uint32_t o[4];
          #pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int f = 8 * w + 2 * xp + q;
            const float2 a = *reinterpret_cast<const float2*>(A.rope + ((size_t)dt * (RD / 2) + f) * 2);
            const float2 b = *reinterpret_cast<const float2*>(A.rope + ((size_t)dt * (RD / 2) + f + 4) * 2);
            o[2 * q] = pack_h2(a.x, b.x); o[2 * q + 1] = pack_h2(a.y, b.y);
          }
          *reinterpret_cast<uint4*>(smem + L::OFF_RELT + (size_t)e * 16) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32) : "memory");

    float acc[HD / 16][4];                                      // O^T: [m-tile][(even | odd channel) x (head 2j | 2j+1)]
    #pragma unroll
    for (int mt = 0; mt < HD / 16; ++mt) { acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f; }
    float m[2] = {-1e30f, -1e30f}, l[2] = {0.f, 0.f}, zacc[2] = {0.f, 0.f};   // heads 2j, 2j+1 (log2 domain); zacc = sum p*vzero

    // per-lane constant offsets: K word i of row g (swizzled chunk), V chunk of rows 2j and 2j+1
    const int swz = HD == 256 ? (g & 7) : ((g >> 1) & 3);
    uint32_t koff[NW];
    #pragma unroll
    for (int i = 0; i < NW; ++i) koff[i] = g * L::ROWB + 16 * (i ^ swz) + 4 * j;
    // V through ldmatrix.trans: lane supplies the row address of matrix lane/8, row lane%8: token (mat&1)*8 + row, 16-byte
    // chunk 2q + (mat>>1) (q = which of the HD/64 loads), XOR-swizzled as the TMA tile is.
    const int vtok = ((lane >> 3) & 1) * 8 + (lane & 7), vch = lane >> 4;
    const uint32_t vrow = vtok * L::ROWB, vsw = HD == 256 ? (vtok & 7) : ((vtok >> 1) & 3);
    const uint32_t qfrag = sbase + L::OFF_QFRAG + lane * 16;
    const uint32_t relt = sbase + L::OFF_RELT + lane * 16;
    const NibK nk = nib_consts();

    // One 32-token group.  TAIL: the open group (fp16 shadow rows, `nvalid` visible tokens); else an int4 group.
    // `st` = stage base, `sub` = which of the unit's four groups (0 for the open group).
    auto group = [&](auto tail_c, const uint32_t st, const int sub, const int nvalid) {
      constexpr bool TAIL = decltype(tail_c)::value;
      const uint32_t s_k = st + L::OFF_K + sub * L::KB, s_v = st + L::OFF_V + sub * L::KB, s_ks = st + L::OFF_KS + sub * L::SCB,
                     s_kz = st + L::OFF_KZ + sub * L::SCB, s_vs = st + L::OFF_VS + sub * 64, s_rope = st + L::OFF_ROPE + sub * L::ROPEB;
      // ---- per-group fold: q' = q*scale (plain channels); Q rotated back by the group's first position (rotary
      //      channels); bias[h] = sum_c q[h][c]*zero[c] as MMA rows that all carry the same vector, so every lane ends up
      //      with the bias of its own two heads.
      uint32_t qf[NW][4], rs[NRd][4], rz[NRd][4];
      float bias[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      #pragma unroll
      for (int i = 0; i < NW; ++i) {
        const uint4 q4 = lds128(qfrag + i * 512);
        const uint32_t qv[4] = {q4.x, q4.y, q4.z, q4.w};
        #pragma unroll
        for (int x = 0; x < 4; ++x) qf[i][x] = qv[x];
        if (!TAIL) {
          const uint4 sc = lds128(s_ks + 16 * (4 * i + j)), zz = lds128(s_kz + 16 * (4 * i + j));
          if (i < NR) { pair_regs(sc, rs[i]); pair_regs(zz, rz[i]); }
          else {
            pair_regs(make_uint4(hmul2(qv[0], sc.x), hmul2(qv[1], sc.y), hmul2(qv[2], sc.z), hmul2(qv[3], sc.w)), qf[i]);
            mma16816(bias[0], zz.x, zz.x, zz.y, zz.y, qv[0], qv[1]);
            mma16816(bias[1], zz.z, zz.z, zz.w, zz.w, qv[2], qv[3]);
          }
        }
      }
      if (RD > 0) {
        #pragma unroll
        for (int i = 0; i < NP; ++i) {
          const uint32_t rp = s_rope + 64 * (4 * i + j);     // 8 frequencies x (cos, sin) fp32
          const uint4 r0 = lds128(rp), r1 = lds128(rp + 16), r2 = lds128(rp + 32), r3 = lds128(rp + 48);
          const uint32_t C[4] = {pack_h2(__uint_as_float(r0.x), __uint_as_float(r2.x)), pack_h2(__uint_as_float(r0.z), __uint_as_float(r2.z)),
                                 pack_h2(__uint_as_float(r1.x), __uint_as_float(r3.x)), pack_h2(__uint_as_float(r1.z), __uint_as_float(r3.z))};
          const uint32_t S[4] = {pack_h2(__uint_as_float(r0.y), __uint_as_float(r2.y)), pack_h2(__uint_as_float(r0.w), __uint_as_float(r2.w)),
                                 pack_h2(__uint_as_float(r1.y), __uint_as_float(r3.y)), pack_h2(__uint_as_float(r1.w), __uint_as_float(r3.w))};
          #pragma unroll
          for (int x = 0; x < 4; ++x) {
            const uint32_t qa = qf[i][x], qb = qf[i + NP][x];
            qf[i][x] = hfma2(qa, C[x], hmul2(qb, S[x]));                 // u = qa*C + qb*S
            qf[i + NP][x] = hfma2(qb, C[x], hneg2(hmul2(qa, S[x])));     // w = qb*C - qa*S
          }
        }
      }
      // Both 16-token tiles of the group go through each step together: twice the independent work between two dependent steps.
      constexpr uint32_t ROW8 = TAIL ? 8 * HD * 2 : 8 * L::ROWB;       // eight K rows further down
      uint32_t ka[NW];                                           // this lane's word i in row g of the group
      #pragma unroll
      for (int i = 0; i < NW; ++i) ka[i] = TAIL ? s_k + g * (HD * 2) + 16 * (4 * i + j) : s_k + koff[i];
      // ---- S^T[32 tok x 8 heads] = K . Q^T.  Three sums a tile: nibbles read at 2^-24 (E), at 2^-20 (O), and true values (R)
      float se[2][4], so[2][4], sr[2][4];
      #pragma unroll
      for (int t = 0; t < 2; ++t)
        #pragma unroll
        for (int x = 0; x < 4; ++x) { se[t][x] = so[t][x] = 0.f; sr[t][x] = bias[0][x] + bias[1][x]; }
      if (RD > 0) {                                              // rotary words: true value, rotated by dt
        #pragma unroll
        for (int t = 0; t < 2; ++t) {
          uint32_t kr[2][NRd][4];
          #pragma unroll
          for (int h = 0; h < 2; ++h)
            #pragma unroll
            for (int i = 0; i < NP; ++i) {
              uint32_t a4[4], b4[4];
              if (TAIL) { pair_regs(lds128(ka[i] + (2 * t + h) * ROW8), a4); pair_regs(lds128(ka[i + NP] + (2 * t + h) * ROW8), b4); }
              else { nib_off_regs(lds32(ka[i] + (2 * t + h) * ROW8), a4, nk); nib_off_regs(lds32(ka[i + NP] + (2 * t + h) * ROW8), b4, nk); }
              const uint32_t ra = relt + (((2 * t + h) * NP + i) * 2) * 512;
              const uint4 t0 = lds128(ra), t1 = lds128(ra + 512);
              const uint32_t cd[4] = {t0.x, t0.z, t1.x, t1.z}, sd[4] = {t0.y, t0.w, t1.y, t1.w};
              #pragma unroll
              for (int x = 0; x < 4; ++x) {
                uint32_t a = a4[x], b = b4[x];
                if (!TAIL) {                                     // (off+n) - off is exact; n*scale + zero rounds once
                  const uint32_t ng = (x & 1) ? NEG_O : NEG_E;
                  a = hfma2(hadd2(a, ng), rs[i][x], rz[i][x]); b = hfma2(hadd2(b, ng), rs[i + NP][x], rz[i + NP][x]);
                }
                kr[h][i][x] = hfma2(a, cd[x], hneg2(hmul2(b, sd[x])));        // a*cd - b*sd
                kr[h][i + NP][x] = hfma2(a, sd[x], hmul2(b, cd[x]));          // a*sd + b*cd
              }
            }
          #pragma unroll
          for (int i = 0; i < NR; ++i) {
            mma16816(sr[t], kr[0][i][0], kr[1][i][0], kr[0][i][1], kr[1][i][1], qf[i][0], qf[i][1]);
            mma16816(sr[t], kr[0][i][2], kr[1][i][2], kr[0][i][3], kr[1][i][3], qf[i][2], qf[i][3]);
          }
        }
      }
      #pragma unroll
      for (int i = NR; i < NW; ++i)
        #pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (TAIL) {
            const uint4 k0 = lds128(ka[i] + 2 * t * ROW8), k1 = lds128(ka[i] + (2 * t + 1) * ROW8);
            mma16816(sr[t], k0.x, k1.x, k0.y, k1.y, qf[i][0], qf[i][1]);
            mma16816(sr[t], k0.z, k1.z, k0.w, k1.w, qf[i][2], qf[i][3]);
          } else {
            const uint32_t k0 = lds32(ka[i] + 2 * t * ROW8), k1 = lds32(ka[i] + (2 * t + 1) * ROW8), k08 = k0 >> 8, k18 = k1 >> 8;
            mma16816(se[t], k0 & NIB_E, k1 & NIB_E, k08 & NIB_E, k18 & NIB_E, qf[i][0], qf[i][2]);
            mma16816(so[t], k0 & NIB_O, k1 & NIB_O, k08 & NIB_O, k18 & NIB_O, qf[i][1], qf[i][3]);
          }
        }
      // V rows of both tiles with their scales and zeros, requested ahead of the softmax
      uint32_t vx[2][HD / 64][4];                                // [tile][load q][tokens 0-7 | 8-15 of chunk 2q, the same of chunk 2q+1]
      #pragma unroll
      for (int t = 0; t < 2; ++t)
        #pragma unroll
        for (int q = 0; q < HD / 64; ++q) ldmatrix_x4_t(s_v + vrow + t * 16 * L::ROWB + 16 * ((2 * q + vch) ^ vsw), vx[t][q]);
      float vs[4], vz[4];                                        // token rows g, g+8, g+16, g+24
      #pragma unroll
      for (int y = 0; y < 4; ++y) {
        const bool v = !TAIL || 8 * y + g < nvalid;
        vs[y] = v ? lds_h(s_vs + 2 * g + 16 * y) : 0.f; vz[y] = v ? lds_h(s_vs + L::UG * 64 + 2 * g + 16 * y) : 0.f;
      }
      // ---- softmax over the group (log2 domain); heads 2j, 2j+1
      float s[4][2];
      #pragma unroll
      for (int y = 0; y < 4; ++y)
        #pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int t = y >> 1, c = 2 * (y & 1) + x;
          s[y][x] = NR < NW && !TAIL ? fmaf(se[t][c], NIB_E_INV, fmaf(so[t][c], NIB_O_INV, sr[t][c])) : sr[t][c];
          if (TAIL && 8 * y + g >= nvalid) s[y][x] = -INFINITY;
        }
      float t0 = fmaxf(fmaxf(s[0][0], s[1][0]), fmaxf(s[2][0], s[3][0])), t1 = fmaxf(fmaxf(s[0][1], s[1][1]), fmaxf(s[2][1], s[3][1]));
      if (__any_sync(0xffffffffu, t0 > m[0] + 8.f || t1 > m[1] + 8.f)) {   // lazy rescale: the running max may lag by 2^8; no shuffle unless it must move
        #pragma unroll
        for (int o = 4; o <= 16; o <<= 1) { t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, o)); t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, o)); }
        const float n0 = fmaxf(m[0], t0), n1 = fmaxf(m[1], t1), a0 = ex2(m[0] - n0), a1 = ex2(m[1] - n1);
        m[0] = n0; m[1] = n1; l[0] *= a0; l[1] *= a1; zacc[0] *= a0; zacc[1] *= a1;
        #pragma unroll
        for (int mt = 0; mt < HD / 16; ++mt) { acc[mt][0] *= a0; acc[mt][1] *= a1; acc[mt][2] *= a0; acc[mt][3] *= a1; }
      }
      // V's per-token scale is folded into P (fp16), its zero point into a per-head scalar: v = vs*n + vz.
      uint32_t pb[4];                                            // B regs per tile: (tokens 2j,2j+1 | head g), (tokens 2j+8,2j+9 | head g)
      #pragma unroll
      for (int y = 0; y < 4; ++y) {
        const bool v = !TAIL || 8 * y + g < nvalid;
        const float p0 = v ? ex2(s[y][0] - m[0]) : 0.f, p1 = v ? ex2(s[y][1] - m[1]) : 0.f;
        l[0] += p0; l[1] += p1;
        zacc[0] = fmaf(p0, vz[y], zacc[0]); zacc[1] = fmaf(p1, vz[y], zacc[1]);
        pb[y] = movmatrix_t(pack_h2(p0 * vs[y], p1 * vs[y]));
      }
      // ---- O^T += V^T P^T.  A transposed 8x8 load hands lane (g, j) the 16-bit element g of token rows 2j and 2j+1 of a
      //      16-byte chunk: four channels (4g .. 4g+3 of the chunk's 32) of two consecutive tokens, which is the pairing along
      //      the contraction that an A register wants.  MMA row g = the channel at bits 3..6 of the shifted word (2^-21), row g+8 = the one at bits 7..10 (2^-17).
      #pragma unroll
      for (int t = 0; t < 2; ++t)
        #pragma unroll
        for (int q = 0; q < HD / 64; ++q)
          #pragma unroll
          for (int p = 0; p < 2; ++p) {
            constexpr uint32_t E = NIB_E << 3, O = NIB_O << 3;
            const uint32_t lo = vx[t][q][2 * p], hi = vx[t][q][2 * p + 1], lo0 = lo << 3, hi0 = hi << 3, lo2 = lo >> 5, hi2 = hi >> 5;
            mma16816(acc[(2 * q + p) * 2], lo0 & E, lo0 & O, hi0 & E, hi0 & O, pb[2 * t], pb[2 * t + 1]);
            mma16816(acc[(2 * q + p) * 2 + 1], lo2 & E, lo2 & O, hi2 & E, hi2 & O, pb[2 * t], pb[2 * t + 1]);
          }
    };

    bool ok = true;
    int k0 = 0;                                                  // units of the items before this one
    for (int n = 0; ; ++n) {                                     // items
    const int nq = it.nq, nu4 = it.nu4, u0 = it.u0, nu = it.nu, len = it.len, r = it.r, kvh = it.kvh, split = it.split;
    const bool has_tail = it.has_tail;
    // Slot kk = (unit kk/4 of this CTA, group kk%4 of the unit), round-robin over the consumer warps: a fixed assignment, so
    // the summation order and with it every bit of the result is the same from run to run (handing slots out from a shared
    // counter was measured: no faster with two warps per scheduler, and not reproducible).
    for (int kk = warp; kk < nu * L::UG && ok; kk += NCW) {
      const int sub = kk % L::UG, u = u0 + kk / L::UG, k = k0 + kk / L::UG, s = k % NSTAGE;
      const bool tail = has_tail && u == nu4, none = tail ? sub != 0 : u * L::UG + sub >= nq;   // the unit holds fewer than four groups
      if (!Q && none) continue;
      const uint32_t st = sbase + L::OFF_STAGES + s * L::STAGE;
      // A wait tells a stage's phases apart by parity only, and a warp has no slot in some units: while such a unit is still on its way, the wait for
      // the next one in its stage would return on the phase before both.  So the unit is seen issued first, which is behind the end of that phase.
      const uint32_t full = bar_full + 8 * s, parity = (k / NSTAGE) & 1;
      uint32_t polls = 0;
      while (s_tag[s] != k && ++polls < WAIT_LIMIT) mbar_try_wait(full, parity);
      if (polls >= WAIT_LIMIT || !mbar_wait(full, parity)) { atomicExch(&g_decode_status, 1); *s_abort = 1; ok = false; break; }
      if (!none) {
        if (tail) group(std::true_type{}, st, 0, len - nq * 32);
        else group(std::false_type{}, st, sub, 32);
      }
      __syncwarp();                                              // no lane still reads the stage or polls its barrier
      if (lane == 0) mbar_arrive(bar_empty + 8 * s);             // one of the four arrivals that free the stage
    }

    // Q: the item after this one, and its queries on their way while this one is merged
    bool more = false;
    uint32_t qnext[Q ? NQE : 1];
    if (Q) {
      int x = 0, y = 0, z = 0;
      if (*s_abort) ok = false;
      if (ok && !mbar_wait(bar_clc + 8 * (n & 1), (n >> 1) & 1)) { atomicExch(&g_decode_status, 1); *s_abort = 1; ok = false; }
      if (ok) more = cancel_result(resp + 16 * (n & 1), x, y, z);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_clc + 16 + 8 * (n & 1));
      if (more) {
        it = item_at(x, y, z);
        #pragma unroll
        for (int i = 0; i < NQE; ++i) qnext[i] = ct + i * NCW * 32 < NW * 32 * 4 ? q_entry(ct + i * NCW * 32, it) : 0u;
      }
    }
    // ---- all consumers done with the item: publish per-warp (m, l, O) into the merge buffer
    #pragma unroll
    for (int o = 4; o <= 16; o <<= 1) {
      l[0] += __shfl_xor_sync(0xffffffffu, l[0], o); l[1] += __shfl_xor_sync(0xffffffffu, l[1], o);
      zacc[0] += __shfl_xor_sync(0xffffffffu, zacc[0], o); zacc[1] += __shfl_xor_sync(0xffffffffu, zacc[1], o);
    }
    // ---- merge the consumer warps and store this split's partial (natural-log m, as the merge kernel expects).  Every warp
    //      scales its own sums by the weight of its maximum and leaves them as they lie in its registers (16 bytes per lane, no bank
    //      conflicts), half of the m-tiles at a time; the sum over the warps runs in warp order.
    if (g == 0) *reinterpret_cast<float4*>(smem + L::OFF_ML + (warp * 4 + j) * 16) = make_float4(m[0], l[0], m[1], l[1]);
    bool bad;                                                    // an abort is seen by all threads or by none
    {
      uint32_t any; const uint32_t mine = !ok || *s_abort;
      asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}" : "=r"(any) : "r"(mine), "n"(NCW * 32) : "memory");
      bad = any != 0;
    }
    if (!bad) {
      float M2[2] = {-1e30f, -1e30f}, L2[2] = {0.f, 0.f};
      float4 ml[NCW];
      #pragma unroll
      for (int w = 0; w < NCW; ++w) {
        ml[w] = *reinterpret_cast<const float4*>(smem + L::OFF_ML + (w * 4 + j) * 16);
        M2[0] = fmaxf(M2[0], ml[w].x); M2[1] = fmaxf(M2[1], ml[w].z);
      }
      const float sc0 = m[0] > -1e29f ? ex2(m[0] - M2[0]) : 0.f, sc1 = m[1] > -1e29f ? ex2(m[1] - M2[1]) : 0.f;
      const size_t p0 = ((size_t)r * A.splits + split) * A.nh + kvh * G;
      if (warp == NCW - 1 && g == 0) {
        #pragma unroll
        for (int w = 0; w < NCW; ++w) {
          L2[0] += (ml[w].x > -1e29f ? ex2(ml[w].x - M2[0]) : 0.f) * ml[w].y;
          L2[1] += (ml[w].z > -1e29f ? ex2(ml[w].z - M2[1]) : 0.f) * ml[w].w;
        }
        #pragma unroll
        for (int x = 0; x < 2; ++x)
          if (2 * j + x < G) { A.pm[p0 + 2 * j + x] = M2[x] > -1e29f ? M2[x] * LN2 : -1e30f; A.pl[p0 + 2 * j + x] = L2[x]; }
      }
      const bool wide = !((uintptr_t)A.pacc & 15);
      float4* mbuf = reinterpret_cast<float4*>(smem + L::OFF_MERGE);
      #pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (half) asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32) : "memory");
        #pragma unroll
        for (int t = 0; t < L::NH; ++t) {                        // m-tile: (even | odd channel) x (head 2j | 2j+1)
          const int mt = half * L::NH + t;
          mbuf[(warp * L::NH + t) * 32 + lane] = make_float4(fmaf(acc[mt][0], VNIB_E_INV, zacc[0]) * sc0, fmaf(acc[mt][1], VNIB_E_INV, zacc[1]) * sc1,
                                                             fmaf(acc[mt][2], VNIB_O_INV, zacc[0]) * sc0, fmaf(acc[mt][3], VNIB_O_INV, zacc[1]) * sc1);
        }
        if (Q && more && half == 0) {                            // nobody still reads the Q fragments of this item
          #pragma unroll
          for (int i = 0; i < NQE; ++i) if (ct + i * NCW * 32 < NW * 32 * 4) reinterpret_cast<uint32_t*>(smem + L::OFF_QFRAG)[ct + i * NCW * 32] = qnext[i];
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32) : "memory");
        if (warp < L::NH / 2) {                                  // a warp per pair of m-tiles: a lane has four channels of two heads
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
          #pragma unroll
          for (int w = 0; w < NCW; ++w) {
            const float4 x = mbuf[(w * L::NH + 2 * warp) * 32 + lane], y = mbuf[(w * L::NH + 2 * warp + 1) * 32 + lane];
            a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w; b.x += y.x; b.y += y.y; b.z += y.z; b.w += y.w;
          }
          const int c = 32 * (half * (L::NH / 2) + warp) + 4 * g;
          float* o0 = A.pacc + (p0 + 2 * j) * HD + c;
          if (wide) {
            if (2 * j < G) *reinterpret_cast<float4*>(o0) = make_float4(a.x, a.z, b.x, b.z);
            if (2 * j + 1 < G) *reinterpret_cast<float4*>(o0 + HD) = make_float4(a.y, a.w, b.y, b.w);
          } else {
            if (2 * j < G) { o0[0] = a.x; o0[1] = a.z; o0[2] = b.x; o0[3] = b.z; }
            if (2 * j + 1 < G) { o0[HD] = a.y; o0[HD + 1] = a.w; o0[HD + 2] = b.y; o0[HD + 3] = b.w; }
          }
        }
      }
    }
    if (!Q || !more || bad) break;
    k0 += nu;
    #pragma unroll
    for (int mt = 0; mt < HD / 16; ++mt) { acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f; }
    m[0] = m[1] = -1e30f;
    l[0] = l[1] = zacc[0] = zacc[1] = 0.f;
    }
  }
}

// ---------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr; cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// 2-D tensor map [rows][cols] of 8- or 16-bit elements, box = box_rows x box_cols.
bool make_map(CUtensorMap* out, const void* base, int elem, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle sw) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * elem};
  const cuuint32_t box[2] = {box_cols, box_rows}, estr[2] = {1, 1};
  return fn(out, elem == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Packed rows in units of 128 tokens, swizzle = row width.
bool make_unit_map(CUtensorMap* out, const void* base, int kvh, int max_ctx, int hd) {
  return make_map(out, base, 1, (uint64_t)kvh * max_ctx, hd / 2, 128, hd / 2, hd == 256 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
}

// The maps of one cache: units of 128 tokens of the packed rows (swizzle = row width), four rows of the group arrays, 128 values of the token arrays.
bool make_maps(Maps* out, const yskn_kv_layer& l, int kvh, int max_ctx, int hd) {
  struct Key {
    const void* p[6]; int kvh, max_ctx, hd;
    bool operator==(const Key& o) const { return memcmp(p, o.p, sizeof(p)) == 0 && kvh == o.kvh && max_ctx == o.max_ctx && hd == o.hd; }
  };
  struct Hash {
    size_t operator()(const Key& k) const {
      size_t h = (size_t)k.max_ctx * 1315423911u ^ (size_t)(k.kvh * 512 + k.hd);
      for (const void* p : k.p) h = (h ^ std::hash<const void*>()(p)) * 0x100000001B3ull;
      return h;
    }
  };
  static std::mutex mu; static std::unordered_map<Key, Maps, Hash> cache;
  std::lock_guard<std::mutex> lk(mu);
  const Key key{{l.kq, l.vq, l.kscale, l.kzero, l.vscale, l.vzero}, kvh, max_ctx, hd};
  auto it = cache.find(key);
  if (it != cache.end()) { *out = it->second; return true; }
  const uint64_t rows = (uint64_t)kvh * max_ctx;
  const CUtensorMapSwizzle none = CU_TENSOR_MAP_SWIZZLE_NONE;
  if (!make_unit_map(&out->k, l.kq, kvh, max_ctx, hd) || !make_unit_map(&out->v, l.vq, kvh, max_ctx, hd) ||
      !make_map(&out->ks, l.kscale, 2, rows / 32, hd, 4, hd, none) || !make_map(&out->kz, l.kzero, 2, rows / 32, hd, 4, hd, none) ||
      !make_map(&out->vs, l.vscale, 2, kvh, max_ctx, 1, 128, none) || !make_map(&out->vz, l.vzero, 2, kvh, max_ctx, 1, 128, none)) return false;
  if (cache.size() > 1024) cache.clear();
  cache.emplace(key, *out);
  return true;
}

// Tensor map over the rope table viewed as one row of RD floats per 32-token group (row stride = 32 table rows), box = 4 rows.
bool make_rope_map(CUtensorMap* out, const float* rope, int rd, uint64_t groups) {
  struct Key { const void* p; uint64_t n; int rd; bool operator==(const Key& o) const { return p == o.p && n == o.n && rd == o.rd; } };
  struct Hash { size_t operator()(const Key& k) const { return std::hash<const void*>()(k.p) ^ (k.n * 2654435761u) ^ (size_t)k.rd; } };
  static std::mutex mu; static std::unordered_map<Key, CUtensorMap, Hash> cache;
  std::lock_guard<std::mutex> lk(mu);
  const Key key{rope, groups, rd};
  auto it = cache.find(key);
  if (it != cache.end()) { *out = it->second; return true; }
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)rd, groups}, strides[1] = {(cuuint64_t)32 * rd * 4};
  const cuuint32_t box[2] = {(cuuint32_t)rd, 4}, estr[2] = {1, 1};
  if (fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(rope), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return false;
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *out);
  return true;
}

template <int HD, int RD, int DT, bool Q, bool multi>
int launch_m(const yskn_attn_g_args& a, int g, Shard sh, int early, const yskn_kv4_ms_rows& ms, const Maps& mp, const CUtensorMap& mr, cudaStream_t st) {
  using L = Lay<HD, RD, Q>;
  auto kern = kv4_decode_mma_kernel<HD, RD, DT, Q, multi>;
  static std::atomic<unsigned long long> attr{0};               // once per device, like the reference's launchers once per process
  if (first_use_on_device(attr)) {
    KV4_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
    KV4_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  }
  DecodeP P{a, sh, g, early, ms};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(a.splits, a.kvh, a.M); cfg.blockDim = dim3(NTHREADS); cfg.dynamicSmemBytes = L::TOTAL; cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  KV4_CUDA(cudaLaunchKernelEx(&cfg, kern, mp, mr, P));
  return launch_status("kv4_decode_mma_kernel");
}

template <int HD, int RD, int DT, bool Q>
int launch_q(const yskn_attn_g_args& a, int g, Shard sh, int early, const yskn_kv4_ms_rows& ms, const Maps& mp, const CUtensorMap& mr, cudaStream_t st) {
  if (ms.pos) return launch_m<HD, RD, DT, Q, true>(a, g, sh, early, ms, mp, mr, st);
  return launch_m<HD, RD, DT, Q, false>(a, g, sh, early, ms, mp, mr, st);
}

// One CTA fills an SM, so a grid of up to one block per SM starts at once and has nothing to take over; a larger one runs as a queue.
template <int HD, int RD, int DT>
int launch_t(const yskn_attn_g_args& a, int g, Shard sh, int early, const yskn_kv4_ms_rows& ms, const Maps& mp, const CUtensorMap& mr, cudaStream_t st) {
  int dev = 0, sms = 0;
  KV4_CUDA(cudaGetDevice(&dev));
  KV4_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if ((long long)a.splits * a.kvh * a.M > sms) return launch_q<HD, RD, DT, true>(a, g, sh, early, ms, mp, mr, st);
  return launch_q<HD, RD, DT, false>(a, g, sh, early, ms, mp, mr, st);
}

template <int HD, int RD>
int launch_dt(const yskn_attn_g_args& a, int g, int dt, Shard sh, int early, const yskn_kv4_ms_rows& ms, const Maps& mp, const CUtensorMap& mr, cudaStream_t st) {
  if (dt == YSKN_KV4_BF16) return launch_t<HD, RD, YSKN_KV4_BF16>(a, g, sh, early, ms, mp, mr, st);
  return launch_t<HD, RD, YSKN_KV4_F16>(a, g, sh, early, ms, mp, mr, st);
}

}  // namespace

bool decode_mma_supports(int g, int hd, int rd, int M) {
  if (g < 1 || g > 8 || M < 1 || M > 8) return false;
  return (hd == 256 && (rd == 64 || rd == 0)) || (hd == 128 && (rd == 128 || rd == 0));
}

// Uploads the table of per-sequence cache arrays and their K / V tensor maps for yskn_kv4_attention_ms (set-up: it copies from host memory).
int ms_prepare(const yskn_kv_layer* h_layers, int n_slots, int kvh, int hd, int max_ctx, yskn_kv_layer* d_layers, void* d_maps, cudaStream_t st) {
  if (!h_layers || !d_layers || !d_maps || n_slots <= 0 || n_slots > 64) KV4_REJECT("yskn_kv4_ms_prepare: bad arguments (n_slots %d)", n_slots);
  if (kvh <= 0 || (hd != 128 && hd != 256) || max_ctx <= 0 || max_ctx % 64) KV4_REJECT("yskn_kv4_ms_prepare: bad shape (kvh %d, hd %d, max_ctx %d)", kvh, hd, max_ctx);
  if ((uintptr_t)d_maps & 127) KV4_REJECT("yskn_kv4_ms_prepare: the map table must be 128-byte aligned");
  std::vector<CUtensorMap> maps(2 * (size_t)n_slots);
  for (int s = 0; s < n_slots; ++s) {
    const yskn_kv_layer& l = h_layers[s];
    const uintptr_t al = (uintptr_t)l.kq | (uintptr_t)l.vq | (uintptr_t)l.kscale | (uintptr_t)l.kzero | (uintptr_t)l.kshadow | (uintptr_t)l.vscale | (uintptr_t)l.vzero;
    if (!l.kq || !l.vq || !l.kscale || !l.kzero || !l.kshadow || !l.vscale || !l.vzero || (al & 15))
      KV4_REJECT("yskn_kv4_ms_prepare: cache arrays of slot %d missing or not 16-byte aligned", s);
    if (!make_unit_map(&maps[2 * s], l.kq, kvh, max_ctx, hd) || !make_unit_map(&maps[2 * s + 1], l.vq, kvh, max_ctx, hd))
      KV4_REJECT("yskn_kv4_ms_prepare: cuTensorMapEncodeTiled failed or is unavailable");
  }
  KV4_CUDA(cudaMemcpyAsync(d_maps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, st));
  KV4_CUDA(cudaMemcpyAsync(d_layers, h_layers, (size_t)n_slots * sizeof(yskn_kv_layer), cudaMemcpyHostToDevice, st));
  KV4_CUDA(cudaStreamSynchronize(st));                            // the host vectors go out of scope
  return 0;
}

int launch_decode_mma(const yskn_attn_g_args& a, int g, int hd, int rd, int act_dtype, Shard sh, int early, cudaStream_t st,
                      const yskn_kv4_ms_rows* ms) {
  const bool multi = ms != nullptr;
  if (multi ? !decode_mma_supports(g, hd, rd, 1) || a.M < 1 || a.M > 64 : !decode_mma_supports(g, hd, rd, a.M))
    KV4_REJECT("yskn_kv4_attention: tensor-core decode does not cover (g %d, hd %d, rd %d, M %d)", g, hd, rd, a.M);
  const uintptr_t al = multi ? (uintptr_t)a.rope
                             : (uintptr_t)a.kv.kq | (uintptr_t)a.kv.vq | (uintptr_t)a.kv.kscale | (uintptr_t)a.kv.kzero | (uintptr_t)a.kv.kshadow |
                               (uintptr_t)a.kv.vscale | (uintptr_t)a.kv.vzero | (uintptr_t)a.rope;
  if (al & 15) KV4_REJECT("yskn_kv4_attention: cache arrays and rope table must be 16-byte aligned");
  Maps mp;
  CUtensorMap mr;
  if (multi) memset(&mp, 0, sizeof(mp));                          // the kernel takes the maps of the row's sequence from ms->maps
  else if (!make_maps(&mp, a.kv, a.kvh, a.max_ctx, hd))
    KV4_REJECT("yskn_kv4_attention: cuTensorMapEncodeTiled failed or is unavailable");
  const yskn_kv4_ms_rows msv = multi ? *ms : yskn_kv4_ms_rows{nullptr, nullptr, nullptr, nullptr, 0};
  if (multi) early = 0;                                           // rows of one sequence in the same pass are appended by the predecessor
  // The rope table must cover positions [0, shard start + shard length); groups past that read as zero and are never used.
  if (rd == 0) mr = mp.k;
  else if (!make_rope_map(&mr, a.rope, rd, ((uint64_t)sh.start + (uint64_t)sh.len) / 32))
    KV4_REJECT("yskn_kv4_attention: cuTensorMapEncodeTiled failed for the rope table");
  if (hd == 256) return rd ? launch_dt<256, 64>(a, g, act_dtype, sh, early, msv, mp, mr, st) : launch_dt<256, 0>(a, g, act_dtype, sh, early, msv, mp, mr, st);
  return rd ? launch_dt<128, 128>(a, g, act_dtype, sh, early, msv, mp, mr, st) : launch_dt<128, 0>(a, g, act_dtype, sh, early, msv, mp, mr, st);
}

int decode_status_fetch(int* out) {
  int v = 0;
  KV4_CUDA(cudaMemcpyFromSymbol(&v, g_decode_status, sizeof(int)));
  const int zero = 0;
  KV4_CUDA(cudaMemcpyToSymbol(g_decode_status, &zero, sizeof(int)));
  *out = v; return 0;
}

}  // namespace kv4
