// KV4 quantize-and-append codec and the RoPE table (sm_100a).
//
// Bit-exact restatement, in new kernels, of the reference's
//   K shadow store            src/post_kernels.cu:48-54
//   per-token V int4          src/post_kernels.cu:64-82
//   32-token K group int4     src/attention_gqa.cu:143-154 (= src/post_kernels.cu:86-96)
//   (cos,sin) table           src/attention_gqa.cu:158-162
// Every arithmetic step that decides a stored bit uses an explicit round-to-nearest intrinsic, so the
// result does not depend on the compiler's FMA contraction (the reference relies on --fmad=false).
//
// Byte movers: every load of a warp is one contiguous 128..512-byte segment.
#include "kv4_common.cuh"
#include <cmath>

namespace kv4 {
namespace {

__device__ __forceinline__ int quant4(float v, float lo, float inv) {
  int q = __float2int_rn(__fmul_rn(__fsub_rn(v, lo), inv));
  return q < 0 ? 0 : (q > 15 ? 15 : q);
}

// Programmatic dependent launch: a decode pass is three short launches, and the start of each is hidden behind the one before.  The
// successor is let in only behind the wait, so what it reads ahead of its own wait (yskn_kv4_attn_ext.early) is
// no newer than the launch before this one.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b) { uint32_t d; asm("min.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) { uint32_t d; asm("max.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
// Channels i, i + 1 of the key rows: fp32 as fp16, 16-bit types as they are; PAIRS: the array is aligned for one load.
template <int DT, bool PAIRS> __device__ __forceinline__ uint32_t load_pair(const void* p, size_t i) {
  if (DT == YSKN_KV4_F32) return (uint32_t)f2h(static_cast<const float*>(p)[i]) | ((uint32_t)f2h(static_cast<const float*>(p)[i + 1]) << 16);
  const uint16_t* h = static_cast<const uint16_t*>(p) + i;
  return PAIRS ? *reinterpret_cast<const uint32_t*>(h) : (uint32_t)h[0] | ((uint32_t)h[1] << 16);
}
// A pair of them as fp16; fp16 too, so that a NaN has one form (x + -0 is x for every other x).
template <int DT> __device__ __forceinline__ uint32_t act_pair(uint32_t u) {
  uint32_t d = u;
  if (DT == YSKN_KV4_BF16) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(u & 0xffff0000u)), "f"(__uint_as_float(u << 16)));
  if (DT == YSKN_KV4_F16) asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(u), "r"(0x80008000u));
  return d;
}

constexpr int KB = 8;                                // key rows of a batch: their loads are in flight together

// Keys: 64 channels of a 32-token group by one warp, two channels a lane.  Rows [first, end) of the pass go to the fp16 shadow; a group that this pass
// completes is quantised: per channel min / max over the 32 rows, fp16 scale and zero, int4 codes (src/attention_gqa.cu:143-154).  The codes
// are formed from the shadow read a second time (a lane's own stores, and lines that were just read): to keep the first walk's values in registers
// the loops would be unrolled, and code that runs once per launch comes from memory itself.
template <int HD, int DT, bool PAIRS>
__device__ __forceinline__ void keys_warp(const yskn_kv_layer& kv, int max_ctx, const void* k_in, int kvh, int pos0, int first, int end, int gi, int head, int c,
                                          bool closes) {
  uint16_t* rows = kv.kshadow + ((size_t)head * max_ctx + (size_t)gi * 32) * HD + c;
  const int f = first - gi * 32, e = end - gi * 32;  // rows of this pass
  uint32_t lo2 = 0x7C007C00u, hi2 = 0xFC00FC00u;
  #pragma unroll 1
  for (int t0 = closes ? 0 : f & ~(KB - 1); t0 < (closes ? 32 : e); t0 += KB) {
    uint32_t v[KB];
    #pragma unroll
    for (int i = 0; i < KB; ++i) {
      const int t = t0 + i;
      const bool mine = t >= f && t < e;
      v[i] = 0u;
      if (mine) v[i] = load_pair<DT, PAIRS>(k_in, ((size_t)(gi * 32 + t - pos0) * kvh + head) * HD + c);
      if (!mine && closes) v[i] = *reinterpret_cast<const uint32_t*>(rows + (size_t)t * HD);
    }
    #pragma unroll
    for (int i = 0; i < KB; ++i) {
      const int t = t0 + i;
      if (t >= f && t < e) {
        v[i] = act_pair<DT>(v[i]);
        *reinterpret_cast<uint32_t*>(rows + (size_t)t * HD) = v[i];
      }
      lo2 = min2(lo2, v[i]); hi2 = max2(hi2, v[i]);
    }
  }
  if (!closes) return;
  float lo[2], inv[2];
  uint32_t s2 = 0, z2 = 0;
  #pragma unroll
  for (int k = 0; k < 2; ++k) {                      // within the bounds that the reference's search starts from
    lo[k] = fminf(1e30f, h2f((uint16_t)(lo2 >> (16 * k))));
    const float hi = fmaxf(-1e30f, h2f((uint16_t)(hi2 >> (16 * k)))), d = __fsub_rn(hi, lo[k]);
    inv[k] = hi > lo[k] ? __fdiv_rn(15.f, d) : 0.f;
    s2 |= (uint32_t)f2h(__fdiv_rn(d, 15.f)) << (16 * k);
    z2 |= (uint32_t)f2h(lo[k]) << (16 * k);
  }
  const size_t gb = (size_t)head * (max_ctx / 32) + gi;
  *reinterpret_cast<uint32_t*>(kv.kscale + gb * HD + c) = s2;
  *reinterpret_cast<uint32_t*>(kv.kzero + gb * HD + c) = z2;
  uint8_t* kq = kv.kq + gb * 32 * (HD / 2) + c / 2;  // a warp's 32 bytes of a row are one sector
  #pragma unroll 1
  for (int t0 = 0; t0 < 32; t0 += KB) {
    uint32_t v[KB];
    #pragma unroll
    for (int i = 0; i < KB; ++i) v[i] = *reinterpret_cast<const uint32_t*>(rows + (size_t)(t0 + i) * HD);
    #pragma unroll
    for (int i = 0; i < KB; ++i)
      kq[(size_t)(t0 + i) * (HD / 2)] = (uint8_t)(quant4(h2f((uint16_t)v[i]), lo[0], inv[0]) | (quant4(h2f((uint16_t)(v[i] >> 16)), lo[1], inv[1]) << 4));
  }
}

// Values: rows first, first + step, .. below end by one warp, each to int4 with its fp16 scale and zero; the next row is on its way meanwhile.
template <int HD, int DT>
__device__ __forceinline__ void values_warp(const yskn_kv_layer& kv, int max_ctx, const void* v_in, int kvh, int pos0, int first, int end, int step, int head, int lane,
                                            bool wide) {
  constexpr int CPL = HD / 32;                       // channels per lane (2, 4 or 8)
  struct Row { uint32_t u[DT == YSKN_KV4_F32 ? CPL : CPL / 2]; };
  auto load = [&](int pos, Row& r) {
    const size_t i = ((size_t)(pos - pos0) * kvh + head) * HD + (size_t)lane * CPL;
    if constexpr (DT == YSKN_KV4_F32) {
      #pragma unroll
      for (int e = 0; e < CPL; ++e) r.u[e] = __float_as_uint(static_cast<const float*>(v_in)[i + e]);
    } else {
      const uint16_t* p = static_cast<const uint16_t*>(v_in) + i;
      if (!wide) {
        #pragma unroll
        for (int e = 0; e < CPL; e += 2) r.u[e / 2] = (uint32_t)p[e] | ((uint32_t)p[e + 1] << 16);
      } else if constexpr (CPL == 8) { const uint4 u = *reinterpret_cast<const uint4*>(p); r.u[0] = u.x; r.u[1] = u.y; r.u[2] = u.z; r.u[3] = u.w; }
      else if constexpr (CPL == 4) { const uint2 u = *reinterpret_cast<const uint2*>(p); r.u[0] = u.x; r.u[1] = u.y; }
      else r.u[0] = *reinterpret_cast<const uint32_t*>(p);
    }
  };
  Row next;
  if (first < end) load(first, next);
  #pragma unroll 1
  for (int pos = first; pos < end; pos += step) {
    const Row row = next;
    if (pos + step < end) load(pos + step, next);
    float y[CPL];
    #pragma unroll
    for (int e = 0; e < CPL; ++e) {
      if (DT == YSKN_KV4_F32) y[e] = round_f16(__uint_as_float(row.u[e]));
      else {
        const uint16_t h = (uint16_t)(row.u[e / 2] >> (16 * (e & 1)));
        y[e] = round_f16(DT == YSKN_KV4_BF16 ? bf2f(h) : h2f(h));
      }
    }
    float lo = y[0], hi = y[0];
    #pragma unroll
    for (int e = 1; e < CPL; ++e) { lo = fminf(lo, y[e]); hi = fmaxf(hi, y[e]); }
    #pragma unroll
    for (int o = 16; o; o >>= 1) { lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o)); hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o)); }
    const float sc = __fdiv_rn(__fsub_rn(hi, lo), 15.f);
    const float inv = hi > lo ? __fdiv_rn(15.f, __fsub_rn(hi, lo)) : 0.f;
    const size_t slot = (size_t)head * max_ctx + pos;
    uint8_t* vq = kv.vq + slot * (HD / 2) + (size_t)lane * (CPL / 2);
    uint32_t packed = 0;
    #pragma unroll
    for (int e = 0; e < CPL; ++e) packed |= (uint32_t)quant4(y[e], lo, inv) << (4 * e);
    if (CPL == 8) *reinterpret_cast<uint32_t*>(vq) = packed;
    else if (CPL == 4) *reinterpret_cast<uint16_t*>(vq) = (uint16_t)packed;
    else *vq = (uint8_t)packed;
    if (lane == 0) { kv.vscale[slot] = f2h(sc); kv.vzero[slot] = f2h(lo); }
  }
}

// One launch for any number of rows: K rows -> fp16 shadow and, where the pass appends a group's 32nd token, the group's int4 keys
// (src/attention_gqa.cu:145-146; in the append launch, as the reference's epilogue does at M = 1: src/post_kernels.cu:55-63); V rows -> int4 + fp16
// scale/zero.  Warps know their work by number: first the keys, (group that the pass touches, kv-head, 64 channels), then the values, (group,
// kv-head, one of `vw` shares of its rows).  Nothing passes between warps.
// Bound by HBM for a prompt (4 KB in, 2.6 KB out per token of four 256-channel heads), by trips to memory for a few rows, and by what room it
// leaves the attention kernel behind it: see append_hd.
template <int HD, int DT, bool PAIRS>
__global__ void __launch_bounds__(256, 4) kv4_append_kernel(yskn_kv_append_args A, int groups, int vw, int wide) {
  const int lane = threadIdx.x & 31, nk = groups * A.kvh * (HD / 64);
  int w = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  pdl_enter();
  const int pos0 = *A.d_pos, last = (int)((unsigned)pos0 + (unsigned)A.M - 1u);
  const bool keys = w < nk;
  if (!keys) w -= nk;
  const int parts = keys ? HD / 64 : vw, part = w % parts, gh = w / parts, gi = (pos0 >> 5) + gh / A.kvh, head = gh % A.kvh, gend = gi * 32 + 31;
  // A group outside the cache is told by its number, which no position makes wrap; positions whose last row would wrap have no other groups.  (A
  // comparison of the position ahead of all this cost every decode step 0.2 us.)
  if (gh >= groups * A.kvh || (unsigned)gi >= (unsigned)A.max_ctx / 32u || gi * 32 > last) return;
  const int first = max(pos0, gi * 32), end = min(last, gend) + 1;               // rows of this pass in the group
  if (keys) keys_warp<HD, DT, PAIRS>(A.kv, A.max_ctx, A.k_in, A.kvh, pos0, first, end, gi, head, part * 64 + 2 * lane, gend >= pos0 && gend <= last);
  else values_warp<HD, DT>(A.kv, A.max_ctx, A.v_in, A.kvh, pos0, first + part, end, vw, head, lane, wide != 0);
}

// The group step alone, from shadow rows that are there: one warp per (candidate group, kv-head, 64 channels).
template <int HD>
__global__ void __launch_bounds__(128) kv4_group_quant_kernel(yskn_kv_quant_args A, int kvh) {
  const int lane = threadIdx.x & 31, w = blockIdx.x * 4 + (threadIdx.x >> 5), part = w % (HD / 64), gh = w / (HD / 64);
  pdl_enter();
  const int pos0 = *A.d_pos, last = (int)((unsigned)pos0 + (unsigned)A.M - 1u), gi = pos0 / 32 + gh / kvh, head = gh % kvh, gend = gi * 32 + 31;
  if (gh >= ((A.M + 31) / 32 + 1) * kvh || (unsigned)gi >= (unsigned)A.max_ctx / 32u || gend < pos0 || gend > last) return;
  keys_warp<HD, YSKN_KV4_F16, true>(A.kv, A.max_ctx, nullptr, kvh, pos0, gi * 32, gi * 32, gi, head, part * 64 + 2 * lane, true);
}

// out[t][i] = (cos, sin)(float(t) * freq_i), freq_i = theta^(-2i/rd).  The fp32 product that defines the
// angle is kept (src/attention_gqa.cu:161); the exponent and the trigonometric functions are taken in double
// and rounded once, which makes the table reproducible on a CPU to the last bit in all but rare cases.
__global__ void kv4_rope_table_kernel(float2* out, int max_ctx, float theta, int rd) {
  const int half = rd / 2;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)max_ctx * half) return;
  const int t = (int)(idx / half), i = (int)(idx % half);
  const float freq = (float)pow((double)theta, -(double)(2 * i) / (double)rd);
  const float ang = __fmul_rn((float)t, freq);
  double s, c; sincos((double)ang, &s, &c);
  out[idx] = make_float2((float)c, (float)s);
}

// Blocks.  The attention kernel is launched while this one runs (programmatic launch) and sets itself up beside it where an SM has room.  Of the decode
// kernel's forms, one CTA of 256 threads an SM, only the single-wave one of head_dim 256 leaves room (232 registers a thread, 61,440 of 65,536 by
// blocks; the queue and the rotary forms of 128 channels take 254 or 255), and there blocks of 64, 128 and 256 threads came out the same for up to
// eight rows (one row 19.8, 11.3 and 81.5 us, five rows 50.4).  The tcgen05 kernel takes all of an SM's registers; blocks of 32 warps on as few SMs
// as possible were slower than its wait for room (64 rows: 9.0 us against 4.0 in blocks of four warps).
template <int HD> int append_hd(const yskn_kv_append_args& a, cudaStream_t st) {
  const int groups = (a.M + 30) / 32 + 1;                        // groups that M rows can touch
  const int vw = a.M < 8 ? a.M : 8;
  const int threads = a.M <= 64 ? 128 : 256;
  const long long warps = (long long)groups * a.kvh * (HD / 64 + vw);
  const dim3 blocks((unsigned)((warps * 32 + threads - 1) / threads));
  const char* who = "kv4_append_kernel";
  const int wide = ((uintptr_t)a.v_in & (HD / 16 - 1)) == 0;     // a lane's HD / 32 values in one load
  const bool pairs = ((uintptr_t)a.k_in & 3) == 0;               // two keys in one load
  switch (a.in_dtype) {
    case YSKN_KV4_F16: return launch_pdl(who, pairs ? kv4_append_kernel<HD, YSKN_KV4_F16, true> : kv4_append_kernel<HD, YSKN_KV4_F16, false>, blocks, threads, 0, st, a, groups, vw, wide);
    case YSKN_KV4_BF16: return launch_pdl(who, pairs ? kv4_append_kernel<HD, YSKN_KV4_BF16, true> : kv4_append_kernel<HD, YSKN_KV4_BF16, false>, blocks, threads, 0, st, a, groups, vw, wide);
    case YSKN_KV4_F32: return launch_pdl(who, kv4_append_kernel<HD, YSKN_KV4_F32, false>, blocks, threads, 0, st, a, groups, vw, wide);
    default: KV4_REJECT("yskn_kv4_append: unknown in_dtype %d", a.in_dtype);
  }
}

// A copy by a kernel, for the few kilobytes a decode step exchanges with the host: either side may be pinned (mapped) host
// memory.  Inside a captured pass a kernel node of this size runs in about 2 us where a memcpy node takes about 6.  Host
// memory is read past the caches (ld.global.cv), so a replayed graph sees what the host wrote since the last replay.
__global__ void __launch_bounds__(256) kv4_copy16_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, size_t n16) {
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i < n16) dst[i] = __ldcv(src + i);
}

}  // namespace

int launch_copy16(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return 0;
  if (!dst || !src) KV4_REJECT("yskn_kv4_copy: null buffer");
  if ((bytes & 15) || (((uintptr_t)dst | (uintptr_t)src) & 15)) KV4_REJECT("yskn_kv4_copy: %zu bytes: size and both addresses must be multiples of 16", bytes);
  if (bytes > ((size_t)1 << 26)) KV4_REJECT("yskn_kv4_copy: %zu bytes: meant for small buffers (at most 64 MiB)", bytes);
  const size_t n16 = bytes / 16;
  kv4_copy16_kernel<<<(unsigned)((n16 + 255) / 256), 256, 0, st>>>(static_cast<const uint4*>(src), static_cast<uint4*>(dst), n16);
  return launch_status("kv4_copy16_kernel");
}

int launch_rope_table(float* d_out, int max_ctx, float theta, int rd, cudaStream_t st) {
  if (!d_out || max_ctx <= 0 || rd <= 0 || (rd & 1)) KV4_REJECT("yskn_kv4_rope_table: bad arguments (max_ctx %d, rd %d)", max_ctx, rd);
  const long long n = (long long)max_ctx * (rd / 2);
  kv4_rope_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(reinterpret_cast<float2*>(d_out), max_ctx, theta, rd);
  return launch_status("kv4_rope_table_kernel");
}

int launch_group_quant(const yskn_kv_quant_args& a, int kvh, int hd, cudaStream_t st) {
  if (a.M <= 0 || kvh <= 0 || !a.d_pos || a.max_ctx % 32) KV4_REJECT("yskn_kv4_group_quant: bad arguments (M %d, kvh %d, max_ctx %d)", a.M, kvh, a.max_ctx);
  const dim3 blocks((unsigned)((((a.M + 31) / 32 + 1) * kvh * (hd / 64) + 3) / 4));
  const char* who = "kv4_group_quant_kernel";
  if (hd == 256) return launch_pdl(who, kv4_group_quant_kernel<256>, blocks, 128, 0, st, a, kvh);
  if (hd == 128) return launch_pdl(who, kv4_group_quant_kernel<128>, blocks, 128, 0, st, a, kvh);
  if (hd == 64) return launch_pdl(who, kv4_group_quant_kernel<64>, blocks, 128, 0, st, a, kvh);
  KV4_REJECT("yskn_kv4_group_quant: unsupported head_dim %d (64, 128, 256)", hd);   // src/attention_gqa.cu:186
}

int launch_append(const yskn_kv_append_args& a, cudaStream_t st) {
  if (!a.k_in || !a.v_in || !a.d_pos || a.M <= 0 || a.kvh <= 0 || a.max_ctx % 32)
    KV4_REJECT("yskn_kv4_append: bad arguments (M %d, kvh %d, max_ctx %d)", a.M, a.kvh, a.max_ctx);
  if (a.hd == 256) return append_hd<256>(a, st);
  if (a.hd == 128) return append_hd<128>(a, st);
  if (a.hd == 64) return append_hd<64>(a, st);
  KV4_REJECT("yskn_kv4_append: unsupported head_dim %d (64, 128, 256)", a.hd);
}

}  // namespace kv4
