// Family-B row codec, step 1: sign-Hadamard-256 rotation + INT8 rows with one fp32 scale per row.
//
// Semantics: the reference's src/kvx_codec.cuh as the shipping engine builds it (rotation on, INT8 payload;
// CMakeLists.txt:56): kvx_sign (:28-32), kvx_rotate (:35-49), kvx_store (:50-70); the decode direction is the one its
// probe runs (src/kvx_probe.cu:15-19).  Bit-exact: every operation is one IEEE fp32 operation in the reference's order.
//
// Mapping: eight lanes per row of 256 (a warp holds four rows); a lane keeps 32 elements in registers, so five of the eight
// butterfly stages pair registers and only three go through shuffles, and every load/store instruction of a row's lanes
// covers one contiguous run.  The stages run in the reference's order h = 1, 2, ... 128.  HBM-bound byte mover by design
// (1,284 B per fp32 row in + out, 772 B per fp16 row).
#include "kvx_rotate.cuh"

namespace kv4 {
namespace {

template <int DT> __device__ __forceinline__ void load_row(const void* base, size_t row, int ll, bool live, float (&v)[32]) {
  #pragma unroll
  for (int k = 0; k < 8; ++k) {
    const size_t d = row * 256 + 32 * k + 4 * ll;
    if (DT == YSKN_KV4_F32) {
      const float4 a = live ? *reinterpret_cast<const float4*>(static_cast<const float*>(base) + d) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[4 * k] = a.x; v[4 * k + 1] = a.y; v[4 * k + 2] = a.z; v[4 * k + 3] = a.w;
    } else {
      const uint2 u = live ? *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + d) : make_uint2(0u, 0u);
      v[4 * k] = DT == YSKN_KV4_F16 ? h2f((uint16_t)u.x) : bf2f((uint16_t)u.x); v[4 * k + 1] = DT == YSKN_KV4_F16 ? h2f((uint16_t)(u.x >> 16)) : bf2f((uint16_t)(u.x >> 16));
      v[4 * k + 2] = DT == YSKN_KV4_F16 ? h2f((uint16_t)u.y) : bf2f((uint16_t)u.y); v[4 * k + 3] = DT == YSKN_KV4_F16 ? h2f((uint16_t)(u.y >> 16)) : bf2f((uint16_t)(u.y >> 16));
    }
  }
}
template <int DT> __device__ __forceinline__ void store_row(void* base, size_t row, int ll, const float (&v)[32]) {
  #pragma unroll
  for (int k = 0; k < 8; ++k) {
    const size_t d = row * 256 + 32 * k + 4 * ll;
    if (DT == YSKN_KV4_F32) *reinterpret_cast<float4*>(static_cast<float*>(base) + d) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    else *reinterpret_cast<uint2*>(static_cast<uint16_t*>(base) + d) =
        make_uint2((uint32_t)act_store16<DT>(v[4 * k]) | ((uint32_t)act_store16<DT>(v[4 * k + 1]) << 16),
                   (uint32_t)act_store16<DT>(v[4 * k + 2]) | ((uint32_t)act_store16<DT>(v[4 * k + 3]) << 16));
  }
}

constexpr int ROWS_PER_BLOCK = 32;                         // 8 warps x 4 rows

// mode 0: rotate, 1: inverse rotate (fp32 in, fp32 out)
__global__ void __launch_bounds__(256) kvx_rotate_kernel(const float* x, float* y, long long rows, int inverse) {
  const int lane = threadIdx.x & 31, ll = lane & 7;
  const long long row = (long long)blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 5) * 4 + (lane >> 3);
  const bool live = row < rows;
  float v[32];
  load_row<YSKN_KV4_F32>(x, (size_t)row, ll, live, v);
  if (!inverse) apply_signs(v, ll);
  hadamard256(v, ll);
  if (inverse) apply_signs(v, ll);
  if (live) store_row<YSKN_KV4_F32>(y, (size_t)row, ll, v);
}

// INT8 codes of a row from its rotated values: scale = max|v| / 127, q = rne(v / scale) clamped to +-127 (src/kvx_codec.cuh:50-70).
struct Int8Scale {
  float scale, inv;
  __device__ __forceinline__ explicit Int8Scale(float amax) { scale = __fdiv_rn(amax, 127.f); inv = scale > 0.f ? __fdiv_rn(1.f, scale) : 0.f; }
  // q = rne(fl(v / scale)).  v * (1 / scale) is within 3.8e-5 of the correctly rounded quotient (|q| <= 127), so rounding it gives
  // the same integer unless it lies that close to a half-integer; only those elements (about one in 10^4) take the exact division.
  __device__ __forceinline__ int code(float v) const {
    const float t = __fmul_rn(v, inv);
    int q = __float2int_rn(t);
    // distance of t from the integer it rounds to; near 0.5 (or NaN: 1/scale overflowed) -> the reference's own arithmetic.
    // |v| <= max|v| makes |v / scale| <= 127 (1 + 2^-23), so the reference's clamp to +-127 can only act on that path.
    if (!(fabsf(__fsub_rn(t, (float)q)) <= 0.5f - 6.2e-5f)) q = max(-127, min(127, scale > 0.f ? __float2int_rn(__fdiv_rn(v, scale)) : 0));
    return q;
  }
};
__device__ __forceinline__ void store_int8_row(const float (&v)[32], int ll, bool live, int8_t* q8, float* scales, size_t row) {
  float amax = 0.f;
  #pragma unroll
  for (int i = 0; i < 32; ++i) amax = fmaxf(amax, fabsf(v[i]));
  #pragma unroll
  for (int m = 4; m; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
  const Int8Scale sc(amax);
  #pragma unroll
  for (int k = 0; k < 8; ++k) {
    uint32_t w = 0u;
    #pragma unroll
    for (int e = 0; e < 4; ++e) w |= ((uint32_t)sc.code(v[4 * k + e]) & 0xFFu) << (8 * e);
    if (live) *reinterpret_cast<uint32_t*>(q8 + row * 256 + 32 * k + 4 * ll) = w;
  }
  if (live && ll == 0) scales[row] = sc.scale;
}

template <int DT>
__global__ void __launch_bounds__(256) kvx_encode_kernel(const void* x, int8_t* q8, float* scales, long long rows) {
  const int lane = threadIdx.x & 31, ll = lane & 7;
  const long long row = (long long)blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 5) * 4 + (lane >> 3);
  const bool live = row < rows;
  float v[32];
  load_row<DT>(x, (size_t)row, ll, live, v);
  apply_signs(v, ll);
  hadamard256(v, ll);
  store_int8_row(v, ll, live, q8, scales, (size_t)row);
}

template <int DT>
__global__ void __launch_bounds__(256) kvx_decode_kernel(const int8_t* q8, const float* scales, void* y, long long rows) {
  const int lane = threadIdx.x & 31, ll = lane & 7;
  const long long row = (long long)blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 5) * 4 + (lane >> 3);
  const bool live = row < rows;
  const float sc = live ? scales[row] : 0.f;
  float v[32];
  #pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t u = live ? *reinterpret_cast<const uint32_t*>(q8 + (size_t)row * 256 + 32 * k + 4 * ll) : 0u;
    #pragma unroll
    for (int e = 0; e < 4; ++e) v[4 * k + e] = __fmul_rn((float)(int8_t)(uint8_t)(u >> (8 * e)), sc);
  }
  hadamard256(v, ll);
  apply_signs(v, ll);
  if (live) store_row<DT>(y, (size_t)row, ll, v);
}

// The attention block's row epilogue over INT8 rows: the reference's q35_attn_post_kernel (src/q35_kernels.cu:1013-1065) from
// the point where a thread holds its bf16-rounded projection value (:1029).  One work item = one row of 256: a query head
// (RMS norm, partial RoPE, rotation -> bf16 q16; its gate half is copied), a key head (the same -> INT8 row at the token's
// position) or a value head (rotation -> INT8 row).  Every operation is the reference's single IEEE operation in its order:
// the sum of squares is the reference's xor-shuffle tree per 32 channels (strides 16, 8, 4 = this layout's lane bits, strides
// 2, 1 = register pairs) followed by the in-order sum of the eight warp sums.  NRH = rotary width / 64.
__device__ __forceinline__ float rbf(float f) { return bf2f(f2bf(f)); }

// One warp per row; lane l owns channels 4l .. 4l + 3 (v[0..3]) and 128 + 4l .. (v[4..7]), so a run of 32 channels is eight lanes.  Bound by instruction issue
// and, for a few tokens, by the length of a warp's straight-line code.  (With eight lanes a row, four rows a warp, a warp had 1,000 instructions and
// the GPU a quarter of the warps: steps of one token over 500 / 32,768 INT8 rows 13.9 / 25.5 us, now 11.4 / 22.8; 100 rows behind 3,000 tokens 40.0, now 32.7.)
template <int NRH>
__global__ void __launch_bounds__(256) kvx_attn_post_kernel(yskn_kvx_attn_post_args A) {
  const int lane = threadIdx.x & 31;
  asm volatile("griddepcontrol.wait;" ::: "memory");           // programmatic dependent launch, both directions
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int per_tok = A.nh + 2 * A.kvh;
  const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= (long long)A.M * per_tok) return;
  const int tok = (int)(item / per_tok), u = (int)(item - (long long)tok * per_tok);
  const int kind = u < A.nh ? 0 : (u < A.nh + A.kvh ? 1 : 2);    // query / key / value head
  const int head = kind == 0 ? u : (kind == 1 ? u - A.nh : u - A.nh - A.kvh);
  const uint16_t* src = (kind == 0 ? A.q_rows + ((size_t)tok * A.nh + head) * 512
                                   : (kind == 1 ? A.k_rows : A.v_rows) + ((size_t)tok * A.kvh + head) * 256) + 4 * lane;
  const uint2 in[2] = {*reinterpret_cast<const uint2*>(src), *reinterpret_cast<const uint2*>(src + 128)};
  const size_t orow = ((size_t)tok * A.nh + head) * 256 + 4 * lane;
  if (kind == 0) {                                               // the gate half of the head's projection, as it is
    const uint2 g0 = *reinterpret_cast<const uint2*>(src + 256), g1 = *reinterpret_cast<const uint2*>(src + 384);
    *reinterpret_cast<uint2*>(A.gate16 + orow) = g0; *reinterpret_cast<uint2*>(A.gate16 + orow + 128) = g1;
  }
  const int pos = *A.d_pos + tok;
  float v[8];
  #pragma unroll
  for (int h = 0; h < 2; ++h) {
    v[4 * h] = __uint_as_float(in[h].x << 16); v[4 * h + 1] = __uint_as_float(in[h].x & 0xffff0000u);
    v[4 * h + 2] = __uint_as_float(in[h].y << 16); v[4 * h + 3] = __uint_as_float(in[h].y & 0xffff0000u);
  }
  if (kind != 2) {
    // ---- RMS norm
    const uint16_t* wn = (kind == 0 ? A.qn_w : A.kn_w) + 4 * lane;
    const uint2 wv[2] = {ld_table(reinterpret_cast<const uint2*>(wn)), ld_table(reinterpret_cast<const uint2*>(wn + 128))};
    float run[2];                                                // sums of squares of runs lane / 8 and 4 + lane / 8
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
      float t[4];
      #pragma unroll
      for (int e = 0; e < 4; ++e) t[e] = __fmul_rn(v[4 * h + e], v[4 * h + e]);
      #pragma unroll
      for (int m = 4; m; m >>= 1)
        #pragma unroll
        for (int e = 0; e < 4; ++e) t[e] = __fadd_rn(t[e], __shfl_xor_sync(0xffffffffu, t[e], m));
      run[h] = __fadd_rn(__fadd_rn(t[0], t[2]), __fadd_rn(t[1], t[3]));
    }
    float tot = 0.f;
    #pragma unroll
    for (int k = 0; k < 8; ++k) tot = __fadd_rn(tot, __shfl_sync(0xffffffffu, run[k >> 2], 8 * (k & 3)));
    const float x = __fadd_rn(__fdiv_rn(tot, 256.f), A.eps);
    const float r = A.pm ? __fdiv_rn(1.f, __fsqrt_rn(x)) : rsqrtf(x);
    #pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t w2 = i & 2 ? wv[i >> 2].y : wv[i >> 2].x;
      const float w = __uint_as_float(i & 1 ? w2 & 0xffff0000u : w2 << 16);
      v[i] = rbf(__fmul_rn(__fmul_rn(v[i], r), __fadd_rn(1.f, w)));
    }
    // ---- rotate-half over the first 64 * NRH channels, pairs (d, d + 32 * NRH): the partner is NRH runs away
    if constexpr (NRH > 0) {
      float p[8];                                                // partners of v
      #pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (NRH == 1 || NRH == 2) p[e] = __shfl_xor_sync(0xffffffffu, v[e], 8 * NRH);
        else if (NRH == 4) { p[e] = v[4 + e]; p[4 + e] = v[e]; }
        else {                                                   // runs 0, 1, 2 with 3, 4, 5: run 3 is the first half's last, 4 and 5 are the second half's first
          const float a = __shfl_sync(0xffffffffu, v[e], lane < 8 ? lane + 24 : lane - 24), b = __shfl_sync(0xffffffffu, v[4 + e], lane - 8);
          p[e] = lane < 8 || lane >= 24 ? a : b;
          p[4 + e] = __shfl_sync(0xffffffffu, v[e], lane + 8);
        }
      }
      #pragma unroll
      for (int h = 0; h < (NRH > 2 ? 2 : 1); ++h) {
        const int d = 128 * h + 4 * lane;
        if (d >= 64 * NRH) continue;
        const bool up = d >= 32 * NRH;                           // the upper channel of its pair
        const float4* rr = reinterpret_cast<const float4*>(A.rope + ((size_t)pos * (32 * NRH) + d - (up ? 32 * NRH : 0)) * 2);
        const float4 c01 = ld_table(rr), c23 = ld_table(rr + 1);
        const float cs[4] = {c01.x, c01.z, c23.x, c23.z}, sn[4] = {c01.y, c01.w, c23.y, c23.w};
        #pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float q = p[4 * h + e];
          v[4 * h + e] = rbf(__fadd_rn(rbf(__fmul_rn(v[4 * h + e], cs[e])), rbf(__fmul_rn(up ? q : -q, sn[e]))));
        }
      }
    }
  }
  // ---- signs and butterflies
  const LaneSigns sg = lane_signs(lane);
  #pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(__float_as_uint(v[i]) ^ (((sg.w[i >> 2] >> (i & 3)) & 1u) << 31));
  hadamard256_warp(v, lane, [](int) { return 0.0625f; });
  if (kind == 0) {
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint2 o;
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.x) : "f"(v[4 * h + 1]), "f"(v[4 * h]));
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.y) : "f"(v[4 * h + 3]), "f"(v[4 * h + 2]));
      *reinterpret_cast<uint2*>(A.q16 + orow + 128 * h) = o;
    }
    return;
  }
  if (pos < 0 || pos >= A.max_ctx) return;                       // a position outside the cache stores nothing
  float amax = 0.f;
  #pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
  #pragma unroll
  for (int m = 16; m; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
  const Int8Scale sc(amax);
  const size_t row = (size_t)head * A.max_ctx + pos;
  int8_t* dst = (kind == 2 ? A.v8 : A.k8) + row * 256 + 4 * lane;
  #pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t w = 0u;
    #pragma unroll
    for (int e = 0; e < 4; ++e) w |= ((uint32_t)sc.code(v[4 * h + e]) & 0xFFu) << (8 * e);
    *reinterpret_cast<uint32_t*>(dst + 128 * h) = w;
  }
  if (lane == 0) (kind == 2 ? A.vs : A.ks)[row] = sc.scale;
}

int grid_for(long long rows, unsigned* grid, const char* who) {
  if (rows < 0 || rows > (1ll << 34)) { set_error("%s: bad row count %lld", who, rows); return -1; }
  *grid = (unsigned)((rows + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK);
  return 0;
}

}  // namespace

int launch_kvx_rotate(const float* x, float* y, long long rows, int inverse, cudaStream_t st) {
  if (rows == 0) return 0;
  if (!x || !y) KV4_REJECT("yskn_kvx_rotate: null buffer");
  if (((uintptr_t)x | (uintptr_t)y) & 15) KV4_REJECT("yskn_kvx_rotate: rows must be 16-byte aligned");
  unsigned grid; if (grid_for(rows, &grid, "yskn_kvx_rotate")) return -1;
  kvx_rotate_kernel<<<grid, 256, 0, st>>>(x, y, rows, inverse ? 1 : 0);
  return launch_status("kvx_rotate_kernel");
}

int launch_kvx_encode(const void* x, int x_dtype, int8_t* q8, float* scales, long long rows, cudaStream_t st) {
  if (rows == 0) return 0;
  if (!x || !q8 || !scales) KV4_REJECT("yskn_kvx_encode: null buffer");
  if (((uintptr_t)x & 15) || ((uintptr_t)q8 & 7)) KV4_REJECT("yskn_kvx_encode: x must be 16-byte and q8 8-byte aligned");
  unsigned grid; if (grid_for(rows, &grid, "yskn_kvx_encode")) return -1;
  if (x_dtype == YSKN_KV4_F32) kvx_encode_kernel<YSKN_KV4_F32><<<grid, 256, 0, st>>>(x, q8, scales, rows);
  else if (x_dtype == YSKN_KV4_F16) kvx_encode_kernel<YSKN_KV4_F16><<<grid, 256, 0, st>>>(x, q8, scales, rows);
  else if (x_dtype == YSKN_KV4_BF16) kvx_encode_kernel<YSKN_KV4_BF16><<<grid, 256, 0, st>>>(x, q8, scales, rows);
  else KV4_REJECT("yskn_kvx_encode: unknown dtype %d", x_dtype);
  return launch_status("kvx_encode_kernel");
}

int launch_kvx_decode(const int8_t* q8, const float* scales, void* y, int y_dtype, long long rows, cudaStream_t st) {
  if (rows == 0) return 0;
  if (!y || !q8 || !scales) KV4_REJECT("yskn_kvx_decode: null buffer");
  if (((uintptr_t)y & 15) || ((uintptr_t)q8 & 7)) KV4_REJECT("yskn_kvx_decode: y must be 16-byte and q8 8-byte aligned");
  unsigned grid; if (grid_for(rows, &grid, "yskn_kvx_decode")) return -1;
  if (y_dtype == YSKN_KV4_F32) kvx_decode_kernel<YSKN_KV4_F32><<<grid, 256, 0, st>>>(q8, scales, y, rows);
  else if (y_dtype == YSKN_KV4_F16) kvx_decode_kernel<YSKN_KV4_F16><<<grid, 256, 0, st>>>(q8, scales, y, rows);
  else if (y_dtype == YSKN_KV4_BF16) kvx_decode_kernel<YSKN_KV4_BF16><<<grid, 256, 0, st>>>(q8, scales, y, rows);
  else KV4_REJECT("yskn_kvx_decode: unknown dtype %d", y_dtype);
  return launch_status("kvx_decode_kernel");
}

int launch_kvx_attn_post(const yskn_kvx_attn_post_args& a, cudaStream_t st) {
  if (a.M == 0) return 0;
  if (!a.q_rows || !a.k_rows || !a.v_rows || !a.qn_w || !a.kn_w || !a.d_pos || !a.q16 || !a.gate16 || !a.k8 || !a.v8 || !a.ks || !a.vs)
    KV4_REJECT("yskn_kvx_attn_post: null buffer");
  if (a.M < 0 || a.nh <= 0 || a.kvh <= 0 || a.max_ctx <= 0) KV4_REJECT("yskn_kvx_attn_post: bad shape (M %d, nh %d, kvh %d, max_ctx %d)", a.M, a.nh, a.kvh, a.max_ctx);
  if (a.rd < 0 || a.rd > 256 || a.rd % 64) KV4_REJECT("yskn_kvx_attn_post: rotary width %d must be a multiple of 64 up to 256", a.rd);
  if (a.rd > 0 && !a.rope) KV4_REJECT("yskn_kvx_attn_post: rotary width %d needs a rope table", a.rd);
  if (((uintptr_t)a.q_rows | (uintptr_t)a.k_rows | (uintptr_t)a.v_rows | (uintptr_t)a.qn_w | (uintptr_t)a.kn_w | (uintptr_t)a.q16 | (uintptr_t)a.gate16 |
       (uintptr_t)a.k8 | (uintptr_t)a.v8) & 7)
    KV4_REJECT("yskn_kvx_attn_post: row arrays must be 8-byte aligned");
  if ((uintptr_t)a.rope & 15) KV4_REJECT("yskn_kvx_attn_post: the rope table must be 16-byte aligned");
  // One-warp blocks spread a few tokens over the SMs; from eight rows an SM on, blocks of eight.
  const long long rows = (long long)a.M * (a.nh + 2 * a.kvh);
  const int threads = rows < 148 * 8 ? 32 : 256;
  if (rows > (1ll << 33)) KV4_REJECT("yskn_kvx_attn_post: bad row count %lld", rows);
  const unsigned grid = (unsigned)((rows + threads / 32 - 1) / (threads / 32));
  switch (a.rd / 64) {
    case 0: return launch_pdl("kvx_attn_post_kernel", kvx_attn_post_kernel<0>, dim3(grid), threads, 0, st, a);
    case 1: return launch_pdl("kvx_attn_post_kernel", kvx_attn_post_kernel<1>, dim3(grid), threads, 0, st, a);
    case 2: return launch_pdl("kvx_attn_post_kernel", kvx_attn_post_kernel<2>, dim3(grid), threads, 0, st, a);
    case 3: return launch_pdl("kvx_attn_post_kernel", kvx_attn_post_kernel<3>, dim3(grid), threads, 0, st, a);
    default: return launch_pdl("kvx_attn_post_kernel", kvx_attn_post_kernel<4>, dim3(grid), threads, 0, st, a);
  }
}

}  // namespace kv4
