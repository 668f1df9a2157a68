// Family-B decode attention over INT8 rows (the cache the row codec of kvx_codec.cu writes): split-K flash-decode on
// the tensor cores for sm_100a, plus the merge with the inverse rotation.
//
// Semantics: the reference's q35_attention_kernel<KV8> (src/q35_kernels.cu:1176-1281) and the tail of its combine
// (src/q35_kernels.cu:1400-1425).  K and V rows are INT8 [Hkv][max_ctx][256] with one fp32 scale per row (ks, vs); Q
// arrives already rotated (kvx_rotate) and is scaled by qscale at load; row r sits at pos = *d_pos + r and sees keys
// 0..pos, all of them INT8 (Family B has no fp16 shadow and rotates K before storing, so nothing happens at read time):
//   s_t = qscale * (q . k8_t) * ks_t,   p_t = softmax(s)_t,   O = sum_t p_t * vs_t * v8_t      (rotated basis)
// Partials (m, l, O) per split in the reference's layout pm/pl [M][S][Hq], pacc [M][S][Hq][256]; the merge divides,
// rotates back (inverse kvx_rotate), rounds to bf16/fp16 and applies the optional sigmoid gate.
//
// Kernel shape: one CTA per (split, kv-head, row); a warp takes 16-token tiles.  Bytes go straight from HBM into
// registers (16-byte loads, K of the next tile and V of this tile in flight while the tensor cores work), because an
// INT8 row needs no staging transform: a lane's 16 K bytes of token g are the A fragments of four k-steps once each byte
// b is read as the fp16 number 1152 + b (byte ^ 0x80 under exponent 2^10, one PRMT per fragment register); the constant
// 1152 leaves through a per-head bias (K) and through 1152 * sum(p') (V).  The contraction index of S is a fixed
// permutation of the channels (slot (w, s, 2j+x) <-> channel 16(4w+j)+4s+x), applied to Q once at set-up; for P.V a lane
// owns channels [32g, 32g+32) of token rows 2j, 2j+1, 2j+8, 2j+9 and PRMT pairs the two tokens of a k-slot.
// HBM-bound: 2,080 bytes per token (4 kv-heads x 2 x 260).
#include "kvx_rotate.cuh"

namespace kv4 {
namespace {

constexpr int KV8_HD = 256;
constexpr int KV8_WARPS = 8;
constexpr int KV8_MS = 260;                               // words of a merge entry
static_assert(KV8_WARPS == 8, "one group of eight lanes holds a head's weights");
constexpr float KV8_LOG2E = 1.4426950408889634f, KV8_LN2 = 0.6931471805599453f;
constexpr uint32_t C64 = 0x64646464u;                      // high bytes of the fp16 pattern 0x64xx = 1024 + xx
constexpr float KV8_OFF = 1152.f;                          // 1024 + 128: a byte b is read as 1152 + b

struct Kv8P { yskn_kv8_attn_args a; int g; };

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_t(uint32_t a) { uint32_t d; asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a)); return d; }
__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) { uint32_t d; asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo)); return d; }
__device__ __forceinline__ uint4 ldg16(const void* p) { return __ldcs(reinterpret_cast<const uint4*>(p)); }   // streamed once

constexpr int KV8_AHEAD = 24;                              // tiles of 16 keys asked into L2 ahead: 96 KB of keys and as much of values a block
template <int DT>
__global__ void __launch_bounds__(KV8_WARPS * 32, 1) kv8_decode_kernel(const Kv8P P) {
  extern __shared__ __align__(16) uint8_t smem[];
  // [16 k-steps][32 lanes] uint2 Q fragments | q sums [4][8] | weights | merge area [warps][8 heads][260]
  uint2* s_q = reinterpret_cast<uint2*>(smem);
  float* s_bias = reinterpret_cast<float*>(smem + 16 * 32 * 8);
  float* s_wgt = s_bias + 32;                              // [8 heads][warps]
  float* s_merge = s_wgt + 64;
  const yskn_kv8_attn_args& A = P.a;
  const int split = blockIdx.x, kvh = blockIdx.y, r = blockIdx.z, G = P.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  // Programmatic dependent launch: this grid may be scheduled while the row epilogue in front of it drains, and waits here before it
  // reads the position, the queries and the new rows; the merge behind it may be scheduled early in turn.
  // One thing is read ahead of that wait: the position, past L1, and for nothing but the address from which the block's first keys are asked into L2 while the
  // epilogue runs.  It may be stale or be written at that moment; held within the cache it then asks for the wrong lines of the cache's own arrays, no more, and
  // all that a result depends on, the position again first of all, is read behind the wait: one token over 32,768 rows 22.8 -> 21.6 us.  (Tried on the int4
  // decode kernel too: behind its append, 2 us, reading the position early costs more than it brings, 19.7 -> 20.8 us.)
  if (threadIdx.x < 2 && r == 0) {
    const int keys = max(0, min(__ldcg(A.d_pos), A.max_ctx)), tl = keys / 16, n = (tl + (int)gridDim.x - 1) / (int)gridDim.x;   // past L1: read again behind the wait
    const int t0 = min(tl, split * n), nt = min(min(n, tl - t0), KV8_AHEAD);
    const int8_t* const p = (threadIdx.x ? A.v8 : A.k8) + ((size_t)kvh * A.max_ctx + 16 * t0) * KV8_HD;
    if (nt > 0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"((uint32_t)nt * 16 * KV8_HD) : "memory");
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int len = *A.d_pos + r + 1;                        // keys 0 .. pos
  const int tiles = (len + 15) / 16, per = (tiles + (int)gridDim.x - 1) / (int)gridDim.x;
  const int ti0 = min(tiles, split * per), ti1 = min(tiles, ti0 + per);

  const size_t plane = (size_t)kvh * A.max_ctx;
  const int8_t* kbase = A.k8 + plane * KV8_HD + 16 * j;    // + token*256 + 64*w : this lane's 16 channels of block w
  const int8_t* vbase = A.v8 + plane * KV8_HD + 32 * g;    // + token*256 (+16)  : this lane's 32 channels
  const float* ksb = A.ks + plane; const float* vsb = A.vs + plane;

  uint4 kx[4], ky[4];                                      // K of the current tile: token g (x) and g+8 (y), blocks w = 0..3
  auto load_k = [&](int ti) {
    const size_t t = (size_t)16 * ti + g;
    #pragma unroll
    for (int w = 0; w < 4; ++w) { kx[w] = ldg16(kbase + t * KV8_HD + 64 * w); ky[w] = ldg16(kbase + (t + 8) * KV8_HD + 64 * w); }
  };
  int ti = ti0 + warp;
  if (ti < ti1) load_k(ti);                                // the first keys are on their way while Q is prepared

  // ---- set-up: Q as B fragments in the slot order of the K loads, scaled by qscale * log2(e); the per-head bias 1152 * sum of the
  //      fp16 values the MMAs multiply by.  A thread keeps one head over its four entries (head = bits 3-5 of e), so the sum is
  //      three shuffles and four partials per head (one thread per head walking the fragments took about 1 us).
  const float qs = A.qscale * KV8_LOG2E;
  float qsum = 0.f;
  for (int e = threadIdx.x; e < 16 * 32 * 2; e += KV8_WARPS * 32) {
    const int x = e & 1, ln = (e >> 1) & 31, kstep = e >> 6, w = kstep >> 2, s = kstep & 3, hh = ln >> 2, jj = ln & 3;
    const int c = 16 * (4 * w + jj) + 4 * s + 2 * x;
    float lo = 0.f, hi = 0.f;
    if (hh < G) {
      const size_t qb = ((size_t)r * A.nh + kvh * G + hh) * KV8_HD + c;
      lo = act_load<DT>(A.q16, qb) * qs; hi = act_load<DT>(A.q16, qb + 1) * qs;
    }
    const uint32_t p = pack_h2(lo, hi);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&p));
    qsum += f.x + f.y;
    reinterpret_cast<uint32_t*>(s_q)[e] = p;
  }
  #pragma unroll
  for (int o = 1; o <= 4; o <<= 1) qsum += __shfl_xor_sync(0xffffffffu, qsum, o);
  if ((lane & 7) == 0) s_bias[(warp >> 1) * 8 + (threadIdx.x >> 3 & 7)] = qsum;
  __syncthreads();
  auto bias_of = [&](int h) { return KV8_OFF * ((s_bias[h] + s_bias[8 + h]) + (s_bias[16 + h] + s_bias[24 + h])); };
  const float bias0 = bias_of(2 * j), bias1 = bias_of(2 * j + 1);

  float acc[16][4];                                        // O^T: [m-tile][(channel 32g+2mt | +1) x (head 2j | 2j+1)]
  #pragma unroll
  for (int mt = 0; mt < 16; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f;
  float m[2] = {-1e30f, -1e30f}, l[2] = {0.f, 0.f}, zs[2] = {0.f, 0.f};   // heads 2j, 2j+1 (log2 domain); zs = sum of rounded p'

  for (; ti < ti1; ti += KV8_WARPS) {
    const int tg = 16 * ti + g;
    const bool v0 = tg < len, v1 = tg + 8 < len;
    // ---- V of this tile and the scales: in flight while S is computed
    uint4 vr[4][2];
    {
      const size_t ta = (size_t)16 * ti + 2 * j;
      const size_t tt[4] = {ta, ta + 1, ta + 8, ta + 9};
      #pragma unroll
      for (int q = 0; q < 4; ++q) { vr[q][0] = ldg16(vbase + tt[q] * KV8_HD); vr[q][1] = ldg16(vbase + tt[q] * KV8_HD + 16); }
    }
    const float ks0 = v0 ? ksb[tg] : 0.f, ks1 = v1 ? ksb[tg + 8] : 0.f;
    const float vs0 = v0 ? vsb[tg] : 0.f, vs1 = v1 ? vsb[tg + 8] : 0.f;
    // ---- S^T[16 tokens x 8 heads] = K . Q^T, two accumulation chains
    float sa[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    #pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint32_t xw[4] = {kx[w].x ^ 0x80808080u, kx[w].y ^ 0x80808080u, kx[w].z ^ 0x80808080u, kx[w].w ^ 0x80808080u};
      const uint32_t yw[4] = {ky[w].x ^ 0x80808080u, ky[w].y ^ 0x80808080u, ky[w].z ^ 0x80808080u, ky[w].w ^ 0x80808080u};
      #pragma unroll
      for (int s = 0; s < 4; ++s) {
        const uint2 qb = s_q[(4 * w + s) * 32 + lane];
        mma16816(sa[s & 1], __byte_perm(xw[s], C64, 0x4140), __byte_perm(yw[s], C64, 0x4140),
                 __byte_perm(xw[s], C64, 0x4342), __byte_perm(yw[s], C64, 0x4342), qb.x, qb.y);
      }
    }
    if (ti + KV8_WARPS < ti1) load_k(ti + KV8_WARPS);       // K of this warp's next tile: in flight during softmax and P.V
    // ---- softmax over the tile (log2 domain); rows g, g+8; heads 2j, 2j+1
    const float s00 = v0 ? (sa[0][0] + sa[1][0] - bias0) * ks0 : -INFINITY, s01 = v0 ? (sa[0][1] + sa[1][1] - bias1) * ks0 : -INFINITY;
    const float s10 = v1 ? (sa[0][2] + sa[1][2] - bias0) * ks1 : -INFINITY, s11 = v1 ? (sa[0][3] + sa[1][3] - bias1) * ks1 : -INFINITY;
    float t0 = fmaxf(s00, s10), t1 = fmaxf(s01, s11);
    #pragma unroll
    for (int o = 4; o <= 16; o <<= 1) { t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, o)); t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, o)); }
    if (__any_sync(0xffffffffu, t0 > m[0] + 8.f || t1 > m[1] + 8.f)) {   // lazy rescale: the running max may lag by 2^8
      const float n0 = fmaxf(m[0], t0), n1 = fmaxf(m[1], t1), a0 = ex2(m[0] - n0), a1 = ex2(m[1] - n1);
      m[0] = n0; m[1] = n1; l[0] *= a0; l[1] *= a1; zs[0] *= a0; zs[1] *= a1;
      #pragma unroll
      for (int mt = 0; mt < 16; ++mt) { acc[mt][0] *= a0; acc[mt][1] *= a1; acc[mt][2] *= a0; acc[mt][3] *= a1; }
    }
    const float p00 = v0 ? ex2(s00 - m[0]) : 0.f, p01 = v0 ? ex2(s01 - m[1]) : 0.f;
    const float p10 = v1 ? ex2(s10 - m[0]) : 0.f, p11 = v1 ? ex2(s11 - m[1]) : 0.f;
    l[0] += p00 + p10; l[1] += p01 + p11;
    // the row scale of V goes into P (fp16); the 1152 offset of the V operand leaves through the sum of the ROUNDED p'
    const uint32_t pp0 = pack_h2(p00 * vs0, p01 * vs0), pp1 = pack_h2(p10 * vs1, p11 * vs1);
    const float2 pr0 = __half22float2(*reinterpret_cast<const __half2*>(&pp0)), pr1 = __half22float2(*reinterpret_cast<const __half2*>(&pp1));
    zs[0] += pr0.x + pr1.x; zs[1] += pr0.y + pr1.y;
    const uint32_t pb0 = movmatrix_t(pp0), pb1 = movmatrix_t(pp1);     // B regs: (tokens 2j,2j+1 | head g), (tokens 2j+8,2j+9 | head g)
    // ---- O^T += V^T P^T: m-tile mt = channels (32g + 2mt, 32g + 2mt + 1) as rows (g, g+8)
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t wa[4] = {vr[0][h].x, vr[0][h].y, vr[0][h].z, vr[0][h].w}, wb[4] = {vr[1][h].x, vr[1][h].y, vr[1][h].z, vr[1][h].w};
      const uint32_t wc[4] = {vr[2][h].x, vr[2][h].y, vr[2][h].z, vr[2][h].w}, wd[4] = {vr[3][h].x, vr[3][h].y, vr[3][h].z, vr[3][h].w};
      #pragma unroll
      for (int wi = 0; wi < 4; ++wi)
        #pragma unroll
        for (int half = 0; half < 2; ++half) {                           // bytes (0,1) then (2,3) of the word
          const uint32_t sel = half ? 0x7362u : 0x5140u;                 // [A.b, B.b, A.b', B.b']
          const uint32_t ab = __byte_perm(wa[wi], wb[wi], sel) ^ 0x80808080u, cd = __byte_perm(wc[wi], wd[wi], sel) ^ 0x80808080u;
          mma16816(acc[8 * h + 2 * wi + half], __byte_perm(ab, C64, 0x4140), __byte_perm(ab, C64, 0x4342),
                   __byte_perm(cd, C64, 0x4140), __byte_perm(cd, C64, 0x4342), pb0, pb1);
        }
    }
  }

  // ---- this warp's (m, l, O) per head: sums over the token lanes, the operand offset removed
  #pragma unroll
  for (int o = 4; o <= 16; o <<= 1) {
    l[0] += __shfl_xor_sync(0xffffffffu, l[0], o); l[1] += __shfl_xor_sync(0xffffffffu, l[1], o);
    zs[0] += __shfl_xor_sync(0xffffffffu, zs[0], o); zs[1] += __shfl_xor_sync(0xffffffffu, zs[1], o);
  }
  // Merge entry of a (warp, head): m, l, -, -, then channel d at slot (d & 31) * 8 + d / 32: the lanes of a store (channels 32g + c, heads 2j)
  // fall into 32 different banks (channels in order gave 8-way conflicts).
  {
    float* mine = s_merge + (size_t)warp * 8 * KV8_MS;
    #pragma unroll
    for (int mt = 0; mt < 16; ++mt) {
      const int c = 4 + 16 * mt + g;                       // channel 32g + 2mt; the next one is 8 further on
      mine[(2 * j) * KV8_MS + c] = acc[mt][0] - KV8_OFF * zs[0]; mine[(2 * j + 1) * KV8_MS + c] = acc[mt][1] - KV8_OFF * zs[1];
      mine[(2 * j) * KV8_MS + c + 8] = acc[mt][2] - KV8_OFF * zs[0]; mine[(2 * j + 1) * KV8_MS + c + 8] = acc[mt][3] - KV8_OFF * zs[1];
    }
    if (g == 0) { mine[(2 * j) * KV8_MS] = m[0]; mine[(2 * j) * KV8_MS + 1] = l[0]; mine[(2 * j + 1) * KV8_MS] = m[1]; mine[(2 * j + 1) * KV8_MS + 1] = l[1]; }
  }
  __syncthreads();
  // ---- merge the warps and store the split's partial (m in the natural-log domain, as the reference's partials)
  if (threadIdx.x < 8 * KV8_WARPS) {                       // the warps' weights, once per head
    const int hh = threadIdx.x / KV8_WARPS, w = threadIdx.x % KV8_WARPS;
    float M2 = -1e30f, L2 = 0.f;
    #pragma unroll
    for (int k = 0; k < KV8_WARPS; ++k) M2 = fmaxf(M2, s_merge[((size_t)k * 8 + hh) * KV8_MS]);
    const float mw = s_merge[((size_t)w * 8 + hh) * KV8_MS], f = mw > -1e29f ? ex2(mw - M2) : 0.f;
    s_wgt[hh * KV8_WARPS + w] = f;
    L2 = f * s_merge[((size_t)w * 8 + hh) * KV8_MS + 1];
    #pragma unroll
    for (int o = 1; o < KV8_WARPS; o <<= 1) L2 += __shfl_xor_sync(0xffffffffu, L2, o);
    const size_t pidx = ((size_t)r * A.splits + split) * A.nh + kvh * G + hh;
    if (w == 0 && hh < G) { A.pm[pidx] = M2 > -1e29f ? M2 * KV8_LN2 : -1e30f; A.pl[pidx] = L2; }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < G * KV8_HD; e += KV8_WARPS * 32) {
    const int hh = e / KV8_HD, i = e % KV8_HD, d = (i & 7) * 32 + (i >> 3);
    float o = 0.f;
    #pragma unroll
    for (int w = 0; w < KV8_WARPS; ++w) o += s_wgt[hh * KV8_WARPS + w] * s_merge[((size_t)w * 8 + hh) * KV8_MS + 4 + i];
    A.pacc[(((size_t)r * A.splits + split) * A.nh + kvh * G + hh) * KV8_HD + d] = o;
  }
}

// ---- merge of the splits + inverse rotation + rounding (+ gate), in two shapes.
// What bounds both is latency, not bytes (a decode step merges 0.9 MB).  The former kernel (one block of 256 threads per row, splits
// walked one after the other, sixteen block barriers for the rotation) took 20 us for 24 rows of 37 splits and 64 us for
// 24,000 rows of one split.
__device__ __forceinline__ float kv8_round(int dt, float v) { return dt == YSKN_KV4_BF16 ? bf2f(f2bf(v)) : h2f(f2h(v)); }
template <int DT> __device__ __forceinline__ float kv8_gated(float y, float gt) {   // y * sigmoid(gate), each factor and the product rounded (src/q35_kernels.cu:1423-1424)
  return kv8_round(DT, __fmul_rn(y, kv8_round(DT, __frcp_rn(__fadd_rn(1.f, expf(-gt))))));
}

// Many splits: one block per (head, row), four runs of splits x 256 channels, every thread's loads issued at once; one warp
// forms the weights meanwhile.  The butterflies (inverse kvx_rotate, src/kvx_codec.cuh:35-49, stages h = 1 ... 128 in order): 1 ... 16 by
// shuffles, 32 ... 128 from one exchange through shared memory, each thread folding the eight values its output depends on.
constexpr int KV8_CQ = 4, KV8_CB = 10;
template <int DT>
__global__ void __launch_bounds__(KV8_CQ * 256) kv8_combine_kernel(const float* pm, const float* pl, const float* pacc, int S, int nh,
                                                                  const void* gate, uint16_t* o16, int inverse_rotate) {
  __shared__ float s_w[64], s_part[KV8_CQ][256], s_buf[256];
  __shared__ float s_L;
  const int head = blockIdx.x, r = blockIdx.y, tid = threadIdx.x, q = tid >> 8, d = tid & 255;
  auto slot = [&](int s) -> size_t { return ((size_t)r * S + s) * nh + head; };
  const int per = (S + KV8_CQ - 1) / KV8_CQ, s0 = min(S, q * per), s1 = min(S, s0 + per);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");       // the attention grid's partials are visible from here on
  const size_t e = ((size_t)r * nh + head) * KV8_HD + d;
  const float gt = gate && q == 0 ? act_load<DT>(gate, e) : 0.f;
  float v[KV8_CB];
  #pragma unroll
  for (int k = 0; k < KV8_CB; ++k) v[k] = s0 + k < s1 ? __ldcg(pacc + slot(s0 + k) * KV8_HD + d) : 0.f;
  if (tid < 32) {                                          // at most 64 splits: two per lane
    const float m0 = tid < S ? __ldcg(pm + slot(tid)) : -1e30f, m1 = tid + 32 < S ? __ldcg(pm + slot(tid + 32)) : -1e30f;
    const float l0 = tid < S ? __ldcg(pl + slot(tid)) : 0.f, l1 = tid + 32 < S ? __ldcg(pl + slot(tid + 32)) : 0.f;
    float mx = fmaxf(m0, m1);
    #pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float w0 = m0 > -1e29f ? expf(m0 - mx) : 0.f, w1 = m1 > -1e29f ? expf(m1 - mx) : 0.f;
    s_w[tid] = w0; s_w[tid + 32] = w1;
    float ls = w0 * l0 + w1 * l1;
    #pragma unroll
    for (int o = 16; o; o >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, o);
    if (tid == 0) s_L = ls;
  }
  __syncthreads();
  float o = 0.f;
  #pragma unroll
  for (int k = 0; k < KV8_CB; ++k) if (s0 + k < s1) o += s_w[s0 + k] * v[k];
  for (int s = s0 + KV8_CB; s < s1; ++s) o += s_w[s] * __ldcg(pacc + slot(s) * KV8_HD + d);     // more than 40 splits
  s_part[q][d] = o;
  __syncthreads();
  if (q != 0) return;
  float y = __fdiv_rn((s_part[0][d] + s_part[1][d]) + (s_part[2][d] + s_part[3][d]), s_L);
  if (inverse_rotate) {
    #pragma unroll
    for (int h = 1; h < 32; h *= 2) {                      // lower index: a + b; upper: lower - upper
      const float other = __shfl_xor_sync(0xffffffffu, y, h);
      y = (d & h) ? __fsub_rn(other, y) : __fadd_rn(y, other);
    }
    s_buf[d] = y;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    float t[8];
    #pragma unroll
    for (int k = 0; k < 8; ++k) t[k] = s_buf[32 * k + (d & 31)];
    const uint32_t f0 = (d & 32) ? 0x80000000u : 0u, f1 = (d & 64) ? 0x80000000u : 0u, f2 = (d & 128) ? 0x80000000u : 0u;
    auto fold = [](float lo, float up, uint32_t flip) { return __fadd_rn(lo, __uint_as_float(__float_as_uint(up) ^ flip)); };
    #pragma unroll
    for (int k = 0; k < 8; k += 2) t[k] = fold(t[k], t[k + 1], f0);
    t[0] = fold(t[0], t[2], f1); t[4] = fold(t[4], t[6], f1);
    y = __fmul_rn(fold(t[0], t[4], f2), 0.0625f);
    if ((c_signs.w[d >> 5] >> (d & 31)) & 1u) y = -y;
  }
  y = kv8_round(DT, y);
  if (gate) y = kv8_gated<DT>(y, gt);
  o16[e] = act_store16<DT>(y);
}

// Many rows: one warp per row, lane l owns channels 4l .. 4l + 3 and 128 + 4l .., no shared memory and no barrier; up to eight splits of loads are in
// flight at once.  Bound by instruction issue for a prompt (56 operations a value, most of them the sigmoid, the butterflies and the quotient), by two trips to
// memory for the rows of a verify pass.  The form it replaces took eight lanes a row (four rows a warp, 32 values a lane: a quarter of the warps, for
// one to four splits only).  Replays over partials in L2, before -> now: 384 rows of 18 splits 7.5 -> 4.1 us, 2,400 of 6 splits 36.5 -> 4.5, 4,032 of 4 splits
// 13.6 -> 5.7, 24,000 of one split 21.3 -> 14.2.
template <int DT, bool ONE>
__global__ void __launch_bounds__(128) kv8_combine_rows_kernel(const float* pm, const float* pl, const float* pacc, int S, int nh, long long rows,
                                                               const void* gate, uint16_t* o16, int inverse_rotate) {
  constexpr int B = ONE ? 1 : 8;
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);          // row = token * nh + head
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (row >= rows) return;
  const long long tok = row / nh;
  const int head = (int)(row - tok * nh);
  const size_t slot0 = (size_t)tok * S * nh + head, step = (size_t)nh * KV8_HD;
  const float* acc = pacc + slot0 * KV8_HD + 4 * lane;
  const size_t e0 = (size_t)row * KV8_HD + 4 * lane;
  float4 a[B][2];
  auto load = [&](int s0) {
    #pragma unroll
    for (int k = 0; k < B; ++k)
      if (s0 + k < S) {
        a[k][0] = __ldcg(reinterpret_cast<const float4*>(acc + (s0 + k) * step));
        a[k][1] = __ldcg(reinterpret_cast<const float4*>(acc + (s0 + k) * step + 128));
      }
  };
  float m0 = -1e30f, m1 = -1e30f, l0 = 0.f, l1 = 0.f, w0, w1 = 0.f, L2;      // of splits `lane` and `lane + 32` (at most 64 splits)
  if (ONE) { m0 = __ldcg(pm + slot0); l0 = __ldcg(pl + slot0); }
  else if (lane < S) { m0 = __ldcg(pm + slot0 + (size_t)lane * nh); l0 = __ldcg(pl + slot0 + (size_t)lane * nh); }
  if (!ONE && lane + 32 < S) { m1 = __ldcg(pm + slot0 + (size_t)(lane + 32) * nh); l1 = __ldcg(pl + slot0 + (size_t)(lane + 32) * nh); }
  load(0);
  uint2 g[2] = {make_uint2(0u, 0u), make_uint2(0u, 0u)};
  if (gate) {
    g[0] = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(gate) + e0);
    g[1] = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(gate) + e0 + 128);
  }
  if (ONE) { w0 = m0 > -1e29f ? 1.f : 0.f; L2 = w0 * l0; }
  else {
    float mx = fmaxf(m0, m1);
    #pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    w0 = m0 > -1e29f ? expf(m0 - mx) : 0.f; w1 = m1 > -1e29f ? expf(m1 - mx) : 0.f;
    L2 = w0 * l0 + w1 * l1;
    #pragma unroll
    for (int o = 16; o; o >>= 1) L2 += __shfl_xor_sync(0xffffffffu, L2, o);
  }
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // v[e] = channel 4 lane + e, v[4 + e] = channel 128 + 4 lane + e
  #pragma unroll 1
  for (int s0 = 0; ; ) {
    #pragma unroll
    for (int k = 0; k < B; ++k) {
      const int s = s0 + k;
      const float w = ONE ? w0 : __shfl_sync(0xffffffffu, s < 32 ? w0 : w1, s & 31);
      if (s < S) {
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
          v[4 * h] += w * a[k][h].x; v[4 * h + 1] += w * a[k][h].y; v[4 * h + 2] += w * a[k][h].z; v[4 * h + 3] += w * a[k][h].w;
        }
      }
    }
    s0 += B;
    if (ONE || s0 >= S) break;
    load(s0);
  }
  // v / L2, correctly rounded.  With r = 1 / L2 rounded and q = v * r, q - (q * L2 - v) * r in two fused steps is the rounded quotient while the values
  // and the residual stay normal (Markstein, IBM J. Res. Dev. 34, 1990; his theorem asks for a q within one unit in the last place, and q may
  // be off by 1.5: the 40.7 million pairs of 24-bit values whose quotient lies near enough to a tie for that to matter were all tried).  Three
  // operations instead of a division per value.  The bounds keep |q| and the residual's last bit normal; the residual has the sign that leaves a
  // zero its own.  Lanes with other values divide.
  const float r = __frcp_rn(L2);
  float big = 0.f;                                         // largest |v|, past NaN, which stays NaN on either way
  uint32_t small = 0xFFFFFFFFu;                            // smallest |v| that is not 0: its bits twice, less 1
  #pragma unroll
  for (int i = 0; i < 8; ++i) { big = fmaxf(big, fabsf(v[i])); small = min(small, 2u * __float_as_uint(v[i]) - 1u); }
  constexpr uint32_t SMALL = 2u * ((127u - 60u) << 23) - 1u;
  if (L2 >= 0x1p-20f && L2 <= 0x1p60f && big <= 0x1p100f && small >= SMALL) {
    #pragma unroll
    for (int i = 0; i < 8; ++i) { const float q = __fmul_rn(v[i], r); v[i] = fmaf(-fmaf(q, L2, -v[i]), r, q); }
  } else {
    #pragma unroll 1
    for (int i = 0; i < 8; ++i) {                          // rolled (rows without keys, sums beyond the range): the values go round by one each time
      const float t = __fdiv_rn(v[0], L2);
      #pragma unroll
      for (int k = 0; k < 7; ++k) v[k] = v[k + 1];
      v[7] = t;
    }
  }
  if (inverse_rotate) {                                    // 1/16 and the signs in one factor
    const LaneSigns sg = lane_signs(lane);
    hadamard256_warp(v, lane, [&](int i) { return __uint_as_float(0x3d800000u | (((sg.w[i >> 2] >> (i & 3)) & 1u) << 31)); });
  }
  auto pack = [](float lo, float hi) {                     // two values rounded to the output type
    uint32_t d;
    if (DT == YSKN_KV4_BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
  };
  auto low = [](uint32_t d) { return DT == YSKN_KV4_BF16 ? __uint_as_float(d << 16) : h2f((uint16_t)d); };
  auto high = [](uint32_t d) { return DT == YSKN_KV4_BF16 ? __uint_as_float(d & 0xffff0000u) : h2f((uint16_t)(d >> 16)); };
  auto sigm = [](float gt) { return __frcp_rn(__fadd_rn(1.f, expf(-gt))); };
  #pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t u[2] = {pack(v[4 * h], v[4 * h + 1]), pack(v[4 * h + 2], v[4 * h + 3])};
    if (gate) {                                            // y * sigmoid(gate): each factor and the product rounded (src/q35_kernels.cu:1423-1424)
      const uint32_t gg[2] = {g[h].x, g[h].y};
      #pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t sg = pack(sigm(low(gg[i])), sigm(high(gg[i])));
        u[i] = pack(__fmul_rn(low(u[i]), low(sg)), __fmul_rn(high(u[i]), high(sg)));
      }
    }
    *reinterpret_cast<uint2*>(o16 + e0 + 128 * h) = make_uint2(u[0], u[1]);
  }
}

template <int DT>
int launch_kv8_combine_dt(const float* pm, const float* pl, const float* pacc, int S, int M, int nh, const void* gate, uint16_t* o16, int inverse_rotate, cudaStream_t st) {
  // The form of a warp per row wants enough rows: up to one block of 1,024 threads per SM the block form's parallel loads win (96 rows of 37 splits 3.1
  // against 4.9 us in replays, 192 rows of 18 splits 5.1 against 3.9).  With more than 32 splits, two weights a lane, the line is two blocks an SM: behind the
  // attention kernel the blocks are resident before it ends, and whole steps of 192 rows in 24 / 37 splits over 8,000 tokens take 48.7 / 55.9 us with blocks and
  // 48.3 / 59.9 with warps (168 rows in 37: 50.4 / 53.9; 288 rows in 33 over 3,000 tokens 30.3 / 28.9, in 37 30.3 / 33.9; 576 rows in 37 37.6 / 36.7).  Warps read
  // 16-byte pieces.
  const long long rows = (long long)M * nh;
  const bool aligned = !((((uintptr_t)pacc) & 15) | (((uintptr_t)o16 | (uintptr_t)gate) & 7));
  if (rows > (S > 32 ? 296 : 148) && aligned)
    return launch_pdl("kv8_combine_rows_kernel", S == 1 ? kv8_combine_rows_kernel<DT, true> : kv8_combine_rows_kernel<DT, false>, dim3((unsigned)((rows + 3) / 4)), 128, 0, st,
                      pm, pl, pacc, S, nh, rows, gate, o16, inverse_rotate);
  return launch_pdl("kv8_combine_kernel", kv8_combine_kernel<DT>, dim3(nh, M), KV8_CQ * 256, 0, st, pm, pl, pacc, S, nh, gate, o16, inverse_rotate);
}

}  // namespace

int launch_kv8_attention(const yskn_kv8_attn_args& a, int act_dtype, cudaStream_t st) {
  if (!a.q16 || !a.k8 || !a.v8 || !a.ks || !a.vs || !a.d_pos || !a.pm || !a.pl || !a.pacc) KV4_REJECT("yskn_kv8_attention: null buffer");
  if (a.kvh <= 0 || a.nh <= 0 || a.nh % a.kvh || a.nh / a.kvh > 8 || a.M <= 0 || a.M > 65535 || a.kvh > 65535 || a.splits <= 0 || a.max_ctx <= 0 || a.max_ctx % 64)
    KV4_REJECT("yskn_kv8_attention: bad shape (kvh %d, nh %d, M %d, splits %d, max_ctx %d): at most 8 query heads per kv-head, max_ctx a multiple of 64",
               a.kvh, a.nh, a.M, a.splits, a.max_ctx);
  if (((uintptr_t)a.k8 | (uintptr_t)a.v8) & 15) KV4_REJECT("yskn_kv8_attention: k8 and v8 must be 16-byte aligned");
  const size_t smem = 16 * 32 * 8 + 32 * 4 + 64 * 4 + (size_t)KV8_WARPS * 8 * KV8_MS * 4;
  Kv8P P{a, a.nh / a.kvh};
  const dim3 grid(a.splits, a.kvh, a.M);
  if (act_dtype == YSKN_KV4_BF16) {
    static std::atomic<unsigned long long> attr{0};
    if (first_use_on_device(attr)) KV4_CUDA(cudaFuncSetAttribute(kv8_decode_kernel<YSKN_KV4_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch_pdl("kv8_decode_kernel", kv8_decode_kernel<YSKN_KV4_BF16>, grid, KV8_WARPS * 32, smem, st, P);
  }
  if (act_dtype == YSKN_KV4_F16) {
    static std::atomic<unsigned long long> attr{0};
    if (first_use_on_device(attr)) KV4_CUDA(cudaFuncSetAttribute(kv8_decode_kernel<YSKN_KV4_F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch_pdl("kv8_decode_kernel", kv8_decode_kernel<YSKN_KV4_F16>, grid, KV8_WARPS * 32, smem, st, P);
  }
  KV4_REJECT("yskn_kv8_attention: q16 is bf16 or fp16 (act_dtype %d)", act_dtype);
}

int launch_kv8_combine(const float* pm, const float* pl, const float* pacc, int splits, int M, int nh, const void* gate, void* o16,
                       int act_dtype, int inverse_rotate, cudaStream_t st) {
  if (!pm || !pl || !pacc || !o16) KV4_REJECT("yskn_kv8_combine: null buffer");
  if (splits <= 0 || splits > 64 || M <= 0 || nh <= 0) KV4_REJECT("yskn_kv8_combine: bad shape (splits %d of at most 64, M %d, nh %d)", splits, M, nh);
  if (M > 65535) KV4_REJECT("yskn_kv8_combine: M %d exceeds the grid limit", M);
  uint16_t* out = static_cast<uint16_t*>(o16);
  if (act_dtype == YSKN_KV4_BF16) return launch_kv8_combine_dt<YSKN_KV4_BF16>(pm, pl, pacc, splits, M, nh, gate, out, inverse_rotate, st);
  if (act_dtype == YSKN_KV4_F16) return launch_kv8_combine_dt<YSKN_KV4_F16>(pm, pl, pacc, splits, M, nh, gate, out, inverse_rotate, st);
  KV4_REJECT("yskn_kv8_combine: o16 is bf16 or fp16 (act_dtype %d)", act_dtype);
}

}  // namespace kv4
