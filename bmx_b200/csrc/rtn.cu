// Plain RTN (round-to-nearest, symmetric, groupwise) packed cache: quantize-on-append, exporter,
// page dequantizer and the split-KV decode kernel.
//   keys  : `rtn_token`  (groups of k_group channels per token)  or
//           `rtn_channel` (groups of k_group tokens per channel, bmx's KIVI-style key arm); post-RoPE
//   values: `rtn_token`  (groups of v_group channels per token)
// Codes are bmx's signed integers (bmx: src/bmx/quant/rtn.py:23-44): keys in two's-complement nibbles,
// values in two's-complement 2-bit fields (a 2-bit symmetric code only takes -1, 0, 1).
//
// Page block per (slot, head), page = 64 or 128 tokens, head dim 128:
//   [ K nibbles page*64 | K scales | V codes page*32 | V scales page*8 ]
//   K nibbles and V codes use the same lane-fragment order as the k2b page (layout.cuh);
//   K scales: rtn_channel -> (page/k_group) x 128 fp16 in k2b_kscale_idx order
//             rtn_token   -> page x 4 fp16, [row][channel group] (unused groups zero)
//   V scales: page x 4 fp16, [row][channel group]
//
// The decode kernel's page blocks arrive by bulk copies in a shared-memory ring; every lane's operands are
// contiguous 16-byte pieces of the block, adjacent between lanes, in mma fragment order.
#include "decode_common.cuh"
#include "f32x2.cuh"

namespace bmxk {

struct RtnGeom {
  int h_kv, n_q_groups, page, k_arm, k_group, v_group, kbits, vbits;
};
constexpr int RTN_TOKEN = 0, RTN_CHANNEL = 1;

BMXK_HD int rtn_kscale_bytes(const RtnGeom& g) { return g.k_arm == RTN_CHANNEL ? (g.page / g.k_group) * 256 : g.page * 8; }
BMXK_HD int rtn_off_kscale(const RtnGeom& g) { return g.page * 64; }
BMXK_HD int rtn_off_vcode(const RtnGeom& g) { return rtn_off_kscale(g) + rtn_kscale_bytes(g); }
BMXK_HD int rtn_off_vscale(const RtnGeom& g) { return rtn_off_vcode(g) + g.page * 32; }
BMXK_HD int rtn_block_bytes(const RtnGeom& g) { return rtn_off_vscale(g) + g.page * 8; }

// ---------------------------------------------------------------------------------------------
// Quantize-on-append.  One block of 256 threads per (item, head).
//   scale = max(absmax, 1e-12) / qmax ; code = clamp(rint(x / scale), -qmax-1, qmax)   (float32)
// What bounds it: warp instructions and the latency of the loads (it read two bytes at a time and divided per value).  Both pages are
// staged with sixteen-byte loads, all in flight together; then a thread owns whole words of the layout: the values are read as the
// channel pairs of the word, codes are summed up at their bit position in float32 (offset binary, at most 16 bits: exact) and a final
// XOR makes them two's complement: no byte codes, no second pass.
// Divisions become products with 1 / scale: t = x (1 / scale) + offset differs from the true quotient, rounded, by at most
// 4.2e-7 + 4.8e-7 + 4.2e-7, so both round alike unless t lies within RTN_NEAR of a half; the eight or sixteen values of a (half)
// word that holds such a value (or a NaN) are divided.  With 16-bit sources exact halves are common (a value that is half of the
// group's maximum: 4e-4 of the values of 2-bit codes), so it matters that no more than a word is done again.  |x| <= absmax keeps
// the codes inside the clamp.
// Two-bit codes of 16-bit sources (all values; keys of the kivi recipe) need no quotient: qmax is 1, the scale is the group's
// maximum s itself, and x / s > 1/2 exactly when x > s / 2 (two 11-bit numbers whose quotient is not 1/2 are 2^-12 away from it, so
// the division's rounding cannot reach it; a tie is code 0 either way): two packed compares per pair.  A group of
// zeros (a padded token, a dead channel) needs nothing else: no value is above a threshold of zero.  A page whose two-bit groups
// include one with a NaN or an infinite or subnormal maximum takes the general way.
// Measured, 4096 blocks (four sequences of 16384 tokens x 8 heads, 2-bit keys per channel, groups of 64, fp16): 417 -> 109 us = 3.0 TB/s,
// the same with a padded token or a dead channel in every page (419, 489 before), 210 us where every page takes the general way;
// 4-bit keys in groups of 32: 413 -> 153 us, half as many blocks 243 -> 82 us (float32 sources 253 -> 121 us).
// ---------------------------------------------------------------------------------------------
constexpr int RTNQ_THREADS = 256;
constexpr float RTN_NEAR = 4e-6f, RTN_MAGIC = 12582912.f;  // 1.5 * 2^23: adding it rounds to an integer, ties to even

template <typename T>
struct RtnSrc;  // a pair of adjacent values, as staged
template <>
struct RtnSrc<__half> {
  typedef uint32_t Pair;
  static __device__ __forceinline__ float2 f(Pair p) { return __half22float2(u32_as_h2(p)); }
  static __device__ __forceinline__ Pair absmax(Pair a, Pair b) { return h2_as_u32(__hmax2(u32_as_h2(a), __habs2(u32_as_h2(b)))); }
  static __device__ __forceinline__ Pair absmax_nan(Pair a, Pair b) { return h2_as_u32(__hmax2_nan(u32_as_h2(a), __habs2(u32_as_h2(b)))); }
  static __device__ __forceinline__ uint32_t above(Pair x, uint32_t t) { return __hgt2_mask(u32_as_h2(x), u32_as_h2(t)); }  // 0xFFFF per half
  static __device__ __forceinline__ uint32_t below(Pair x, uint32_t t) { return __hlt2_mask(u32_as_h2(x), __hneg2(u32_as_h2(t))); }
  static __device__ __forceinline__ uint32_t halves(float a, float b) { return h2_as_u32(__floats2half2_rn(0.5f * a, 0.5f * b)); }
  static __device__ __forceinline__ bool plain(float m) { return m == 0.f || (m >= 2.5e-4f && m <= 65504.f); }  // m / 2 is zero or a normal number of the type
};
template <>
struct RtnSrc<__nv_bfloat16> {
  typedef uint32_t Pair;
  static __device__ __forceinline__ float2 f(Pair p) { return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xFFFF0000u)); }
  static __device__ __forceinline__ Pair absmax(Pair a, Pair b) {
    const __nv_bfloat162 r = __hmax2(bf2(a), __habs2(bf2(b)));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ Pair absmax_nan(Pair a, Pair b) {
    const __nv_bfloat162 r = __hmax2_nan(bf2(a), __habs2(bf2(b)));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ __nv_bfloat162 bf2(uint32_t a) { return *reinterpret_cast<__nv_bfloat162*>(&a); }
  static __device__ __forceinline__ uint32_t above(Pair x, uint32_t t) { return __hgt2_mask(bf2(x), bf2(t)); }
  static __device__ __forceinline__ uint32_t below(Pair x, uint32_t t) { return __hlt2_mask(bf2(x), __hneg2(bf2(t))); }
  static __device__ __forceinline__ uint32_t halves(float a, float b) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(0.5f * a, 0.5f * b);
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ bool plain(float m) { return m == 0.f || (m >= 1e-30f && m <= 3.3e38f); }
};
template <>
struct RtnSrc<float> {
  typedef float2 Pair;
  static __device__ __forceinline__ float2 f(Pair p) { return p; }
  static __device__ __forceinline__ Pair absmax(Pair a, Pair b) { return make_float2(fmaxf(a.x, fabsf(b.x)), fmaxf(a.y, fabsf(b.y))); }
  static __device__ __forceinline__ Pair absmax_nan(Pair a, Pair b) { return absmax(a, b); }
  static __device__ __forceinline__ uint32_t above(Pair, uint32_t) { return 0u; }  // not used: float sources take the general way
  static __device__ __forceinline__ uint32_t below(Pair, uint32_t) { return 0u; }
  static __device__ __forceinline__ uint32_t halves(float, float) { return 0u; }
  static __device__ __forceinline__ bool plain(float) { return true; }
};
// Two codes plus `offset` (8 or 2), times weight, added to acc; `far`: the largest distance from a rounded value so far.
__device__ __forceinline__ F2 rtn_add_codes(F2 acc, float2 x, F2 inv, float offset, float weight, float& far) {
  const F2 t = f2_fma(f2_pack(x.x, x.y), inv, f2_pack(offset, offset));
  const F2 q = f2_add(f2_add(t, f2_pack(RTN_MAGIC, RTN_MAGIC)), f2_pack(-RTN_MAGIC, -RTN_MAGIC));
  float d0, d1;
  f2_unpack(f2_fma(q, f2_pack(-1.f, -1.f), t), d0, d1);
  far = max_nan(far, max_nan(fabsf(d0), fabsf(d1)));
  return f2_fma(q, f2_pack(weight, weight), acc);
}
// Out of line: it runs for about 1 % of the words.
__device__ __noinline__ float rtn_code_divided(float x, float scale, float qmax) { return fminf(fmaxf(rintf(x / scale), -qmax - 1.f), qmax); }

template <typename T, int PAGE>
struct RtnQuantSmem {
  static constexpr int ROW = HEAD_DIM * (int)sizeof(T);  // bytes per staged row; its 16-byte chunks are XORed with the row's low bits (rtn_at)
  static constexpr int SC = (PAGE / 32) * HEAD_DIM;            // scales: [token group][channel] or [row][4 channel groups], whichever is used
  static constexpr int SC_WORDS = SC > PAGE * 4 ? SC : PAGE * 4;
  static constexpr int BYTES = 2 * PAGE * ROW + 4 * SC_WORDS * 4;  // both pages, both scales and their inverses
};

// Byte `b` of staged row `r`: consecutive rows' equal chunks lie in different banks, and three blocks of 16-bit pages share an SM.
template <int ROW>
__device__ __forceinline__ int rtn_at(int r, int b) { return r * ROW + (b ^ ((r & 7) << 4)); }

template <typename T, int PAGE>
__global__ void __launch_bounds__(RTNQ_THREADS, sizeof(T) == 2 ? 3 : 1) rtn_quant_page_kernel(RtnGeom g, const T* __restrict__ k, const T* __restrict__ v,
                                                                      int64_t stride_seq, int64_t stride_head, int64_t stride_tok,
                                                                      const int32_t* __restrict__ slots, int n_pages,
                                                                      uint8_t* __restrict__ pages, int vec) {
  typedef RtnSrc<T> S;
  typedef typename S::Pair Pair;
  constexpr int ROW = RtnQuantSmem<T, PAGE>::ROW;
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* kst = smem;                       // [PAGE][ROW]
  uint8_t* vst = kst + PAGE * ROW;           // [PAGE][ROW]
  float* ksc = reinterpret_cast<float*>(vst + PAGE * ROW);
  float* vsc = ksc + RtnQuantSmem<T, PAGE>::SC_WORDS;  // [row][4]
  float* kinv = vsc + RtnQuantSmem<T, PAGE>::SC_WORDS;  // 1 / scale
  float* vinv = kinv + RtnQuantSmem<T, PAGE>::SC_WORDS;
  const int item = blockIdx.x / g.h_kv, h = blockIdx.x % g.h_kv;
  const int seq = item / n_pages, pg = item % n_pages, tid = threadIdx.x;
  uint8_t* blk = pages + ((int64_t)slots[item] * g.h_kv + h) * rtn_block_bytes(g);
  const T* ksrc = k + seq * stride_seq + h * stride_head + (int64_t)pg * PAGE * stride_tok;
  const T* vsrc = v + seq * stride_seq + h * stride_head + (int64_t)pg * PAGE * stride_tok;
  __half* kscale = reinterpret_cast<__half*>(blk + rtn_off_kscale(g));
  __half* vscale = reinterpret_cast<__half*>(blk + rtn_off_vscale(g));
  const float kq = (float)((1 << (g.kbits - 1)) - 1), vq = (float)((1 << (g.vbits - 1)) - 1);

  __shared__ int odd_s;
  if (tid == 0) odd_s = 0;
  // ---- staging ----
  if (vec & 1) {
    constexpr int PER_ROW = HEAD_DIM * (int)sizeof(T) / 16, N = PAGE * PER_ROW / RTNQ_THREADS, PER = 16 / (int)sizeof(T);
    uint4 a[N], b[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int o = i * RTNQ_THREADS + tid, r = o / PER_ROW, c = o % PER_ROW;
      a[i] = *reinterpret_cast<const uint4*>(ksrc + r * stride_tok + c * PER);
      b[i] = *reinterpret_cast<const uint4*>(vsrc + r * stride_tok + c * PER);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int o = i * RTNQ_THREADS + tid, r = o / PER_ROW, c = o % PER_ROW;
      *reinterpret_cast<uint4*>(kst + rtn_at<ROW>(r, c * 16)) = a[i];
      *reinterpret_cast<uint4*>(vst + rtn_at<ROW>(r, c * 16)) = b[i];
    }
  } else {
#pragma unroll 8
    for (int o = tid; o < PAGE * HEAD_DIM; o += RTNQ_THREADS) {
      const int r = o >> 7, c = o & 127;
      const int at = rtn_at<ROW>(r, c * (int)sizeof(T));
      *reinterpret_cast<T*>(kst + at) = ksrc[r * stride_tok + c];
      *reinterpret_cast<T*>(vst + at) = vsrc[r * stride_tok + c];
    }
  }
  __syncthreads();

  // ---- scales; beside them 1 / scale, or (two-bit codes of 16-bit sources) half the scale as a pair of the source's type ----
  constexpr bool V2 = sizeof(T) == 2;
  const bool k2 = sizeof(T) == 2 && g.kbits == 2;
  bool odd = false;  // a group that the packed compares do not cover
  auto token_scales = [&](const uint8_t* st, int grp, float qmax, bool two, float* sc, float* inv, __half* out) {  // four lanes per row, 32 channels each
    constexpr int CH = 2 * (int)sizeof(T);  // sixteen-byte chunks of 32 channels
    for (int u = tid; u < PAGE * 4; u += RTNQ_THREADS) {
      const int r = u >> 2, qt = u & 3;
      Pair m = Pair{};
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const uint4 w = *reinterpret_cast<const uint4*>(st + rtn_at<ROW>(r, 16 * (CH * qt + ((i + qt * (CH / 4)) & (CH - 1)))));  // the lanes of a row start in different banks
#pragma unroll
        for (int e = 0; e < 16 / (int)sizeof(Pair); ++e) m = S::absmax_nan(m, reinterpret_cast<const Pair*>(&w)[e]);
      }
      float2 mf = S::f(m);
      if (mf.x != mf.x || mf.y != mf.y) {  // the reference's maximum passes over NaN
        m = Pair{};
        odd |= two;
        for (int i = 0; i < 16; ++i) m = S::absmax(m, *reinterpret_cast<const Pair*>(st + rtn_at<ROW>(r, (16 * qt + i) * (int)sizeof(Pair))));
        mf = S::f(m);
      }
      float am = fmaxf(mf.x, mf.y);
      if (grp >= 64) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
      if (grp == 128) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
      const float s = fmaxf(am, 1e-12f) / qmax;
      sc[u] = s;  // [row][32-channel quarter]
      odd |= two && !S::plain(am);
      if (two) reinterpret_cast<uint32_t*>(inv)[u] = S::halves(s, s);
      else inv[u] = 1.f / s;
      const int per = grp / 32;
      if (qt % per == 0) out[r * 4 + qt / per] = __float2half_rn(s);
      if (qt >= HEAD_DIM / grp) out[r * 4 + qt] = __float2half_rn(0.f);
    }
  };
  if (g.k_arm == RTN_CHANNEL) {  // thread = (channel pair, 32 tokens), maxima of 32-token blocks, then of whole groups
    for (int u = tid; u < 64 * (PAGE / 32); u += RTNQ_THREADS) {
      const int c2 = u & 63, rb = u >> 6;
      Pair m = Pair{};
#pragma unroll 16
      for (int r = 0; r < 32; ++r) m = S::absmax_nan(m, *reinterpret_cast<const Pair*>(kst + rtn_at<ROW>(32 * rb + r, c2 * (int)sizeof(Pair))));
      float2 mf = S::f(m);
      if (mf.x != mf.x || mf.y != mf.y) {
        m = Pair{};
        odd |= k2;
        for (int r = 0; r < 32; ++r) m = S::absmax(m, *reinterpret_cast<const Pair*>(kst + rtn_at<ROW>(32 * rb + r, c2 * (int)sizeof(Pair))));
        mf = S::f(m);
      }
      *reinterpret_cast<float2*>(ksc + rb * HEAD_DIM + 2 * c2) = mf;
    }
    __syncthreads();
    const int per = g.k_group / 32, c = tid & 127;
    float sc[PAGE / 64];
#pragma unroll
    for (int n = 0; n < PAGE / 64; ++n) {
      const int rb = (tid >> 7) + 2 * n, g0 = rb / per * per;
      float am = 0.f;
      for (int i = 0; i < per; ++i) am = fmaxf(am, ksc[(g0 + i) * HEAD_DIM + c]);
      sc[n] = fmaxf(am, 1e-12f) / kq;
      odd |= k2 && !S::plain(am);
      if (rb == g0) kscale[k2b_kscale_idx(rb / per, c)] = __float2half_rn(sc[n]);
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < PAGE / 64; ++n) {
      const int o = ((tid >> 7) + 2 * n) * HEAD_DIM + c;
      ksc[o] = sc[n];
      if (k2) {  // channel pairs: [32-token block][64]
        const float other = __shfl_xor_sync(0xffffffffu, sc[n], 1);
        if (!(c & 1)) reinterpret_cast<uint32_t*>(kinv)[o >> 1] = S::halves(sc[n], other);
      } else {
        kinv[o] = 1.f / sc[n];
      }
    }
  } else {
    token_scales(kst, g.k_group, kq, k2, ksc, kinv, kscale);
  }
  token_scales(vst, g.v_group, vq, V2, vsc, vinv, vscale);
  if (odd) odd_s = 1;
  __syncthreads();
  const bool packed = odd_s == 0;

  // ---- keys: thread = (16-row block, row g and g + 8, lane t of the quad): channels 8n + 2t, + 1 of two rows, 16 bytes each ----
  for (int u = tid; u < PAGE * 2; u += RTNQ_THREADS) {
    const int wr = u >> 5, gg = (u >> 2) & 7, t = u & 3;
    uint32_t out[2][4];
#pragma unroll
    for (int th = 0; th < 2; ++th) {
      const int r = 16 * wr + 8 * th + gg;
      const int chan = (r >> 5) * HEAD_DIM + 2 * t;
      auto pair = [&](int n) { return S::f(*reinterpret_cast<const Pair*>(kst + rtn_at<ROW>(r, (4 * n + t) * (int)sizeof(Pair)))); };
      if (k2 && packed) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t w = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const Pair x = *reinterpret_cast<const Pair*>(kst + rtn_at<ROW>(r, (4 * (4 * q + i) + t) * (int)sizeof(Pair)));
            const uint32_t thr = reinterpret_cast<const uint32_t*>(kinv)[g.k_arm == RTN_CHANNEL ? (chan >> 1) + 4 * (4 * q + i) : 4 * r + q];
            const uint32_t up = S::above(x, thr), dn = S::below(x, thr);
            w |= ((up | dn) & (0x00010001u << (4 * i))) | (dn & (0x000E000Eu << (4 * i)));  // 0001 or 1111
          }
          out[th][q] = w;
        }
      } else
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        F2 acc = f2_pack(8388608.f, 8388608.f);  // 2^23: the sum sits in the low bits
        float far = 0.f;
        const float rs = g.k_arm == RTN_CHANNEL ? 0.f : k2 ? 1.f / ksc[4 * r + q] : kinv[4 * r + q];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          F2 inv;
          if (g.k_arm == RTN_CHANNEL && k2) inv = f2_pack(1.f / ksc[chan + 8 * (4 * q + i)], 1.f / ksc[chan + 8 * (4 * q + i) + 1]);
          else if (g.k_arm == RTN_CHANNEL) inv.v = *reinterpret_cast<const unsigned long long*>(kinv + chan + 8 * (4 * q + i));
          else inv = f2_pack(rs, rs);
          acc = rtn_add_codes(acc, pair(4 * q + i), inv, 8.f, (float)(1 << (4 * i)), far);
        }
        if (!(far < 0.5f - RTN_NEAR)) {
          acc = f2_pack(8388608.f, 8388608.f);
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            const float2 x = pair(4 * q + i);
            const float* sc = g.k_arm == RTN_CHANNEL ? ksc + chan + 8 * (4 * q + i) : ksc + 4 * r + q;
            const float w = (float)(1 << (4 * i));
            acc = f2_fma(f2_pack(rtn_code_divided(x.x, sc[0], kq) + 8.f, rtn_code_divided(x.y, sc[g.k_arm == RTN_CHANNEL], kq) + 8.f), f2_pack(w, w), acc);
          }
        }
        float lo, hi;
        f2_unpack(acc, lo, hi);
        out[th][q] = prmt(__float_as_uint(lo), __float_as_uint(hi), 0x5410u) ^ 0x88888888u;
      }
      uint32_t* dst = reinterpret_cast<uint32_t*>(blk) + ((wr * 2 + th) * 32 + 4 * gg + t) * 4;
      if (vec & 2) *reinterpret_cast<uint4*>(dst) = make_uint4(out[th][0], out[th][1], out[th][2], out[th][3]);
      else
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[q] = out[th][q];
    }
  }
  // ---- values: thread = (16-row block, channels 8m + 2g2, + 1, lane t of the quad, half of the words) ----
  uint32_t* vout = reinterpret_cast<uint32_t*>(blk + rtn_off_vcode(g));
  for (int u = tid; u < PAGE * 2; u += RTNQ_THREADS) {
    const int wr = u >> 5, g2 = (u >> 3) & 3, t = (u >> 1) & 3, jh = u & 1;
    const int r0 = 16 * wr + 2 * t;
    uint32_t words[2][2];  // [channel of the pair][word of the half]
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      const int j = 2 * jh + jj;
      if (V2 && packed) {
        uint32_t w[2];  // 16 bits of each of the two channels' words
#pragma unroll
        for (int hs = 0; hs < 2; ++hs) {
          w[hs] = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int e = k & 1, chi = (k >> 1) & 1, thi = k >> 2, row = r0 + 8 * thi + e, bit = 4 * (2 * chi + e) + 2 * thi;
            const Pair x = *reinterpret_cast<const Pair*>(vst + rtn_at<ROW>(row, (16 * j + 8 * hs + 4 * chi + g2) * (int)sizeof(Pair)));
            const uint32_t thr = reinterpret_cast<const uint32_t*>(vinv)[4 * row + j];
            const uint32_t up = S::above(x, thr), dn = S::below(x, thr);
            w[hs] |= ((up | dn) & (0x00010001u << bit)) | (dn & (0x00020002u << bit));  // 01 or 11
          }
        }
        words[0][jj] = prmt(w[0], w[1], 0x5410u), words[1][jj] = prmt(w[0], w[1], 0x7632u);
        continue;
      }
      float half_lo[2], half_hi[2];
#pragma unroll
      for (int hs = 0; hs < 2; ++hs) {
        // value k = (thi, chi, e): row r0 + 8 thi + e, channels 32 j + 16 hs + 8 chi + 2 g2, + 1
        auto pair = [&](int chi, int row) { return S::f(*reinterpret_cast<const Pair*>(vst + rtn_at<ROW>(r0 + row, (16 * j + 8 * hs + 4 * chi + g2) * (int)sizeof(Pair)))); };
        F2 acc = f2_pack(8388608.f, 8388608.f);
        float far = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int e = k & 1, chi = (k >> 1) & 1, thi = k >> 2, row = 8 * thi + e;
          const float inv = V2 ? 1.f / vsc[4 * (r0 + row) + j] : vinv[4 * (r0 + row) + j];
          acc = rtn_add_codes(acc, pair(chi, row), f2_pack(inv, inv), 2.f, (float)(1 << (4 * (2 * chi + e) + 2 * thi)), far);
        }
        if (!(far < 0.5f - RTN_NEAR)) {
          acc = f2_pack(8388608.f, 8388608.f);
#pragma unroll 1
          for (int k = 0; k < 8; ++k) {
            const int e = k & 1, chi = (k >> 1) & 1, thi = k >> 2, row = 8 * thi + e;
            const float2 x = pair(chi, row);
            const float sc = vsc[4 * (r0 + row) + j], w = (float)(1 << (4 * (2 * chi + e) + 2 * thi));
            acc = f2_fma(f2_pack(rtn_code_divided(x.x, sc, vq) + 2.f, rtn_code_divided(x.y, sc, vq) + 2.f), f2_pack(w, w), acc);
          }
        }
        f2_unpack(acc, half_lo[hs], half_hi[hs]);
      }
      words[0][jj] = prmt(__float_as_uint(half_lo[0]), __float_as_uint(half_lo[1]), 0x5410u) ^ 0xAAAAAAAAu;
      words[1][jj] = prmt(__float_as_uint(half_hi[0]), __float_as_uint(half_hi[1]), 0x5410u) ^ 0xAAAAAAAAu;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t* dst = vout + (wr * 32 + 4 * (2 * g2 + c) + t) * 4 + 2 * jh;
      if (vec & 2) *reinterpret_cast<uint2*>(dst) = make_uint2(words[c][0], words[c][1]);
      else dst[0] = words[c][0], dst[1] = words[c][1];
    }
  }
}

__device__ __forceinline__ int rtn_read_kcode(const uint32_t* kw, int r, int c) {
  int w, b;
  k2b_kres_loc(r, c, w, b);
  return (((kw[w] >> b) & 0xF) ^ 8) - 8;
}
__device__ __forceinline__ int rtn_read_vcode(const uint32_t* vw, int r, int c) {
  int w, b;
  k2b_vcode_loc(r, c, w, b);
  return (((vw[w] >> b) & 3) ^ 2) - 2;
}
__device__ __forceinline__ float rtn_kscale_at(const RtnGeom& g, const __half* ks, int r, int c) {
  return __half2float(g.k_arm == RTN_CHANNEL ? ks[k2b_kscale_idx(r / g.k_group, c)] : ks[r * 4 + c / g.k_group]);
}

// Exporter / dequantizer: one block per (page, head).  Codes go out as int8 in bmx's containers
// (bmx: src/bmx/cache/triton_dequant_attention.py:1390-1451 for token arms; the (C, page) block-dict
// layout of src/bmx/cache/codecs.py:723-725 for channel-grouped keys); dequant = code * fp16 scale.
__global__ void rtn_export_kernel(RtnGeom g, const uint8_t* __restrict__ pages, const int32_t* __restrict__ slots,
                                  int8_t* __restrict__ k_codes, __half* __restrict__ k_scales, int8_t* __restrict__ v_codes,
                                  __half* __restrict__ v_scales, float* __restrict__ k_deq, float* __restrict__ v_deq) {
  const int n = blockIdx.x / g.h_kv, h = blockIdx.x % g.h_kv, page = g.page, C = g.h_kv * HEAD_DIM;
  const uint8_t* blk = pages + ((int64_t)slots[n] * g.h_kv + h) * rtn_block_bytes(g);
  const uint32_t* kw = reinterpret_cast<const uint32_t*>(blk);
  const __half* ks = reinterpret_cast<const __half*>(blk + rtn_off_kscale(g));
  const uint32_t* vw = reinterpret_cast<const uint32_t*>(blk + rtn_off_vcode(g));
  const __half* vs = reinterpret_cast<const __half*>(blk + rtn_off_vscale(g));
  const int nkg = HEAD_DIM / g.k_group, nvg = HEAD_DIM / g.v_group, ntg = page / g.k_group;
  for (int o = threadIdx.x; o < page * HEAD_DIM; o += blockDim.x) {
    const int r = o / HEAD_DIM, c = o % HEAD_DIM;
    const int kc = rtn_read_kcode(kw, r, c), vc = rtn_read_vcode(vw, r, c);
    if (k_codes) {
      if (g.k_arm == RTN_TOKEN) k_codes[(((int64_t)n * g.h_kv + h) * page + r) * HEAD_DIM + c] = (int8_t)kc;
      else k_codes[((int64_t)n * C + h * HEAD_DIM + c) * page + r] = (int8_t)kc;
    }
    if (v_codes) v_codes[(((int64_t)n * g.h_kv + h) * page + r) * HEAD_DIM + c] = (int8_t)vc;
    if (k_deq) k_deq[((int64_t)n * page + r) * C + h * HEAD_DIM + c] = (float)kc * rtn_kscale_at(g, ks, r, c);
    if (v_deq) v_deq[((int64_t)n * page + r) * C + h * HEAD_DIM + c] = (float)vc * __half2float(vs[r * 4 + c / g.v_group]);
  }
  if (k_scales) {
    if (g.k_arm == RTN_TOKEN) {
      for (int o = threadIdx.x; o < page * nkg; o += blockDim.x)
        k_scales[(((int64_t)n * g.h_kv + h) * page + o / nkg) * nkg + o % nkg] = ks[(o / nkg) * 4 + o % nkg];
    } else {
      for (int o = threadIdx.x; o < HEAD_DIM * ntg; o += blockDim.x)
        k_scales[((int64_t)n * C + h * HEAD_DIM + o / ntg) * ntg + o % ntg] = ks[k2b_kscale_idx(o % ntg, o / ntg)];
    }
  }
  if (v_scales)
    for (int o = threadIdx.x; o < page * nvg; o += blockDim.x)
      v_scales[(((int64_t)n * g.h_kv + h) * page + o / nvg) * nvg + o % nvg] = vs[(o / nvg) * 4 + o % nvg];
}

// ---------------------------------------------------------------------------------------------
// Page dequantizer of the dense prompt route: code * fp16 scale rounded once to the model's 16-bit type, written straight into
// (batch, h_kv, row_stride, 128) tensors with the fp16 window behind the pages.  One block per (sequence, page, head); the last
// blocks of a sequence copy 128 window rows each.  What bounds it: the writes (512 bytes per token and head, 112 read).  A thread
// decodes the words of the layout and drops channel pairs into swizzled rows in shared memory, which leave as sixteen-byte stores.
// Measured, 8192 tokens and 128 of the window x 8 heads: 285 -> 10.6 us to fp16 (3.9 TB/s), 297 -> 12.6 us to bf16 (a float32 dequantizer, casts and
// concatenations before).
// ---------------------------------------------------------------------------------------------
constexpr int RTND_THREADS = 256;
template <typename OutT>
struct RtnOut;
template <>
struct RtnOut<__half> {
  static __device__ __forceinline__ uint32_t scaled(__half2 code, __half2 sc) { return h2_as_u32(__hmul2(code, sc)); }  // one rounding
  static __device__ __forceinline__ uint4 copied(uint4 w) { return w; }
};
template <>
struct RtnOut<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t two(float2 x) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(x.x, x.y);
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  static __device__ __forceinline__ uint32_t scaled(__half2 code, __half2 sc) {  // the product of a code and an fp16 scale is exact in float32
    const float2 a = __half22float2(code), b = __half22float2(sc);
    return two(make_float2(a.x * b.x, a.y * b.y));
  }
  static __device__ __forceinline__ uint4 copied(uint4 w) {
    return make_uint4(two(__half22float2(u32_as_h2(w.x))), two(__half22float2(u32_as_h2(w.y))), two(__half22float2(u32_as_h2(w.z))),
                      two(__half22float2(u32_as_h2(w.w))));
  }
};

template <typename OutT, int PAGE>
__global__ void __launch_bounds__(RTND_THREADS) rtn_dequant_dense_kernel(RtnGeom g, const uint8_t* __restrict__ pages,
                                                                         const int32_t* __restrict__ page_table, int table_stride, int n_pg,
                                                                         const __half* __restrict__ k_tail, const __half* __restrict__ v_tail,
                                                                         int tail_len, int tail_cap, OutT* __restrict__ k_out,
                                                                         OutT* __restrict__ v_out, int64_t row_stride) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t *kst = smem, *vst = smem + PAGE * 256;
  const int per_seq = n_pg + (tail_len + 127) / 128, b = blockIdx.x / per_seq, j = blockIdx.x % per_seq, h = blockIdx.y, tid = threadIdx.x;
  const int64_t bh = (int64_t)b * g.h_kv + h;
  if (j >= n_pg) {  // window rows
    const int t0 = (j - n_pg) * 128, n = min(128, tail_len - t0);
    const uint4* ks = reinterpret_cast<const uint4*>(k_tail + (bh * tail_cap + t0) * HEAD_DIM);
    const uint4* vs = reinterpret_cast<const uint4*>(v_tail + (bh * tail_cap + t0) * HEAD_DIM);
    uint4* kd = reinterpret_cast<uint4*>(k_out + (bh * row_stride + (int64_t)n_pg * PAGE + t0) * HEAD_DIM);
    uint4* vd = reinterpret_cast<uint4*>(v_out + (bh * row_stride + (int64_t)n_pg * PAGE + t0) * HEAD_DIM);
    for (int o = tid; o < n * 16; o += RTND_THREADS) kd[o] = RtnOut<OutT>::copied(ks[o]), vd[o] = RtnOut<OutT>::copied(vs[o]);
    return;
  }
  const uint8_t* blk = pages + ((int64_t)page_table[(int64_t)b * table_stride + j] * g.h_kv + h) * rtn_block_bytes(g);
  const __half* ks = reinterpret_cast<const __half*>(blk + rtn_off_kscale(g));
  const __half* vs = reinterpret_cast<const __half*>(blk + rtn_off_vscale(g));
  const __half2 c1032 = __floats2half2_rn(1032.f, 1032.f), c16th = __floats2half2_rn(0.0625f, 0.0625f), cm72 = __floats2half2_rn(-72.f, -72.f);
  // keys: thread = (16-row block, row g and g + 8, lane t): channels 8n + 2t, + 1
  for (int u = tid; u < PAGE * 2; u += RTND_THREADS) {
    const int wr = u >> 5, gg = (u >> 2) & 7, t = u & 3;
    uint4 sc4[4];  // rtn_channel: the scales of the token group, both rows
    if (g.k_arm == RTN_CHANNEL) {
#pragma unroll
      for (int q = 0; q < 4; ++q) sc4[q] = *reinterpret_cast<const uint4*>(ks + ((16 * wr) / g.k_group) * 128 + q * 32 + t * 8);
    }
#pragma unroll
    for (int th = 0; th < 2; ++th) {
      const int r = 16 * wr + 8 * th + gg;
      const uint4 w4 = *reinterpret_cast<const uint4*>(blk + ((wr * 2 + th) * 32 + 4 * gg + t) * 16);
      const uint32_t ww[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t lo = ww[q], hi = ww[q] >> 8;
        __half2 c[4] = {__hsub2(u32_as_h2(lop3<0x6A>(lo, 0x000F000Fu, 0x64086408u)), c1032),
                        __hfma2(u32_as_h2(lop3<0x6A>(lo, 0x00F000F0u, 0x64806480u)), c16th, cm72),
                        __hsub2(u32_as_h2(lop3<0x6A>(hi, 0x000F000Fu, 0x64086408u)), c1032),
                        __hfma2(u32_as_h2(lop3<0x6A>(hi, 0x00F000F0u, 0x64806480u)), c16th, cm72)};
        const uint32_t chan[4] = {sc4[q].x, sc4[q].y, sc4[q].z, sc4[q].w};
        const __half2 tok = g.k_arm == RTN_CHANNEL ? __half2half2(__ushort_as_half(0)) : __half2half2(ks[r * 4 + (32 * q) / g.k_group]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint32_t*>(kst + rtn_at<256>(r, (4 * (4 * q + i) + t) * 4)) =
              RtnOut<OutT>::scaled(c[i], g.k_arm == RTN_CHANNEL ? u32_as_h2(chan[i]) : tok);
      }
    }
  }
  // values: thread = (16-row block, channels 8m + 2g2, + 1, lane t, half of the words)
  for (int u = tid; u < PAGE * 2; u += RTND_THREADS) {
    const int wr = u >> 5, g2 = (u >> 3) & 3, t = (u >> 1) & 3, jh = u & 1, r0 = 16 * wr + 2 * t;
    const uint2 wa = *reinterpret_cast<const uint2*>(blk + rtn_off_vcode(g) + (wr * 32 + 8 * g2 + t) * 16 + 8 * jh);
    const uint2 wb = *reinterpret_cast<const uint2*>(blk + rtn_off_vcode(g) + (wr * 32 + 8 * g2 + 4 + t) * 16 + 8 * jh);
    const uint32_t lut = 0xBCC03C00u;  // high bytes of 0, 1, -2, -1 as fp16
#pragma unroll
    for (int jj = 0; jj < 2; ++jj)
#pragma unroll
      for (int hs = 0; hs < 2; ++hs)
#pragma unroll
        for (int thi = 0; thi < 2; ++thi) {
          const uint32_t sa = ((jj ? wa.y : wa.x) >> (16 * hs + 2 * thi)) & 0x3333u, sb = ((jj ? wb.y : wb.x) >> (16 * hs + 2 * thi)) & 0x3333u;
          const uint32_t ha = prmt(lut, 0u, sa), hb = prmt(lut, 0u, sb);  // bytes: (chi 0, e 0), (0, 1), (1, 0), (1, 1)
          const uint32_t c0 = prmt(ha, hb, 0x5140u), c1 = prmt(ha, hb, 0x7362u);
#pragma unroll
          for (int chi = 0; chi < 2; ++chi)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int r = r0 + 8 * thi + e, c = 32 * (2 * jh + jj) + 16 * hs + 8 * chi + 2 * g2;
              const __half2 code = u32_as_h2(prmt(chi ? c1 : c0, 0u, e ? 0x3424u : 0x1404u));
              *reinterpret_cast<uint32_t*>(vst + rtn_at<256>(r, 2 * c)) =
                  RtnOut<OutT>::scaled(code, __half2half2(vs[r * 4 + (32 * (2 * jh + jj)) / g.v_group]));
            }
        }
  }
  __syncthreads();
  uint4* kd = reinterpret_cast<uint4*>(k_out + (bh * row_stride + (int64_t)j * PAGE) * HEAD_DIM);
  uint4* vd = reinterpret_cast<uint4*>(v_out + (bh * row_stride + (int64_t)j * PAGE) * HEAD_DIM);
  for (int o = tid; o < PAGE * 16; o += RTND_THREADS) {
    const int at = rtn_at<256>(o >> 4, (o & 15) * 16);
    kd[o] = *reinterpret_cast<const uint4*>(kst + at), vd[o] = *reinterpret_cast<const uint4*>(vst + at);
  }
}

// ---------------------------------------------------------------------------------------------
// Split-KV decode.  Persistent grid, one CTA per SM; score warp w and value warp w own token rows 16w..16w+15 of every
// 128-token tile of their CTA's range; same flat decomposition, partial record and merge kernel as k2b.
// ---------------------------------------------------------------------------------------------
struct RtnDecodeParams {
  RtnGeom g;
  const __half* q;
  const uint8_t* pages;
  const int32_t* page_table;
  int table_stride;
  const int32_t* n_pages;
  int batch;
  float scale_log2;
  float* part;
  int32_t* status;
  int n_stages;
  long long wait_limit;  // cycles after which a wait gives up
  int lost;              // self-test: the tile of every range whose copy is left out, or -1
};

constexpr int RTN_WARPS = 8;                             // score warps, and as many value warps
constexpr int RTN_THREADS = (2 * RTN_WARPS + 1) * 32;    // and one warp that issues the copies
constexpr int RTN_MAX_STAGES = 8;
constexpr int RTN_S_BYTES = RTN_WARPS * 32 * 16;         // scores of a tile, beside its stage of the ring
constexpr int RTN_FIXED_SMEM = (8 * 8 * HEAD_DIM + 128) * 4 + (2 + RTN_WARPS) * RTN_MAX_STAGES * 8;  // range reduction, barriers
constexpr int RTN_SMEM = 200 * 1024;                     // most that the ring may grow to

// Bounded wait that reports where it ran out.  It does not look at the status word first: this entry point never asked for a
// cleared workspace, so what the word holds before the call means nothing.  A warp whose wait ran out hands nothing on, so the waits of
// those that depend on it run out as well: the copy warp never fills a stage that was not given back, and waits for the copies in
// flight before it ends.
__device__ __forceinline__ bool rtn_wait(uint64_t* bar, uint32_t parity, const RtnDecodeParams& p, int where) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t spin = 1;; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 255u) == 0u && clock64() - t0 > p.wait_limit) {
      p.status[0] = 1, p.status[1] = blockIdx.x, p.status[2] = where;
      return false;
    }
  }
}
__device__ __forceinline__ bool rtn_warp_wait(uint64_t* bar, uint32_t parity, const RtnDecodeParams& p, int where) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;  // the usual case, without divergence
  return __all_sync(0xffffffffu, rtn_wait(bar, parity, p, where));
}
__device__ __forceinline__ void rtn_value_warps_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// A score maximum as the running maximum takes it: rounded to fp16, and from 8192 on as it is (there the rounding would be off by
// more than 2, and a weight of 2^(8 + error) times a value scale leaves the range of fp16).
__device__ __forceinline__ float rtn_coarse(float x) { return fabsf(x) <= 8192.f ? __half2float(__float2half_rn(x)) : x; }

// What bounds it: latency and instruction issue, not bytes (112 per token and head with groups of 32).  One warp issues the copies of
// whole page blocks, up to n_stages tiles ahead (a register prefetch of one tile left the page-table lookup and the DRAM latency on the
// path of every tile).  The work on 16 token rows is split over two warps, so that the dependent products of one tile's scores run
// beside the value lookups of the tile before: a score warp hands its four scores per lane on through shared memory.  One CTA per SM:
// a range is walked in one piece, so the running maximum and the sums see the tiles in one order whatever the overlap.  The arm and
// the groups are template parameters, so that every operand index is a constant.
//   keys    code * scale rounded once to fp16 (the stored scale is fp16: subnormal scales lose nothing), against the queries as they
//           come: the scores do not depend on how the other heads of the group are scaled.
//   values  codes 0, 1, -2, -1 as fp16 have zero low bytes: one byte-permute lookup yields the high bytes of four codes.
// The running maximum moves only when a score passes it by more than 8 (log2): that test needs no cross-lane reduction.
// Measured, 8 heads, 4-bit keys per channel, groups of 32, step with merge, passes back to back: 16 sequences x 8192 tokens 122.0 ->
// 60.8 us, one sequence of 4096 tokens 12.4 -> 10.4, one of 12000 20.6 -> 17.4 (both warps' work in one warp, two CTAs per SM, nibbles
// as integers against queries that carry the scales: 82.9, 16.7, 22.6 us, and scores that depend on the other heads' magnitudes).
template <int PAGE, int ARM, int KG, int VG>
__global__ void __launch_bounds__(RTN_THREADS, 1) rtn_decode_kernel(const RtnDecodeParams p) {
  constexpr int PAGES_PER_TILE = TILE_TOKENS / PAGE, WR_PER_PAGE = PAGE / 16;
  extern __shared__ __align__(16) uint8_t smem[];
  const RtnGeom g = p.g;
  const int G = g.n_q_groups, PB = rtn_block_bytes(g), stage_bytes = PB * PAGES_PER_TILE;
  uint8_t* ring = smem;
  float* red = reinterpret_cast<float*>(smem + p.n_stages * stage_bytes);  // [8 warps][8 q][128]
  float* red_m = red + 8 * 8 * HEAD_DIM;                                    // [8][8]
  float* red_l = red_m + 64;
  float4* s_sm = reinterpret_cast<float4*>(red_l + 64);                     // [n_stages][8 warps][32 lanes] scores, log2 units
  uint64_t* full = reinterpret_cast<uint64_t*>(s_sm + p.n_stages * RTN_WARPS * 32);  // [RTN_MAX_STAGES] a tile's blocks have landed
  uint64_t* empty = full + RTN_MAX_STAGES;                                  // [RTN_MAX_STAGES] all value warps (and so all score warps) are done with it
  uint64_t* scored = empty + RTN_MAX_STAGES;                                // [RTN_MAX_STAGES][8] a score warp is done with its rows
  int* cum = reinterpret_cast<int*>(scored + RTN_MAX_STAGES * RTN_WARPS);   // [batch + 1]
  int* npg_sm = cum + p.batch + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t4 = lane & 3;
  asm volatile("griddepcontrol.launch_dependents;");  // the merge kernel is this kernel's programmatic dependent (see launch_merge)
  if (warp == 0) fill_cum(cum, p.n_pages, p.batch, g.h_kv, PAGE, lane);
  if (tid == 32) {
    for (int i = 0; i < p.n_stages; ++i) mbar_init(full + i, 1), mbar_init(empty + i, RTN_WARPS);
    for (int i = 0; i < p.n_stages * RTN_WARPS; ++i) mbar_init(scored + i, 1);
    fence_barrier_init();
  }
  for (int i = tid; i < p.batch; i += RTN_THREADS) npg_sm[i] = p.n_pages[i];
  __syncthreads();
  const int total = cum[p.batch];
  const int per_cta = (total + gridDim.x - 1) / gridDim.x;
  const int f_begin = min(total, (int)blockIdx.x * per_cta), f_end = min(total, f_begin + per_cta);
  if (f_begin >= f_end) return;
  TileCursor cur;
  cur.init(cum, npg_sm, f_begin, PAGE);

  if (warp == 2 * RTN_WARPS) {
    // ===================== copies: the lanes hold the slots of the next 32 pages of the sequence =====================
    int st = 0, issued = 0, slots = 0, slots_b = -1, slots_j = 0;
    uint32_t ph = 1;  // parity to wait for on `empty`: the first pass over the ring finds every stage free
    for (int f = f_begin; f < f_end; ++f) {
      const int page0 = cur.j * PAGES_PER_TILE, pages_here = min(PAGES_PER_TILE, npg_sm[cur.b] - page0);
      if (cur.b != slots_b || page0 < slots_j || page0 + PAGES_PER_TILE > slots_j + 32) {
        slots_b = cur.b, slots_j = page0;
        slots = page0 + lane < npg_sm[cur.b] ? p.page_table[(int64_t)cur.b * p.table_stride + page0 + lane] : 0;
      }
      if (!rtn_warp_wait(empty + st, ph, p, 60)) break;
      const bool copies = lane == 0 && f - f_begin != p.lost;
      if (copies) mbar_arrive_expect_tx(full + st, (uint32_t)(pages_here * PB));
#pragma unroll
      for (int i = 0; i < PAGES_PER_TILE; ++i) {
        const int slot = __shfl_sync(0xffffffffu, slots, page0 - slots_j + i);
        if (copies && i < pages_here)
          bulk_g2s(ring + st * stage_bytes + i * PB, p.pages + ((int64_t)slot * g.h_kv + cur.h) * PB, (uint32_t)PB, full + st);
      }
      ++issued;
      cur.next(npg_sm, g.h_kv, PAGE, p.batch);
      if (++st == p.n_stages) st = 0, ph ^= 1;
    }
    for (int i = max(0, issued - p.n_stages); i < issued; ++i)  // no copy is in flight when this CTA ends, whatever became of its readers
      rtn_warp_wait(full + i % p.n_stages, (uint32_t)(i / p.n_stages) & 1u, p, 62);
    return;
  }

  const int w8 = warp & (RTN_WARPS - 1);  // 16 rows of the tile
  const int sub_page = w8 / WR_PER_PAGE, wr = w8 % WR_PER_PAGE;
  int st = 0;
  uint32_t ph = 0;

  if (warp < RTN_WARPS) {
    // ===================== scores =====================
    // byte offsets of this lane's pieces inside a tile's stage
    const int off_k = sub_page * PB + (wr * 64 + lane) * 16;
    const int off_ks = sub_page * PB + rtn_off_kscale(g) + (ARM == RTN_CHANNEL ? (((16 * wr) / KG) * 128 + t4 * 8) * 2 : (16 * wr + gq) * 8);
    const __half2 c1032 = __floats2half2_rn(1032.f, 1032.f), c16th = __floats2half2_rn(0.0625f, 0.0625f), cm72 = __floats2half2_rn(-72.f, -72.f);
    uint32_t qb[16];  // B operands: channel pairs (8n + 2t, + 1) of query g
    int cur_bh = -1;
    for (int f = f_begin; f < f_end; ++f) {
      const int bh = cur.b * g.h_kv + cur.h;
      const bool valid = PAGES_PER_TILE == 1 || cur.j * PAGES_PER_TILE + sub_page < npg_sm[cur.b];
      if (bh != cur_bh) {
        cur_bh = bh;
        const __half* qp = p.q + ((int64_t)bh * G + gq) * HEAD_DIM + 2 * t4;
#pragma unroll
        for (int n = 0; n < 16; ++n) qb[n] = (gq < G) ? *reinterpret_cast<const uint32_t*>(qp + 8 * n) : 0u;
      }
      if (!rtn_warp_wait(full + st, ph, p, 61)) break;
      if (valid) {
        const uint8_t* tile = ring + st * stage_bytes;
        const uint4 k0 = *reinterpret_cast<const uint4*>(tile + off_k), k1 = *reinterpret_cast<const uint4*>(tile + off_k + 512);
        const uint32_t ww[2][4] = {{k0.x, k0.y, k0.z, k0.w}, {k1.x, k1.y, k1.z, k1.w}};
        uint32_t tsc[4];  // rtn_token: the four scales of row g, then those of row g + 8
        if (ARM == RTN_TOKEN) {
          const uint2 x = *reinterpret_cast<const uint2*>(tile + off_ks), y = *reinterpret_cast<const uint2*>(tile + off_ks + 64);
          tsc[0] = x.x, tsc[1] = x.y, tsc[2] = y.x, tsc[3] = y.y;
        }
        float S[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {  // channels 32 qd .. 32 qd + 31
          uint32_t a[4][2];
          uint4 s4 = make_uint4(0u, 0u, 0u, 0u);
          if (ARM == RTN_CHANNEL) s4 = *reinterpret_cast<const uint4*>(tile + off_ks + 64 * qd);
          const uint32_t sw[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
          for (int c = 0; c < 2; ++c) {  // rows g, g + 8
            const uint32_t lo = ww[c][qd], hi = ww[c][qd] >> 8;
            const __half2 code[4] = {__hsub2(u32_as_h2(lop3<0x6A>(lo, 0x000F000Fu, 0x64086408u)), c1032),
                                     __hfma2(u32_as_h2(lop3<0x6A>(lo, 0x00F000F0u, 0x64806480u)), c16th, cm72),
                                     __hsub2(u32_as_h2(lop3<0x6A>(hi, 0x000F000Fu, 0x64086408u)), c1032),
                                     __hfma2(u32_as_h2(lop3<0x6A>(hi, 0x00F000F0u, 0x64806480u)), c16th, cm72)};
            const int gi = (32 * qd) / KG;
            const uint32_t tok = ARM == RTN_TOKEN ? prmt(tsc[2 * c + (gi >> 1)], 0u, (gi & 1) ? 0x3232u : 0x1010u) : 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i][c] = h2_as_u32(__hmul2(code[i], u32_as_h2(ARM == RTN_CHANNEL ? sw[i] : tok)));
          }
          mma_f32acc(S[0], S[1], S[2], S[3], a[0][0], a[0][1], a[1][0], a[1][1], qb[4 * qd], qb[4 * qd + 1]);
          mma_f32acc(S[0], S[1], S[2], S[3], a[2][0], a[2][1], a[3][0], a[3][1], qb[4 * qd + 2], qb[4 * qd + 3]);
        }
        // the place's last scores were read before this stage was filled again
        s_sm[(st * RTN_WARPS + w8) * 32 + lane] = make_float4(S[0] * p.scale_log2, S[1] * p.scale_log2, S[2] * p.scale_log2, S[3] * p.scale_log2);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(scored + st * RTN_WARPS + w8);
      cur.next(npg_sm, g.h_kv, PAGE, p.batch);
      if (++st == p.n_stages) st = 0, ph ^= 1;
    }
    return;
  }

  // ===================== weights and values =====================
  const int off_v = sub_page * PB + rtn_off_vcode(g) + (wr * 32 + lane) * 16, off_vs = sub_page * PB + rtn_off_vscale(g) + (16 * wr + gq) * 8;
  float O[8][4];
  float m0 = 0.f, m1 = 0.f, l0 = 0.f, l1 = 0.f;
  int cur_bh = -1, cur_b = 0, cur_h = 0;
  // two's-complement 2-bit value codes as fp16: 0, 1, -2, -1 (high bytes; the low bytes are zero)
  const uint32_t lut_hi = 0xBCC03C00u;

  auto flush = [&](int b_, int h_) {
#pragma unroll
    for (int m = 4; m <= 16; m <<= 1) l0 += __shfl_xor_sync(0xffffffffu, l0, m), l1 += __shfl_xor_sync(0xffffffffu, l1, m);
    if (gq == 0) {
      red_m[w8 * 8 + 2 * t4] = m0, red_m[w8 * 8 + 2 * t4 + 1] = m1;
      red_l[w8 * 8 + 2 * t4] = l0, red_l[w8 * 8 + 2 * t4 + 1] = l1;
    }
#pragma unroll
    for (int mt = 0; mt < 8; ++mt) {
      float* o = red + (w8 * 8) * HEAD_DIM;
      o[(2 * t4) * HEAD_DIM + 16 * mt + gq] = O[mt][0];
      o[(2 * t4 + 1) * HEAD_DIM + 16 * mt + gq] = O[mt][1];
      o[(2 * t4) * HEAD_DIM + 16 * mt + gq + 8] = O[mt][2];
      o[(2 * t4 + 1) * HEAD_DIM + 16 * mt + gq + 8] = O[mt][3];
    }
    rtn_value_warps_sync();
    float* dst = p.part + ((int64_t)(blockIdx.x + b_ * g.h_kv + h_) * G) * PART_STRIDE;
    for (int o = tid - 32 * RTN_WARPS; o < G * HEAD_DIM; o += 256) {
      const int qi = o / HEAD_DIM, ch = o % HEAD_DIM;
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < 8; ++w) M = fmaxf(M, red_m[w * 8 + qi]);
      float acc = 0.f, l = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float mw = red_m[w * 8 + qi];
        const float f = (mw == -INFINITY) ? 0.f : ex2_approx(mw - M);
        acc += red[(w * 8 + qi) * HEAD_DIM + ch] * f;
        l += red_l[w * 8 + qi] * f;
      }
      dst[qi * PART_STRIDE + 2 + ch] = acc;
      if (ch == 0) dst[qi * PART_STRIDE] = M, dst[qi * PART_STRIDE + 1] = l;
    }
    rtn_value_warps_sync();
  };

  bool alive = true;  // false once a wait ran out: nothing is read or handed back any more, the barriers of flush() are still met
  for (int f = f_begin;; ++f) {
    const int b = cur.b, h = cur.h, bh = f < f_end ? cur.b * g.h_kv + cur.h : -1;
    if (bh != cur_bh) {
      if (cur_bh >= 0) flush(cur_b, cur_h);
      if (f == f_end) break;
      cur_bh = bh, cur_b = b, cur_h = h;
      m0 = (2 * t4 < G) ? -INFINITY : 0.f, m1 = (2 * t4 + 1 < G) ? -INFINITY : 0.f, l0 = l1 = 0.f;
#pragma unroll
      for (int mt = 0; mt < 8; ++mt) O[mt][0] = O[mt][1] = O[mt][2] = O[mt][3] = 0.f;
    }
    const bool valid = PAGES_PER_TILE == 1 || cur.j * PAGES_PER_TILE + sub_page < npg_sm[b];
    if (alive) alive = rtn_warp_wait(full + st, ph, p, 64);
    uint2 vs0 = make_uint2(0u, 0u), vs1 = vs0;
    uint4 vc = make_uint4(0u, 0u, 0u, 0u);
    if (alive && valid) {
      const uint8_t* tile = ring + st * stage_bytes;
      vs0 = *reinterpret_cast<const uint2*>(tile + off_vs), vs1 = *reinterpret_cast<const uint2*>(tile + off_vs + 64);
      vc = *reinterpret_cast<const uint4*>(tile + off_v);
    }
    if (alive) alive = rtn_warp_wait(scored + st * RTN_WARPS + w8, ph, p, 63);
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
    if (alive) {
      if (valid) S = s_sm[(st * RTN_WARPS + w8) * 32 + lane];
      __syncwarp();
      if (lane == 0) mbar_arrive(empty + st);  // this pair of warps holds all it needs of the stage
    }
    if (alive && valid) {
      // ---- online softmax (base 2, lazy rescale), this lane owns queries 2t and 2t+1 ----
      float t0 = rtn_coarse(fmaxf(S.x, S.z)), t1 = rtn_coarse(fmaxf(S.y, S.w));
      if (__any_sync(0xffffffffu, t0 > m0 + 8.f || t1 > m1 + 8.f)) {
#pragma unroll
        for (int m = 4; m <= 16; m <<= 1) t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, m)), t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, m));
        const float n0 = t0 > m0 + 8.f ? t0 + 0.5f : m0, n1 = t1 > m1 + 8.f ? t1 + 0.5f : m1;
        const float f0 = (m0 == -INFINITY) ? 0.f : ex2_approx(m0 - n0), f1 = (m1 == -INFINITY) ? 0.f : ex2_approx(m1 - n1);
        l0 *= f0, l1 *= f1, m0 = n0, m1 = n1;
#pragma unroll
        for (int mt = 0; mt < 8; ++mt) O[mt][0] *= f0, O[mt][1] *= f1, O[mt][2] *= f0, O[mt][3] *= f1;
      }
      const float p0 = ex2_approx(S.x - m0), p1 = ex2_approx(S.y - m1), p2 = ex2_approx(S.z - m0), p3 = ex2_approx(S.w - m1);
      l0 += p0 + p2, l1 += p1 + p3;
      // ---- values: weights times the per-(row, channel group) scale, one B fragment per group ----
      constexpr int NV = HEAD_DIM / VG;
      uint32_t pb[NV][2];
      const uint32_t vsw[4] = {vs0.x, vs0.y, vs1.x, vs1.y};
#pragma unroll
      for (int gi = 0; gi < NV; ++gi) {
        const float2 a2 = __half22float2(u32_as_h2(vsw[gi >> 1])), b2 = __half22float2(u32_as_h2(vsw[2 + (gi >> 1)]));
        const float sa = (gi & 1) ? a2.y : a2.x, sb = (gi & 1) ? b2.y : b2.x;
        pb[gi][0] = movmatrix_trans(h2_as_u32(__floats2half2_rn(p0 * sa, p1 * sa)));
        pb[gi][1] = movmatrix_trans(h2_as_u32(__floats2half2_rn(p2 * sb, p3 * sb)));
      }
      const uint32_t vv[4] = {vc.x, vc.y, vc.z, vc.w};
#pragma unroll
      for (int jw = 0; jw < 4; ++jw) {
        const uint32_t x0 = vv[jw] & 0x33333333u, x1 = (vv[jw] >> 2) & 0x33333333u;
#pragma unroll
        for (int hs = 0; hs < 2; ++hs) {
          const uint32_t hi0 = prmt(lut_hi, 0u, hs ? (x0 >> 16) : x0), hi1 = prmt(lut_hi, 0u, hs ? (x1 >> 16) : x1);
          constexpr int MT_PER = VG / 16;
          const int mt = 2 * jw + hs, gi = mt / MT_PER;
          mma_f32acc(O[mt][0], O[mt][1], O[mt][2], O[mt][3], prmt(hi0, 0u, 0x1404u), prmt(hi0, 0u, 0x3424u), prmt(hi1, 0u, 0x1404u),
                     prmt(hi1, 0u, 0x3424u), pb[gi][0], pb[gi][1]);
        }
      }
    }
    cur.next(npg_sm, g.h_kv, PAGE, p.batch);
    if (++st == p.n_stages) st = 0, ph ^= 1;
  }
}

template <int PAGE, int ARM, int KG, int VG>
static int launch_rtn_decode(const RtnDecodeParams& prm, int grid, size_t smem, cudaStream_t s) {
  static PerDeviceOnce configured;
  if (configured.first()) {
    const cudaError_t e = cudaFuncSetAttribute(rtn_decode_kernel<PAGE, ARM, KG, VG>, cudaFuncAttributeMaxDynamicSharedMemorySize, RTN_SMEM);
    if (e != cudaSuccess) {
      configured.retract();
      set_error("bmxk_rtn_decode: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return BMXK_ERR_CUDA;
    }
  }
  rtn_decode_kernel<PAGE, ARM, KG, VG><<<grid, RTN_THREADS, smem, s>>>(prm);
  return check_launch("bmxk_rtn_decode");
}
template <int PAGE, int ARM, int KG>
static int launch_rtn_decode_v(const RtnDecodeParams& prm, int grid, size_t smem, cudaStream_t s) {
  if (prm.g.v_group == 32) return launch_rtn_decode<PAGE, ARM, KG, 32>(prm, grid, smem, s);
  if (prm.g.v_group == 64) return launch_rtn_decode<PAGE, ARM, KG, 64>(prm, grid, smem, s);
  return launch_rtn_decode<PAGE, ARM, KG, 128>(prm, grid, smem, s);
}
template <int PAGE>
static int launch_rtn_decode_k(const RtnDecodeParams& prm, int grid, size_t smem, cudaStream_t s) {
  const int kg = prm.g.k_group;
  if (prm.g.k_arm == RTN_CHANNEL) {
    if (kg == 32) return launch_rtn_decode_v<PAGE, RTN_CHANNEL, 32>(prm, grid, smem, s);
    if constexpr (PAGE == 128)  // a token group never spans pages
      if (kg == 128) return launch_rtn_decode_v<PAGE, RTN_CHANNEL, 128>(prm, grid, smem, s);
    return launch_rtn_decode_v<PAGE, RTN_CHANNEL, 64>(prm, grid, smem, s);
  }
  if (kg == 32) return launch_rtn_decode_v<PAGE, RTN_TOKEN, 32>(prm, grid, smem, s);
  if (kg == 64) return launch_rtn_decode_v<PAGE, RTN_TOKEN, 64>(prm, grid, smem, s);
  return launch_rtn_decode_v<PAGE, RTN_TOKEN, 128>(prm, grid, smem, s);
}

static int check_rtn_geom(const bmxk_rtn_geom* g, const char* who) {
  BMXK_REQUIRE(g != nullptr, "%s: null geometry", who);
  BMXK_REQUIRE(g->h_kv >= 1 && g->h_kv <= 64 && g->n_q_groups >= 1 && g->n_q_groups <= 8, "%s: h_kv=%d n_q_groups=%d", who,
               g->h_kv, g->n_q_groups);
  BMXK_REQUIRE(g->page == 64 || g->page == 128, "%s: page=%d must be 64 or 128", who, g->page);
  BMXK_REQUIRE(g->k_arm == RTN_TOKEN || g->k_arm == RTN_CHANNEL, "%s: k_arm=%d (0 = rtn_token, 1 = rtn_channel)", who, g->k_arm);
  BMXK_REQUIRE(g->k_group == 32 || g->k_group == 64 || g->k_group == 128, "%s: k_group=%d must be 32, 64 or 128", who, g->k_group);
  BMXK_REQUIRE(g->k_arm == RTN_TOKEN || g->page % g->k_group == 0, "%s: k_group=%d must divide page=%d", who, g->k_group, g->page);
  BMXK_REQUIRE(g->v_group == 32 || g->v_group == 64 || g->v_group == 128, "%s: v_group=%d must be 32, 64 or 128", who, g->v_group);
  BMXK_REQUIRE(g->kbits >= 2 && g->kbits <= 4, "%s: kbits=%d must be in 2..4 (nibble container)", who, g->kbits);
  BMXK_REQUIRE(g->vbits == 2, "%s: vbits=%d (only 2-bit value codes have a kernel)", who, g->vbits);
  return BMXK_OK;
}
static RtnGeom to_rtn(const bmxk_rtn_geom* g) {
  RtnGeom o;
  o.h_kv = g->h_kv, o.n_q_groups = g->n_q_groups, o.page = g->page, o.k_arm = g->k_arm, o.k_group = g->k_group;
  o.v_group = g->v_group, o.kbits = g->kbits, o.vbits = g->vbits;
  return o;
}

template <typename T, int PAGE>
static int launch_rtn_quant(const RtnGeom& g, const T* k, const T* v, int64_t ss, int64_t sh, int64_t st, const int32_t* slots, int blocks,
                            int n_pages, uint8_t* pages, int vec, cudaStream_t s) {
  constexpr int smem = RtnQuantSmem<T, PAGE>::BYTES;
  static PerDeviceOnce configured;
  if (configured.first()) {
    const cudaError_t e = cudaFuncSetAttribute(rtn_quant_page_kernel<T, PAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
      configured.retract();
      set_error("bmxk_rtn_append: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return BMXK_ERR_CUDA;
    }
  }
  rtn_quant_page_kernel<T, PAGE><<<blocks, RTNQ_THREADS, smem, s>>>(g, k, v, ss, sh, st, slots, n_pages, pages, vec);
  return check_launch("bmxk_rtn_append");
}
template <typename T>
static int rtn_append_impl(const RtnGeom& g, const void* k, const void* v, int64_t ss, int64_t sh, int64_t st, const int32_t* slots, int n_seq,
                           int n_pages, uint8_t* pages, cudaStream_t s) {
  constexpr int64_t PER = 16 / sizeof(T);  // sixteen-byte loads need every row start aligned to them
  const int loads = ((uintptr_t)k | (uintptr_t)v) % 16 == 0 && (n_seq == 1 || ss % PER == 0) && (g.h_kv == 1 || sh % PER == 0) && st % PER == 0;
  const int vec = loads | ((uintptr_t)pages % 16 == 0 ? 2 : 0);  // bit 0: wide loads, bit 1: wide stores
  const int blocks = n_seq * n_pages * g.h_kv;
  if (g.page == 128) return launch_rtn_quant<T, 128>(g, (const T*)k, (const T*)v, ss, sh, st, slots, blocks, n_pages, pages, vec, s);
  return launch_rtn_quant<T, 64>(g, (const T*)k, (const T*)v, ss, sh, st, slots, blocks, n_pages, pages, vec, s);
}

template <typename OutT, int PAGE>
static int launch_rtn_dense(const RtnGeom& g, int blocks, const uint8_t* pages, const int32_t* page_table, int table_stride, int n_pages,
                            const __half* k_tail, const __half* v_tail, int tail_len, int tail_cap, OutT* k_out, OutT* v_out, int64_t row_stride,
                            cudaStream_t s) {
  constexpr int smem = 2 * PAGE * 256;
  static PerDeviceOnce configured;
  if (configured.first()) {
    const cudaError_t e = cudaFuncSetAttribute(rtn_dequant_dense_kernel<OutT, PAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
      configured.retract();
      set_error("bmxk_rtn_dequant_dense: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return BMXK_ERR_CUDA;
    }
  }
  rtn_dequant_dense_kernel<OutT, PAGE><<<dim3((unsigned)blocks, (unsigned)g.h_kv), RTND_THREADS, smem, s>>>(
      g, pages, page_table, table_stride, n_pages, k_tail, v_tail, tail_len, tail_cap, k_out, v_out, row_stride);
  return check_launch("bmxk_rtn_dequant_dense");
}

}  // namespace bmxk

using namespace bmxk;

extern "C" {

size_t bmxk_rtn_page_block_bytes(const bmxk_rtn_geom* g) { return g ? (size_t)rtn_block_bytes(to_rtn(g)) : 0; }

size_t bmxk_rtn_decode_workspace_bytes(const bmxk_rtn_geom* g, int batch, int max_pages) {
  if (!g || batch <= 0) return 0;
  (void)max_pages;
  return 256 + ((size_t)num_sms() + (size_t)batch * g->h_kv) * g->n_q_groups * PART_STRIDE * sizeof(float);
}

int bmxk_rtn_append(const bmxk_rtn_geom* g, const void* k, const void* v, int src_dtype, int64_t stride_seq,
                    int64_t stride_head, int64_t stride_tok, const int32_t* slots, int n_seq, int n_pages, void* pages,
                    void* stream) {
  int rc = check_rtn_geom(g, "bmxk_rtn_append");
  if (rc) return rc;
  BMXK_REQUIRE(n_seq >= 0 && n_pages >= 0, "bmxk_rtn_append: negative counts");
  if (n_seq == 0 || n_pages == 0) return BMXK_OK;
  BMXK_REQUIRE(k && v && slots && pages, "bmxk_rtn_append: null pointer");
  BMXK_REQUIRE(stride_tok >= HEAD_DIM, "bmxk_rtn_append: stride_tok=%lld < 128", (long long)stride_tok);
  const RtnGeom gg = to_rtn(g);
  cudaStream_t s = (cudaStream_t)stream;
  uint8_t* dst = (uint8_t*)pages;
  switch (src_dtype) {
    case BMXK_DTYPE_F16:
      return rtn_append_impl<__half>(gg, k, v, stride_seq, stride_head, stride_tok, slots, n_seq, n_pages, dst, s);
    case BMXK_DTYPE_BF16:
      return rtn_append_impl<__nv_bfloat16>(gg, k, v, stride_seq, stride_head, stride_tok, slots, n_seq, n_pages, dst, s);
    case BMXK_DTYPE_F32:
      return rtn_append_impl<float>(gg, k, v, stride_seq, stride_head, stride_tok, slots, n_seq, n_pages, dst, s);
    default:
      set_error("bmxk_rtn_append: unknown src_dtype %d", src_dtype);
      return BMXK_ERR_INVALID;
  }
}

int bmxk_rtn_export(const bmxk_rtn_geom* g, const void* pages, const int32_t* slots, int n, int8_t* k_codes, void* k_scales,
                    int8_t* v_codes, void* v_scales, float* k_deq, float* v_deq, void* stream) {
  int rc = check_rtn_geom(g, "bmxk_rtn_export");
  if (rc) return rc;
  BMXK_REQUIRE(n >= 0, "bmxk_rtn_export: n < 0");
  if (n == 0) return BMXK_OK;
  BMXK_REQUIRE(pages && slots, "bmxk_rtn_export: null pointer");
  rtn_export_kernel<<<n * g->h_kv, 256, 0, (cudaStream_t)stream>>>(to_rtn(g), (const uint8_t*)pages, slots, k_codes,
                                                                  (__half*)k_scales, v_codes, (__half*)v_scales, k_deq, v_deq);
  return check_launch("bmxk_rtn_export");
}

int bmxk_rtn_dequant_dense(const bmxk_rtn_geom* g, const void* pages, const int32_t* page_table, int table_stride, int n_pages, int batch,
                           const void* k_tail, const void* v_tail, int tail_len, int tail_cap, void* k_out, void* v_out,
                           int64_t row_stride, int out_dtype, void* stream) {
  int rc = check_rtn_geom(g, "bmxk_rtn_dequant_dense");
  if (rc) return rc;
  BMXK_REQUIRE(n_pages >= 0 && batch >= 1 && tail_len >= 0 && tail_len <= tail_cap, "bmxk_rtn_dequant_dense: n_pages=%d batch=%d tail_len=%d of %d",
               n_pages, batch, tail_len, tail_cap);
  const int64_t blocks = ((int64_t)n_pages + (tail_len + 127) / 128) * batch;
  if (blocks == 0) return BMXK_OK;
  BMXK_REQUIRE(blocks <= 0x7fffffff, "bmxk_rtn_dequant_dense: too many pages in one call");
  BMXK_REQUIRE(k_out && v_out && (n_pages == 0 || (pages && page_table && table_stride >= n_pages)) && (tail_len == 0 || (k_tail && v_tail)),
               "bmxk_rtn_dequant_dense: null pointer or table_stride=%d < n_pages", table_stride);
  BMXK_REQUIRE(row_stride >= (int64_t)n_pages * g->page + tail_len, "bmxk_rtn_dequant_dense: row_stride=%lld below the rows written",
               (long long)row_stride);
  BMXK_REQUIRE(out_dtype == BMXK_DTYPE_F16 || out_dtype == BMXK_DTYPE_BF16, "bmxk_rtn_dequant_dense: out_dtype=%d (fp16 or bf16)", out_dtype);
  BMXK_REQUIRE((((uintptr_t)pages | (uintptr_t)k_out | (uintptr_t)v_out | (uintptr_t)k_tail | (uintptr_t)v_tail) & 15) == 0,
               "bmxk_rtn_dequant_dense: misaligned buffer");
  const RtnGeom gg = to_rtn(g);
  cudaStream_t s = (cudaStream_t)stream;
#define BMXK_RTN_DENSE(OutT, PAGE)                                                                                                      \
  launch_rtn_dense<OutT, PAGE>(gg, (int)blocks, (const uint8_t*)pages, page_table, table_stride, n_pages, (const __half*)k_tail,        \
                               (const __half*)v_tail, tail_len, tail_cap, (OutT*)k_out, (OutT*)v_out, row_stride, s)
  if (out_dtype == BMXK_DTYPE_F16) return g->page == 128 ? BMXK_RTN_DENSE(__half, 128) : BMXK_RTN_DENSE(__half, 64);
  return g->page == 128 ? BMXK_RTN_DENSE(__nv_bfloat16, 128) : BMXK_RTN_DENSE(__nv_bfloat16, 64);
#undef BMXK_RTN_DENSE
}

static int rtn_decode_impl(const bmxk_rtn_geom* g, const void* q, const void* pages, const int32_t* page_table, int table_stride,
                           const int32_t* n_pages, int batch, int max_pages, const void* k_tail, const void* v_tail,
                           const int32_t* tail_len, int tail_cap, float sm_scale, void* workspace, size_t workspace_bytes, void* out,
                           int out_dtype, float* partial_out, long long wait_limit, int lost, void* stream) {
  int rc = check_rtn_geom(g, "bmxk_rtn_decode");
  if (rc) return rc;
  BMXK_REQUIRE(batch >= 1 && (int64_t)batch * g->h_kv <= MAX_BH, "bmxk_rtn_decode: batch*h_kv out of range");
  BMXK_REQUIRE(max_pages >= 0 && tail_cap >= 0, "bmxk_rtn_decode: negative sizes");
  BMXK_REQUIRE(q && n_pages && workspace, "bmxk_rtn_decode: null pointer");
  BMXK_REQUIRE(max_pages == 0 || (pages && page_table), "bmxk_rtn_decode: null page pool / table");
  BMXK_REQUIRE(tail_cap == 0 || (k_tail && v_tail && tail_len), "bmxk_rtn_decode: null tail");
  BMXK_REQUIRE(out || partial_out, "bmxk_rtn_decode: no output");
  BMXK_REQUIRE(out_dtype == BMXK_DTYPE_F16 || out_dtype == BMXK_DTYPE_F32, "bmxk_rtn_decode: out_dtype=%d", out_dtype);
  BMXK_REQUIRE(workspace_bytes >= bmxk_rtn_decode_workspace_bytes(g, batch, max_pages), "bmxk_rtn_decode: workspace too small");
  BMXK_REQUIRE(((uintptr_t)pages & 15) == 0, "bmxk_rtn_decode: the page pool must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  float* part = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(workspace) + 256);
  const int64_t max_tiles = (int64_t)batch * g->h_kv * (((int64_t)max_pages * g->page + TILE_TOKENS - 1) / TILE_TOKENS);
  const int grid = (int)(max_tiles < num_sms() ? (max_tiles < 1 ? 1 : max_tiles) : num_sms());
  const float scale_log2 = sm_scale * 1.4426950408889634f;
  if (max_pages > 0) {
    RtnDecodeParams prm;
    prm.g = to_rtn(g), prm.q = (const __half*)q, prm.pages = (const uint8_t*)pages, prm.page_table = page_table;
    prm.table_stride = table_stride, prm.n_pages = n_pages, prm.batch = batch, prm.scale_log2 = scale_log2, prm.part = part;
    prm.status = reinterpret_cast<int32_t*>(workspace), prm.wait_limit = wait_limit, prm.lost = lost;
    // batches of thousands of sequences (page counts in shared memory) get a shorter ring
    const size_t fixed = RTN_FIXED_SMEM + (size_t)(2 * batch + 1) * 4 + 16, stage = (size_t)rtn_block_bytes(prm.g) * (TILE_TOKENS / g->page) + RTN_S_BYTES;
    prm.n_stages = 2;
    while (prm.n_stages < RTN_MAX_STAGES && fixed + (prm.n_stages + 1) * stage <= RTN_SMEM) ++prm.n_stages;
    const size_t smem = fixed + prm.n_stages * stage;
    rc = g->page == 128 ? launch_rtn_decode_k<128>(prm, grid, smem, s) : launch_rtn_decode_k<64>(prm, grid, smem, s);
    if (rc) return rc;
  }
  K2bMergeParams mp;
  mp.g.h_kv = g->h_kv, mp.g.n_q_groups = g->n_q_groups, mp.g.page = g->page, mp.g.rank = 0, mp.g.group = g->k_group;
  mp.g.n_coef_heads = 0, mp.g.kbits = g->kbits, mp.g.vbits = g->vbits, mp.g.layout = 0;
  mp.n_sub = 1;
  mp.q = (const __half*)q, mp.n_pages = n_pages, mp.batch = batch, mp.main_grid = grid, mp.part = part;
  mp.k_tail = (const __half*)k_tail, mp.v_tail = (const __half*)v_tail, mp.tail_len = tail_cap > 0 ? tail_len : nullptr;
  mp.tail_cap = tail_cap, mp.signs = nullptr, mp.scale_log2 = scale_log2, mp.out = out, mp.out_dtype = out_dtype;
  mp.partial_out = partial_out;
  return launch_merge(mp, s, max_pages > 0);
}

int bmxk_rtn_decode(const bmxk_rtn_geom* g, const void* q, const void* pages, const int32_t* page_table, int table_stride,
                    const int32_t* n_pages, int batch, int max_pages, const void* k_tail, const void* v_tail,
                    const int32_t* tail_len, int tail_cap, float sm_scale, void* workspace, size_t workspace_bytes, void* out,
                    int out_dtype, float* partial_out, void* stream) {
  return rtn_decode_impl(g, q, pages, page_table, table_stride, n_pages, batch, max_pages, k_tail, v_tail, tail_len, tail_cap, sm_scale, workspace,
                         workspace_bytes, out, out_dtype, partial_out, WAIT_LIMIT_CYCLES, -1, stream);
}

int bmxk_selftest_rtn_lost_copy(const bmxk_rtn_geom* g, const void* q, const void* pages, const int32_t* page_table, int table_stride,
                                const int32_t* n_pages, int batch, int max_pages, float sm_scale, void* workspace, size_t workspace_bytes,
                                void* out, int lost_tile, int64_t limit_cycles, void* stream) {
  BMXK_REQUIRE(lost_tile >= 0, "bmxk_selftest_rtn_lost_copy: lost_tile=%d", lost_tile);
  BMXK_REQUIRE(limit_cycles >= 1000 && limit_cycles <= 200000000,
               "bmxk_selftest_rtn_lost_copy: limit of %lld cycles outside [1e3, 2e8] (this test must end within a fraction of a second)",
               (long long)limit_cycles);
  return rtn_decode_impl(g, q, pages, page_table, table_stride, n_pages, batch, max_pages, nullptr, nullptr, nullptr, 0, sm_scale, workspace,
                         workspace_bytes, out, BMXK_DTYPE_F16, nullptr, (long long)limit_cycles, lost_tile, stream);
}

}  // extern "C"
