// Value codec of one 128-token page of one head, layout 1, for 16-bit sources: Hadamard + 2-bit Lloyd codes
//   n = fp16(max(||v||, 1e-12)); u = v / n; y = fwht(u * signs); idx = #{mid_k < y * sqrt(128)}   (bmx: src/bmx/cache/codecs.py:616-636)
// with the codes of quant_value_token() below, bit for bit, at a fraction of its instructions.  Shared by the k2b page quantizer and
// the value-block quantizer (256 threads per page and head).
//
// What bounds it: warp instructions; the shuffles of a butterfly over lanes cost four issue cycles each and the divisions about nine
// instructions.  So the transform runs on the raw values: 128 = 16 x 8, the 16-point part as one mma.sync per 16 tokens and
// 16 channels (operands +-1 and v: products exact, fp32 accumulators), the 8-point part as packed fp32 adds in registers, and no
// division at all: z = fwht(v * signs), unnormalised, is compared with mid_k * n.  Where z lies so close to a threshold that the two
// computations could disagree, the token is done again by quant_value_token(): about 1 % of the tokens.
//   near: |z - mid_k n| < VQ_EPS n.  In units of n, with sum|u| <= sqrt(128) ||u||: quant_value_token errs by at most
//   2^-24 (11.4 (1 + 7) + 2 * 11.4) = 7e-6 (division, seven levels, the division by and product with sqrt(128)), the products below by
//   16 * 2^-23 * 11.4 = 2.2e-5 (16 terms added in fp32, truncation allowed for) + 3 * 2^-24 * 11.4 = 2e-6: 3.1e-5 in all, VQ_EPS = 4e-5.
//   The bound needs ||u|| = 1 to within the rounding of n to fp16: tokens whose norm is below the fp16 normal range, infinite or NaN
//   always go to quant_value_token().
// The product of the three distances decides both the code's low bit (its sign) and "near" (its size).
// A row of an mma tile can be any token: tile i takes tokens 16 g + i and 16 g + 8 + i for lane group g, so that a thread
// ends up with the tokens of one 16-token word of the layout and shifts the two bits of a code straight into place.
// The channel bits are dealt out for 16-byte operand loads: bits 0, 1, 3, 4 are the 16-point part (pair, operand half, lane of
// the quad), bits 2, 5, 6 the 8-point part.
#pragma once
#include "f32x2.cuh"

namespace bmxk {

constexpr float VQ_EPS = 4e-5f;
constexpr int VQ_THREADS = 256;
constexpr int VQ_STAGE_BYTES = 128 * 256;  // staged page: 16-byte chunk c of row r at r * 256 + ((c ^ vq_key(r)) * 16)
constexpr int VQ_WORDS_BYTES = 128 * 32;   // code words of the page block
constexpr int VQ_SMEM_BYTES = VQ_STAGE_BYTES + VQ_WORDS_BYTES + 128 * 4 + 16;

__device__ __forceinline__ int vq_key(int r) { return ((r >> 4) & 1) * 4 + (r >> 5); }  // eight lanes of a 128-bit read: distinct banks

__device__ __forceinline__ float vq_half_round(float x) { return __half2float(__float2half_rn(x)); }

// One token by one warp, lane = channels 4 lane .. 4 lane + 3: the reference's operation sequence.  Returns the four codes, one per byte.
__device__ __forceinline__ uint32_t quant_value_token(float (&x)[4], const float (&sg)[4], float m0, float m1, float m2, int lane, float& n) {
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) ss = fmaf(x[k], x[k], ss);
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) ss = ss + __shfl_xor_sync(0xffffffffu, ss, m);
  n = vq_half_round(fmaxf(sqrtf(ss), 1e-12f));
#pragma unroll
  for (int k = 0; k < 4; ++k) x[k] = (x[k] / n) * sg[k];
  fwht128_warp(x, lane);
  const float sqrt_d = 11.313708498984761f;
  uint32_t packed4 = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float y = x[k] * sqrt_d;
    packed4 |= (uint32_t)((y > m0) + (y > m1) + (y > m2)) << (8 * k);
  }
  return packed4;
}

template <typename T>
__device__ __forceinline__ float2 vq_unpack(uint32_t w);
template <>
__device__ __forceinline__ float2 vq_unpack<__half>(uint32_t w) { return __half22float2(u32_as_h2(w)); }
template <>
__device__ __forceinline__ float2 vq_unpack<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
template <typename T>
__device__ __forceinline__ void vq_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void vq_mma<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  mma_f32acc(c[0], c[1], c[2], c[3], a0, a1, a2, a3, b0, b1);
}
template <>
__device__ __forceinline__ void vq_mma<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <typename T>
struct VqOne;
template <>
struct VqOne<__half> { static constexpr uint32_t bits = 0x3C00u; };
template <>
struct VqOne<__nv_bfloat16> { static constexpr uint32_t bits = 0x3F80u; };

// Stages the page (128 rows of 128 elements, stride_tok apart).  vec16: rows start on 16-byte boundaries.
template <typename T>
__device__ __forceinline__ void vq_stage(const T* src, int64_t stride_tok, bool vec16, uint8_t* stage, int tid) {
  if (vec16) {
    uint4 u[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {  // eight wide loads in flight per thread
      const int o = k * VQ_THREADS + tid;
      u[k] = *reinterpret_cast<const uint4*>(src + (o >> 4) * stride_tok + 8 * (o & 15));
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int o = k * VQ_THREADS + tid, r = o >> 4;
      *reinterpret_cast<uint4*>(stage + r * 256 + (((o & 15) ^ vq_key(r)) << 4)) = u[k];
    }
  } else {
    for (int o = tid; o < 128 * 128; o += VQ_THREADS) {
      const int r = o >> 7, c = o & 127;
      reinterpret_cast<T*>(stage + r * 256 + (((c >> 3) ^ vq_key(r)) << 4))[c & 7] = src[r * stride_tok + c];
    }
  }
}

// Codes of the staged page into words[1024] (layout 1 order) and norms into vnorm[128] (global).  All 256 threads; the staged page
// must be visible (a barrier after vq_stage), and the words are complete after the caller's next barrier.
template <typename T>
__device__ __forceinline__ void vq_quant_page(const uint8_t* stage, uint32_t* words, float* norms, uint32_t* redo, const float* signs,
                                              const float* codebook, __half* vnorm, int tid) {
  const int lane = tid & 31, warp = tid >> 5, gq = lane >> 2, t4 = lane & 3;
  const float c0 = codebook[0], c1 = codebook[1], c2 = codebook[2], c3 = codebook[3];
  const float m0 = (c0 + c1) / 2.f, m1 = (c1 + c2) / 2.f, m2 = (c2 + c3) / 2.f;
  if (tid < 4) redo[tid] = 0u;
  // the low bit of a code is the sign of the product of the three distances only for sorted thresholds; the products take signs of +-1
  const int plain = __syncthreads_and(m0 <= m1 && m1 <= m2 && fabsf(signs[tid & 127]) == 1.f);
  // ---- norms: warp i takes tokens 16 g + i and 16 g + 8 + i; the sums run in the order of quant_value_token ----
  {
    float ssr[2];
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int r = 16 * gq + 8 * rr + warp;
      float p[4][2];
#pragma unroll
      for (int kh = 0; kh < 4; ++kh) {
        const uint4 u = *reinterpret_cast<const uint4*>(stage + r * 256 + (((4 * kh + t4) ^ vq_key(r)) << 4));
        const float2 x0 = vq_unpack<T>(u.x), x1 = vq_unpack<T>(u.y), x2 = vq_unpack<T>(u.z), x3 = vq_unpack<T>(u.w);
        p[kh][0] = fmaf(x1.y, x1.y, fmaf(x1.x, x1.x, fmaf(x0.y, x0.y, fmaf(x0.x, x0.x, 0.f))));
        p[kh][1] = fmaf(x3.y, x3.y, fmaf(x3.x, x3.x, fmaf(x2.y, x2.y, fmaf(x2.x, x2.x, 0.f))));
      }
      float s[2];
#pragma unroll
      for (int a = 0; a < 2; ++a) {  // channel bits 6, 5 (registers), 4, 3 (lanes), 2 (registers)
        s[a] = (p[0][a] + p[2][a]) + (p[1][a] + p[3][a]);
        s[a] = s[a] + __shfl_xor_sync(0xffffffffu, s[a], 2);
        s[a] = s[a] + __shfl_xor_sync(0xffffffffu, s[a], 1);
      }
      ssr[rr] = s[0] + s[1];
    }
    if (t4 < 2) {
      const int r = 16 * gq + 8 * t4 + warp;
      const float ss = t4 ? ssr[1] : ssr[0];
      const float n = vq_half_round(fmaxf(sqrtf(ss), 1e-12f));
      norms[r] = n;
      vnorm[r] = __float2half_rn(n);
      if (!(n >= 6.2e-5f && n <= 65504.f && ss <= 3.0e38f)) atomicOr(redo + (r >> 5), 1u << (r & 31));
    }
  }
  __syncthreads();
  // ---- codes: warp = (channel bit 4, pair of tiles) ----
  {
    const int nh = warp & 1, pr = warp >> 1;
    uint32_t bm[8][2];  // +-1 operand of each 16-channel block, signs included
#pragma unroll
    for (int ks = 0; ks < 8; ++ks)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t w = 0;
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
          const int ch = 32 * (ks >> 1) + 8 * t4 + 4 * (ks & 1) + 2 * hf + pp;
          // output column g: channel bits 0, 1 = g >> 1, bit 3 = g & 1, bit 4 = nh
          const int par = (pp & (gq >> 1)) ^ (hf & (gq >> 2)) ^ (t4 & gq) ^ ((t4 >> 1) & nh);
          const uint32_t neg = (uint32_t)(par & 1) ^ (signs[ch] < 0.f ? 1u : 0u);
          w |= (VqOne<T>::bits | (neg << 15)) << (16 * pp);
        }
        bm[ks][hf] = w;
      }
    // near-threshold bound on the product of the distances, in units of n^3
    const float d01 = m1 - m0, d12 = m2 - m1, d02 = m2 - m0, eps = VQ_EPS + 3e-7f * fmaxf(fabsf(m0), fabsf(m2));
    const float e01 = d01 + eps, e12 = d12 + eps, e02 = d02 + eps;
    const float bound = 1.001f * eps * fmaxf(fmaxf(e01 * e02, e01 * e12), e02 * e12);
    uint32_t word[8][2];
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) word[nb][0] = word[nb][1] = 0u;
#pragma unroll 1
    for (int ii = 1; ii >= 0; --ii) {
      const int i = 2 * pr + ii, r0 = 16 * gq + i, r1 = r0 + 8;
      F2 z[2][8];  // [row][block], two channels each
#pragma unroll
      for (int kh = 0; kh < 4; ++kh) {
        const uint4 u0 = *reinterpret_cast<const uint4*>(stage + r0 * 256 + (((4 * kh + t4) ^ vq_key(r0)) << 4));
        const uint4 u1 = *reinterpret_cast<const uint4*>(stage + r1 * 256 + (((4 * kh + t4) ^ vq_key(r1)) << 4));
        float ca[4] = {0.f, 0.f, 0.f, 0.f}, cb[4] = {0.f, 0.f, 0.f, 0.f};
        vq_mma<T>(ca, u0.x, u1.x, u0.y, u1.y, bm[2 * kh][0], bm[2 * kh][1]);
        vq_mma<T>(cb, u0.z, u1.z, u0.w, u1.w, bm[2 * kh + 1][0], bm[2 * kh + 1][1]);
        z[0][2 * kh] = f2_pack(ca[0], ca[1]), z[1][2 * kh] = f2_pack(ca[2], ca[3]);
        z[0][2 * kh + 1] = f2_pack(cb[0], cb[1]), z[1][2 * kh + 1] = f2_pack(cb[2], cb[3]);
      }
      const F2 minus1 = f2_pack(-1.f, -1.f);
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
#pragma unroll
        for (int m = 1; m < 8; m <<= 1)
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (!(k & m)) {
              const F2 a = z[rr][k], b = z[rr][k | m];
              z[rr][k] = f2_add(a, b), z[rr][k | m] = f2_fma(b, minus1, a);
            }
      }
      // row 8 + g first: its bits end up above those of row g
#pragma unroll
      for (int rr = 1; rr >= 0; --rr) {
        const int r = rr ? r1 : r0;
        const float n = norms[r];
        const float a0 = m0 * n, a1 = m1 * n, a2 = m2 * n;
        const F2 A0 = f2_pack(a0, a0), A1 = f2_pack(a1, a1), A2 = f2_pack(a2, a2);
        float least = 3.0e38f;
#pragma unroll
        for (int nb = 0; nb < 8; ++nb) {
          const F2 f0 = f2_fma(z[rr][nb], minus1, A0), f1 = f2_fma(z[rr][nb], minus1, A1), f2 = f2_fma(z[rr][nb], minus1, A2);
          const F2 pq = f2_mul(f2_mul(f0, f1), f2);
          float h0, h1, p0, p1;
          f2_unpack(f1, h0, h1), f2_unpack(pq, p0, p1);
          word[nb][0] = __funnelshift_l(__float_as_uint(p0), __funnelshift_l(__float_as_uint(h0), word[nb][0], 1), 1);
          word[nb][1] = __funnelshift_l(__float_as_uint(p1), __funnelshift_l(__float_as_uint(h1), word[nb][1], 1), 1);
          least = fminf(least, fminf(fabsf(p0), fabsf(p1)));
        }
        if (!(least >= bound * n * n * n)) atomicOr(redo + (r >> 5), 1u << (r & 31));
      }
    }
    // eight bits per word and warp: byte pr of word (16-token group g, channel)
    uint8_t* wb = reinterpret_cast<uint8_t*>(words);
#pragma unroll
    for (int nb = 0; nb < 8; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int ch = t4 + 4 * (nb & 1) + 8 * e + 16 * nh + 32 * (nb >> 1);
        wb[((((gq >> 2) * 128 + ch) * 4 + (gq & 3)) << 2) + pr] = (uint8_t)word[nb][e];
      }
  }
  __syncthreads();
  // ---- tokens near a threshold (or with an extreme norm): the exact sequence ----
  {
    uint32_t rd[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) rd[k] = plain ? redo[k] : 0xffffffffu;
    if (rd[0] | rd[1] | rd[2] | rd[3]) {
      float sg[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) sg[k] = signs[4 * lane + k];
      int seen = 0;
#pragma unroll 1
      for (int k = 0; k < 4; ++k)
        for (uint32_t left = rd[k]; left; left &= left - 1) {
          if ((seen++ & 7) != warp) continue;
          const int r = 32 * k + __ffs(left) - 1;
          const uint2 u = *reinterpret_cast<const uint2*>(stage + r * 256 + (((lane >> 1) ^ vq_key(r)) << 4) + 8 * (lane & 1));
          const float2 xa = vq_unpack<T>(u.x), xb = vq_unpack<T>(u.y);
          float x[4] = {xa.x, xa.y, xb.x, xb.y}, n;
          const uint32_t codes = quant_value_token(x, sg, m0, m1, m2, lane, n);
          const int tau = r & 15, bit = tau < 8 ? 4 * tau : 4 * (tau - 8) + 2;
#pragma unroll
          for (int c = 0; c < 4; ++c) {  // other tokens of the same word may be in other warps' hands
            uint32_t* w = words + ((r >> 6) * 128 + 4 * lane + c) * 4 + ((r & 63) >> 4);
            const uint32_t want = (codes >> (8 * c)) & 3u, is = (*reinterpret_cast<volatile uint32_t*>(w) >> bit) & 3u;
            if (want != is) atomicXor(w, (want ^ is) << bit);
          }
        }
    }
  }
}

}  // namespace bmxk
