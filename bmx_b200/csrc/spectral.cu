// K4 spectral key codec, per-head packs (128 x 128 encoder / decoder, per-direction bit tiers):
// quantize-on-append and page dequantizer.
//   encode   Y = M @ enc                                   (bmx: src/bmx/cache/spectral.py:798)
//   per direction j with b_j > 0 bits, per group of `group` tokens: symmetric RTN with the step refined
//   by 10 alternating-minimisation rounds                  (bmx: src/bmx/quant/rtn.py:10-44, mse_scale=True)
//   decode   M_hat = Y_hat @ dec^T                          (bmx: src/bmx/cache/spectral.py:812-839)
// Containers follow bmx (spectral.py:703-739): 2- and 4-bit tiers offset-binary at exact width, the 3-bit
// tier as two's-complement nibbles, 5/6/8-bit tiers as int8; all packed along tokens.
//
// Page block per (slot, head): for every direction with bits, its code row (page * container_bits / 8
// bytes) at the byte offset the host assigns (directions sorted by tier), then float32 scales
// [direction][page / group].  Sums run in ascending index order with one accumulator (fmaf for the two
// matrix products; separate multiply and add inside the step refinement, as the reference does), which
// makes the result independent of launch shape.  Compiled with -fmad=false.
#include "value_quant.cuh"

namespace bmxk {

struct SpectralGeom {
  int h_kv, page, group, block_bytes, scale_off;
};

__device__ __forceinline__ int container_bits(int b) { return b == 0 ? 0 : (b == 2 ? 2 : (b <= 4 ? 4 : 8)); }

// Round-to-nearest-even of a float of magnitude below 2^22, as the low bits of (x + RINT_MAGIC); minus RINT_MAGIC: rintf(x).
constexpr float RINT_MAGIC = 12582912.f;

// code = clamp(rint(x / scale)) of two values, by the product with r = 1 / scale.  |x r - x / scale| <= 2^-23 |x r| and the true
// division rounds by another 2^-24, so both round alike unless x r lies within (qmax + 2) 2^-22 of a half; `far` collects the
// largest distance from the rounded value, and a caller that finds it above 0.5 - (qmax + 2) 2^-22 divides instead.  (Values
// clamped to -qmax - 1 or qmax are at distance 0.)
__device__ __forceinline__ F2 codes_by_product(F2 x, F2 r, float lo, float hi, float& far) {
  const F2 magic = f2_pack(RINT_MAGIC, RINT_MAGIC), unmagic = f2_pack(-RINT_MAGIC, -RINT_MAGIC), minus1 = f2_pack(-1.f, -1.f);
  float t0, t1, d0, d1;
  f2_unpack(f2_mul(x, r), t0, t1);
  const F2 t = f2_pack(fminf(fmaxf(t0, lo), hi), fminf(fmaxf(t1, lo), hi));
  const F2 q = f2_add(f2_add(t, magic), unmagic);
  f2_unpack(f2_fma(q, minus1, t), d0, d1);
  far = fmaxf(far, fmaxf(fabsf(d0), fabsf(d1)));
  return q;
}
__device__ __forceinline__ float code_by_division(float x, float scale, float lo, float hi) { return fminf(fmaxf(rintf(x / scale), lo), hi); }

// One block of 256 threads per (item, head), two blocks per SM.
// What bounds it: the fp32 pipe.  Y = M @ enc is 2 million fused multiply-adds per block that have to stay float32 sums in ascending
// order (the scales are float32 numbers derived from every value), the refinement about seven fp32 operations per value and round.
//   encode      keys transposed in shared memory, 32 encoder rows at a time beside them (the next 32 travel in registers); a warp
//               owns 16 of the directions that carry bits (the others are never computed), a thread PAGE / 16 rows x 8 directions.
//   refinement  thread = chain (direction, token group), num and den in the reference's order (den is a sum of small integers: exact
//               in any).  A round whose scale comes out as it went in is a fixed point: the remaining rounds would repeat it and are
//               skipped.  Chains need 3 to 10 rounds (mean 6), the slowest of 32 nearly always 10: after rounds 4, 6 and 8 the chains
//               that still move are packed to the front of the block (after every round costs more in barriers than it saves).
//               Divisions become products with the reciprocal (codes_by_product); rounds with a value near a half divide.
// Measured, 2048 blocks (four sequences of 8192 tokens x 8 heads, 104 of 128 directions with bits, groups of 64): 927 -> 320 us (with
// the value blocks of value_blocks.cu 1013 -> 374 us), of which about 150 are the product (104 at the fp32 peak), 90 the refinement, 50
// the loads, 20 the codes.
// Packed fp32 pairs for the product (409 us with the values: operand bandwidth), 64-row blocks at three or four per SM (397, 427 us) are
// slower.
constexpr int SQ_THREADS = 256, SQ_CHUNK = 32;
__host__ __device__ constexpr int sq_stride(int page) { return page + 4; }  // floats per channel row: 128-bit reads of consecutive rows hit distinct banks
__host__ __device__ constexpr int sq_smem(int page) { return (HEAD_DIM * sq_stride(page) + 2 * SQ_CHUNK * HEAD_DIM + 2 * HEAD_DIM + 16) * 4; }

template <typename T, int PAGE>
__global__ void __launch_bounds__(SQ_THREADS, 2) spectral_quant_page_kernel(SpectralGeom g, const T* __restrict__ k, int64_t stride_seq,
                                                                            int64_t stride_head, int64_t stride_tok,
                                                                            const float* __restrict__ enc, const int32_t* __restrict__ col_bits,
                                                                            const int32_t* __restrict__ col_off,
                                                                            const int32_t* __restrict__ slots, int n_pages,
                                                                            uint8_t* __restrict__ pages, int vec) {
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr int STR = sq_stride(PAGE), RPT = PAGE / 16, RB = PAGE / 32;
  float* Ms = reinterpret_cast<float*>(smem);         // [128 channels][STR] keys, later [direction in the list][STR] Y
  float* es = Ms + HEAD_DIM * STR;                     // [2][SQ_CHUNK][128] encoder rows, columns of the list
  float* scale_s = es;                                 // [256] later: scales of the chains at hand,
  uint8_t* list = reinterpret_cast<uint8_t*>(scale_s + SQ_THREADS);  // [2][256] and the chains that still move
  int* cols = reinterpret_cast<int*>(es + 2 * SQ_CHUNK * HEAD_DIM);  // list of the directions with bits, ascending: direction | bits << 8
  int* offs = cols + HEAD_DIM;                         // their code rows' byte offsets
  int* moved = offs + HEAD_DIM;                        // [8] chains of each warp that still move (first: directions per warp)
  const int item = blockIdx.x / g.h_kv, h = blockIdx.x % g.h_kv;
  const int seq = item / n_pages, pg = item % n_pages, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // every global read that the rest waits for is issued here together
  const int my_bits = tid < HEAD_DIM ? col_bits[h * HEAD_DIM + tid] : 0, my_off = tid < HEAD_DIM ? col_off[h * HEAD_DIM + tid] : 0;
  uint8_t* blk = pages + ((int64_t)slots[item] * g.h_kv + h) * g.block_bytes;
  {  // keys: a lane takes 16 * RB channels of one row
    const int r = 32 * (warp % RB) + lane, c_base = (warp / RB) * 16 * RB;
    const T* src = k + seq * stride_seq + h * stride_head + ((int64_t)pg * PAGE + r) * stride_tok + c_base;
    if (vec) {
      constexpr int PER = 16 / (int)sizeof(T);
      uint4 u[16 * RB / PER];
#pragma unroll
      for (int i = 0; i < 16 * RB / PER; ++i) u[i] = *reinterpret_cast<const uint4*>(src + i * PER);
#pragma unroll
      for (int i = 0; i < 16 * RB; ++i) Ms[(c_base + i) * STR + r] = load_as_float<T>(reinterpret_cast<const T*>(u) + i);
    } else {
#pragma unroll 8
      for (int i = 0; i < 16 * RB; ++i) Ms[(c_base + i) * STR + r] = load_as_float<T>(src + i);
    }
  }
  const uint32_t used_mask = __ballot_sync(0xffffffffu, my_bits != 0);
  if (lane == 0) moved[warp] = __popc(used_mask);
  __syncthreads();
  const int n_used = moved[0] + moved[1] + moved[2] + moved[3];
  if (my_bits != 0) {
    int n = __popc(used_mask & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) n += moved[w];
    cols[n] = tid | (my_bits << 8), offs[n] = my_off;
  }
  __syncthreads();
  const float* e = enc + (int64_t)h * HEAD_DIM * HEAD_DIM;
  // ---- Y[:, list] ----
  {
    const int jl = tid & 127, cl = tid >> 7, col = jl < n_used ? cols[jl] & 0xFF : -1;
    float nxt[SQ_CHUNK / 2];
    auto fetch = [&](int c0) {
#pragma unroll
      for (int i = 0; i < SQ_CHUNK / 2; ++i) nxt[i] = col >= 0 ? e[(c0 + cl + 2 * i) * HEAD_DIM + col] : 0.f;
    };
    auto put = [&](float* dst) {
#pragma unroll
      for (int i = 0; i < SQ_CHUNK / 2; ++i) dst[(cl + 2 * i) * HEAD_DIM + jl] = nxt[i];
    };
    const bool works = 16 * warp < n_used;
    const int rg = lane & 15, j0 = 16 * warp + 8 * (lane >> 4);  // rows 4 rg .. + 3 (and 64 + 4 rg ..): a quarter-warp reads 128 bytes on end
    float acc[RPT][8];
#pragma unroll
    for (int a = 0; a < RPT; ++a)
#pragma unroll
      for (int b = 0; b < 8; ++b) acc[a][b] = 0.f;
    fetch(0);
    put(es);
    __syncthreads();
#pragma unroll 1
    for (int c0 = 0; c0 < HEAD_DIM; c0 += SQ_CHUNK) {
      const float* eb = es + ((c0 / SQ_CHUNK) & 1) * SQ_CHUNK * HEAD_DIM;
      if (c0 + SQ_CHUNK < HEAD_DIM) fetch(c0 + SQ_CHUNK);
      if (works) {
#pragma unroll 2
        for (int c = 0; c < SQ_CHUNK; ++c) {
          float m[RPT], w[8];
#pragma unroll
          for (int a = 0; a < RPT; a += 4) {
            const float4 t = *reinterpret_cast<const float4*>(Ms + (c0 + c) * STR + 4 * rg + 16 * a);
            m[a] = t.x, m[a + 1] = t.y, m[a + 2] = t.z, m[a + 3] = t.w;
          }
#pragma unroll
          for (int b = 0; b < 8; b += 4) {
            const float4 t = *reinterpret_cast<const float4*>(eb + c * HEAD_DIM + j0 + b);
            w[b] = t.x, w[b + 1] = t.y, w[b + 2] = t.z, w[b + 3] = t.w;
          }
#pragma unroll
          for (int a = 0; a < RPT; ++a)
#pragma unroll
            for (int b = 0; b < 8; ++b) acc[a][b] = fmaf(m[a], w[b], acc[a][b]);
        }
      }
      if (c0 + SQ_CHUNK < HEAD_DIM) put(es + (((c0 / SQ_CHUNK) + 1) & 1) * SQ_CHUNK * HEAD_DIM);
      __syncthreads();  // the chunk read here is overwritten two rounds on; after the last one Y may replace the keys
    }
    if (works)
#pragma unroll
      for (int b = 0; b < 8; ++b)
#pragma unroll
        for (int a = 0; a < RPT; a += 4)
          *reinterpret_cast<float4*>(Ms + (j0 + b) * STR + 4 * rg + 16 * a) = make_float4(acc[a][b], acc[a + 1][b], acc[a + 2][b], acc[a + 3][b]);
  }
  __syncthreads();
  // ---- scales and codes: chain = (token group, direction), up to 256 at a time ----
  const int n_grp = PAGE / g.group;
  for (int q0 = 0; q0 < n_used * n_grp; q0 += SQ_THREADS) {
    const int n_here = min(SQ_THREADS, n_used * n_grp - q0);
    if (tid < n_here) {
      const int q = q0 + tid, grp = q / n_used, jl = q - grp * n_used, b = cols[jl] >> 8;
      const float* x = Ms + jl * STR + grp * g.group;
      float amax = 0.f;
      for (int r = 0; r < g.group; r += 4) {
        const float4 t = *reinterpret_cast<const float4*>(x + r);
        amax = fmaxf(fmaxf(fmaxf(amax, fabsf(t.x)), fmaxf(fabsf(t.y), fabsf(t.z))), fabsf(t.w));
      }
      scale_s[tid] = fmaxf(amax, 1e-12f) / (float)((1 << (b - 1)) - 1);
      list[tid] = (uint8_t)tid;
    }
    __syncthreads();
    int n_act = n_here;
    for (int seg = 0; seg < 4 && n_act > 0; ++seg) {  // rounds 0..3, 4..5, 6..7, 8..9
      const uint8_t* cur = list + (seg & 1) * SQ_THREADS;
      uint8_t* nxt = list + ((seg & 1) ^ 1) * SQ_THREADS;
      bool moves = false;
      int id = 0;
      if (tid < n_act) {
        id = cur[tid];
        const int q = q0 + id, grp = q / n_used, jl = q - grp * n_used, b = cols[jl] >> 8;
        const float qmax = (float)((1 << (b - 1)) - 1), lo = -qmax - 1.f, hi = qmax, near_half = 0.5f - (qmax + 2.f) * 2.384185791015625e-7f;
        const float* x = Ms + jl * STR + grp * g.group;
        float scale = scale_s[id];
        moves = true;
#pragma unroll 1
        for (int it = seg ? 2 : 4; it > 0 && moves; --it) {
          float num = 0.f, den = 0.f, far = 0.f;
          const bool recip = scale < 1e30f;  // 1 / scale is a normal number
          if (recip) {
            const float inv = 1.f / scale;
            const F2 r2 = f2_pack(inv, inv);
            F2 d2 = f2_pack(0.f, 0.f);
#pragma unroll 4
            for (int r = 0; r < g.group; r += 4) {
              const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(x + r);
              F2 xa, xb;
              xa.v = t.x, xb.v = t.y;
              const F2 qa = codes_by_product(xa, r2, lo, hi, far), qb = codes_by_product(xb, r2, lo, hi, far);
              float p0, p1, p2, p3;
              f2_unpack(f2_mul(xa, qa), p0, p1), f2_unpack(f2_mul(xb, qb), p2, p3);
              num = num + p0, num = num + p1, num = num + p2, num = num + p3;
              d2 = f2_fma(qa, qa, d2), d2 = f2_fma(qb, qb, d2);
            }
            float e0, e1;
            f2_unpack(d2, e0, e1);
            den = e0 + e1;
          }
          if (!recip || !(far < near_half)) {
            num = den = 0.f;
            for (int r = 0; r < g.group; ++r) {
              const float c = code_by_division(x[r], scale, lo, hi);
              num = num + x[r] * c;
              den = den + c * c;
            }
          }
          const float now = fmaxf(num / fmaxf(den, 1e-12f), 1e-12f);
          moves = now != scale;
          scale = now;
        }
        scale_s[id] = scale;
      }
      // the chains that moved, packed to the front: whole warps fall idle instead of waiting for their slowest lane
      const uint32_t mask = __ballot_sync(0xffffffffu, moves);
      if (lane == 0) moved[warp] = __popc(mask);
      __syncthreads();
      int before = 0, all = 0;
#pragma unroll
      for (int w = 0; w < SQ_THREADS / 32; ++w) {
        const int m = moved[w];
        before += w < warp ? m : 0, all += m;
      }
      if (moves) nxt[before + __popc(mask & ((1u << lane) - 1u))] = (uint8_t)id;
      n_act = all;
      __syncthreads();
    }
    if (tid < n_here) {
      const int q = q0 + tid, grp = q / n_used, jl = q - grp * n_used, j = cols[jl] & 0xFF, r0 = grp * g.group;
      const int b = cols[jl] >> 8, cb = container_bits(b);
      const float qmax = (float)((1 << (b - 1)) - 1), lo = -qmax - 1.f, hi = qmax, near_half = 0.5f - (qmax + 2.f) * 2.384185791015625e-7f;
      const float* x = Ms + jl * STR + r0;
      const float scale = scale_s[tid];
      reinterpret_cast<float*>(blk + g.scale_off)[j * n_grp + grp] = scale;
      uint8_t* row = blk + offs[jl] + r0 * cb / 8;
      const float inv = 1.f / scale;
      const F2 r2 = f2_pack(inv, inv), magic = f2_pack(RINT_MAGIC, RINT_MAGIC);
      const uint32_t off = (b == 2 || b == 4) ? 1u << (b - 1) : 0u, mask = (1u << cb) - 1u;
      const bool wide = ((uintptr_t)row & 7) == 0;
      for (int r = 0; r < g.group; r += 8) {  // eight codes: cb bytes
        F2 qv[4];
        float far = 0.f;
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(x + r + 2 * u);
          F2 xa, xb;
          xa.v = t.x, xb.v = t.y;
          qv[u] = codes_by_product(xa, r2, lo, hi, far), qv[u + 1] = codes_by_product(xb, r2, lo, hi, far);
        }
        if (!(scale < 1e30f) || !(far < near_half))
#pragma unroll
          for (int u = 0; u < 4; ++u) qv[u] = f2_pack(code_by_division(x[r + 2 * u], scale, lo, hi), code_by_division(x[r + 2 * u + 1], scale, lo, hi));
        uint32_t w0 = 0, w1 = 0;  // codes 0..3 and 4..7, cb bits each
#pragma unroll
        for (int u = 3; u >= 0; --u) {
          float a, c;
          f2_unpack(f2_add(qv[u], magic), a, c);  // the code sits in the low bits
          const uint32_t f0 = (__float_as_uint(a) + off) & mask, f1 = (__float_as_uint(c) + off) & mask;
          uint32_t& w = u >= 2 ? w1 : w0;
          w = (((w << cb) | f1) << cb) | f0;
        }
        uint8_t* dst = row + r * cb / 8;
        if (cb == 8) {
          if (wide) *reinterpret_cast<uint2*>(dst) = make_uint2(w0, w1);
          else
            for (int i = 0; i < 8; ++i) dst[i] = (uint8_t)((i < 4 ? w0 : w1) >> (8 * (i & 3)));
        } else {
          const uint32_t w = w0 | (w1 << (4 * cb));
          if (!wide)
            for (int i = 0; i < cb; ++i) dst[i] = (uint8_t)(w >> (8 * i));
          else if (cb == 4) *reinterpret_cast<uint32_t*>(dst) = w;
          else *reinterpret_cast<uint16_t*>(dst) = (uint16_t)w;
        }
      }
    }
    __syncthreads();  // the next 256 chains take over the lists
  }
}

template <typename T, int PAGE>
static int launch_spectral_quant(const SpectralGeom& g, const T* k, int64_t ss, int64_t sh, int64_t st, const float* enc, const int32_t* col_bits,
                                 const int32_t* col_off, const int32_t* slots, int blocks, int n_pages, uint8_t* pages, int vec, cudaStream_t s) {
  static PerDeviceOnce configured;
  if (configured.first()) {
    const cudaError_t e = cudaFuncSetAttribute(spectral_quant_page_kernel<T, PAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, sq_smem(PAGE));
    if (e != cudaSuccess) {
      configured.retract();
      set_error("bmxk_spectral_append: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return BMXK_ERR_CUDA;
    }
  }
  spectral_quant_page_kernel<T, PAGE><<<blocks, SQ_THREADS, sq_smem(PAGE), s>>>(g, k, ss, sh, st, enc, col_bits, col_off, slots, n_pages, pages, vec);
  return check_launch("bmxk_spectral_append");
}
template <typename T>
static int spectral_append_impl(const SpectralGeom& g, const void* k, int64_t ss, int64_t sh, int64_t st, const float* enc, const int32_t* col_bits,
                                const int32_t* col_off, const int32_t* slots, int n_seq, int n_pages, uint8_t* pages, cudaStream_t s) {
  constexpr int64_t PER = 16 / sizeof(T);  // sixteen-byte loads need every row start aligned to them
  const int vec = (uintptr_t)k % 16 == 0 && (n_seq == 1 || ss % PER == 0) && (g.h_kv == 1 || sh % PER == 0) && st % PER == 0;
  const int blocks = n_seq * n_pages * g.h_kv;
  if (g.page == 128) return launch_spectral_quant<T, 128>(g, (const T*)k, ss, sh, st, enc, col_bits, col_off, slots, blocks, n_pages, pages, vec, s);
  return launch_spectral_quant<T, 64>(g, (const T*)k, ss, sh, st, enc, col_bits, col_off, slots, blocks, n_pages, pages, vec, s);
}

__device__ __forceinline__ int spectral_code(const uint8_t* row, int r, int b) {
  const int cb = container_bits(b);
  if (cb == 8) return (int)(int8_t)row[r];
  const uint32_t f = (row[r * cb / 8] >> (cb * (r % (8 / cb)))) & ((1u << cb) - 1u);
  if (b == 3) return (int)((f ^ 8u)) - 8;          // two's-complement nibble
  return (int)f - (1 << (b - 1));                  // offset binary (2- and 4-bit tiers)
}

// One block per (page, head): codes as int8 (n, h, 128 directions, page), scales float32, and/or
// M_hat = Y_hat @ dec^T as float32 (n, page, h*128).
__global__ void __launch_bounds__(128) spectral_dequant_kernel(SpectralGeom g, const uint8_t* __restrict__ pages,
                                                               const float* __restrict__ dec, const int32_t* __restrict__ col_bits,
                                                               const int32_t* __restrict__ col_off, const int32_t* __restrict__ slots,
                                                               int8_t* __restrict__ codes, float* __restrict__ scales_out,
                                                               float* __restrict__ k_out) {
  extern __shared__ __align__(16) uint8_t smem[];
  float* Ys = reinterpret_cast<float*>(smem);  // [page][128]
  const int n = blockIdx.x / g.h_kv, h = blockIdx.x % g.h_kv, page = g.page, j = threadIdx.x, ngrp = page / g.group;
  const uint8_t* blk = pages + ((int64_t)slots[n] * g.h_kv + h) * g.block_bytes;
  const int b = col_bits[h * HEAD_DIM + j];
  const uint8_t* row = blk + col_off[h * HEAD_DIM + j];
  const float* sc = reinterpret_cast<const float*>(blk + g.scale_off) + j * ngrp;
  for (int r = 0; r < page; ++r) {
    const int q = b ? spectral_code(row, r, b) : 0;
    Ys[r * HEAD_DIM + j] = b ? (float)q * sc[r / g.group] : 0.f;
    if (codes) codes[(((int64_t)n * g.h_kv + h) * HEAD_DIM + j) * page + r] = (int8_t)q;
  }
  if (scales_out)
    for (int grp = 0; grp < ngrp; ++grp) scales_out[(((int64_t)n * g.h_kv + h) * HEAD_DIM + j) * ngrp + grp] = b ? sc[grp] : 0.f;
  __syncthreads();
  if (k_out) {
    const float* d = dec + (int64_t)h * HEAD_DIM * HEAD_DIM + (int64_t)j * HEAD_DIM;  // dec[c = j][:]
    for (int r = 0; r < page; ++r) {
      float acc = 0.f;
      for (int i = 0; i < HEAD_DIM; ++i) acc = fmaf(Ys[r * HEAD_DIM + i], d[i], acc);
      k_out[((int64_t)n * page + r) * (g.h_kv * HEAD_DIM) + h * HEAD_DIM + j] = acc;
    }
  }
}

static int check_sgeom(const bmxk_spectral_geom* g, const char* who) {
  BMXK_REQUIRE(g != nullptr, "%s: null geometry", who);
  BMXK_REQUIRE(g->h_kv >= 1 && g->h_kv <= 64, "%s: h_kv=%d", who, g->h_kv);
  BMXK_REQUIRE(g->page == 64 || g->page == 128, "%s: page=%d must be 64 or 128", who, g->page);
  BMXK_REQUIRE(g->group >= 8 && g->page % g->group == 0 && g->group % 8 == 0, "%s: group=%d must divide page and be a multiple of 8", who,
               g->group);
  BMXK_REQUIRE(g->block_bytes > 0 && g->scale_off >= 0 && g->scale_off % 4 == 0 &&
                   g->scale_off + HEAD_DIM * (g->page / g->group) * 4 <= g->block_bytes,
               "%s: inconsistent block_bytes=%d / scale_off=%d", who, g->block_bytes, g->scale_off);
  return BMXK_OK;
}
static SpectralGeom to_s(const bmxk_spectral_geom* g) {
  SpectralGeom o;
  o.h_kv = g->h_kv, o.page = g->page, o.group = g->group, o.block_bytes = g->block_bytes, o.scale_off = g->scale_off;
  return o;
}

}  // namespace bmxk

using namespace bmxk;

extern "C" {

int bmxk_spectral_append(const bmxk_spectral_geom* g, const void* k_pre, int src_dtype, int64_t stride_seq, int64_t stride_head,
                         int64_t stride_tok, const float* enc, const int32_t* col_bits, const int32_t* col_off,
                         const int32_t* slots, int n_seq, int n_pages, void* pages, void* stream) {
  int rc = check_sgeom(g, "bmxk_spectral_append");
  if (rc) return rc;
  BMXK_REQUIRE(n_seq >= 0 && n_pages >= 0, "bmxk_spectral_append: negative counts");
  if (n_seq == 0 || n_pages == 0) return BMXK_OK;
  BMXK_REQUIRE(k_pre && enc && col_bits && col_off && slots && pages, "bmxk_spectral_append: null pointer");
  const SpectralGeom gg = to_s(g);
  cudaStream_t s = (cudaStream_t)stream;
  uint8_t* dst = (uint8_t*)pages;
  if (src_dtype == BMXK_DTYPE_F16)
    return spectral_append_impl<__half>(gg, k_pre, stride_seq, stride_head, stride_tok, enc, col_bits, col_off, slots, n_seq, n_pages, dst, s);
  if (src_dtype == BMXK_DTYPE_BF16)
    return spectral_append_impl<__nv_bfloat16>(gg, k_pre, stride_seq, stride_head, stride_tok, enc, col_bits, col_off, slots, n_seq, n_pages, dst, s);
  if (src_dtype == BMXK_DTYPE_F32)
    return spectral_append_impl<float>(gg, k_pre, stride_seq, stride_head, stride_tok, enc, col_bits, col_off, slots, n_seq, n_pages, dst, s);
  set_error("bmxk_spectral_append: unknown src_dtype %d", src_dtype);
  return BMXK_ERR_INVALID;
}

int bmxk_spectral_dequant_pages(const bmxk_spectral_geom* g, const void* pages, const float* dec, const int32_t* col_bits,
                                const int32_t* col_off, const int32_t* slots, int n, int8_t* codes, float* scales, float* k_out,
                                void* stream) {
  int rc = check_sgeom(g, "bmxk_spectral_dequant_pages");
  if (rc) return rc;
  BMXK_REQUIRE(n >= 0, "bmxk_spectral_dequant_pages: n < 0");
  if (n == 0) return BMXK_OK;
  BMXK_REQUIRE(pages && col_bits && col_off && slots && (!k_out || dec), "bmxk_spectral_dequant_pages: null pointer");
  static PerDeviceOnce configured;
  if (configured.first()) cudaFuncSetAttribute(spectral_dequant_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
  spectral_dequant_kernel<<<n * g->h_kv, 128, (size_t)g->page * HEAD_DIM * 4, (cudaStream_t)stream>>>(
      to_s(g), (const uint8_t*)pages, dec, col_bits, col_off, slots, codes, scales, k_out);
  return check_launch("bmxk_spectral_dequant_pages");
}

}  // extern "C"
