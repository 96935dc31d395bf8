// Activation / weight quantizers and block-scale packers (HBM-bound, SIMT).
//
// Row quantizers: one CTA of 64 to 256 threads per row, 128-bit loads, the row cached in registers
// (8192 elements at most on the cached path), warp-shuffle + shared-memory reductions, and the
// producer op (GELU table, AdaLN modulation, LayerNorm, RMSNorm, gated residual) fused in front
// of the absmax so the bf16 intermediate never round-trips through HBM.
//
// All divisions and reciprocals that define a stored scale or code use the IEEE-rounded
// intrinsics (__fdiv_rn, __frcp_rn); this file must not be built with fast-math.

#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <type_traits>

#include "rk_blockscale.cuh"
#include "rk_common.cuh"
#include "rk_host.h"

namespace rk {
namespace {

constexpr int kRowThreads = 256;
constexpr int kMaxVec = 4;                              // 8-element vectors cached per thread
constexpr int kCachedK = kRowThreads * kMaxVec * 8;     // 8192

__device__ __forceinline__ float block_reduce(float v, bool is_max, float* scratch) {
  v = is_max ? warp_max(v) : warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();  // scratch may still be read from a previous reduction
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float r = scratch[0];
  for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) r = is_max ? fmaxf(r, scratch[w]) : r + scratch[w];
  return r;
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, bool vec, int valid, float (&v)[8]) {
  if (vec && valid >= 8) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = bf16_bits_to_float(w[i] & 0xFFFFu);
      v[2 * i + 1] = bf16_bits_to_float(w[i] >> 16);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < valid ? __bfloat162float(p[i]) : 0.0f;
  }
}

// eight values that are already bf16-representable (or are to be rounded to nearest even) as one 16-byte store
__device__ __forceinline__ void store8(__nv_bfloat16* p, bool vec, int valid, const float (&v)[8]) {
  if (vec && valid >= 8) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < valid) p[i] = __float2bfloat16_rn(v[i]);
  }
}

// clamp(rint(v / scale)) as an int in [-limit, limit]
__device__ __forceinline__ int quant_code(float v, float scale, float limit) {
  float q = rintf(__fdiv_rn(v, scale));
  q = fminf(fmaxf(q, -limit), limit);
  return __float2int_rn(q);
}

// Writes eight codes starting at element index `idx` of a padded row.
template <int BITS>
__device__ __forceinline__ void store_codes8(uint8_t* qrow, int idx, const int (&c)[8]) {
  if constexpr (BITS == 8) {
    uint2 o;
    o.x = (c[0] & 255) | ((c[1] & 255) << 8) | ((c[2] & 255) << 16) | ((c[3] & 255) << 24);
    o.y = (c[4] & 255) | ((c[5] & 255) << 8) | ((c[6] & 255) << 16) | ((c[7] & 255) << 24);
    *reinterpret_cast<uint2*>(qrow + idx) = o;
  } else {
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) o |= static_cast<uint32_t>(c[i] & 15) << (4 * i);
    *reinterpret_cast<uint32_t*>(qrow + idx / 2) = o;
  }
}

// Eight bf16 values as four packed pairs.
struct Packed8 {
  uint32_t w[4];
};
__device__ __forceinline__ float2 bf16_pair(uint32_t w) { return make_float2(bf16_lo(w), bf16_hi(w)); }
__device__ __forceinline__ float2 splat2(float v) { return make_float2(v, v); }
// the larger magnitude of the two; NaN if either is
__device__ __forceinline__ float absmax_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(fabsf(a)), "f"(fabsf(b)));
  return r;
}

// Eight codes at once, bit-identical to quant_code() on every element but without a division, a
// round instruction and a float -> int conversion per element (those made the row quantizers
// instruction-bound: ~31 instructions per element at 17% of DRAM bandwidth).
//   u = v * rcp, rcp = fl(1 / scale), lies within 3 * 2^-24 * |q| <= 2.3e-5 of the correctly rounded
//   quotient; t = u + 1.5 * 2^23 rounds u to the nearest integer (ties to even) and leaves that
//   integer in the low mantissa bits, so the low byte (nibble) of t IS the two's-complement code.  No
//   clamp: `scale` comes from this row's own maximum, so |q| <= limit * (1 + 2^-22).  Only if some u
//   lies within 4e-5 of a tie (or is not a number, or infinite) could the exact quotient give another
//   code; then all eight take the exact sequence (about one group of eight in a thousand).
// In packed fp32 (two elements an instruction) and with one comparison for the eight: in the norm kernels, with their sums
// and normalisation packed as well, 3264 rows of 2048 with a gated residual went from 17.1 to 15.2 us, 1764 from 9.1 to 8.6.
// Should the compiler make the product and the sum one operation, r differs only where u is near a tie.
// Elements at and beyond `k` must already be zero.
template <int BITS>
__device__ __forceinline__ void quantize_store8(uint8_t* qrow, int idx, const Packed8& p, float scale, float rcp, float limit) {
  const float2 magic = splat2(12582912.0f), minus_magic = splat2(-12582912.0f);  // 1.5 * 2^23, bits 0x4B400000
  const float2 rcp2 = splat2(rcp), minus_one = splat2(-1.0f);
  uint32_t t[8];
  float worst = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // two at a time, each lane rounded as the single operation is
    const float2 u = __fmul2_rn(bf16_pair(p.w[i]), rcp2);
    const float2 r = __fadd2_rn(u, magic);
    const float2 e = __ffma2_rn(__fadd2_rn(r, minus_magic), minus_one, u);  // exact: distance of u from the integer it rounded to
    worst = absmax_nan(absmax_nan(worst, e.x), e.y);
    t[2 * i] = __float_as_uint(r.x), t[2 * i + 1] = __float_as_uint(r.y);
  }
  if (!(worst < 0.49996f)) {
    int c[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      c[2 * i] = quant_code(bf16_lo(p.w[i]), scale, limit);
      c[2 * i + 1] = quant_code(bf16_hi(p.w[i]), scale, limit);
    }
    store_codes8<BITS>(qrow, idx, c);
    return;
  }
  // low bytes of t gathered four to a word
  const uint32_t lo = __byte_perm(__byte_perm(t[0], t[1], 0x0040u), __byte_perm(t[2], t[3], 0x0040u), 0x5410u);
  const uint32_t hi = __byte_perm(__byte_perm(t[4], t[5], 0x0040u), __byte_perm(t[6], t[7], 0x0040u), 0x5410u);
  if constexpr (BITS == 8) {
    *reinterpret_cast<uint2*>(qrow + idx) = make_uint2(lo, hi);
  } else {
    // bytes b0 b1 b2 b3 -> (b0 & 15) | (b1 & 15) << 4 | ...: fold the odd byte of each pair onto the even one
    const uint32_t l = lo & 0x0F0F0F0Fu, h = hi & 0x0F0F0F0Fu;
    const uint32_t lf = l | (l >> 4), hf = h | (h >> 4);
    *reinterpret_cast<uint32_t*>(qrow + idx / 2) = __byte_perm(lf, hf, 0x6420u);
  }
}

__device__ __forceinline__ float row_scale_from_max(float maximum, float limit, bool true_division) {
  if (!(maximum > 0.0f)) return 1.0f;
  // activations: max * fl32(1/limit); weights: max / limit
  return true_division ? __fdiv_rn(maximum, limit) : __fmul_rn(maximum, static_cast<float>(1.0 / limit));
}

// ---- rows held as packed bf16 pairs -----------------------------------------------------------------
// A thread keeps VEC vectors of eight bf16 values as four 32-bit words each.  Products and sums of two
// bf16 values are taken two at a time in bf16 arithmetic: one rounding of the exact result.  That is
// what rounding the fp32 result to bf16 gives too - 24 >= 2 * 8 + 2 bits make the second rounding
// innocuous - except for products below the normal range, where one rounding is the closer one.
// The row kernels are bound by instructions per element (36 -> about 17 for the modulated norm), not by
// bytes: see the launch rule below for the figures.
// The narrow shapes are picked for many rows: 768 resident threads per SM (1764 rows of 64 threads in one wave).
constexpr int row_min_blocks(int threads, int vecs) { return threads < kRowThreads && threads * vecs >= 256 ? 768 / threads : 1; }
// eight bf16 values; those at and beyond `valid` read as zero
__device__ __forceinline__ Packed8 load8p(const __nv_bfloat16* p, bool vec, int valid) {
  Packed8 r;
  if (vec && valid >= 8) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    r.w[0] = u.x, r.w[1] = u.y, r.w[2] = u.z, r.w[3] = u.w;
  } else {
    const unsigned short* s = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t lo = 2 * i < valid ? s[2 * i] : 0u, hi = 2 * i + 1 < valid ? s[2 * i + 1] : 0u;
      r.w[i] = lo | (hi << 16);
    }
  }
  return r;
}
__device__ __forceinline__ void store8p(__nv_bfloat16* p, bool vec, int valid, const Packed8& v) {
  if (vec && valid >= 8) {
    *reinterpret_cast<uint4*>(p) = make_uint4(v.w[0], v.w[1], v.w[2], v.w[3]);
  } else {
    unsigned short* s = reinterpret_cast<unsigned short*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < valid) s[i] = static_cast<unsigned short>(v.w[i >> 1] >> (16 * (i & 1)));
  }
}
// zeroes the elements at and beyond `valid`
__device__ __forceinline__ void mask8(Packed8& p, int valid) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (2 * i >= valid) p.w[i] = 0u;
    else if (2 * i + 1 >= valid) p.w[i] &= 0xFFFFu;
  }
}

// Row sum over a CTA of THREADS threads in the summation order of a 256-thread CTA (thread t of that CTA
// adds its elements, a warp's lanes are added by shuffles, the eight warps in order), so that the number
// of threads a launch picks never changes a result.  Vector j of thread t is vector j * THREADS + t of the
// row, i.e. it belongs to accumulator j % (256 / THREADS).  `scratch`: eight words, not reused.
template <int THREADS>
__device__ __forceinline__ float row_sum256(float (&acc)[kRowThreads / THREADS], float* scratch) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < kRowThreads / THREADS; ++r) {
    const float s = warp_sum(acc[r]);
    if (lane == 0) scratch[r * (THREADS / 32) + warp] = s;
  }
  __syncthreads();
  float total = scratch[0];
#pragma unroll
  for (int w = 1; w < kRowThreads / 32; ++w) total += scratch[w];
  return total;
}

// A thread's part of a row sum for row_sum256: adds the elements `get(vector, pair)` (or their squares) of its VEC vectors in
// order, vector j to accumulator j % R.  Two accumulators at a time in packed fp32 where there are two: the same sums, rounded
// identically.
template <bool SQUARES, int VEC, int R, typename Get>
__device__ __forceinline__ void add_vectors(Get get, float (&acc)[R]) {
  if constexpr (R >= 2 && VEC >= 2) {
    float2 acc2[R / 2];
#pragma unroll
    for (int r = 0; r < R / 2; ++r) acc2[r] = splat2(0.0f);
#pragma unroll
    for (int it = 0; it < VEC; it += 2) {
      float2& a = acc2[(it % R) / 2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f0 = get(it, i), f1 = get(it + 1, i);
        const float2 lo = make_float2(f0.x, f1.x), hi = make_float2(f0.y, f1.y);
        a = SQUARES ? __ffma2_rn(lo, lo, a) : __fadd2_rn(a, lo);
        a = SQUARES ? __ffma2_rn(hi, hi, a) : __fadd2_rn(a, hi);
      }
    }
#pragma unroll
    for (int r = 0; r < R / 2; ++r) acc[2 * r] = acc2[r].x, acc[2 * r + 1] = acc2[r].y;
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0f;
#pragma unroll
    for (int it = 0; it < VEC; ++it)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = get(it, i);
        float& a = acc[it % R];
        a = SQUARES ? __fmaf_rn(f.x, f.x, a) : a + f.x;
        a = SQUARES ? __fmaf_rn(f.y, f.y, a) : a + f.y;
      }
  }
}

// Common tail: absmax over the cached values, scale, quantize, store (zero padding to kpad).  `threads`: the CTA size.
template <int BITS, int VEC>
__device__ __forceinline__ void finish_row(Packed8 (&vals)[VEC], int threads, int k, int kpad, uint8_t* qrow, float* scale_out,
                                           bool true_division, float* scratch) {
  const float limit = static_cast<float>((1 << (BITS - 1)) - 1);
  uint32_t m = 0u;
#pragma unroll
  for (int it = 0; it < VEC; ++it) {
    const int idx = (it * threads + static_cast<int>(threadIdx.x)) * 8;
    if (idx + 8 > k) mask8(vals[it], k - idx);  // ragged end of the row: codes beyond k are zero
#pragma unroll
    for (int i = 0; i < 4; ++i) m = absmax_bf16x2(m, vals[it].w[i]);
  }
  const float local = warp_max(fmaxf(bf16_lo(m), bf16_hi(m)));
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = local;
  __syncthreads();
  float maximum = scratch[0];
  for (int w = 1; w < (threads >> 5); ++w) maximum = fmaxf(maximum, scratch[w]);
  const float scale = row_scale_from_max(maximum, limit, true_division);
  if (threadIdx.x == 0) *scale_out = scale;
  const float rcp = __frcp_rn(scale);
#pragma unroll
  for (int it = 0; it < VEC; ++it) {
    const int idx = (it * threads + static_cast<int>(threadIdx.x)) * 8;
    if (idx < kpad) quantize_store8<BITS>(qrow, idx, vals[it], scale, rcp, limit);
  }
}

// ------------------------------------------------------------------ plain / GELU-table rows
// VEC vectors of eight elements per thread; rows longer than blockDim.x * VEC vectors (VEC == 4 only) take two passes
template <int BITS, int MODE, int VEC>
__global__ void __launch_bounds__(kRowThreads)
quant_rows_kernel(const __nv_bfloat16* __restrict__ x, long long x_stride, const __nv_bfloat16* __restrict__ up,
                  long long up_stride, const __nv_bfloat16* __restrict__ lut, int k, int kpad, int n_rows,
                  uint8_t* __restrict__ q, float* __restrict__ scales, int true_division, int vec_ok) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  __shared__ float scratch[kRowThreads / 32];
  const int row = blockIdx.x;
  const int qbytes = BITS == 8 ? kpad : kpad / 2;
  uint8_t* qrow = q + static_cast<long long>(row) * qbytes;
  if (row >= n_rows) {  // padding row of a weight matrix: zero codes, unit scale
    for (int i = threadIdx.x * 4; i < qbytes; i += static_cast<int>(blockDim.x) * 4) *reinterpret_cast<uint32_t*>(qrow + i) = 0;
    if (threadIdx.x == 0) scales[row] = 1.0f;
    return;
  }
  const __nv_bfloat16* xr = x + row * x_stride;
  const __nv_bfloat16* ur = MODE == RK_ACT_LUT_MUL ? up + row * up_stride : nullptr;
  const unsigned short* table = reinterpret_cast<const unsigned short*>(lut);
  auto activate = [&](Packed8& v, const Packed8& u) {
    if constexpr (MODE != RK_ACT_PLAIN) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v.w[i] = static_cast<uint32_t>(__ldg(table + (v.w[i] & 0xFFFFu))) | (static_cast<uint32_t>(__ldg(table + (v.w[i] >> 16))) << 16);
        if constexpr (MODE == RK_ACT_LUT_MUL) v.w[i] = mul_bf16x2(v.w[i], u.w[i]);
      }
    }
  };
  const int threads = static_cast<int>(blockDim.x);  // 64, 128 or 256: see row_threads
  if (VEC < kMaxVec || k <= threads * VEC * 8) {
    Packed8 vals[VEC], ups[MODE == RK_ACT_LUT_MUL ? VEC : 1];
#pragma unroll
    for (int it = 0; it < VEC; ++it) {  // all loads first: they overlap
      const int idx = (it * threads + threadIdx.x) * 8;
      vals[it] = load8p(xr + idx, vec_ok, k - idx);
      if constexpr (MODE == RK_ACT_LUT_MUL) ups[it] = load8p(ur + idx, vec_ok, k - idx);
    }
#pragma unroll
    for (int it = 0; it < VEC; ++it) {
      const int idx = (it * threads + threadIdx.x) * 8;
      if (MODE != RK_ACT_PLAIN && idx < k) activate(vals[it], ups[MODE == RK_ACT_LUT_MUL ? it : 0]);
    }
    finish_row<BITS, VEC>(vals, threads, k, kpad, qrow, scales + row, true_division != 0, scratch);
  } else {
    // long rows: two passes over global memory (the second one hits L2)
    auto values_at = [&](int idx) {
      Packed8 v = load8p(xr + idx, vec_ok, k - idx), u{};
      if constexpr (MODE == RK_ACT_LUT_MUL) u = load8p(ur + idx, vec_ok, k - idx);
      activate(v, u);
      if (idx + 8 > k) mask8(v, k - idx);
      return v;
    };
    const float limit = static_cast<float>((1 << (BITS - 1)) - 1);
    uint32_t m = 0u;
    for (int idx = threadIdx.x * 8; idx < k; idx += threads * 8) {
      const Packed8 v = values_at(idx);
#pragma unroll
      for (int i = 0; i < 4; ++i) m = absmax_bf16x2(m, v.w[i]);
    }
    const float maximum = block_reduce(fmaxf(bf16_lo(m), bf16_hi(m)), true, scratch);
    const float scale = row_scale_from_max(maximum, limit, true_division != 0);
    if (threadIdx.x == 0) scales[row] = scale;
    const float rcp = __frcp_rn(scale);
    for (int idx = threadIdx.x * 8; idx < kpad; idx += threads * 8) {
      Packed8 v{};
      if (idx < k) v = values_at(idx);
      quantize_store8<BITS>(qrow, idx, v, scale, rcp, limit);
    }
  }
}

// ------------------------------------------------------------------ table activations with the table on chip
// A gather of 32 random entries of the 128 KB table takes an SM's L1 about 20 cycles (one tag look-up per line) and
// bounds the kernels above once there is enough work; from shared memory it takes three or four (bank conflicts
// only).  So for large tensors one CTA of 1024 threads per SM copies the whole table first and then walks the rows.
constexpr int kTableThreads = 1024;
constexpr int kTableBytes = 65536 * 2;
// Elements from which the table pays (long rows leave the L1 form few CTAs).  Measured, table in L1 against on chip - row
// quantizer: 300 x 8192 8.1 -> 6.9 us, 1764 x 8192 17.9 -> 15.0, 196 x 8192 7.7 -> 7.0, 100 x 8192 5.4 -> 6.7, 1764 x 2048
// 8.6 -> 6.9, 1300 x 2048 7.9 -> 6.7, 1000 x 2048 6.4 -> 6.8; product and maximum: 400 x 4096 5.2 -> 4.3, 816 x 2048
// 5.1 -> 4.3, 1764 x 2048 7.4 -> 5.3, 400 x 1024 3.6 -> 3.6, 50 x 4096 3.1 -> 3.6.
constexpr int64_t kTableRowsLine = 2400000, kTableLongRowsLine = 1300000;  // k up to 4096, beyond
constexpr int64_t kTableProductLine = 1ll << 20;

// every thread of the CTA: starts copying the table (eight 16-byte pieces each); table_arrive() completes it
__device__ __forceinline__ void table_copy(const __nv_bfloat16* lut, uint8_t* smem) {
  const uint32_t dst = smem_u32(smem);
#pragma unroll
  for (int i = 0; i < kTableBytes / 16 / kTableThreads; ++i) {
    const uint32_t off = (i * kTableThreads + threadIdx.x) * 16;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + off), "l"(reinterpret_cast<const uint8_t*>(lut) + off)
                 : "memory");
  }
}
__device__ __forceinline__ void table_arrive() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}
__device__ __forceinline__ uint32_t table_pair(const unsigned short* table, uint32_t w) {
  return static_cast<uint32_t>(table[w & 0xFFFFu]) | (static_cast<uint32_t>(table[w >> 16]) << 16);
}

// GROUP threads per row, four vectors of eight each (k <= GROUP * 32): the CTA holds 1024 / GROUP rows at a time and every
// group walks on by itself (named barriers).  Values, codes and scales are those of quant_rows_kernel.
template <int BITS, int MODE, int GROUP>
__global__ void __launch_bounds__(kTableThreads, 1)
quant_rows_table_kernel(const __nv_bfloat16* __restrict__ x, long long x_stride, const __nv_bfloat16* __restrict__ up,
                        long long up_stride, const __nv_bfloat16* __restrict__ lut, int k, int kpad, int n_rows,
                        uint8_t* __restrict__ q, float* __restrict__ scales, int vec_ok) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  extern __shared__ __align__(16) uint8_t smem_table[];
  __shared__ float scratch[kTableThreads / 32];
  table_copy(lut, smem_table);
  const unsigned short* const table = reinterpret_cast<const unsigned short*>(smem_table);
  constexpr int kGroups = kTableThreads / GROUP, kWarps = GROUP / 32;
  // One named barrier per group.  A CTA has sixteen, 0 to 15, and GROUP = 64 needs them all: group 0 takes barrier 0, which is
  // free again because its only other use, table_arrive(), lies before the first group_sync() of every thread.
  static_assert(kGroups <= 16, "a CTA has sixteen named barriers");
  const int group = threadIdx.x / GROUP, t = threadIdx.x % GROUP;
  float* const part = scratch + group * kWarps;
  auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(group), "n"(GROUP) : "memory"); };
  const float limit = static_cast<float>((1 << (BITS - 1)) - 1);
  bool first = true;
  for (int row0 = blockIdx.x * kGroups; row0 < n_rows; row0 += gridDim.x * kGroups) {  // uniform over the CTA
    const int row = row0 + group;
    const bool live = row < n_rows;
    Packed8 v[kMaxVec], u[MODE == RK_ACT_LUT_MUL ? kMaxVec : 1];
#pragma unroll
    for (int it = 0; it < kMaxVec; ++it) {
      const int idx = (it * GROUP + t) * 8, valid = live ? k - idx : 0;
      v[it] = load8p(x + row * x_stride + idx, vec_ok, valid);
      if constexpr (MODE == RK_ACT_LUT_MUL) u[it] = load8p(up + row * up_stride + idx, vec_ok, valid);
    }
    if (first) table_arrive();  // the first rows are on their way meanwhile
    first = false;
    if (!live) continue;
    uint32_t m = 0u;
#pragma unroll
    for (int it = 0; it < kMaxVec; ++it) {
      const int idx = (it * GROUP + t) * 8;
      if (idx >= k) continue;  // zeros stay zeros, whatever the table says
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[it].w[i] = table_pair(table, v[it].w[i]);
        if constexpr (MODE == RK_ACT_LUT_MUL) v[it].w[i] = mul_bf16x2(v[it].w[i], u[it].w[i]);
      }
      if (idx + 8 > k) mask8(v[it], k - idx);
#pragma unroll
      for (int i = 0; i < 4; ++i) m = absmax_bf16x2(m, v[it].w[i]);
    }
    const float local = warp_max(fmaxf(bf16_lo(m), bf16_hi(m)));
    group_sync();  // the previous row's maxima have been read
    if ((t & 31) == 0) part[t >> 5] = local;
    group_sync();
    float maximum = part[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) maximum = fmaxf(maximum, part[w]);
    const float scale = row_scale_from_max(maximum, limit, false);
    if (t == 0) scales[row] = scale;
    const float rcp = __frcp_rn(scale);
    uint8_t* const qrow = q + static_cast<long long>(row) * (BITS == 8 ? kpad : kpad / 2);
#pragma unroll
    for (int it = 0; it < kMaxVec; ++it) {
      const int idx = (it * GROUP + t) * 8;
      if (idx < kpad) quantize_store8<BITS>(qrow, idx, v[it], scale, rcp, limit);
    }
  }
}

// ------------------------------------------------------------------ table activation * up -> bf16 + tensor amax
// out = bf16(table[x] * up) element by element (the arithmetic of the GELU-table mode of the row
// quantizer above) and the absolute maximum of the finite results, for a per-tensor scale that a
// block packer needs before it can run.  Eight elements per thread and step; rows may be strided.
// ON_CHIP: 1024 threads per CTA, the table in shared memory (see quant_rows_table_kernel); else 256 threads, the table
// gathered through L1.
template <bool ON_CHIP>
__global__ void __launch_bounds__(ON_CHIP ? kTableThreads : 256, 1)
lut_mul_amax_kernel(const __nv_bfloat16* __restrict__ x, long long x_stride, const __nv_bfloat16* __restrict__ up,
                    long long up_stride, const __nv_bfloat16* __restrict__ lut, long long rows, int k,
                    __nv_bfloat16* __restrict__ out, unsigned* __restrict__ staging) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  constexpr int kUnroll = 2;
  extern __shared__ __align__(16) uint8_t smem_table[];
  __shared__ uint32_t scratch[kTableThreads / 32];
  const unsigned short* table = reinterpret_cast<const unsigned short*>(lut);
  if constexpr (ON_CHIP) {
    table_copy(lut, smem_table);
    table = reinterpret_cast<const unsigned short*>(smem_table);
  }
  const int per_row = k >> 3;
  const long long total = rows * per_row;
  const bool short_index = total < (1ll << 32);  // a 64-bit division costs as much as four gathers
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  uint32_t m = 0u;
  bool first = true;
  // the trip count is the same for every thread of the CTA: the first trip holds a barrier
  for (long long base = static_cast<long long>(blockIdx.x) * blockDim.x; base < total; base += kUnroll * step) {
    uint4 xv[kUnroll], uv[kUnroll];
    long long dst[kUnroll];
#pragma unroll
    for (int j = 0; j < kUnroll; ++j) {
      const long long i = base + j * step + threadIdx.x;
      dst[j] = -1;
      if (i < total) {
        const long long row = short_index ? static_cast<unsigned>(i) / static_cast<unsigned>(per_row) : i / per_row;
        const int col = static_cast<int>(i - row * per_row) << 3;
        xv[j] = *reinterpret_cast<const uint4*>(x + row * x_stride + col);
        uv[j] = *reinterpret_cast<const uint4*>(up + row * up_stride + col);
        dst[j] = row * k + col;
      }
    }
    if (ON_CHIP && first) table_arrive();
    first = false;
#pragma unroll
    for (int j = 0; j < kUnroll; ++j) {
      if (dst[j] < 0) continue;
      uint32_t w[4] = {xv[j].x, xv[j].y, xv[j].z, xv[j].w};
      const uint32_t u[4] = {uv[j].x, uv[j].y, uv[j].z, uv[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        w[i] = mul_bf16x2(table_pair(table, w[i]), u[i]);
        // magnitudes order like their bit patterns; infinities and NaN count as zero
        const uint32_t lo = w[i] & 0x7FFFu, hi = (w[i] >> 16) & 0x7FFFu;
        m = max(m, lo < 0x7F80u ? lo : 0u);
        m = max(m, hi < 0x7F80u ? hi : 0u);
      }
      *reinterpret_cast<uint4*>(out + dst[j]) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  if (staging != nullptr) {
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
      m = threadIdx.x < (blockDim.x >> 5) ? scratch[threadIdx.x] : 0u;
      m = __reduce_max_sync(0xffffffffu, m);
      if (threadIdx.x == 0 && m != 0u) atomicMax(staging, m << 16);  // the float of those upper bits
    }
  }
}

// ------------------------------------------------------------------ AdaLN modulation (+LayerNorm, +gated residual)
// The modulation vectors are requested before the statistics are reduced, so that their latency hides behind it.
template <int BITS, int THREADS, int VEC>
__global__ void __launch_bounds__(THREADS, row_min_blocks(THREADS, VEC))
quant_rows_modulated_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ mod_scale,
                            const __nv_bfloat16* __restrict__ mod_shift, int k, int kpad, int tokens, int layer_norm,
                            float eps, const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ gate,
                            __nv_bfloat16* __restrict__ residual_out, uint8_t* __restrict__ q,
                            float* __restrict__ scales) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  constexpr int R = kRowThreads / THREADS;
  __shared__ float scratch[3][kRowThreads / 32];
  const int row = blockIdx.x;
  const long long xoff = static_cast<long long>(row) * k;
  const long long moff = static_cast<long long>(row / tokens) * k;
  uint8_t* qrow = q + static_cast<long long>(row) * (BITS == 8 ? kpad : kpad / 2);
  const bool vec = (k % 8) == 0;
  Packed8 vals[VEC];
  if (y != nullptr) {
    Packed8 yv[VEC], gv[VEC];
#pragma unroll
    for (int it = 0; it < VEC; ++it) {
      const int idx = (it * THREADS + threadIdx.x) * 8;
      vals[it] = load8p(x + xoff + idx, vec, k - idx);
      yv[it] = load8p(y + xoff + idx, vec, k - idx);
      gv[it] = load8p(gate + moff + idx, vec, k - idx);
    }
#pragma unroll
    for (int it = 0; it < VEC; ++it) {
      const int idx = (it * THREADS + threadIdx.x) * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i)  // residual = bf16(x + bf16(y * gate))
        vals[it].w[i] = add_bf16x2(vals[it].w[i], mul_bf16x2(yv[it].w[i], gv[it].w[i]));
      if (idx < k) store8p(residual_out + xoff + idx, vec, k - idx, vals[it]);
    }
  } else {
#pragma unroll
    for (int it = 0; it < VEC; ++it) {
      const int idx = (it * THREADS + threadIdx.x) * 8;
      vals[it] = load8p(x + xoff + idx, vec, k - idx);
    }
  }
  Packed8 sc[VEC], sh[VEC];
#pragma unroll
  for (int it = 0; it < VEC; ++it) {
    const int idx = (it * THREADS + threadIdx.x) * 8;
    sc[it] = load8p(mod_scale + moff + idx, vec, k - idx);
    sh[it] = load8p(mod_shift + moff + idx, vec, k - idx);
  }
  if (layer_norm) {
    // The centred values in fp32 stay in registers for rows of up to 2048 elements; beyond, 32 registers more than the launch
    // has cost more than computing them twice (3264 x 4096 with a gated residual 20.8 -> 21.9 us).
    constexpr bool kHold = THREADS * VEC <= 256;
    float2 f[kHold ? VEC : 1][4];
    float acc[R];
    add_vectors<false, VEC, R>([&](int it, int i) { return bf16_pair(vals[it].w[i]); }, acc);  // elements beyond k are zero
    const float mean = __fdiv_rn(row_sum256<THREADS>(acc, scratch[0]), static_cast<float>(k));
    const float2 minus_mean = splat2(-mean);
    auto centred = [&](int it, int i) {
      float2 c = __fadd2_rn(bf16_pair(vals[it].w[i]), minus_mean);
      const int at = (it * THREADS + static_cast<int>(threadIdx.x)) * 8 + 2 * i;  // what lies beyond k adds nothing
      if (at >= k) c.x = 0.0f;
      if (at + 1 >= k) c.y = 0.0f;
      return c;
    };
    if constexpr (kHold) {
#pragma unroll
      for (int it = 0; it < VEC; ++it) {
        const int idx = (it * THREADS + threadIdx.x) * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) f[it][i] = __fadd2_rn(bf16_pair(vals[it].w[i]), minus_mean);
        if (idx + 8 > k) {  // ragged end
#pragma unroll
          for (int i = 0; i < 4; ++i) f[it][i] = centred(it, i);
        }
      }
    }
    auto value = [&](int it, int i) {
      if constexpr (kHold) return f[it][i];
      else return centred(it, i);
    };
    add_vectors<true, VEC, R>(value, acc);
    const float var = __fdiv_rn(row_sum256<THREADS>(acc, scratch[1]), static_cast<float>(k));
    const float2 inv = splat2(rsqrtf(var + eps));
#pragma unroll
    for (int it = 0; it < VEC; ++it)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 n = __fmul2_rn(value(it, i), inv);
        vals[it].w[i] = pack_bf16x2(n.x, n.y);
      }
  }
#pragma unroll
  for (int it = 0; it < VEC; ++it)
#pragma unroll
    for (int i = 0; i < 4; ++i)  // bf16(bf16(x * bf16(1 + scale)) + shift)
      vals[it].w[i] = add_bf16x2(mul_bf16x2(vals[it].w[i], add_bf16x2(0x3F803F80u, sc[it].w[i])), sh[it].w[i]);
  finish_row<BITS, VEC>(vals, THREADS, k, kpad, qrow, scales + row, false, scratch[2]);
}

// ------------------------------------------------------------------ RMSNorm (Gemma) -> quantize
// n = bf16( fl(fl(s * inv) * fl(1 + a)) + b ), inv = rsqrt(mean(s^2) + eps);
//   plain:    a = weight[k], b absent;  adaptive: a = scale[row / tokens, k], b = shift[row / tokens, k].
template <int BITS, int THREADS, int VEC>
__global__ void __launch_bounds__(THREADS, row_min_blocks(THREADS, VEC))
rmsnorm_quant_rows_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                          const __nv_bfloat16* __restrict__ gate,
                          const __nv_bfloat16* __restrict__ a_ptr, const __nv_bfloat16* __restrict__ b_ptr,
                          int tokens, int k, int kpad, float eps, __nv_bfloat16* __restrict__ sum_out,
                          __nv_bfloat16* __restrict__ norm_out, uint8_t* __restrict__ q, float* __restrict__ scales) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  constexpr int R = kRowThreads / THREADS;
  __shared__ float scratch[2][kRowThreads / 32];
  const int row = blockIdx.x;
  const long long xoff = static_cast<long long>(row) * k;
  const long long aoff = tokens > 0 ? static_cast<long long>(row / tokens) * k : 0;
  uint8_t* qrow = BITS == 16 ? q : q + static_cast<long long>(row) * (BITS == 8 ? kpad : kpad / 2);
  const bool vec = (k % 8) == 0;
  Packed8 vals[VEC];
#pragma unroll
  for (int it = 0; it < VEC; ++it) {
    const int idx = (it * THREADS + threadIdx.x) * 8;
    vals[it] = load8p(x + xoff + idx, vec, k - idx);
  }
  if (residual != nullptr) {
    Packed8 rv[VEC];
#pragma unroll
    for (int it = 0; it < VEC; ++it) {
      const int idx = (it * THREADS + threadIdx.x) * 8;
      rv[it] = load8p(residual + xoff + idx, vec, k - idx);
    }
    if (gate != nullptr) {  // gated residual: the branch is scaled per (batch entry, channel) first
#pragma unroll
      for (int it = 0; it < VEC; ++it) {
        const int idx = (it * THREADS + threadIdx.x) * 8;
        const Packed8 gv = load8p(gate + aoff + idx, vec, k - idx);
#pragma unroll
        for (int i = 0; i < 4; ++i) rv[it].w[i] = mul_bf16x2(rv[it].w[i], gv.w[i]);
      }
    }
#pragma unroll
    for (int it = 0; it < VEC; ++it)
#pragma unroll
      for (int i = 0; i < 4; ++i) vals[it].w[i] = add_bf16x2(vals[it].w[i], rv[it].w[i]);
  }
  Packed8 av[VEC], bv[VEC];
#pragma unroll
  for (int it = 0; it < VEC; ++it) {
    const int idx = (it * THREADS + threadIdx.x) * 8;
    av[it] = load8p(a_ptr + aoff + idx, vec, k - idx);
    if (b_ptr != nullptr) bv[it] = load8p(b_ptr + aoff + idx, vec, k - idx);
  }
  // fp32 values held in registers, or (with a bf16 result, whose norm keeps more) unpacked again: 16384 x 2048 38.5 -> 39.9 us held
  constexpr bool kHold = BITS != 16;
  float2 f[kHold ? VEC : 1][4];
  auto value = [&](int it, int i) {
    if constexpr (kHold) return f[it][i];
    else return bf16_pair(vals[it].w[i]);
  };
#pragma unroll
  for (int it = 0; it < VEC; ++it) {
    const int idx = (it * THREADS + threadIdx.x) * 8;
    if (sum_out != nullptr && idx < k) store8p(sum_out + xoff + idx, vec, k - idx, vals[it]);
    if constexpr (kHold) {
#pragma unroll
      for (int i = 0; i < 4; ++i) f[it][i] = bf16_pair(vals[it].w[i]);  // elements beyond k are zero
    }
  }
  float acc[R];
  add_vectors<true, VEC, R>(value, acc);
  const float var = __fdiv_rn(row_sum256<THREADS>(acc, scratch[0]), static_cast<float>(k));
  const float2 inv = splat2(rsqrtf(var + eps)), one = splat2(1.0f);
  uint32_t m = 0u;
#pragma unroll
  for (int it = 0; it < VEC; ++it) {
    const int idx = (it * THREADS + threadIdx.x) * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 n = __fmul2_rn(value(it, i), inv), w = __fadd2_rn(one, bf16_pair(av[it].w[i]));
      float t0 = __fmul_rn(n.x, w.x), t1 = __fmul_rn(n.y, w.y);  // not packed: a packed product and sum may be made one operation
      if (b_ptr != nullptr) {
        t0 = __fadd_rn(t0, bf16_lo(bv[it].w[i]));
        t1 = __fadd_rn(t1, bf16_hi(bv[it].w[i]));
      }
      vals[it].w[i] = pack_bf16x2(t0, t1);
    }
    if (idx + 8 > k) mask8(vals[it], k - idx);
    if (norm_out != nullptr && idx < k) store8p(norm_out + xoff + idx, vec, k - idx, vals[it]);
  }
  if constexpr (BITS == 16) {
    // no row quantizer: the bf16 result is the output (norm_out) and the tensor's absolute maximum
    // (finite values only) is collected for a per-tensor scale; `q` is that staging word, or null
    if (q != nullptr) {
#pragma unroll
      for (int it = 0; it < VEC; ++it)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // magnitudes order like their bit patterns; infinities and NaN count as zero
          const uint32_t lo = vals[it].w[i] & 0x7FFFu, hi = (vals[it].w[i] >> 16) & 0x7FFFu;
          m = max(m, lo < 0x7F80u ? lo : 0u);
          m = max(m, hi < 0x7F80u ? hi : 0u);
        }
      m = __reduce_max_sync(0xffffffffu, m);
      if ((threadIdx.x & 31) == 0) scratch[1][threadIdx.x >> 5] = __uint_as_float(m << 16);
      __syncthreads();
      if (threadIdx.x == 0) {
        float row_max = scratch[1][0];
        for (int w = 1; w < THREADS / 32; ++w) row_max = fmaxf(row_max, scratch[1][w]);
        atomicMax(reinterpret_cast<unsigned*>(q), __float_as_uint(row_max));
      }
    }
  } else {
    finish_row<BITS, VEC>(vals, THREADS, k, kpad, qrow, scales + row, false, scratch[1]);
  }
}

// ------------------------------------------------------------------ W4 group-128 weight packer
// One warp per (row, group of 128): four consecutive elements per lane.
__global__ void __launch_bounds__(256)
pack_w4_g128_kernel(const __nv_bfloat16* __restrict__ w, int n, int k, uint8_t* __restrict__ q,
                    __nv_bfloat16* __restrict__ scales) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const int groups = k / 128;
  const long long gw = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= static_cast<long long>(n) * groups) return;
  const int row = static_cast<int>(gw / groups);
  const int g = static_cast<int>(gw % groups);
  const __nv_bfloat16* src = w + static_cast<long long>(row) * k + g * 128 + lane * 4;
  const uint2 u = *reinterpret_cast<const uint2*>(src);
  float v[4] = {bf16_bits_to_float(u.x & 0xFFFFu), bf16_bits_to_float(u.x >> 16), bf16_bits_to_float(u.y & 0xFFFFu),
                bf16_bits_to_float(u.y >> 16)};
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  amax = warp_max(amax);
  // s = bf16(amax / 7) (1.0 for an all-zero group); codes use float(s)
  __nv_bfloat16 sb = __float2bfloat16_rn(amax > 0.0f ? __fdiv_rn(amax, 7.0f) : 1.0f);
  if (!(__bfloat162float(sb) > 0.0f)) sb = __float2bfloat16_rn(1.0f);  // amax / 7 flushed to zero in bf16
  const float s = __bfloat162float(sb);
  if (lane == 0) scales[static_cast<long long>(g) * n + row] = sb;
  // Eight consecutive weights k0..k7 share one 32-bit word whose byte b holds k_b in its low nibble
  // and k_{b+4} in its high nibble (the order the GEMM's expansion step consumes cheapest).  An
  // even lane owns k0..k3, its odd neighbour k4..k7.
  uint32_t spread = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) spread |= static_cast<uint32_t>(quant_code(v[i], s, 7.0f) & 15) << (8 * i);
  const uint32_t upper = __shfl_xor_sync(0xffffffffu, spread, 1);
  if (!(lane & 1))
    *reinterpret_cast<uint32_t*>(q + static_cast<long long>(row) * (k / 2) + g * 64 + (lane >> 1) * 4) =
        spread | (upper << 4);
}

// ------------------------------------------------------------------ per-tensor FP8
__global__ void __launch_bounds__(256)
amax_finite_kernel(const __nv_bfloat16* __restrict__ x, long long elements, unsigned* __restrict__ amax_bits) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  __shared__ float scratch[8];
  float local = 0.0f;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x * 8;
  for (long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8; idx < elements;
       idx += stride) {
    float v[8];
    const long long left = elements - idx;
    load8(x + idx, true, left >= 8 ? 8 : static_cast<int>(left), v);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float a = fabsf(v[i]);
      if (a <= 3.4028234664e38f) local = fmaxf(local, a);  // skips inf and NaN
    }
  }
  local = warp_max(local);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    float r = scratch[0];
    for (int w = 1; w < 8; ++w) r = fmaxf(r, scratch[w]);
    atomicMax(amax_bits, __float_as_uint(r));  // non-negative floats order like their bit patterns
  }
}

// scale = max(amax / divisor, 1e-12); also clears the staging word for the next call
__global__ void finalize_scale_kernel(unsigned* amax_bits, float divisor, float* scale_out) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const float amax = __uint_as_float(*amax_bits);
  *scale_out = fmaxf(__fdiv_rn(amax, divisor), 1e-12f);
  *amax_bits = 0u;
}

// eight e4m3 codes of clamp(v * inverse, +-448), two conversions per instruction (a NaN becomes -448, as fmaxf leaves it)
__device__ __forceinline__ uint2 to_fp8x8(const float (&v)[8], float inverse) {
  uint32_t c[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float lo = fminf(448.0f, fmaxf(-448.0f, __fmul_rn(v[2 * i], inverse)));
    const float hi = fminf(448.0f, fmaxf(-448.0f, __fmul_rn(v[2 * i + 1], inverse)));
    c[i] = __nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
  }
  return make_uint2(c[0] | (c[1] << 16), c[2] | (c[3] << 16));
}

// the first `count` (below eight) of eight codes
__device__ __forceinline__ void store_codes(uint8_t* q, uint2 codes, int count) {
#pragma unroll
  for (int i = 0; i < 7; ++i)
    if (i < count) q[i] = static_cast<uint8_t>((i < 4 ? codes.x : codes.y) >> (8 * (i & 3)));
}

// Sixteen elements per thread and step: two 16-byte loads in flight, one 16-byte store (maximum and conversion of
// 816 x 32768: 26.6 -> 20.1 us against eight elements and scalar conversions).
__global__ void __launch_bounds__(256)
to_fp8_kernel(const __nv_bfloat16* __restrict__ x, long long elements, const float* __restrict__ scale,
              uint8_t* __restrict__ q, int q16) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const float inverse = __fdiv_rn(1.0f, *scale);
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x * 16;
  for (long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 16; idx < elements;
       idx += stride) {
    const long long left = elements - idx;
    const int valid = left >= 16 ? 16 : static_cast<int>(left);
    float v[8], w[8];
    load8(x + idx, true, valid, v);
    load8(x + idx + 8, true, valid - 8, w);
    const uint2 a = to_fp8x8(v, inverse), b = to_fp8x8(w, inverse);
    if (valid == 16 && q16) {  // `q16`: the codes are 16-byte aligned; else they are 8-byte aligned
      *reinterpret_cast<uint4*>(q + idx) = make_uint4(a.x, a.y, b.x, b.y);
    } else if (valid >= 8) {
      *reinterpret_cast<uint2*>(q + idx) = a;
      if (valid == 16) *reinterpret_cast<uint2*>(q + idx + 8) = b;
      else store_codes(q + idx + 8, b, valid - 8);
    } else {
      store_codes(q + idx, a, valid);
    }
  }
}

// ------------------------------------------------------------------ block-scale packers
// MXFP8: eight lanes per 32-element block, four elements per lane.  The thread grid covers the
// padded scale-factor domain so that every byte of the SF buffer is written.
// SWIGLU: x is [rows, 2 k] (gate first, then up) and the packed value is bf16(table[gate] * up), `table`
// being SiLU on all 65536 bf16 bit patterns (blackwell/csrc/mxfp8_swiglu.cu:20-78).
template <bool SWIGLU>
__global__ void __launch_bounds__(256)
pack_mxfp8_kernel(const __nv_bfloat16* __restrict__ x, long long rows, long long k, uint8_t* __restrict__ q,
                  uint8_t* __restrict__ sf, const __nv_bfloat16* __restrict__ table) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const long long groups_padded = (k + 127) / 128 * 4;
  const long long rows_padded = (rows + 127) / 128 * 128;
  const long long thread = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long block_index = thread / 8;
  const int lane8 = static_cast<int>(thread % 8);
  const long long row = block_index / groups_padded;
  const long long group = block_index % groups_padded;
  if (row >= rows_padded) return;
  const long long sfi = sf_offset(row, group, groups_padded / 4);
  if (row >= rows || group * 32 >= k) {
    if (lane8 == 0) sf[sfi] = 0;
    return;
  }
  const long long base = row * k + group * 32 + lane8 * 4;
  float v[4];
  if constexpr (SWIGLU) {
    const long long in = row * 2 * k + group * 32 + lane8 * 4;
    const uint2 g = *reinterpret_cast<const uint2*>(x + in);
    const uint2 u = *reinterpret_cast<const uint2*>(x + in + k);
    const uint32_t gb[4] = {g.x & 0xFFFFu, g.x >> 16, g.y & 0xFFFFu, g.y >> 16};
    const uint32_t ub[4] = {u.x & 0xFFFFu, u.x >> 16, u.y & 0xFFFFu, u.y >> 16};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = round_bf16(__fmul_rn(__bfloat162float(table[gb[i]]), bf16_bits_to_float(ub[i])));
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(x + base);
    v[0] = bf16_bits_to_float(u.x & 0xFFFFu), v[1] = bf16_bits_to_float(u.x >> 16);
    v[2] = bf16_bits_to_float(u.y & 0xFFFFu), v[3] = bf16_bits_to_float(u.y >> 16);
  }
  float amax = 0.0f;
  unsigned invalid = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    amax = fmaxf(amax, fabsf(v[i]));
    invalid |= !(fabsf(v[i]) <= 3.4028234664e38f);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o, 8));
    invalid |= __shfl_xor_sync(0xffffffffu, invalid, o, 8);
  }
  const uint32_t e = mxfp8_block_scale(amax, invalid != 0);
  if (lane8 == 0) sf[sfi] = static_cast<uint8_t>(e);
  const float inverse = mxfp8_inverse_scale(e);
  uint32_t out = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    out |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(__fmul_rn(v[i], inverse), __NV_SATFINITE, __NV_E4M3)) << (8 * i);
  *reinterpret_cast<uint32_t*>(q + base) = out;
}

// The scale of the W4A8-MX formats: the smallest power of two >= v, as a UE8M0 exponent byte (1.0 for
// v <= 0 or NaN; blackwell/csrc/fp4_mx_cutlass_linear.cu:47-58, `ceil_power_of_two`).
__device__ __forceinline__ uint32_t ceil_pow2_ue8m0(float v) {
  if (!(v > 0.0f)) return 127u;
  const uint32_t bits = __float_as_uint(v);
  uint32_t e = bits >> 23;             // biased exponent (v > 0: no sign bit)
  if (e == 0u) return 1u;              // subnormal input: below 2^-126, the smallest normal scale covers it
  if (bits & 0x7FFFFFu) ++e;           // not a power of two: round up
  return e > 254u ? 254u : e;
}

// W4A8-MX, 32-element blocks, eight lanes per block (four elements per lane); FMT 0: MXFP8 activations
// q = e4m3(clamp(x / s, +-448)), s = ceil_pow2(amax / 448); FMT 1: MXFP4 weights q = e2m1(x / s),
// s = ceil_pow2(amax / 6), two codes per byte, low nibble = even k.  Reference:
// blackwell/csrc/fp4_mx_cutlass_linear.cu:59-132.  Every byte of the scale buffer is written.
template <int FMT>
__global__ void __launch_bounds__(256)
pack_mx_ceil_kernel(const __nv_bfloat16* __restrict__ x, long long rows, long long k, uint8_t* __restrict__ q,
                    uint8_t* __restrict__ sf) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const long long groups_padded = (k + 127) / 128 * 4;
  const long long rows_padded = (rows + 127) / 128 * 128;
  const long long thread = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long block_index = thread / 8;
  const int lane8 = static_cast<int>(thread % 8);
  const long long row = block_index / groups_padded;
  const long long group = block_index % groups_padded;
  if (row >= rows_padded) return;
  const long long sfi = sf_offset(row, group, groups_padded / 4);
  if (row >= rows || group * 32 >= k) {
    if (lane8 == 0) sf[sfi] = 0;
    return;
  }
  const long long base = row * k + group * 32 + lane8 * 4;
  const uint2 u = *reinterpret_cast<const uint2*>(x + base);
  const float v[4] = {bf16_bits_to_float(u.x & 0xFFFFu), bf16_bits_to_float(u.x >> 16), bf16_bits_to_float(u.y & 0xFFFFu),
                      bf16_bits_to_float(u.y >> 16)};
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o, 8));
  const uint32_t e = ceil_pow2_ue8m0(__fdiv_rn(amax, FMT == 0 ? 448.0f : 6.0f));
  if (lane8 == 0) sf[sfi] = static_cast<uint8_t>(e);
  const float inverse = __uint_as_float((254u - e) << 23);  // 2^(127 - e), e in 1..254
  if constexpr (FMT == 0) {
    uint32_t out = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float t = fminf(448.0f, fmaxf(-448.0f, __fmul_rn(v[i], inverse)));
      out |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(t, __NV_SATFINITE, __NV_E4M3)) << (8 * i);
    }
    *reinterpret_cast<uint32_t*>(q + base) = out;
  } else {
    const uint32_t lo = __nv_cvt_float2_to_fp4x2(make_float2(__fmul_rn(v[0], inverse), __fmul_rn(v[1], inverse)), __NV_E2M1,
                                                 cudaRoundNearest);
    const uint32_t hi = __nv_cvt_float2_to_fp4x2(make_float2(__fmul_rn(v[2], inverse), __fmul_rn(v[3], inverse)), __NV_E2M1,
                                                 cudaRoundNearest);
    *reinterpret_cast<unsigned short*>(q + base / 2) = static_cast<unsigned short>((lo & 0xFFu) | ((hi & 0xFFu) << 8));
  }
}

// NVFP4: one thread per 16-element block (two 128-bit loads, one 64-bit store).
__global__ void __launch_bounds__(256)
pack_nvfp4_kernel(const __nv_bfloat16* __restrict__ x, long long rows, long long k, const float* __restrict__ global,
                  uint8_t* __restrict__ q, uint8_t* __restrict__ sf) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const long long groups = k / 16;
  const long long groups_padded = (groups + 3) / 4 * 4;
  const long long rows_padded = (rows + 127) / 128 * 128;
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long row = idx / groups_padded;
  const long long group = idx % groups_padded;
  if (row >= rows_padded) return;
  const long long sfi = sf_offset(row, group, groups_padded / 4);
  if (row >= rows || group >= groups) {
    sf[sfi] = 0;
    return;
  }
  float v[16];
  load8(x + row * k + group * 16, true, 8, *reinterpret_cast<float(*)[8]>(&v[0]));
  load8(x + row * k + group * 16 + 8, true, 8, *reinterpret_cast<float(*)[8]>(&v[8]));
  if (global != nullptr) {
    // v / g for sixteen values and one divisor.  With r = fl(1 / g) correctly rounded, q = fl(v r)
    // corrected by its exact residual - e = fma(-q, g, v), q' = fma(e, r, q) - IS the correctly rounded
    // quotient (Markstein's theorem) unless the significand of g is all ones; the magnitude window
    // keeps every intermediate in the normal range.  Everything else (zeros, whose sign the division
    // keeps, tiny and huge values, such a divisor) takes the IEEE division.  16 divisions cost ~10
    // instructions each and made this kernel instruction bound.
    const float g = *global;
    const float r = __frcp_rn(g);
    const bool divisor_ok = (__float_as_uint(g) & 0x7FFFFFu) != 0x7FFFFFu && g >= 0x1p-40f && g <= 0x1p40f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float a = fabsf(v[i]);
      if (divisor_ok && a >= 0x1p-60f && a <= 0x1p60f) {
        const float q = __fmul_rn(v[i], r);
        v[i] = __fmaf_rn(__fmaf_rn(-q, g, v[i]), r, q);
      } else {
        v[i] = __fdiv_rn(v[i], g);
      }
    }
  }
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
  const float scale = amax > 0.0f ? __fdiv_rn(amax, 6.0f) : 1.0f;
  const uint8_t code = static_cast<uint8_t>(__nv_cvt_float_to_fp8(scale, __NV_SATFINITE, __NV_E4M3)) & 0x7F;
  float deq = __half2float(__half(__nv_cvt_fp8_to_halfraw(code, __NV_E4M3)));
  if (!(deq > 0.0f)) deq = scale;
  const float reciprocal = __fdiv_rn(1.0f, deq);
  unsigned long long packed = 0;
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const __nv_fp4x2_storage_t pair = __nv_cvt_float2_to_fp4x2(
        make_float2(__fmul_rn(v[i], reciprocal), __fmul_rn(v[i + 1], reciprocal)), __NV_E2M1, cudaRoundNearest);
    packed |= static_cast<unsigned long long>(static_cast<uint8_t>(pair)) << (4 * i);
  }
  *reinterpret_cast<unsigned long long*>(q + row * (k / 2) + group * 8) = packed;
  sf[sfi] = code;
}

// ------------------------------------------------------------------ fused producers for the FP8 / NVFP4 GEMMs
// SwiGLU in fp32, as the reference's per-tensor FP8 producer evaluates it
// (blackwell/csrc/fp8_cutlass_linear.cu:271-279): bf16( gate / (1 + exp(-gate)) * up ).
__device__ __forceinline__ float swiglu_f32(float gate, float up) {
  return round_bf16(__fmul_rn(__fdiv_rn(gate, __fadd_rn(1.0f, expf(-gate))), up));
}
// Eight consecutive fp32-step SwiGLU outputs (bf16 values) of row-major gate_up [rows, 2 * inter], gate first.  A 64-bit
// division costs as much as an activation, so the row is found with a 32-bit one wherever the index fits.
__device__ __forceinline__ void load8_swiglu(const __nv_bfloat16* gate_up, long long inter, long long idx, float (&v)[8]) {
  const long long row = idx < (1ll << 32) ? static_cast<unsigned>(idx) / static_cast<unsigned>(inter) : idx / inter;
  const long long col = idx - row * inter;
  const __nv_bfloat16* g = gate_up + row * 2 * inter + col;
  float gv[8], uv[8];
  const bool vec = (inter % 8) == 0;
  load8(g, vec, 8, gv);
  load8(g + inter, vec, 8, uv);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = swiglu_f32(gv[i], uv[i]);
}
// Eight consecutive outputs of `row` in bf16 steps: gate first, then up; or `interleaved`: blocks of 128 columns, 64 up
// values followed by their 64 gate values (the layout a fused gate/up projection writes:
// blackwell/csrc/fp4_cutlass_linear.cu:958-965).  inter % 8 == 0.
__device__ __forceinline__ void load8_swiglu_bf16(const __nv_bfloat16* gate_up, long long inter, long long row, long long col,
                                                  uint32_t* v, bool interleaved) {
  const __nv_bfloat16* g = gate_up + row * 2 * inter + col;
  const __nv_bfloat16* u = g + inter;
  if (interleaved) {  // eight consecutive columns never straddle a 64-column block
    u = gate_up + row * 2 * inter + (col >> 6) * 128 + (col & 63);
    g = u + 64;
  }
  const uint4 gw = *reinterpret_cast<const uint4*>(g), uw = *reinterpret_cast<const uint4*>(u);
  v[0] = swiglu_bf16x2_steps(gw.x, uw.x), v[1] = swiglu_bf16x2_steps(gw.y, uw.y);
  v[2] = swiglu_bf16x2_steps(gw.z, uw.z), v[3] = swiglu_bf16x2_steps(gw.w, uw.w);
}

// SwiGLU -> MXFP8 with power-of-two (ceil) block scales, the activation side of W4A8-MX
// (blackwell/csrc/fp4_mx_cutlass_linear.cu:134-179, `pack_swiglu_mxfp8_warp_kernel`): the product
// gate / (1 + exp(-gate)) * up stays in fp32 (no bf16 rounding) before the block quantizer.
__global__ void __launch_bounds__(256)
swiglu_pack_mxfp8_ceil_kernel(const __nv_bfloat16* __restrict__ gate_up, long long rows, long long inter, int interleaved,
                              uint8_t* __restrict__ q, uint8_t* __restrict__ sf) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const long long groups_padded = (inter + 127) / 128 * 4;
  const long long rows_padded = (rows + 127) / 128 * 128;
  const long long thread = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long block_index = thread / 8;
  const int lane8 = static_cast<int>(thread % 8);
  const long long row = block_index / groups_padded;
  const long long group = block_index % groups_padded;
  if (row >= rows_padded) return;
  const long long sfi = sf_offset(row, group, groups_padded / 4);
  if (row >= rows || group * 32 >= inter) {
    if (lane8 == 0) sf[sfi] = 0;
    return;
  }
  const long long col = group * 32 + lane8 * 4;
  const __nv_bfloat16* g = gate_up + row * 2 * inter + col;
  const __nv_bfloat16* u = g + inter;
  if (interleaved) {
    u = gate_up + row * 2 * inter + (col >> 6) * 128 + (col & 63);
    g = u + 64;
  }
  const uint2 gw = *reinterpret_cast<const uint2*>(g), uw = *reinterpret_cast<const uint2*>(u);
  const float gv[4] = {bf16_bits_to_float(gw.x & 0xFFFFu), bf16_bits_to_float(gw.x >> 16), bf16_bits_to_float(gw.y & 0xFFFFu),
                       bf16_bits_to_float(gw.y >> 16)};
  const float uv[4] = {bf16_bits_to_float(uw.x & 0xFFFFu), bf16_bits_to_float(uw.x >> 16), bf16_bits_to_float(uw.y & 0xFFFFu),
                       bf16_bits_to_float(uw.y >> 16)};
  float v[4], amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = __fmul_rn(__fdiv_rn(gv[i], __fadd_rn(1.0f, expf(-gv[i]))), uv[i]);
    amax = fmaxf(amax, fabsf(v[i]));
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o, 8));
  const uint32_t e = ceil_pow2_ue8m0(__fdiv_rn(amax, 448.0f));
  if (lane8 == 0) sf[sfi] = static_cast<uint8_t>(e);
  const float inverse = __uint_as_float((254u - e) << 23);
  uint32_t out = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float t = fminf(448.0f, fmaxf(-448.0f, __fmul_rn(v[i], inverse)));
    out |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(t, __NV_SATFINITE, __NV_E4M3)) << (8 * i);
  }
  *reinterpret_cast<uint32_t*>(q + row * inter + col) = out;
}

// The maximum of the finite outputs, and with `product` the outputs themselves: [rows, inter] bf16, so that the conversion
// that needs the maximum does not evaluate the activation a second time.
__global__ void __launch_bounds__(256)
swiglu_amax_kernel(const __nv_bfloat16* __restrict__ gate_up, long long rows, long long inter,
                   unsigned* __restrict__ amax_bits, __nv_bfloat16* __restrict__ product) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  __shared__ uint32_t scratch[8];
  uint32_t m = 0u;
  const long long elements = rows * inter;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x * 8;
  for (long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8; idx < elements;
       idx += stride) {
    float v[8];
    load8_swiglu(gate_up, inter, idx, v);  // inter % 8 == 0: a vector never straddles rows
    Packed8 p;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p.w[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
      // magnitudes order like their bit patterns; infinities and NaN count as zero
      const uint32_t lo = p.w[i] & 0x7FFFu, hi = (p.w[i] >> 16) & 0x7FFFu;
      m = max(m, lo < 0x7F80u ? lo : 0u);
      m = max(m, hi < 0x7F80u ? hi : 0u);
    }
    if (product != nullptr) store8p(product + idx, true, 8, p);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = max(m, scratch[w]);
    atomicMax(amax_bits, m << 16);  // the float of those upper bits
  }
}

__global__ void __launch_bounds__(256)
swiglu_to_fp8_kernel(const __nv_bfloat16* __restrict__ gate_up, long long rows, long long inter,
                     const float* __restrict__ scale, uint8_t* __restrict__ q) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const float inverse = __fdiv_rn(1.0f, *scale);
  const long long elements = rows * inter;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x * 8;
  for (long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8; idx < elements;
       idx += stride) {
    float v[8];
    load8_swiglu(gate_up, inter, idx, v);
    *reinterpret_cast<uint2*>(q + idx) = to_fp8x8(v, inverse);
  }
}

// SwiGLU -> NVFP4: one thread per 16-element block of the [rows, inter] activation.
__global__ void __launch_bounds__(256)
swiglu_pack_nvfp4_kernel(const __nv_bfloat16* __restrict__ gate_up, long long rows, long long inter, int interleaved,
                         uint8_t* __restrict__ q, uint8_t* __restrict__ sf) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const long long groups = inter / 16;
  const long long groups_padded = (groups + 3) / 4 * 4;
  const long long rows_padded = (rows + 127) / 128 * 128;
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long row = idx / groups_padded;
  const long long group = idx % groups_padded;
  if (row >= rows_padded) return;
  const long long sfi = sf_offset(row, group, groups_padded / 4);
  if (row >= rows || group >= groups) {
    sf[sfi] = 0;
    return;
  }
  uint32_t v[8];
  load8_swiglu_bf16(gate_up, inter, row, group * 16, &v[0], interleaved != 0);
  load8_swiglu_bf16(gate_up, inter, row, group * 16 + 8, &v[4], interleaved != 0);
  uint8_t code;
  const unsigned long long packed = nvfp4_block(v, &code);
  *reinterpret_cast<unsigned long long*>(q + row * (inter / 2) + group * 8) = packed;
  sf[sfi] = code;
}

// SwiGLU alone, bf16 in the reference's bf16x2 steps (blackwell/csrc/fp4_cutlass_linear.cu:944-995,
// `silu_mul_bf16`): eight outputs per thread; either gate/up layout.
__global__ void __launch_bounds__(256)
silu_mul_bf16_kernel(const __nv_bfloat16* __restrict__ gate_up, long long rows, long long inter, int interleaved,
                     __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const long long total = rows * inter;
  for (long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 8; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x * 8) {
    Packed8 v;
    const long long row = idx / inter;
    load8_swiglu_bf16(gate_up, inter, row, idx - row * inter, v.w, interleaved != 0);  // inter % 8 == 0: one row per vector
    store8p(out + idx, true, 8, v);
  }
}

// (residual add +) RMSNorm feeding a per-tensor FP8 quantizer (FMT 0: writes the bf16 results and the
// tensor's absolute maximum), an NVFP4 packer (FMT 1: packs straight from registers) or nothing (FMT 2: the
// plain norm of blackwell/csrc/fp4_cutlass_linear.cu:429-476).  Arithmetic
// of blackwell/csrc/fp8_cutlass_linear.cu:145-203 and blackwell/csrc/fp4_cutlass_linear.cu:843-929:
// s = bf16(x + residual); r = rsqrt(mean(s^2) + eps); y = bf16( bf16(s * r) * weight ).
// One CTA per row (FMT 1: per row of the 128-row padded scale-factor domain), row cached in registers.
template <int FMT>
__global__ void __launch_bounds__(kRowThreads)
rmsnorm_producer_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                        const __nv_bfloat16* __restrict__ weight, int rows, int k, float eps,
                        __nv_bfloat16* __restrict__ sum_out, __nv_bfloat16* __restrict__ norm_out,
                        unsigned* __restrict__ amax_bits, uint8_t* __restrict__ q, uint8_t* __restrict__ sf) {
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  __shared__ float scratch[kRowThreads / 32];
  const int row = blockIdx.x;
  const int groups = k / 16;
  const int groups_padded = (groups + 3) / 4 * 4;
  if (row >= rows) {  // FMT 1 only: padding rows of the scale-factor buffer read as zero
    for (int g = threadIdx.x; g < groups_padded; g += kRowThreads) sf[sf_offset(row, g, groups_padded / 4)] = 0;
    return;
  }
  const long long xoff = static_cast<long long>(row) * k;
  float vals[kMaxVec][8];
  float sq = 0.0f;
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int idx = (it * kRowThreads + threadIdx.x) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) vals[it][i] = 0.0f;
    if (idx < k) {  // k % 16 == 0: whole vectors only
      load8(x + xoff + idx, true, 8, vals[it]);
      if (residual != nullptr) {
        float rv[8];
        load8(residual + xoff + idx, true, 8, rv);
#pragma unroll
        for (int i = 0; i < 8; ++i) vals[it][i] = round_bf16(__fadd_rn(vals[it][i], rv[i]));
        if (sum_out != nullptr) store8(sum_out + xoff + idx, true, 8, vals[it]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) sq = fmaf(vals[it][i], vals[it][i], sq);
    }
  }
  const float inv = rsqrtf(__fadd_rn(__fdiv_rn(block_reduce(sq, false, scratch), static_cast<float>(k)), eps));
  float local_max = 0.0f;
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int idx = (it * kRowThreads + threadIdx.x) * 8;
    if (idx < k) {
      float wv[8];
      load8(weight + idx, true, 8, wv);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float y = round_bf16(__fmul_rn(round_bf16(__fmul_rn(vals[it][i], inv)), wv[i]));
        vals[it][i] = y;
        const float a = fabsf(y);
        if (a <= 3.4028234664e38f) local_max = fmaxf(local_max, a);
      }
      if (norm_out != nullptr) store8(norm_out + xoff + idx, true, 8, vals[it]);
    }
  }
  if (FMT == 2) return;  // the plain norm: the bf16 result is the output
  if (FMT == 0) {
    const float m = block_reduce(local_max, true, scratch);
    if (threadIdx.x == 0) atomicMax(amax_bits, __float_as_uint(m));
    return;
  }
  // FMT 1: a 16-element block is held by an even thread (low half) and its odd neighbour (high half)
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int idx = (it * kRowThreads + threadIdx.x) * 8;  // warp-uniform validity: k % 256 handled by the mask below
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t own = pack_bf16x2(vals[it][2 * i], vals[it][2 * i + 1]);  // bf16 values already: nothing is rounded
      const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
      v[i] = (threadIdx.x & 1) ? other : own;
      v[4 + i] = (threadIdx.x & 1) ? own : other;
    }
    if (idx < k) {
      uint8_t code;
      const unsigned long long packed = nvfp4_block(v, &code);
      const int group = idx / 16;
      // each thread stores the four code bytes of its own eight values
      const uint32_t mine = static_cast<uint32_t>((threadIdx.x & 1) ? (packed >> 32) : packed);
      *reinterpret_cast<uint32_t*>(q + static_cast<long long>(row) * (k / 2) + idx / 2) = mine;
      if (!(threadIdx.x & 1)) sf[sf_offset(row, group, groups_padded / 4)] = code;
    }
  }
  // scale factors of the padded groups of this row
  for (int g = groups + threadIdx.x; g < groups_padded; g += kRowThreads) sf[sf_offset(row, g, groups_padded / 4)] = 0;
}

__global__ void probe_rcp_kernel(uint32_t* out) { *out = __float_as_uint(rcp_approx_ftz(448.0f)); }

// Threads per row of the row kernels: as many as the row has vectors of eight (64 to 256), halved further (at most four
// vectors per thread) while the rows would need more than one wave of resident threads (1536 per SM with one vector
// each, about 1024 with more).  With few rows the latency of a thread decides; with many, fewer warps per row mean
// fewer barriers and more rows in flight.  Against 256 threads for every row, four vectors each (most of them masked)
// and fp32 arithmetic per element - LayerNorm + modulation + gated residual to int8: 50 x 1024 4.3 -> 2.4 us, 816 x 2048
// 11.7 -> 5.0, 1764 x 2048 21.9 -> 9.0 (2.8 TB/s), 16384 x 2048 234 -> 74; adaptive RMSNorm: 50 x 1024 3.6 -> 2.3,
// 400 x 1024 4.4 -> 3.4, 1764 x 2048 13.9 -> 8.6; add + RMSNorm + tensor maximum: 816 x 2048 6.4 -> 3.9; plain rows:
// 50 x 4096 2.9 -> 2.5, 1764 x 8192 15.2 -> 12.5.  One wave against two: 816 x 2048 5.0 us with 256 threads, 5.7 with 128;
// threads without a vector: 400 x 1024 3.9 us with 256 threads, 3.5 with 128.
int row_threads(int64_t rows, int64_t kpad) {
  int threads = kRowThreads;
  while (threads > 64 && threads * 4 >= kpad) threads /= 2;
  while (threads > 64 && rows * threads > 148 * (kpad <= threads * 8 ? 1536 : 1024) && (threads / 2) * kMaxVec * 8 >= kpad)
    threads /= 2;
  return threads;
}
// vectors of eight per thread: 1, 2 or 4 (longer rows loop in the kernels that take them)
int row_vectors(int threads, int64_t kpad) { return kpad <= threads * 8 ? 1 : (kpad <= threads * 16 ? 2 : 4); }

// Calls `f` with the (threads, vectors) pair of the rule above as compile-time constants; kpad <= kCachedK.
template <typename F>
void with_row_shape(int64_t rows, int64_t kpad, F&& f) {
  const int threads = row_threads(rows, kpad), vecs = row_vectors(threads, kpad);
  using std::integral_constant;
  auto pick = [&](auto t) {
    if (vecs == 1) f(t, integral_constant<int, 1>{});
    else if (vecs == 2) f(t, integral_constant<int, 2>{});
    else f(t, integral_constant<int, 4>{});
  };
  if (threads == 64) pick(integral_constant<int, 64>{});
  else if (threads == 128) pick(integral_constant<int, 128>{});
  else pick(integral_constant<int, 256>{});
}

// Table in shared memory or gathered through L1?  Copying it costs an SM about 2 us and leaves it one CTA, so there must be
// enough work: `line` elements.
bool table_on_chip(const void* lut, int64_t rows, int64_t k, int64_t line) { return aligned16(lut) && rows * k >= line; }
// one CTA per SM (at most `blocks`) of a kernel whose dynamic shared memory is the table
template <typename... KArgs, typename... Args>
int launch_with_table(void (*kernel)(KArgs...), int64_t blocks, cudaStream_t st, Args&&... args) {
  const cudaError_t set = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes);
  if (set != cudaSuccess) return fail(RK_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(set));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(std::min<int64_t>(blocks, 148)));
  cfg.blockDim = dim3(kTableThreads);
  cfg.dynamicSmemBytes = kTableBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
  return check_launch("table kernel");
}

template <int BITS>
int launch_quant_rows(const void* x, int64_t rows, int64_t total_rows, int64_t k, int64_t xs, const void* up,
                      int64_t us, const void* lut, int mode, void* q, float* scales, int true_division,
                      cudaStream_t st) {
  const int kpad = static_cast<int>(round_up(k, 128));
  const int vec_ok = aligned16(x) && xs % 8 == 0 && (mode != RK_ACT_LUT_MUL || (aligned16(up) && us % 8 == 0));
  auto xb = static_cast<const __nv_bfloat16*>(x);
  auto ub = static_cast<const __nv_bfloat16*>(up);
  auto lb = static_cast<const __nv_bfloat16*>(lut);
  auto qb = static_cast<uint8_t*>(q);
  const dim3 grid(static_cast<unsigned>(total_rows));
  if (mode != RK_ACT_PLAIN && total_rows == rows && !true_division && kpad <= kCachedK && table_on_chip(lut, rows, k, k > 4096 ? kTableLongRowsLine : kTableRowsLine)) {
    auto launch_table = [&](auto kernel, int group) {
      return launch_with_table(kernel, (rows + kTableThreads / group - 1) / (kTableThreads / group), st, xb, xs, ub, us, lb,
                               static_cast<int>(k), kpad, static_cast<int>(rows), qb, scales, vec_ok);
    };
    auto by_group = [&](auto mode_c) {
      constexpr int kMode = decltype(mode_c)::value;
      if (kpad <= 64 * 32) return launch_table(quant_rows_table_kernel<BITS, kMode, 64>, 64);
      if (kpad <= 128 * 32) return launch_table(quant_rows_table_kernel<BITS, kMode, 128>, 128);
      return launch_table(quant_rows_table_kernel<BITS, kMode, 256>, 256);
    };
    return mode == RK_ACT_LUT_MUL ? by_group(std::integral_constant<int, RK_ACT_LUT_MUL>{})
                                  : by_group(std::integral_constant<int, RK_ACT_LUT>{});
  }
  const int threads = row_threads(total_rows, kpad);
  const int vecs = row_vectors(threads, kpad);
  auto launch = [&](auto kernel) {
    launch_pdl(kernel, grid, threads, st, xb, xs, ub, us, lb, static_cast<int>(k), kpad, static_cast<int>(rows), qb, scales,
               true_division, vec_ok);
  };
  auto by_vectors = [&](auto mode_c) {
    constexpr int kMode = decltype(mode_c)::value;
    if (vecs == 1) launch(quant_rows_kernel<BITS, kMode, 1>);
    else if (vecs == 2) launch(quant_rows_kernel<BITS, kMode, 2>);
    else launch(quant_rows_kernel<BITS, kMode, 4>);
  };
  switch (mode) {
    case RK_ACT_PLAIN: by_vectors(std::integral_constant<int, RK_ACT_PLAIN>{}); break;
    case RK_ACT_LUT_MUL: by_vectors(std::integral_constant<int, RK_ACT_LUT_MUL>{}); break;
    default: by_vectors(std::integral_constant<int, RK_ACT_LUT>{});
  }
  return check_launch("quant_rows");
}

}  // namespace
}  // namespace rk

namespace rk {
int launch_finalize_scale(unsigned* staging, float divisor, float* scale_out, cudaStream_t stream) {
  launch_pdl(finalize_scale_kernel, 1, 1, stream, staging, divisor, scale_out);
  return check_launch("finalize_scale");
}
}  // namespace rk

using namespace rk;

extern "C" int rk_quant_rows(const void* x, int64_t rows, int64_t k, int64_t x_stride, const void* up,
                             int64_t up_stride, const void* lut, int mode, int bits, void* q, float* scales,
                             void* stream) {
  if (!x || !q || !scales) return fail(RK_EINVAL, "rk_quant_rows: null pointer");
  if (bits != 4 && bits != 8) return fail(RK_EINVAL, "rk_quant_rows: bits must be 4 or 8");
  if (rows < 1 || k < 1 || k > 65536) return fail(RK_EINVAL, "rk_quant_rows: unsupported activation dimensions");
  if (mode < 0 || mode > 2) return fail(RK_EINVAL, "rk_quant_rows: unknown mode");
  if (mode != RK_ACT_PLAIN && !lut) return fail(RK_EINVAL, "rk_quant_rows: table required");
  if (mode == RK_ACT_LUT_MUL && !up) return fail(RK_EINVAL, "rk_quant_rows: gated mode needs `up`");
  if (x_stride < k || (mode == RK_ACT_LUT_MUL && up_stride < k)) return fail(RK_EINVAL, "rk_quant_rows: row stride < k");
  return bits == 8 ? launch_quant_rows<8>(x, rows, rows, k, x_stride, up, up_stride, lut, mode, q, scales, 0,
                                          as_stream(stream))
                   : launch_quant_rows<4>(x, rows, rows, k, x_stride, up, up_stride, lut, mode, q, scales, 0,
                                          as_stream(stream));
}

extern "C" int rk_quant_weight_int(const void* w, int64_t n, int64_t k, int bits, void* q, float* scales,
                                   void* stream) {
  if (!w || !q || !scales) return fail(RK_EINVAL, "rk_quant_weight_int: null pointer");
  if (bits != 4 && bits != 8) return fail(RK_EINVAL, "rk_quant_weight_int: bits must be 4 or 8");
  if (n < 1 || k < 1 || k > 65536) return fail(RK_EINVAL, "rk_quant_weight_int: unsupported weight dimensions");
  const int64_t npad = round_up(n, 8);
  return bits == 8 ? launch_quant_rows<8>(w, n, npad, k, k, nullptr, 0, nullptr, RK_ACT_PLAIN, q, scales, 1,
                                          as_stream(stream))
                   : launch_quant_rows<4>(w, n, npad, k, k, nullptr, 0, nullptr, RK_ACT_PLAIN, q, scales, 1,
                                          as_stream(stream));
}

extern "C" int rk_quant_rows_modulated(const void* x, const void* scale, const void* shift, int64_t rows, int64_t k,
                                       int64_t tokens, int layer_norm, float eps, const void* y, const void* gate,
                                       void* residual_out, int bits, void* q, float* scales, void* stream) {
  if (!x || !scale || !shift || !q || !scales) return fail(RK_EINVAL, "rk_quant_rows_modulated: null pointer");
  if (bits != 4 && bits != 8) return fail(RK_EINVAL, "rk_quant_rows_modulated: bits must be 4 or 8");
  if (rows < 1 || k < 1 || tokens < 1 || rows % tokens != 0)
    return fail(RK_EINVAL, "rk_quant_rows_modulated: rows must be a positive multiple of tokens");
  if (k > kCachedK) return fail(RK_EUNSUPPORTED, "rk_quant_rows_modulated: k > %d", kCachedK);
  if ((y == nullptr) != (gate == nullptr) || (y != nullptr && residual_out == nullptr))
    return fail(RK_EINVAL, "rk_quant_rows_modulated: y, gate and residual_out go together");
  if (!aligned16(x) || !aligned16(scale) || !aligned16(shift) || (y && (!aligned16(y) || !aligned16(gate))) ||
      (residual_out && !aligned16(residual_out)))
    return fail(RK_EINVAL, "rk_quant_rows_modulated: pointers must be 16-byte aligned");
  const int kpad = static_cast<int>(round_up(k, 128));
  auto b = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  auto launch = [&](auto kernel, int threads) {
    launch_pdl(kernel, static_cast<unsigned>(rows), threads, as_stream(stream), b(x), b(scale), b(shift), static_cast<int>(k),
               kpad, static_cast<int>(tokens), layer_norm, eps, b(y), b(gate), static_cast<__nv_bfloat16*>(residual_out),
               static_cast<uint8_t*>(q), scales);
  };
  with_row_shape(rows, kpad, [&](auto t, auto v) {
    constexpr int kT = decltype(t)::value, kV = decltype(v)::value;
    if (bits == 8) launch(quant_rows_modulated_kernel<8, kT, kV>, kT);
    else launch(quant_rows_modulated_kernel<4, kT, kV>, kT);
  });
  return check_launch("quant_rows_modulated");
}

namespace {
int launch_rmsnorm_quant_rows(const char* who, const void* x, const void* residual, const void* gate, const void* scale,
                              const void* shift, int64_t tokens, int64_t rows, int64_t k, float eps, int bits,
                              void* sum_out, void* norm_out, void* q, float* scales, void* stream) {
  if (!x || !scale || !q || !scales) return fail(RK_EINVAL, "%s: null pointer", who);
  if (bits != 4 && bits != 8) return fail(RK_EINVAL, "%s: bits must be 4 or 8", who);
  if (rows < 1 || k < 1 || tokens < 0 || (tokens > 0 && rows % tokens != 0))
    return fail(RK_EINVAL, "%s: bad row / token counts", who);
  if (gate && (!residual || tokens < 1)) return fail(RK_EINVAL, "%s: a gate needs a residual branch and tokens > 0", who);
  if (k > kCachedK) return fail(RK_EUNSUPPORTED, "%s: k > %d", who, kCachedK);
  if (!aligned16(x) || !aligned16(scale) || (residual && !aligned16(residual)) || (shift && !aligned16(shift)) ||
      (gate && !aligned16(gate)) || (sum_out && !aligned16(sum_out)) || (norm_out && !aligned16(norm_out)))
    return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  const int kpad = static_cast<int>(round_up(k, 128));
  auto b = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  auto launch = [&](auto kernel, int threads) {
    launch_pdl(kernel, static_cast<unsigned>(rows), threads, as_stream(stream), b(x), b(residual), b(gate), b(scale), b(shift),
               static_cast<int>(tokens), static_cast<int>(k), kpad, eps, static_cast<__nv_bfloat16*>(sum_out),
               static_cast<__nv_bfloat16*>(norm_out), static_cast<uint8_t*>(q), scales);
  };
  with_row_shape(rows, kpad, [&](auto t, auto v) {
    constexpr int kT = decltype(t)::value, kV = decltype(v)::value;
    if (bits == 8) launch(rmsnorm_quant_rows_kernel<8, kT, kV>, kT);
    else launch(rmsnorm_quant_rows_kernel<4, kT, kV>, kT);
  });
  return check_launch(who);
}
}  // namespace

extern "C" int rk_rmsnorm_quant_rows(const void* x, const void* residual, const void* scale, const void* shift,
                                     int64_t tokens, int64_t rows, int64_t k, float eps, int bits, void* sum_out,
                                     void* norm_out, void* q, float* scales, void* stream) {
  return launch_rmsnorm_quant_rows("rk_rmsnorm_quant_rows", x, residual, nullptr, scale, shift, tokens, rows, k, eps, bits,
                                   sum_out, norm_out, q, scales, stream);
}

extern "C" int rk_gated_rmsnorm_quant_rows(const void* x, const void* branch, const void* gate, const void* scale,
                                           const void* shift, int64_t tokens, int64_t rows, int64_t k, float eps,
                                           int bits, void* sum_out, void* norm_out, void* q, float* scales,
                                           void* stream) {
  if (!branch || !gate) return fail(RK_EINVAL, "rk_gated_rmsnorm_quant_rows: null pointer");
  return launch_rmsnorm_quant_rows("rk_gated_rmsnorm_quant_rows", x, branch, gate, scale, shift, tokens, rows, k, eps,
                                   bits, sum_out, norm_out, q, scales, stream);
}

extern "C" int rk_rmsnorm_tensor_scale(const void* x, const void* residual, const void* scale, const void* shift,
                                       int64_t tokens, int64_t rows, int64_t k, float eps, float divisor, void* sum_out,
                                       void* norm_out, float* scale_out, void* workspace, size_t workspace_bytes,
                                       void* stream) {
  const char* who = "rk_rmsnorm_tensor_scale";
  if (!x || !scale || !norm_out) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || k < 1 || tokens < 0 || (tokens > 0 && rows % tokens != 0))
    return fail(RK_EINVAL, "%s: bad row / token counts", who);
  if (k > kCachedK) return fail(RK_EUNSUPPORTED, "%s: k > %d", who, kCachedK);
  if (!aligned16(x) || !aligned16(scale) || !aligned16(norm_out) || (residual && !aligned16(residual)) ||
      (shift && !aligned16(shift)) || (sum_out && !aligned16(sum_out)))
    return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  unsigned* staging = nullptr;
  if (scale_out != nullptr) {
    if (!(divisor > 0.0f)) return fail(RK_EINVAL, "%s: the divisor must be positive", who);
    if (!workspace || workspace_bytes < RK_WORKSPACE_HEADER) return fail(RK_EWORKSPACE, "%s: workspace too small", who);
    staging = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(workspace) + 64);  // zero between calls
  }
  auto b = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  with_row_shape(rows, k, [&](auto t, auto v) {
    constexpr int kT = decltype(t)::value, kV = decltype(v)::value;
    launch_pdl(rmsnorm_quant_rows_kernel<16, kT, kV>, static_cast<unsigned>(rows), kT, as_stream(stream), b(x), b(residual),
               nullptr, b(scale), b(shift), static_cast<int>(tokens), static_cast<int>(k), 0, eps,
               static_cast<__nv_bfloat16*>(sum_out), static_cast<__nv_bfloat16*>(norm_out), reinterpret_cast<uint8_t*>(staging),
               nullptr);
  });
  if (staging != nullptr) launch_pdl(finalize_scale_kernel, 1, 1, as_stream(stream), staging, divisor, scale_out);
  return check_launch(who);
}

extern "C" int rk_lut_mul_tensor_scale(const void* x, int64_t x_stride, const void* up, int64_t up_stride,
                                       const void* lut, int64_t rows, int64_t k, float divisor, void* out,
                                       float* scale_out, void* workspace, size_t workspace_bytes, void* stream) {
  const char* who = "rk_lut_mul_tensor_scale";
  if (!x || !up || !lut || !out) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || k < 8 || k % 8 != 0 || k > (1 << 30)) return fail(RK_EINVAL, "%s: rows >= 1 and k a multiple of 8", who);
  if (x_stride < k || up_stride < k || x_stride % 8 != 0 || up_stride % 8 != 0)
    return fail(RK_EINVAL, "%s: row strides must be multiples of 8 and >= k", who);
  if (!aligned16(x) || !aligned16(up) || !aligned16(out)) return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  unsigned* staging = nullptr;
  if (scale_out != nullptr) {
    if (!(divisor > 0.0f)) return fail(RK_EINVAL, "%s: the divisor must be positive", who);
    if (!workspace || workspace_bytes < RK_WORKSPACE_HEADER) return fail(RK_EWORKSPACE, "%s: workspace too small", who);
    staging = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(workspace) + 64);  // zero between calls
  }
  const long long vectors = rows * (k / 8);
  auto b = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  if (table_on_chip(lut, rows, k, kTableProductLine)) {
    const int rc = launch_with_table(lut_mul_amax_kernel<true>, (vectors + kTableThreads - 1) / kTableThreads, as_stream(stream),
                                     b(x), x_stride, b(up), up_stride, b(lut), rows, static_cast<int>(k),
                                     static_cast<__nv_bfloat16*>(out), staging);
    if (rc != RK_OK) return rc;
  } else {
    const unsigned blocks = static_cast<unsigned>(std::min<long long>((vectors + 255) / 256, 148LL * 8));
    launch_pdl(lut_mul_amax_kernel<false>, blocks, 256, as_stream(stream), b(x), x_stride, b(up), up_stride, b(lut), rows,
               static_cast<int>(k), static_cast<__nv_bfloat16*>(out), staging);
  }
  if (staging != nullptr) launch_pdl(finalize_scale_kernel, 1, 1, as_stream(stream), staging, divisor, scale_out);
  return check_launch(who);
}

extern "C" int rk_pack_w4_g128(const void* w, int64_t n, int64_t k, void* q, void* scales, void* stream) {
  if (!w || !q || !scales) return fail(RK_EINVAL, "rk_pack_w4_g128: null pointer");
  if (n < 1 || k < 128 || k % 128 != 0) return fail(RK_EINVAL, "rk_pack_w4_g128: k must be a positive multiple of 128");
  if (!aligned16(w)) return fail(RK_EINVAL, "rk_pack_w4_g128: w must be 16-byte aligned");
  const long long warps = static_cast<long long>(n) * (k / 128);
  const unsigned blocks = static_cast<unsigned>((warps + 7) / 8);
  launch_pdl(pack_w4_g128_kernel, blocks, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(w), static_cast<int>(n),
                                                             static_cast<int>(k), static_cast<uint8_t*>(q),
                                                             static_cast<__nv_bfloat16*>(scales));
  return check_launch("pack_w4_g128");
}

namespace {
int tensor_amax_scale(const void* x, int64_t elements, float divisor, float* scale_out, void* workspace,
                      size_t workspace_bytes, cudaStream_t st, const char* who) {
  if (!x || !scale_out) return fail(RK_EINVAL, "%s: null pointer", who);
  if (!workspace || workspace_bytes < RK_WORKSPACE_HEADER) return fail(RK_EWORKSPACE, "%s: workspace too small", who);
  if (elements < 1 || !aligned16(x)) return fail(RK_EINVAL, "%s: bad size or alignment", who);
  unsigned* staging = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(workspace) + 64);
  long long blocks = (elements + 2047) / 2048;
  if (blocks > 1184) blocks = 1184;  // 148 SMs x 8 CTAs
  launch_pdl(amax_finite_kernel, static_cast<unsigned>(blocks), 256, st, static_cast<const __nv_bfloat16*>(x), elements,
                                                                    staging);
  launch_pdl(finalize_scale_kernel, 1, 1, st, staging, divisor, scale_out);
  return check_launch(who);
}
}  // namespace

extern "C" int rk_quant_tensor_fp8_with_scale(const void* x, int64_t elements, const float* scale, void* q,
                                              void* stream) {
  if (!x || !scale || !q) return fail(RK_EINVAL, "rk_quant_tensor_fp8_with_scale: null pointer");
  if (elements < 1 || !aligned16(x) || (reinterpret_cast<uintptr_t>(q) & 7u))
    return fail(RK_EINVAL, "rk_quant_tensor_fp8_with_scale: bad size or alignment");
  long long blocks = (elements + 4095) / 4096;
  if (blocks > 1184) blocks = 1184;
  launch_pdl(to_fp8_kernel, static_cast<unsigned>(blocks), 256, as_stream(stream), static_cast<const __nv_bfloat16*>(x),
             elements, scale, static_cast<uint8_t*>(q), aligned16(q) ? 1 : 0);
  return check_launch("to_fp8");
}

extern "C" int rk_quant_tensor_fp8(const void* x, int64_t elements, void* q, float* scale_out, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  int rc = tensor_amax_scale(x, elements, 448.0f, scale_out, workspace, workspace_bytes, as_stream(stream),
                             "rk_quant_tensor_fp8");
  if (rc != RK_OK) return rc;
  return rk_quant_tensor_fp8_with_scale(x, elements, scale_out, q, stream);
}

extern "C" int rk_nvfp4_global_scale(const void* x, int64_t elements, float* scale_out, void* workspace,
                                     size_t workspace_bytes, void* stream) {
  return tensor_amax_scale(x, elements, 6.0f * 448.0f, scale_out, workspace, workspace_bytes, as_stream(stream),
                           "rk_nvfp4_global_scale");
}

extern "C" size_t rk_sf_bytes(int64_t rows, int64_t groups) {
  if (rows < 1 || groups < 1) return 0;
  return static_cast<size_t>(((rows + 127) / 128) * ((groups + 3) / 4) * 512);
}

extern "C" int rk_pack_mxfp8(const void* x, int64_t rows, int64_t k, void* q, void* sf, void* stream) {
  if (!x || !q || !sf) return fail(RK_EINVAL, "rk_pack_mxfp8: null pointer");
  if (rows < 1 || k < 32 || k % 32 != 0) return fail(RK_EINVAL, "rk_pack_mxfp8: k must be a positive multiple of 32");
  if (!aligned16(x) || !aligned16(q)) return fail(RK_EINVAL, "rk_pack_mxfp8: pointers must be 16-byte aligned");
  const long long blocks32 = ((rows + 127) / 128 * 128) * ((k + 127) / 128 * 4);
  const unsigned grid = static_cast<unsigned>((blocks32 * 8 + 255) / 256);
  launch_pdl(pack_mxfp8_kernel<false>, grid, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(x), rows, k,
             static_cast<uint8_t*>(q), static_cast<uint8_t*>(sf), nullptr);
  return check_launch("pack_mxfp8");
}

extern "C" int rk_swiglu_pack_mxfp8(const void* gate_up, int64_t rows, int64_t inter, const void* silu_table, void* q,
                                    void* sf, void* stream) {
  const char* who = "rk_swiglu_pack_mxfp8";
  if (!gate_up || !silu_table || !q || !sf) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || inter < 32 || inter % 32 != 0) return fail(RK_EINVAL, "%s: the intermediate size must be a positive multiple of 32", who);
  if (!aligned16(gate_up) || !aligned16(q)) return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  const long long blocks32 = ((rows + 127) / 128 * 128) * ((inter + 127) / 128 * 4);
  const unsigned grid = static_cast<unsigned>((blocks32 * 8 + 255) / 256);
  launch_pdl(pack_mxfp8_kernel<true>, grid, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(gate_up), rows, inter,
             static_cast<uint8_t*>(q), static_cast<uint8_t*>(sf), static_cast<const __nv_bfloat16*>(silu_table));
  return check_launch(who);
}

extern "C" int rk_pack_nvfp4(const void* x, int64_t rows, int64_t k, const float* global_scale, void* q, void* sf,
                             void* stream) {
  if (!x || !q || !sf) return fail(RK_EINVAL, "rk_pack_nvfp4: null pointer");
  if (rows < 1 || k < 32 || k % 32 != 0) return fail(RK_EINVAL, "rk_pack_nvfp4: k must be a positive multiple of 32");
  if (!aligned16(x) || !aligned16(q)) return fail(RK_EINVAL, "rk_pack_nvfp4: pointers must be 16-byte aligned");
  const long long threads = ((rows + 127) / 128 * 128) * ((k / 16 + 3) / 4 * 4);
  const unsigned grid = static_cast<unsigned>((threads + 255) / 256);
  launch_pdl(pack_nvfp4_kernel, grid, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(x), rows, k, global_scale,
                                                         static_cast<uint8_t*>(q), static_cast<uint8_t*>(sf));
  return check_launch("pack_nvfp4");
}

extern "C" int rk_rmsnorm_quant_fp8(const void* x, const void* residual, const void* weight, int64_t rows, int64_t k,
                                    float eps, void* sum_out, void* norm_out, void* q, float* scale_out,
                                    void* workspace, size_t workspace_bytes, void* stream) {
  const char* who = "rk_rmsnorm_quant_fp8";
  if (!x || !weight || !norm_out || !q || !scale_out) return fail(RK_EINVAL, "%s: null pointer", who);
  if (!workspace || workspace_bytes < RK_WORKSPACE_HEADER) return fail(RK_EWORKSPACE, "%s: workspace too small", who);
  if (rows < 1 || k < 16 || k % 16 != 0 || k > rk::kCachedK) return fail(RK_EINVAL, "%s: k must be a multiple of 16, at most %d", who, rk::kCachedK);
  if (!aligned16(x) || !aligned16(weight) || (residual && !aligned16(residual)) || !aligned16(norm_out) ||
      (sum_out && !aligned16(sum_out)))
    return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  cudaStream_t st = as_stream(stream);
  unsigned* staging = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(workspace) + 64);
  auto b = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  launch_pdl(rk::rmsnorm_producer_kernel<0>, static_cast<unsigned>(rows), rk::kRowThreads, st, 
      b(x), b(residual), b(weight), static_cast<int>(rows), static_cast<int>(k), eps,
      static_cast<__nv_bfloat16*>(sum_out), static_cast<__nv_bfloat16*>(norm_out), staging, nullptr, nullptr);
  launch_pdl(rk::finalize_scale_kernel, 1, 1, st, staging, 448.0f, scale_out);
  int rc = check_launch(who);
  if (rc != RK_OK) return rc;
  return rk_quant_tensor_fp8_with_scale(norm_out, rows * k, scale_out, q, stream);
}

extern "C" int rk_swiglu_quant_fp8(const void* gate_up, int64_t rows, int64_t inter, const float* scale_in, void* q,
                                   float* scale_out, void* workspace, size_t workspace_bytes, void* stream) {
  const char* who = "rk_swiglu_quant_fp8";
  if (!gate_up || !q || (!scale_in && !scale_out)) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || inter < 16 || inter % 16 != 0) return fail(RK_EINVAL, "%s: the intermediate size must be a multiple of 16", who);
  if (!aligned16(gate_up) || (reinterpret_cast<uintptr_t>(q) & 7u)) return fail(RK_EINVAL, "%s: bad alignment", who);
  cudaStream_t st = as_stream(stream);
  const long long elements = rows * inter;
  long long blocks = (elements + 2047) / 2048;
  if (blocks > 2368) blocks = 2368;
  const float* scale = scale_in;
  if (scale_in == nullptr) {
    if (!workspace || workspace_bytes < RK_WORKSPACE_HEADER) return fail(RK_EWORKSPACE, "%s: workspace too small", who);
    unsigned* staging = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(workspace) + 64);
    launch_pdl(rk::swiglu_amax_kernel, static_cast<unsigned>(blocks > 1184 ? 1184 : blocks), 256, st, 
        static_cast<const __nv_bfloat16*>(gate_up), rows, inter, staging, nullptr);
    launch_pdl(rk::finalize_scale_kernel, 1, 1, st, staging, 448.0f, scale_out);
    scale = scale_out;
  }
  launch_pdl(rk::swiglu_to_fp8_kernel, static_cast<unsigned>(blocks), 256, st, static_cast<const __nv_bfloat16*>(gate_up), rows,
                                                                          inter, scale, static_cast<uint8_t*>(q));
  return check_launch(who);
}

extern "C" int rk_swiglu_quant_fp8_product(const void* gate_up, int64_t rows, int64_t inter, void* product, void* q,
                                           float* scale_out, void* workspace, size_t workspace_bytes, void* stream) {
  const char* who = "rk_swiglu_quant_fp8_product";
  if (!gate_up || !product || !q || !scale_out) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || inter < 16 || inter % 16 != 0) return fail(RK_EINVAL, "%s: the intermediate size must be a multiple of 16", who);
  if (!aligned16(gate_up) || !aligned16(product) || (reinterpret_cast<uintptr_t>(q) & 7u)) return fail(RK_EINVAL, "%s: bad alignment", who);
  if (!workspace || workspace_bytes < RK_WORKSPACE_HEADER) return fail(RK_EWORKSPACE, "%s: workspace too small", who);
  cudaStream_t st = as_stream(stream);
  unsigned* staging = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(workspace) + 64);
  const long long blocks = (rows * inter + 2047) / 2048;
  launch_pdl(rk::swiglu_amax_kernel, static_cast<unsigned>(blocks > 1184 ? 1184 : blocks), 256, st,
             static_cast<const __nv_bfloat16*>(gate_up), rows, inter, staging, static_cast<__nv_bfloat16*>(product));
  launch_pdl(rk::finalize_scale_kernel, 1, 1, st, staging, 448.0f, scale_out);
  return rk_quant_tensor_fp8_with_scale(product, rows * inter, scale_out, q, stream);
}

extern "C" int rk_rmsnorm_pack_nvfp4(const void* x, const void* residual, const void* weight, int64_t rows, int64_t k,
                                     float eps, void* sum_out, void* norm_out, void* q, void* sf, void* stream) {
  const char* who = "rk_rmsnorm_pack_nvfp4";
  if (!x || !weight || !q || !sf) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || k < 32 || k % 32 != 0 || k > rk::kCachedK) return fail(RK_EINVAL, "%s: k must be a multiple of 32, at most %d", who, rk::kCachedK);
  if (!aligned16(x) || !aligned16(weight) || (residual && !aligned16(residual)) || !aligned16(q) ||
      (sum_out && !aligned16(sum_out)) || (norm_out && !aligned16(norm_out)))
    return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  auto b = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  const unsigned rows_padded = static_cast<unsigned>((rows + 127) / 128 * 128);
  launch_pdl(rk::rmsnorm_producer_kernel<1>, rows_padded, rk::kRowThreads, as_stream(stream), 
      b(x), b(residual), b(weight), static_cast<int>(rows), static_cast<int>(k), eps,
      static_cast<__nv_bfloat16*>(sum_out), static_cast<__nv_bfloat16*>(norm_out), nullptr, static_cast<uint8_t*>(q),
      static_cast<uint8_t*>(sf));
  return check_launch(who);
}

extern "C" int rk_rmsnorm_bf16(const void* x, const void* residual, const void* weight, int64_t rows, int64_t k, float eps,
                               void* sum_out, void* norm_out, void* stream) {
  const char* who = "rk_rmsnorm_bf16";
  if (!x || !weight || !norm_out || (residual && !sum_out)) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || k < 16 || k % 16 != 0 || k > rk::kCachedK) return fail(RK_EINVAL, "%s: k must be a multiple of 16, at most %d", who, rk::kCachedK);
  if (!aligned16(x) || !aligned16(weight) || (residual && !aligned16(residual)) || !aligned16(norm_out) ||
      (sum_out && !aligned16(sum_out)))
    return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  auto b = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  launch_pdl(rk::rmsnorm_producer_kernel<2>, static_cast<unsigned>(rows), rk::kRowThreads, as_stream(stream),
             b(x), b(residual), b(weight), static_cast<int>(rows), static_cast<int>(k), eps,
             static_cast<__nv_bfloat16*>(sum_out), static_cast<__nv_bfloat16*>(norm_out), nullptr, nullptr, nullptr);
  return check_launch(who);
}

extern "C" int rk_silu_mul_bf16(const void* gate_up, int64_t rows, int64_t inter, int interleaved, void* out, void* stream) {
  const char* who = "rk_silu_mul_bf16";
  if (!gate_up || !out) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || inter < 8 || inter % 8 != 0) return fail(RK_EINVAL, "%s: the intermediate size must be a positive multiple of 8", who);
  if (interleaved && inter % 64 != 0) return fail(RK_EINVAL, "%s: the interleaved layout needs a multiple of 64 columns", who);
  if (!aligned16(gate_up) || !aligned16(out)) return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  const long long vectors = rows * inter / 8;
  const unsigned blocks = static_cast<unsigned>(std::min<long long>((vectors + 255) / 256, 148LL * 8));
  launch_pdl(rk::silu_mul_bf16_kernel, blocks, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(gate_up), rows, inter,
             interleaved, static_cast<__nv_bfloat16*>(out));
  return check_launch(who);
}

extern "C" int rk_swiglu_pack_nvfp4_layout(const void* gate_up, int64_t rows, int64_t inter, int interleaved, void* q,
                                           void* sf, void* stream) {
  const char* who = "rk_swiglu_pack_nvfp4";
  if (!gate_up || !q || !sf) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || inter < 32 || inter % 32 != 0) return fail(RK_EINVAL, "%s: the intermediate size must be a multiple of 32", who);
  if (interleaved && inter % 64 != 0) return fail(RK_EINVAL, "%s: the interleaved layout needs a multiple of 64 columns", who);
  if (!aligned16(gate_up) || !aligned16(q)) return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  const long long threads = ((rows + 127) / 128 * 128) * ((inter / 16 + 3) / 4 * 4);
  const unsigned grid = static_cast<unsigned>((threads + 255) / 256);
  launch_pdl(rk::swiglu_pack_nvfp4_kernel, grid, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(gate_up), rows, inter,
                                                                   interleaved ? 1 : 0, static_cast<uint8_t*>(q),
                                                                   static_cast<uint8_t*>(sf));
  return check_launch(who);
}

extern "C" int rk_swiglu_pack_nvfp4(const void* gate_up, int64_t rows, int64_t inter, void* q, void* sf, void* stream) {
  return rk_swiglu_pack_nvfp4_layout(gate_up, rows, inter, 0, q, sf, stream);
}

static int pack_mx_ceil(const void* x, int64_t rows, int64_t k, int fmt, void* q, void* sf, void* stream, const char* who) {
  if (!x || !q || !sf) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || k < 32 || k % 32 != 0) return fail(RK_EINVAL, "%s: k must be a positive multiple of 32", who);
  if (!aligned16(x) || !aligned16(q)) return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  const long long blocks32 = ((rows + 127) / 128 * 128) * ((k + 127) / 128 * 4);
  const unsigned grid = static_cast<unsigned>((blocks32 * 8 + 255) / 256);
  if (fmt == 0)
    launch_pdl(rk::pack_mx_ceil_kernel<0>, grid, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(x), rows, k,
                                                                   static_cast<uint8_t*>(q), static_cast<uint8_t*>(sf));
  else
    launch_pdl(rk::pack_mx_ceil_kernel<1>, grid, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(x), rows, k,
                                                                   static_cast<uint8_t*>(q), static_cast<uint8_t*>(sf));
  return check_launch(who);
}

extern "C" int rk_swiglu_pack_mxfp8_w4a8(const void* gate_up, int64_t rows, int64_t inter, int interleaved, void* q, void* sf,
                                         void* stream) {
  const char* who = "rk_swiglu_pack_mxfp8_w4a8";
  if (!gate_up || !q || !sf) return fail(RK_EINVAL, "%s: null pointer", who);
  if (rows < 1 || inter < 32 || inter % 32 != 0) return fail(RK_EINVAL, "%s: the intermediate size must be a multiple of 32", who);
  if (interleaved && inter % 64 != 0) return fail(RK_EINVAL, "%s: the interleaved layout needs a multiple of 64 columns", who);
  if (!aligned16(gate_up) || !aligned16(q)) return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  const long long blocks32 = ((rows + 127) / 128 * 128) * ((inter + 127) / 128 * 4);
  const unsigned grid = static_cast<unsigned>((blocks32 * 8 + 255) / 256);
  launch_pdl(rk::swiglu_pack_mxfp8_ceil_kernel, grid, 256, as_stream(stream), static_cast<const __nv_bfloat16*>(gate_up), rows, inter,
                                                                        interleaved ? 1 : 0, static_cast<uint8_t*>(q),
                                                                        static_cast<uint8_t*>(sf));
  return check_launch(who);
}

extern "C" int rk_pack_mxfp8_act_w4a8(const void* x, int64_t rows, int64_t k, void* q, void* sf, void* stream) {
  return pack_mx_ceil(x, rows, k, 0, q, sf, stream, "rk_pack_mxfp8_act_w4a8");
}

extern "C" int rk_pack_mxfp4_weight(const void* w, int64_t rows, int64_t k, void* q, void* sf, void* stream) {
  return pack_mx_ceil(w, rows, k, 1, q, sf, stream, "rk_pack_mxfp4_weight");
}

extern "C" int rk_probe_rcp_approx_448(uint32_t* bits) {
  if (!bits) return fail(RK_EINVAL, "rk_probe_rcp_approx_448: null pointer");
  uint32_t* d = nullptr;
  if (cudaMalloc(&d, 4) != cudaSuccess) return fail(RK_ECUDA, "rk_probe_rcp_approx_448: cudaMalloc failed");
  probe_rcp_kernel<<<1, 1>>>(d);
  cudaError_t e = cudaMemcpy(bits, d, 4, cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return fail(RK_ECUDA, "rk_probe_rcp_approx_448: %s", cudaGetErrorString(e));
  return RK_OK;
}
