// Device helpers shared by the packers (rk_quant.cu) and by GEMM epilogues that re-quantize their
// output: the 128 x 4 scale-factor layout, one NVFP4 block, SwiGLU in the reference's bf16 steps.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include <cstdint>

#include "rk_common.cuh"

namespace rk {
namespace {

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// byte offset of the factor of (row, group) in the swizzled scale-factor buffer; kt = 512-byte chunks per 128-row block
__device__ __forceinline__ long long sf_offset(long long row, long long group, long long kt) {
  return ((row / 128) * kt + group / 4) * 512 + (row % 32) * 16 + ((row % 128) / 32) * 4 + group % 4;
}

__device__ __forceinline__ float rcp_approx_ftz(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// smallest power of two >= x as a biased exponent byte (x >= 0, finite)
__device__ __forceinline__ uint32_t ue8m0_roundup(float x) {
  const uint32_t b = __float_as_uint(x);
  const uint32_t e = (b >> 23) & 0xFFu, mant = b & 0x7FFFFFu;
  uint32_t r = e == 0 ? (mant > 0x400000u ? 1u : 0u) : e + (mant != 0u ? 1u : 0u);
  return r > 254u ? 254u : r;
}

// MXFP8 block of 32 (blackwell/csrc/mxfp8_common.cuh:12-32): the UE8M0 scale byte of a block with absolute
// maximum `amax` (255 when the block holds a non-finite value), and the multiplier 2^(127 - e) that goes with it,
// built as the exponent byte 254 - e (255 stays NaN, 0 becomes the subnormal 2^-127).
__device__ __forceinline__ uint32_t mxfp8_block_scale(float amax, bool invalid) {
  return invalid ? 255u : ue8m0_roundup(__fmul_rn(amax, rcp_approx_ftz(448.0f)));
}
__device__ __forceinline__ float mxfp8_inverse_scale(uint32_t e) {
  const uint32_t ie = (254u - e) & 255u;
  return ie == 255u ? __uint_as_float(0x7FC00000u) : (ie == 0u ? __uint_as_float(0x00400000u) : __uint_as_float(ie << 23));
}

// ---- two bf16 values at a time.  One rounding of the exact product or sum: the same as rounding the fp32 result to
// bf16 (24 >= 2 * 8 + 2 bits make that second rounding innocuous), except for products below the normal range, where one
// rounding is the closer one.
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hadd2_rn(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// running maximum of magnitudes; like fmaxf, a NaN loses against a number
__device__ __forceinline__ uint32_t absmax_bf16x2(uint32_t m, uint32_t v) {
  v &= 0x7FFF7FFFu;
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&m), *reinterpret_cast<const __nv_bfloat162*>(&v));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// SwiGLU in bf16 steps, as the reference's NVFP4 producer evaluates it with packed bf16 arithmetic
// (blackwell/csrc/fp4_cutlass_linear.cu:1029-1033): every intermediate is rounded to bf16.  Two at a time.
// The reciprocal of a bf16 value d >= 1 is rounded to bf16 at once, so the approximate one (1 ulp of fp32) serves: with
// eight significant bits in d and nine in a rounding boundary, 1 / d is at least 2^-17 (relative) away from every
// boundary unless it lies on one, which only a power of two's reciprocal could, and that is exact.
__device__ __forceinline__ uint32_t swiglu_bf16x2_steps(uint32_t gate, uint32_t up) {
  const uint32_t e = pack_bf16x2(expf(-bf16_lo(gate)), expf(-bf16_hi(gate)));
  const uint32_t d = add_bf16x2(0x3F803F80u, e);
  float r0, r1;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r0) : "f"(bf16_lo(d)));
  asm("rcp.approx.f32 %0, %1;" : "=f"(r1) : "f"(bf16_hi(d)));
  return mul_bf16x2(mul_bf16x2(gate, pack_bf16x2(r0, r1)), up);
}

// One 16-element NVFP4 block: UE4M3 scale byte and eight code bytes (two E2M1 codes each, low nibble first).
// Same arithmetic as pack_nvfp4_kernel (blackwell/csrc/fp4_cutlass_linear.cu:789-841, no per-tensor scale).
// `v`: eight words of two bf16 values.
__device__ __forceinline__ unsigned long long nvfp4_block(const uint32_t (&v)[8], uint8_t* code_out) {
  uint32_t m = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) m = absmax_bf16x2(m, v[i]);
  const float amax = fmaxf(bf16_lo(m), bf16_hi(m));
  const float scale = amax > 0.0f ? __fdiv_rn(amax, 6.0f) : 1.0f;
  const uint8_t code = static_cast<uint8_t>(__nv_cvt_float_to_fp8(scale, __NV_SATFINITE, __NV_E4M3)) & 0x7F;
  float deq = __half2float(__half(__nv_cvt_fp8_to_halfraw(code, __NV_E4M3)));
  if (!(deq > 0.0f)) deq = scale;
  const float reciprocal = __frcp_rn(deq);  // == 1 / deq, correctly rounded
  uint32_t half[2] = {0u, 0u};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __nv_fp4x2_storage_t pair = __nv_cvt_float2_to_fp4x2(
        make_float2(__fmul_rn(bf16_lo(v[i]), reciprocal), __fmul_rn(bf16_hi(v[i]), reciprocal)), __NV_E2M1, cudaRoundNearest);
    half[i >> 2] |= static_cast<uint32_t>(static_cast<uint8_t>(pair)) << (8 * (i & 3));
  }
  *code_out = code;
  return static_cast<unsigned long long>(half[0]) | (static_cast<unsigned long long>(half[1]) << 32);
}

}  // namespace
}  // namespace rk
