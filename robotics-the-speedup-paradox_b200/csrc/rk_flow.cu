// What stands between two denoising steps of the flow-matching action expert, in one launch: the last layer's
// pending update, the final adaptive RMS norm, the fp32 output projection, the Euler step and the fp32 input
// projection of the next step (models/pi05/modeling_pi05.py:673-720, 793-889; models/pi05/modeling_gemma.py:62-106).
//
// As tensor ops and library GEMMs these are some twenty dependent launches of 1.5 to 26 us each (76 us of a step with 50 rows:
// the [50, 1024] x [32, 1024] fp32 GEMM alone 26); the work is 0.1 MB of rows and two 128 KB weights.
// Arithmetic of the tensor ops, rounding for rounding; only the order of the fp32 sums is this kernel's own:
//   x' = bf16(x + bf16(branch * gate));  h = bf16(x' * rsqrt(mean(x'^2) + eps) * (1 + scale) + shift)
//   x_next = x_t + dt * (h . w_out + b_out);  tokens = bf16(x_next . w_in + b_in)
//
// One CTA takes R rows, so that its 256 KB of weights from L2 serve R rows: one row each while there are SMs for
// them, then two, then four.  Bound by latency: five dependent phases, each near one L2 round trip, and at 400 rows by the
// weights' way from L2 (25 MB).  In the chunk: 76 -> 9 us a step with 50 rows, 85 -> 16 us with 400.

#include <cuda_bf16.h>

#include <type_traits>

#include "rk_common.cuh"
#include "rk_host.h"

namespace rk {
namespace {

constexpr int kFlowThreads = 256;
constexpr int kFlowMaxK = 2048;
constexpr int kFlowMaxD = 64;

struct FlowParams {
  const __nv_bfloat16 *x, *branch, *gate;  // [rows, k], [rows, k] or null, [rows / tokens, k] or null
  const float *scale, *shift;              // rows of the modulation, mod_stride apart
  long long mod_stride;
  const float *w_out, *b_out;              // [d, k], [d]
  const float *w_in, *b_in;                // [k, d], [k]
  const float* x_t;                        // [rows, d]
  float* x_next;                           // [rows, d]
  __nv_bfloat16* tokens_out;               // [rows, k] or null
  int rows, tokens, k, d;
  float eps, dt;
};

// U: float4 of input weights per lane of a group of eight (d <= 32 U)
template <int R, int U>
__global__ void __launch_bounds__(kFlowThreads)
flow_step_tail_kernel(const FlowParams p) {
  __shared__ __align__(16) float h[R][kFlowMaxK];
  __shared__ __align__(16) float xs[R][kFlowMaxD];
  __shared__ float partial[R][kFlowThreads / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * R;
  pdl_launch_dependents();
  {
    // the weights, last read a whole step ago, start their way from HBM to L2 while the kernels before this one drain:
    // a request to L2 alone, each CTA a share
    const long long lines = static_cast<long long>(p.k) * p.d / 32;  // 128-byte lines of each weight
    for (long long i = static_cast<long long>(blockIdx.x) * kFlowThreads + threadIdx.x; i < lines; i += static_cast<long long>(gridDim.x) * kFlowThreads) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w_out + i * 32));
      if (p.tokens_out != nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w_in + i * 32));  // the last step may come without
    }
  }
  pdl_wait();

  // ---- update and norm: thread t holds elements 4 t .. 4 t + 3 of every 1024
  constexpr int kParts = kFlowMaxK / (4 * kFlowThreads);
  float v[R][kParts][4];
  float sum[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = min(row0 + r, p.rows - 1);
    const long long at = static_cast<long long>(row) * p.k;
    const long long gat = static_cast<long long>(row / p.tokens) * p.k;
    sum[r] = 0.0f;
#pragma unroll
    for (int q = 0; q < kParts; ++q) {
      const int c = q * 4 * kFlowThreads + threadIdx.x * 4;
      v[r][q][0] = v[r][q][1] = v[r][q][2] = v[r][q][3] = 0.0f;
      if (c >= p.k) continue;
      const uint2 w = *reinterpret_cast<const uint2*>(p.x + at + c);
      float e[4] = {bf16_bits_to_float(w.x & 0xFFFFu), __uint_as_float(w.x & 0xFFFF0000u), bf16_bits_to_float(w.y & 0xFFFFu),
                    __uint_as_float(w.y & 0xFFFF0000u)};
      if (p.branch != nullptr) {
        const uint2 bw = *reinterpret_cast<const uint2*>(p.branch + at + c);
        float u[4] = {bf16_bits_to_float(bw.x & 0xFFFFu), __uint_as_float(bw.x & 0xFFFF0000u), bf16_bits_to_float(bw.y & 0xFFFFu),
                      __uint_as_float(bw.y & 0xFFFF0000u)};
        if (p.gate != nullptr) {
          const uint2 gw = *reinterpret_cast<const uint2*>(p.gate + gat + c);
          const float g[4] = {bf16_bits_to_float(gw.x & 0xFFFFu), __uint_as_float(gw.x & 0xFFFF0000u),
                              bf16_bits_to_float(gw.y & 0xFFFFu), __uint_as_float(gw.y & 0xFFFF0000u)};
#pragma unroll
          for (int i = 0; i < 4; ++i) u[i] = __bfloat162float(__float2bfloat16_rn(__fmul_rn(u[i], g[i])));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = __bfloat162float(__float2bfloat16_rn(__fadd_rn(e[i], u[i])));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[r][q][i] = e[i];
        sum[r] = __fmaf_rn(e[i], e[i], sum[r]);
      }
    }
  }
  float4 sc[R][kParts], sh[R][kParts];  // asked for before the sums are reduced
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const long long mod = static_cast<long long>(min(row0 + r, p.rows - 1) / p.tokens) * p.mod_stride;
#pragma unroll
    for (int q = 0; q < kParts; ++q) {
      const int c = q * 4 * kFlowThreads + threadIdx.x * 4;
      if (c >= p.k) continue;
      sc[r][q] = *reinterpret_cast<const float4*>(p.scale + mod + c);
      sh[r][q] = *reinterpret_cast<const float4*>(p.shift + mod + c);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    sum[r] = warp_sum(sum[r]);
    if (lane == 0) partial[r][warp] = sum[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < kFlowThreads / 32; ++w) total += partial[r][w];
    const float inv = rsqrtf(__fadd_rn(__fdiv_rn(total, static_cast<float>(p.k)), p.eps));
#pragma unroll
    for (int q = 0; q < kParts; ++q) {
      const int c = q * 4 * kFlowThreads + threadIdx.x * 4;
      if (c >= p.k) continue;
      const float s4[4] = {sc[r][q].x, sc[r][q].y, sc[r][q].z, sc[r][q].w};
      const float t4[4] = {sh[r][q].x, sh[r][q].y, sh[r][q].z, sh[r][q].w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        h[r][c + i] = __bfloat162float(__float2bfloat16_rn(
            __fadd_rn(__fmul_rn(__fmul_rn(v[r][q][i], inv), __fadd_rn(1.0f, s4[i])), t4[i])));
    }
  }
  __syncthreads();

  // ---- output projection and Euler step: a warp takes four dimensions at a time, a lane every 32nd float4 of K
  for (int d0 = warp * 4; d0 < p.d; d0 += kFlowThreads / 32 * 4) {
    float acc[4][R], old[R], bias = 0.0f;
    if (lane < 4) bias = p.b_out[d0 + lane];
#pragma unroll
    for (int r = 0; r < R; ++r) old[r] = lane < 4 ? p.x_t[static_cast<long long>(min(row0 + r, p.rows - 1)) * p.d + d0 + lane] : 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[j][r] = 0.0f;
#pragma unroll 4
    for (int c = lane * 4; c < p.k; c += 128) {
      float4 hv[R];
#pragma unroll
      for (int r = 0; r < R; ++r) hv[r] = *reinterpret_cast<const float4*>(&h[r][c]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // d is a multiple of four
        const float4 w = __ldg(reinterpret_cast<const float4*>(p.w_out + static_cast<long long>(d0 + j) * p.k + c));
#pragma unroll
        for (int r = 0; r < R; ++r)
          acc[j][r] = fmaf(w.w, hv[r].w, fmaf(w.z, hv[r].z, fmaf(w.y, hv[r].y, fmaf(w.x, hv[r].x, acc[j][r]))));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[j][r] = warp_sum(acc[j][r]);
    if (lane < 4) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float dot = lane == 0 ? acc[0][r] : lane == 1 ? acc[1][r] : lane == 2 ? acc[2][r] : acc[3][r];
        const int dim = d0 + lane;
        const long long at = static_cast<long long>(min(row0 + r, p.rows - 1)) * p.d + dim;
        const float next = __fadd_rn(old[r], __fmul_rn(p.dt, __fadd_rn(dot, bias)));
        xs[r][dim] = next;
        if (row0 + r < p.rows) p.x_next[at] = next;
      }
    }
  }
  if (p.tokens_out == nullptr) return;
  __syncthreads();

  // ---- input projection of the next step: eight lanes share an output channel (a float4 or two of its weights each), so that
  // a warp's loads are dense; a channel per thread, each with a line of its own, took 9.4 us of a 16.6 us launch
  const int sub = lane & 7;
  float4 xv[U][R];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int r = 0; r < R; ++r)
      xv[u][r] = 4 * (sub + 8 * u) < p.d ? *reinterpret_cast<const float4*>(&xs[r][4 * (sub + 8 * u)]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  constexpr int kBatch = 8;                      // channels of a lane group in flight
  constexpr int kStep = kFlowThreads / 8;        // channels that the CTA takes at a time
  for (int c0 = warp * 4 + (lane >> 3); c0 - (lane >> 3) < p.k; c0 += kBatch * kStep) {
    float4 w[kBatch][U];
    float bias[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int c = min(c0 + i * kStep, p.k - 1);
      const float* const src = p.w_in + static_cast<long long>(c) * p.d;
#pragma unroll
      for (int u = 0; u < U; ++u)
        w[i][u] = 4 * (sub + 8 * u) < p.d ? __ldg(reinterpret_cast<const float4*>(src) + sub + 8 * u) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      bias[i] = p.b_in[c];
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int c = c0 + i * kStep;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float acc = 0.0f;
#pragma unroll
        for (int u = 0; u < U; ++u)
          acc = fmaf(w[i][u].w, xv[u][r].w, fmaf(w[i][u].z, xv[u][r].z, fmaf(w[i][u].y, xv[u][r].y, fmaf(w[i][u].x, xv[u][r].x, acc))));
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        if (sub == 0 && c < p.k && row0 + r < p.rows)
          p.tokens_out[static_cast<long long>(row0 + r) * p.k + c] = __float2bfloat16_rn(__fadd_rn(acc, bias[i]));
      }
    }
  }
}

}  // namespace
}  // namespace rk

extern "C" int rk_flow_step_tail(const void* x, const void* branch, const void* gate, const float* scale, const float* shift,
                                 int64_t mod_stride, int64_t tokens, int64_t rows, int64_t k, float eps, const float* w_out,
                                 const float* b_out, int64_t d, const float* x_t, float dt, const float* w_in,
                                 const float* b_in, float* x_next, void* tokens_out, void* stream) {
  using namespace rk;
  const char* who = "rk_flow_step_tail";
  if (!x || !scale || !shift || !w_out || !b_out || !x_t || !x_next || (tokens_out && (!w_in || !b_in)))
    return fail(RK_EINVAL, "%s: null pointer", who);
  if (gate && !branch) return fail(RK_EINVAL, "%s: a gate needs a branch", who);
  if (rows < 1 || rows > (1 << 24) || tokens < 1 || rows % tokens != 0) return fail(RK_EINVAL, "%s: bad row / token counts", who);
  if (k < 4 || k % 4 != 0 || d < 4 || d % 4 != 0 || (k * d) % 32 != 0) return fail(RK_EINVAL, "%s: k and d must be multiples of 4, k * d of 32", who);
  if (k > kFlowMaxK || d > kFlowMaxD) return fail(RK_EUNSUPPORTED, "%s: k <= %d and d <= %d", who, kFlowMaxK, kFlowMaxD);
  if (mod_stride < k || mod_stride % 4 != 0) return fail(RK_EINVAL, "%s: modulation rows must cover k and be a multiple of 4 apart", who);
  for (const void* ptr : {x, branch, gate, static_cast<const void*>(scale), static_cast<const void*>(shift),
                          static_cast<const void*>(w_out), static_cast<const void*>(w_in)})
    if (!aligned16(ptr)) return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  FlowParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.branch = static_cast<const __nv_bfloat16*>(branch);
  p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.scale = scale;
  p.shift = shift;
  p.mod_stride = mod_stride;
  p.w_out = w_out;
  p.b_out = b_out;
  p.w_in = w_in;
  p.b_in = b_in;
  p.x_t = x_t;
  p.x_next = x_next;
  p.tokens_out = static_cast<__nv_bfloat16*>(tokens_out);
  p.rows = static_cast<int>(rows);
  p.tokens = static_cast<int>(tokens);
  p.k = static_cast<int>(k);
  p.d = static_cast<int>(d);
  p.eps = eps;
  p.dt = dt;
  constexpr int kSms = 148;
  auto launch = [&](auto r) {
    constexpr int R = decltype(r)::value;
    const dim3 grid(static_cast<unsigned>((rows + R - 1) / R));
    if (d <= 32) launch_pdl(flow_step_tail_kernel<R, 1>, grid, dim3(kFlowThreads), as_stream(stream), p);
    else launch_pdl(flow_step_tail_kernel<R, 2>, grid, dim3(kFlowThreads), as_stream(stream), p);
  };
  if (rows <= kSms) launch(std::integral_constant<int, 1>{});
  else if (rows <= 2 * kSms) launch(std::integral_constant<int, 2>{});
  else launch(std::integral_constant<int, 4>{});
  return check_launch(who);
}
