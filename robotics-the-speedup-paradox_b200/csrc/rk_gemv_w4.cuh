// W4A16 group-wise int4 products with a handful of activation rows (decode batches of one to sixteen).
//
// Byte-streaming work: two flops per weight and row.  The tensor-memory kernels of rk_gemm_w4.cuh take 128 output channels
// per CTA and expand them through one ring, which leaves them at the latency of that ring; here every warp streams its own
// weights straight into registers and expands them there, and the warps of an SM hide each other's latency.  The
// expanded weights are the A operand of warp-level m16n8k16 MMAs (bf16, fp32 accumulation): sixteen output channels by
// eight activation rows, so that up to eight rows cost what one does.  tcgen05 has nothing to offer at this size: its A
// tile is 128 channels from shared or tensor memory.
//
// A warp owns sixteen output channels and a contiguous share of K's groups; `share` warps of a CTA split a channel tile
// along K and add their totals through shared memory in a fixed order.  Lane (g, t) = (lane / 4, lane % 4) loads the 16
// bytes t of a group's 64 for channels g and g + 8: 32 consecutive weights of each, which are also the K positions that
// the MMA fragments of lane t stand for (any order of K serves, as long as both operands use the same).  The loads
// of four groups are in flight while two are computed.  The activations lie in shared memory in fragment order.
//
// Arithmetic of the kernels above it: nibbles to exact bf16 integers, the group's partial sum in fp32, times the group
// scale in fp32, summed in fp32.
//
// Bound by the integer pipe (7 of some 14 instructions per eight weights are masks and byte permutes) and by the launch
// and the first loads.  16384 x 2048, one row 8.3 -> 7.1 us, 1024 x 1024 2.9 -> 2.1, 2048 x 16384 8.3 -> 7.9, against a kernel that
// multiplied on the FMA pipe (a byte permute and half a packed FMA per weight); eight rows against rk_gemm_w4.cuh 9.1 -> 8.0, 5.4
// -> 2.4 and 13.0 (their activations do not fit here).  Deeper batches (four groups) and three CTAs per SM measured slower.
//
// Packed word format as everywhere: byte b of a word holds weights k_b (low nibble) and k_{b+4}.
#pragma once

#include <cuda_bf16.h>

#include "rk_common.cuh"
#include "rk_gemm_w4.cuh"

namespace rk {

constexpr int kGemvRows = 16;   // output channels per warp
constexpr int kGemvBatch = 2;   // groups per batch of loads; two batches are in flight
// activations and totals of a CTA: two CTAs of eight warps or one of sixteen share an SM
__host__ __device__ constexpr int gemv_smem_limit(int warps) { return warps == 8 ? 96 * 1024 : 200 * 1024; }

struct GemvParams {
  const uint8_t* q;              // [n, k / 2]
  const __nv_bfloat16* scales;   // [k / 128, n]
  const __nv_bfloat16* x;        // [m, k]
  const __nv_bfloat16* bias;     // [n] or null
  __nv_bfloat16* out;            // [m, n]
  int m, n, k;
  int share;                     // warps per channel tile (a power of two up to the warps of a CTA)
};

// bytes of one activation row in fragment order: 64 more than the row, so that the eight rows of a fragment spread over the banks
__host__ __device__ constexpr int gemv_row_bytes(int k) { return 2 * k + 64; }
// activation rows (one of zeros behind them where they do not fill the fragments), then the totals
__host__ __device__ constexpr int gemv_sums_offset(int m, int k) { return (m + (m % 8 != 0 ? 1 : 0)) * gemv_row_bytes(k); }
__host__ __device__ constexpr int gemv_smem(int m, int k, int tiles8, int warps) { return gemv_sums_offset(m, k) + warps * tiles8 * 8 * kGemvRows * 4; }

__device__ __forceinline__ void mma_m16n8k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct GemvBatch {
  uint4 w[kGemvBatch][2];             // the 32 weights of channels g and g + 8
  unsigned short scale[kGemvBatch][2];
};

// TILES8: blocks of eight activation rows (m <= 8 * TILES8)
template <int TILES8, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
rk_gemv_w4a16_kernel(const GemvParams p) {
  extern __shared__ __align__(16) uint8_t gemv_smem_dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int tiles_per_cta = WARPS / p.share;
  const int part = warp % p.share;                                  // which share of K
  const int n0 = (blockIdx.x * tiles_per_cta + warp / p.share) * kGemvRows;
  const int groups = p.k >> 7;
  const int first = groups * part / p.share, last = n0 < p.n ? groups * (part + 1) / p.share : 0;
  const long long row_bytes = p.k >> 1;
  // channels beyond n (a multiple of eight: the tile's second half) read the last channel and are not stored
  const int ch[2] = {min(n0 + g, p.n - 1), min(n0 + g + 8, p.n - 1)};
  pdl_launch_dependents();
  if (lane < kGemvRows && n0 + lane < p.n && first < last) {
    // this warp's rows start their way to L2 while the preceding kernel drains (a request to L2 alone)
    const uint8_t* const row = p.q + (n0 + lane) * row_bytes + first * 64;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row), "r"((last - first) * 64) : "memory");
  }
  pdl_wait();  // the activations (and, in tests, freshly packed weights) come from the preceding kernel

  const uint8_t* src[2] = {p.q + ch[0] * row_bytes + first * 64 + t * 16, p.q + ch[1] * row_bytes + first * 64 + t * 16};
  const unsigned short* scale[2] = {reinterpret_cast<const unsigned short*>(p.scales) + static_cast<long long>(first) * p.n + ch[0],
                                    reinterpret_cast<const unsigned short*>(p.scales) + static_cast<long long>(first) * p.n + ch[1]};
  // loads the next `count` groups (the same in all lanes) and moves on
  auto load = [&](GemvBatch& b, int count) {
#pragma unroll
    for (int j = 0; j < kGemvBatch; ++j) {
      if (j >= count) break;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        b.w[j][h] = __ldcs(reinterpret_cast<const uint4*>(src[h]));
        b.scale[j][h] = __ldg(scale[h]);
        src[h] += 64;
        scale[h] += p.n;
      }
    }
  };
  GemvBatch batch[2];
  load(batch[0], last - first);
  load(batch[1], last - first - kGemvBatch);

  // activations in fragment order: eight elements (one word's weights) of group j, lane t, word w at j * 256 + w * 64 + t * 16;
  // the fragment's rows beyond m read a row of zeros
  const int pitch = gemv_row_bytes(p.k);
  for (int i = threadIdx.x; i < p.m * (p.k >> 3); i += WARPS * 32) {
    const int r = i / (p.k >> 3), c = i - r * (p.k >> 3);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;"
                 ::"r"(smem_u32(gemv_smem_dyn) + r * pitch + (c >> 4) * 256 + (c & 3) * 64 + ((c >> 2) & 3) * 16),
                   "l"(p.x + static_cast<long long>(r) * p.k + c * 8) : "memory");
  }
  if (p.m % 8 != 0)
    for (int i = threadIdx.x; i < p.k >> 3; i += WARPS * 32)
      *reinterpret_cast<uint4*>(gemv_smem_dyn + p.m * pitch + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  const uint8_t* xrow[TILES8];
  float total[TILES8][4];
#pragma unroll
  for (int u = 0; u < TILES8; ++u) {
    xrow[u] = gemv_smem_dyn + min(u * 8 + g, p.m) * pitch + first * 256 + t * 16;
    total[u][0] = total[u][1] = total[u][2] = total[u][3] = 0.0f;
  }
  auto compute = [&](const GemvBatch& b, int count) {
#pragma unroll
    for (int j = 0; j < kGemvBatch; ++j) {
      if (j >= count) break;
      const uint32_t lo[4] = {b.w[j][0].x, b.w[j][0].y, b.w[j][0].z, b.w[j][0].w};
      const uint32_t hi[4] = {b.w[j][1].x, b.w[j][1].y, b.w[j][1].z, b.w[j][1].w};
      float acc[TILES8][2][4];  // two chains, so that an MMA does not wait for the one before it
#pragma unroll
      for (int u = 0; u < TILES8; ++u)
#pragma unroll
        for (int c = 0; c < 2; ++c) acc[u][c][0] = acc[u][c][1] = acc[u][c][2] = acc[u][c][3] = 0.0f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const uint4 a = w4_unpack8(lo[w]), c = w4_unpack8(hi[w]);
#pragma unroll
        for (int u = 0; u < TILES8; ++u) {
          const uint4 x = *reinterpret_cast<const uint4*>(xrow[u] + w * 64);
          mma_m16n8k16(acc[u][0], a.x, c.x, a.y, c.y, x.x, x.y);
          mma_m16n8k16(acc[u][1], a.z, c.z, a.w, c.w, x.z, x.w);
        }
      }
      const float s0 = bf16_bits_to_float(b.scale[j][0]), s1 = bf16_bits_to_float(b.scale[j][1]);
#pragma unroll
      for (int u = 0; u < TILES8; ++u) {
        xrow[u] += 256;
        total[u][0] = fmaf(s0, acc[u][0][0] + acc[u][1][0], total[u][0]);
        total[u][1] = fmaf(s0, acc[u][0][1] + acc[u][1][1], total[u][1]);
        total[u][2] = fmaf(s1, acc[u][0][2] + acc[u][1][2], total[u][2]);
        total[u][3] = fmaf(s1, acc[u][0][3] + acc[u][1][3], total[u][3]);
      }
    }
  };
  for (int left = last - first; left > 0; left -= 2 * kGemvBatch) {
    compute(batch[0], left);
    load(batch[0], left - 2 * kGemvBatch);
    compute(batch[1], left - kGemvBatch);
    load(batch[1], left - 3 * kGemvBatch);
  }

  // totals to shared memory as [warp][activation row][channel], then added over the shares of K in order
  float* const sums = reinterpret_cast<float*>(gemv_smem_dyn + gemv_sums_offset(p.m, p.k));
#pragma unroll
  for (int u = 0; u < TILES8; ++u) {
    float* const dst = sums + (warp * TILES8 + u) * 8 * kGemvRows;
    dst[2 * t * kGemvRows + g] = total[u][0];
    dst[(2 * t + 1) * kGemvRows + g] = total[u][1];
    dst[2 * t * kGemvRows + g + 8] = total[u][2];
    dst[(2 * t + 1) * kGemvRows + g + 8] = total[u][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < tiles_per_cta * p.m * kGemvRows; i += WARPS * 32) {
    const int channel = i & (kGemvRows - 1), rest = i / kGemvRows;
    const int tile = rest / p.m, row = rest - tile * p.m;
    const int n = (blockIdx.x * tiles_per_cta + tile) * kGemvRows + channel;
    if (n >= p.n) continue;
    float sum = 0.0f;
    for (int s = 0; s < p.share; ++s) sum += sums[((tile * p.share + s) * TILES8 * 8 + row) * kGemvRows + channel];
    if (p.bias != nullptr) sum += __bfloat162float(p.bias[n]);
    p.out[static_cast<long long>(row) * p.n + n] = __float2bfloat16_rn(sum);
  }
}

}  // namespace rk
