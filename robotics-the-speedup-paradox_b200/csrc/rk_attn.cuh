// Attention of a short block of fresh query tokens over a long cached key / value prefix: the
// action expert's 50 chunk tokens x 8 heads against 816 + 50 keys of one shared KV head
// (models/pi05/modeling_gemma.py:247-274, eager_attention_forward).  Non-causal, no mask.
//
// Arithmetic follows the reference's eager path step by step:
//   s = bf16(q . k) * scaling          (matmul output rounded to bf16, then the bf16 scale)
//   p = bf16( softmax_fp32(s) )        (fp32 max / exp / sum over ALL keys, probabilities to bf16)
//   o = bf16( sum_j p_j v_j )          (fp32 accumulation)
//
// Work decomposition.  The query rows of `G` heads that share a KV head form one 128-lane tile
// (row = token * G + head_in_tile, G * tokens <= 128).  The keys are cut into KS equal slices and a
// thread-block cluster of KS CTAs shares one tile, one slice each, so that 8 x 4 tiles become
// 128 CTAs.  Per CTA:
//   1. S = Q K^T for its slice with tcgen05 kind::f16 MMAs (Q and the K slice staged by TMA in the
//      128-byte swizzle), fp32 accumulators in TMEM;
//   2. softmax threads (two per row) find the maximum m_t of their own scores, take exp(score - m_t) once
//      per score and sum it to l_t; ONE exchange of the pairs (m_t, l_t) through distributed shared memory
//      gives every thread the row's maximum m and sum l = sum_t l_t exp(m_t - m), and its own
//      probabilities are exp(score - m_t) * (exp(m_t - m) / l);
//   3. p is written back to TMEM as packed bf16 (over the scores it replaces) and is the TMEM
//      A operand of the second MMA, O_slice = P V, against V^T tiles (keys contiguous) from TMA;
//   4. the partial outputs are summed across the cluster in rank order; each CTA finishes 256 / KS of the
//      head's columns and stores bf16 rows.  Every warp sends its rows' share of each peer's columns as one
//      bulk copy into that peer's shared memory, counted on an mbarrier there (tiles of at most 104 rows and
//      192 keys); larger tiles park the outputs in their own shared memory and fetch from each other.
// No global scratch, no atomics, fixed summation order.  Every wait is bounded.
//
// Bound by latency: loads, four short MMA phases, three passes over a row and two exchanges, one after the other
// (clock cycles of one CTA, 50 rows, 613 keys in four slices: scores complete 2900, exponentials 5500, statistics exchanged
// 6000, output accumulated 10100, received 12200, stored 14100).  Measured before -> after: scores kept in
// registers, two at a time through packed conversions, statistics written to every peer, outputs by bulk copies: one
// environment, 613 keys 13.0 -> 11.4 us (9.3 with tiles of 50 rows); eight, 866 keys 17.2 -> 15.8.  Fetching the outputs 16
// bytes per thread from the peers took 5000 of 24000 cycles, the packed conversions 2400.
//
// Warp roles (320 threads): warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer, warps 2..9 =
// softmax / epilogue: warp w works on TMEM lanes 32 * (w % 4) .. + 31 (one thread per query row) and
// two warps share each row, taking alternate 32-column chunks.  The softmax stream is latency
// bound (long dependent chains per row), so two warps per scheduler nearly halve it.
#pragma once

#include <cuda.h>

#include "rk_gemm_tc.cuh"

namespace rk {

constexpr int kAttnThreads = 320;
constexpr int kAttnSoftmaxThreads = 256;
constexpr int kAttnDim = 256;                 // head dimension this kernel is built for
constexpr int kAttnQBytes = 128 * 128;        // one 64-element column block of the query tile
constexpr int kAttnSlotBytes = 256 * 128;     // ring slot: a K block (keys x 128 B) or a V^T block (256 x 128 B)
constexpr int kAttnSlots = 4;
constexpr int kAttnPartPitch = kAttnDim + 4;  // floats between two rows of a parked partial output
constexpr int kAttnRingOffset = 4 * kAttnQBytes + 8192;  // the query tile and, after the scores, part of the receive area
constexpr int kAttnSmem = kAttnRingOffset + kAttnSlots * kAttnSlotBytes + 1024;
// Exchange by bulk copies: the query tile, the pad behind it and ring slot 0 (104 KB, all dead once every CTA has its
// scores) receive one KB per row of the tile; slots 1 to 3 hold the value blocks and then what is sent.
constexpr int kAttnPushRows = 104, kAttnPushKeys = 192;

struct AttnParams {
  int tokens, heads, kv_heads, group;  // group = query heads per tile (share one KV head)
  int kv_len;        // valid keys
  int keys;          // keys per slice (multiple of 32, <= 256)
  int splits;        // slices == cluster size
  int push;          // partial outputs travel by bulk copies (rows <= kAttnPushRows, keys <= kAttnPushKeys)
  float scaling;     // applied to the bf16-rounded scores
  int scaling_pow2;  // the scale is a power of two
  __nv_bfloat16* out;  // [batch, tokens, heads, 256]
  int* status;
};

__device__ __forceinline__ float attn_round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
// score as the reference's bf16 tensor ops leave it: the matmul output rounded to bf16, times the scale, rounded again
__device__ __forceinline__ float attn_score(uint32_t acc_bits, float scaling) {
  return attn_round_bf16(attn_round_bf16(__uint_as_float(acc_bits)) * scaling);
}

__device__ __forceinline__ float attn_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void tmem_st_16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ float dsmem_ld_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
  return v;
}

__global__ void __launch_bounds__(kAttnThreads, 1)
rk_attn_prefix_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_vt, const AttnParams p) {
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t bar_q;                    // the query tile has landed
  __shared__ __align__(8) uint64_t bar_full[kAttnSlots];   // K blocks complete phase 0 of slots 0..3, V^T blocks phase 1
  __shared__ __align__(8) uint64_t bar_empty[kAttnSlots];
  __shared__ __align__(8) uint64_t bar_s_full, bar_p_full, bar_o_full;
  __shared__ __align__(8) uint64_t bar_recv;                 // the other slices' partial outputs have arrived (push)
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ int verdict[2];
  __shared__ float2 row_stats[16][128];  // (maximum, sum) per key slice and warp of a row pair, written by every CTA of the cluster

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  uint8_t* const smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
  const uint32_t ring_base = smem_base + kAttnRingOffset;
  const int split = static_cast<int>(cluster_ctarank());
  const int tile = blockIdx.y;                      // head group
  const int b = blockIdx.z;
  const int head0 = tile * p.group;
  const int kv_head = head0 / (p.heads / p.kv_heads);
  const int key0 = split * p.keys;
  const int rows_valid = p.group * p.tokens;
  const int kblocks_v = (p.keys + 63) >> 6;         // V^T blocks of 64 keys

  pdl_launch_dependents();
  if (threadIdx.x == 64) {
    // the cached keys and values start their way from DRAM to L2 while the kernel before this one appends to them
    // (L2 is the coherence point: an early fetch is never stale)
    for (int i = 0; i < 4; ++i)
      asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];"
                   ::"l"(reinterpret_cast<uint64_t>(&tm_k)), "r"(i * 64), "r"(key0), "r"(b * p.kv_heads + kv_head) : "memory");
    for (int i = 0; i < kblocks_v; ++i)
      asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];"
                   ::"l"(reinterpret_cast<uint64_t>(&tm_vt)), "r"(key0 + i * 64), "r"(0), "r"(b * p.kv_heads + kv_head) : "memory");
  }
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar_q), 1);
    for (int s = 0; s < kAttnSlots; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_s_full), 1);
    mbar_init(smem_u32(&bar_p_full), kAttnSoftmaxThreads);
    mbar_init(smem_u32(&bar_o_full), 1);
    mbar_init(smem_u32(&bar_recv), 1);
    abort_flag = 0;
    fence_barrier_init();
    if (p.push) mbar_arrive_expect_tx(smem_u32(&bar_recv), static_cast<uint32_t>((p.splits - 1) * rows_valid * (1024 / p.splits)));
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_vt);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_slot), 512u);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // every CTA of the cluster runs: its shared memory may be written
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem_base = tmem_base_slot;
  const uint32_t tmem_s = tmem_base;         // scores (fp32, `keys` columns), later the packed probabilities
  const uint32_t tmem_o = tmem_base + 256;   // output accumulator, 256 columns

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    const uint32_t on = elect_one();
    const uint64_t pol_keep = l2_policy_evict_last();  // Q is read by KS CTAs, K / V by every tile of the batch row
    mbar_arrive_expect_tx(smem_u32(&bar_q), static_cast<uint32_t>(4 * rows_valid * 128), on);
    for (int kb = 0; kb < 4; ++kb)
      asm volatile(
          "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %7, 0;\n\t"
          "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
          " [%0], [%1, {%3, %4, %5}], [%2], %6;\n\t}"
          ::"r"(smem_base + kb * kAttnQBytes), "l"(reinterpret_cast<uint64_t>(&tm_q)), "r"(smem_u32(&bar_q)), "r"(kb * 64),
            "r"(head0), "r"(b * p.tokens), "l"(pol_keep), "r"(on)
          : "memory");
    // four K blocks (64 of the 256 dimensions each), then the V^T blocks (64 keys each) as the slots free up
    for (int i = 0; i < 4 + kblocks_v; ++i) {
      const int s = (i + (i >= kAttnSlots ? p.push : 0)) & (kAttnSlots - 1);
      if (i >= kAttnSlots &&
          !mbar_wait_bounded(smem_u32(&bar_empty[s]), ((i / kAttnSlots) & 1) ^ 1, &abort_flag, p.status, RK_DEV_TIMEOUT_EMPTY))
        break;
      const uint32_t full = smem_u32(&bar_full[s]);
      const uint32_t dst = ring_base + s * kAttnSlotBytes;
      if (i < 4) {
        mbar_arrive_expect_tx(full, static_cast<uint32_t>(p.keys * 128), on);
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %7, 0;\n\t"
            "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
            " [%0], [%1, {%3, %4, %5}], [%2], %6;\n\t}"
            ::"r"(dst), "l"(reinterpret_cast<uint64_t>(&tm_k)), "r"(full), "r"(i * 64), "r"(key0),
              "r"(b * p.kv_heads + kv_head), "l"(pol_keep), "r"(on)
            : "memory");
      } else {
        mbar_arrive_expect_tx(full, static_cast<uint32_t>(kAttnSlotBytes), on);
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %7, 0;\n\t"
            "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
            " [%0], [%1, {%3, %4, %5}], [%2], %6;\n\t}"
            ::"r"(dst), "l"(reinterpret_cast<uint64_t>(&tm_vt)), "r"(full), "r"(key0 + (i - 4) * 64), "r"(0),
              "r"(b * p.kv_heads + kv_head), "l"(pol_keep), "r"(on)
            : "memory");
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t on = elect_one();
    bool alive = mbar_wait_bounded(smem_u32(&bar_q), 0, &abort_flag, p.status, RK_DEV_TIMEOUT_FULL);
    tc_fence_after();
    const uint32_t idesc_s = umma_idesc(DFMT_F32, FMT_BF16, FMT_BF16, 128, static_cast<uint32_t>(p.keys));
    const uint32_t idesc_o = umma_idesc(DFMT_F32, FMT_BF16, FMT_BF16, 128, 256);
    // S = Q K^T: four column blocks of 64 dimensions, four MMAs (16 dimensions) each
    for (int kb = 0; kb < 4 && alive; ++kb) {
      if (!mbar_wait_bounded(smem_u32(&bar_full[kb]), 0, &abort_flag, p.status, RK_DEV_TIMEOUT_FULL)) {
        alive = false;
        break;
      }
      tc_fence_after();
      const uint64_t ad = umma_desc_k128(smem_base + kb * kAttnQBytes);
      const uint64_t bd = umma_desc_k128(ring_base + kb * kAttnSlotBytes);
#pragma unroll
      for (int k = 0; k < 4; ++k) mma_f16(tmem_s, ad + k * 2, bd + k * 2, idesc_s, (kb > 0 || k > 0) ? 1u : 0u, on);
      tc_commit(smem_u32(&bar_empty[kb]), on);  // the slot may take a V^T block
    }
    if (alive) tc_commit(smem_u32(&bar_s_full), on);
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // #1
    // O = P V: the probabilities are the TMEM A operand (two bf16 per column), V^T blocks of 64 keys
    alive = alive && mbar_wait_bounded(smem_u32(&bar_p_full), 0, &abort_flag, p.status, RK_DEV_TIMEOUT_XFORM);
    tc_fence_after();
    const int mmas = p.keys >> 4;  // 16 keys per MMA
    for (int j = 0; j < kblocks_v && alive; ++j) {
      const int i = 4 + j, s = (i + p.push) & (kAttnSlots - 1);
      if (!mbar_wait_bounded(smem_u32(&bar_full[s]), (i / kAttnSlots) & 1, &abort_flag, p.status, RK_DEV_TIMEOUT_FULL)) {
        alive = false;
        break;
      }
      tc_fence_after();
      const uint64_t bd = umma_desc_k128(ring_base + s * kAttnSlotBytes);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int kk = j * 4 + k;
        if (kk < mmas) mma_f16_ts(tmem_o, tmem_s + kk * 8, bd + k * 2, idesc_o, kk > 0 ? 1u : 0u, on);
      }
      tc_commit(smem_u32(&bar_empty[s]), on);
    }
    if (alive) tc_commit(smem_u32(&bar_o_full), on);
  } else {
    // ------------------------------------------------------------ softmax / epilogue: two threads per query row
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;  // which of the row's two threads: chunks half, half + 2, ...
    const int r = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const float log2e = 1.4426950408889634f;
    const int valid = min(p.keys, p.kv_len - key0);  // keys of this slice that exist (may be <= 0 for a trailing slice)
    const bool active = quad * 32 < rows_valid;
    bool ok = mbar_wait_group(smem_u32(&bar_s_full), 0, threadIdx.x == 64, 1, kAttnSoftmaxThreads, &abort_flag, p.status,
                              RK_DEV_TIMEOUT_ACC, verdict, 0);
    tc_fence_after();
    // The thread's scores (up to four chunks of 32 columns) are read from tensor memory once and stay in registers through
    // all three passes.  Warps whose 32 rows lie beyond the tile's rows have nothing to do but take part in the barriers.
    uint32_t s[4][32];
    float m_own = -INFINITY, l_own = 0.0f;
    if (active) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c0 = half * 32 + i * 64;
        __syncwarp();
        if (c0 < p.keys) tmem_ld_32(tmem_s + lane_addr + c0, s[i]);
      }
      tc_wait_ld();
      // pass 1: the maximum of this thread's chunks.  Rounding to bf16 and the positive scale are
      // monotonic, so the maximum of the scores is the score of the largest raw accumulator.
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int left = valid - (half * 32 + i * 64);  // keys of this chunk that exist
        if (left >= 32) {
#pragma unroll
          for (int j = 0; j < 32; ++j) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(s[i][j]));
        } else if (left > 0) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < left) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(s[i][j]));
        }
      }
      const float m_raw = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      m_own = m_raw > -INFINITY ? attn_score(__float_as_uint(m_raw), p.scaling) : -INFINITY;
      // pass 2: e = exp(score - m_own) once per score, summed, kept in place of the score.  A share of -infinities,
      // or of scores so low (below -2.3e38) that m_own * log2e overflows, gives e = 0 and a sum of zero, not infinity - infinity:
      // beside any larger score of the row it weighs nothing.
      const float mneg = fminf(-m_own * log2e, 3.4028234664e38f);
      float2 l01 = make_float2(0.0f, 0.0f), l23 = l01;
      // A scale that is a power of two makes the second rounding of the score the identity and folds into log2e, exactly:
      // one packed conversion and one packed FMA serve two scores (the general form pays two conversions for each).
      const float factor = p.scaling * log2e;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c0 = half * 32 + i * 64;
        const int left = valid - c0;
        if (c0 >= p.keys) continue;
        if (p.scaling_pow2) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const uint32_t w0 = pack_bf16x2(__uint_as_float(s[i][j]), __uint_as_float(s[i][j + 1]));
            const uint32_t w1 = pack_bf16x2(__uint_as_float(s[i][j + 2]), __uint_as_float(s[i][j + 3]));
            const float2 f2 = make_float2(factor, factor), n2 = make_float2(mneg, mneg);
            const float2 x0 = __ffma2_rn(make_float2(__uint_as_float(w0 << 16), __uint_as_float(w0 & 0xFFFF0000u)), f2, n2);
            const float2 x1 = __ffma2_rn(make_float2(__uint_as_float(w1 << 16), __uint_as_float(w1 & 0xFFFF0000u)), f2, n2);
            s[i][j] = __float_as_uint(attn_ex2(x0.x)), s[i][j + 1] = __float_as_uint(attn_ex2(x0.y));
            s[i][j + 2] = __float_as_uint(attn_ex2(x1.x)), s[i][j + 3] = __float_as_uint(attn_ex2(x1.y));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            s[i][j] = __float_as_uint(attn_ex2(fmaf(attn_score(s[i][j], p.scaling), log2e, mneg)));
        }
        if (left < 32) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j >= left) s[i][j] = 0u;
        }
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          l01 = __fadd2_rn(l01, make_float2(__uint_as_float(s[i][j]), __uint_as_float(s[i][j + 1])));
          l23 = __fadd2_rn(l23, make_float2(__uint_as_float(s[i][j + 2]), __uint_as_float(s[i][j + 3])));
        }
      }
      l_own = (l01.x + l01.y) + (l23.x + l23.y);
      // the pair goes to every CTA of the cluster: after the barrier each reads the row's pairs from its own shared memory
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q < p.splits) {
          uint32_t dst;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_u32(&row_stats[2 * split + half][r])), "r"(q));
          asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dst), "f"(m_own), "f"(l_own) : "memory");
        }
      }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // #1
    if (active) {
      // the row's 2 * KS pairs (maximum, sum)
      float2 part[16];
      float m_glob = -INFINITY;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        part[q] = make_float2(-INFINITY, 0.0f);
        if (q < 2 * p.splits) part[q] = row_stats[q][r];
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) m_glob = fmaxf(m_glob, part[q].x);
      float l_glob = 0.0f;
#pragma unroll
      for (int q = 0; q < 16; ++q)  // fixed order: slice 0 (even chunks, odd chunks), slice 1, ...; a part without keys adds zero
        if (q < 2 * p.splits) l_glob = fmaf(part[q].y, part[q].x > -INFINITY ? attn_ex2((part[q].x - m_glob) * log2e) : 0.0f, l_glob);
      const float own = m_own > -INFINITY ? attn_ex2((m_own - m_glob) * log2e) : 0.0f;
      // a row with nothing above those lowest scores has no probabilities: NaN, as softmax of all -infinity gives
      const float inv_l = l_glob > 0.0f ? __fdiv_rn(own, l_glob) : (m_glob < 0.0f ? __uint_as_float(0x7FC00000u) : 0.0f);
      // pass 3: probabilities as packed bf16 over the scores (packed column j covers the fp32 columns 2j, 2j + 1; every
      // thread of the row has read its scores before the barrier).
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c0 = half * 32 + i * 64;
        if (c0 >= p.keys) continue;
        uint32_t w[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
          w[j] = pack_bf16x2(__uint_as_float(s[i][2 * j]) * inv_l, __uint_as_float(s[i][2 * j + 1]) * inv_l);
        __syncwarp();
        tmem_st_16(tmem_s + lane_addr + (c0 >> 1), w);
      }
    }
    tc_wait_st();
    tc_fence_before();
    mbar_arrive(smem_u32(&bar_p_full));
    ok = mbar_wait_group(smem_u32(&bar_o_full), 0, threadIdx.x == 64, 1, kAttnSoftmaxThreads, &abort_flag, p.status,
                         RK_DEV_TIMEOUT_ACC, verdict, 1) && ok;
    tc_fence_after();
    if (p.push) {
      // Each of the row's two threads takes 128 columns, slice by slice: a slice is [rows][256 / splits] fp32 with its 16-byte
      // chunks permuted by row (bank conflicts), the same at its source and destination.  A warp's rows are contiguous: it
      // sends them itself, one bulk copy per peer.  Always sent, also after a failed wait: the peers count the bytes.
      const int slice_bytes = 1024 / p.splits;
      const int per_warp = p.splits >= 2 ? p.splits >> 1 : 1;  // slices that this thread's columns span
      const int cols = 256 / p.splits;
      const int warp_rows = min(32, rows_valid - quad * 32);
      for (int u = 0; u < per_warp && active; ++u) {
        const int dest = half * per_warp + u;
        const uint32_t slot = static_cast<uint32_t>(rows_valid * slice_bytes);
        const uint32_t local = dest == split ? split * slot : kAttnRingOffset + kAttnSlotBytes + (dest < split ? dest : dest - 1) * slot;
        uint8_t* const row = smem_gen + local + r * slice_bytes;
        for (int c0 = 0; c0 < cols; c0 += 32) {
          uint32_t a[32];
          __syncwarp();
          tmem_ld_32(tmem_o + lane_addr + dest * cols + c0, a);
          tc_wait_ld();
          if (r < rows_valid) {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              *reinterpret_cast<uint4*>(row + ((((c0 + j) >> 2) ^ (r & 7)) << 4)) =
                  ok ? make_uint4(a[j], a[j + 1], a[j + 2], a[j + 3]) : make_uint4(0u, 0u, 0u, 0u);
          }
        }
        if (dest == split) continue;
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          uint32_t dst, bar;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_base + split * slot + quad * 32 * slice_bytes), "r"(dest));
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_u32(&bar_recv)), "r"(dest));
          asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       ::"r"(dst), "r"(smem_base + local + quad * 32 * slice_bytes), "r"(warp_rows * slice_bytes), "r"(bar) : "memory");
        }
        __syncwarp();
      }
    } else {
      // park this slice's partial output by rows ([128][kAttnPartPitch] fp32; the pitch spreads a column's 16-byte
      // stores over all banks) over the operand buffers: every MMA that read them has completed.  Each of the row's two
      // threads takes 128 columns.
      float* const part = reinterpret_cast<float*>(smem_gen) + r * kAttnPartPitch;
      for (int c0 = half * 128; c0 < half * 128 + 128 && active; c0 += 32) {
        uint32_t a[32];
        __syncwarp();
        tmem_ld_32(tmem_o + lane_addr + c0, a);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<uint4*>(part + c0 + j) = ok ? make_uint4(a[j], a[j + 1], a[j + 2], a[j + 3]) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }
  if (warp == 0) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // #1
  }

  // ---------------------------------------------------------------- sum the slices across the cluster
  // this CTA finishes 256 / splits columns of every row: an item is four columns of a row, summed in slice order
  const int quads = 64 / p.splits;           // items per row: 64, 32, 16 or 8
  const int shift = 31 - __clz(quads);
  const int c_lo = split * 4 * quads;
  auto store_item = [&](int r, int c, const float4& x) {
    const int token = r / p.group, head = head0 + r % p.group;
    *reinterpret_cast<uint2*>(p.out + ((static_cast<long long>(b) * p.tokens + token) * p.heads + head) * kAttnDim + c) =
        make_uint2(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w));
  };
  __syncthreads();
  if (p.push) {
    // The peers send whatever became of their own waits, so this one does not give up before its limit when a role of this
    // CTA has: nobody may leave while copies to it are in flight.
    if (threadIdx.x == 0) {
      int never = 0;
      if (!mbar_wait_bounded(smem_u32(&bar_recv), 0, &never, p.status, RK_DEV_TIMEOUT_ACC)) abort_flag = 1;
    }
    __syncthreads();
    // what this CTA sent has arrived once its receivers have passed here; it stays until then (the wait is at the end)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // #2 orders no data, only the exits
    const uint32_t slot = static_cast<uint32_t>(rows_valid) << (shift + 4);
    const bool dead = *reinterpret_cast<volatile int*>(&abort_flag) != 0;
    for (int i = threadIdx.x; i < (rows_valid << shift) && !dead; i += kAttnThreads) {
      const int r = i >> shift, ch = i & (quads - 1);
      const uint8_t* const src = smem_gen + (r << (shift + 4)) + ((ch ^ (r & 7)) << 4);
      float4 x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < p.splits) x[q] = *reinterpret_cast<const float4*>(src + q * slot);
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (q < p.splits) x[0].x += x[q].x, x[0].y += x[q].y, x[0].z += x[q].z, x[0].w += x[q].w;
      store_item(r, c_lo + ch * 4, x[0]);
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // #2
  } else {
    cluster_sync_all();  // #2: every CTA's partial output is in its shared memory
    uint32_t peer[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      peer[q] = 0;
      if (q < p.splits) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer[q]) : "r"(smem_base), "r"(q));
    }
    const bool dead = *reinterpret_cast<volatile int*>(&abort_flag) != 0;
    for (int i = threadIdx.x; i < (rows_valid << shift) && !dead; i += kAttnThreads) {
      const int r = i >> shift, c = c_lo + (i & (quads - 1)) * 4;
      float4 x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // all loads first, then the sums in slice order
        x[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (q < p.splits)
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(x[q].x), "=f"(x[q].y), "=f"(x[q].z), "=f"(x[q].w)
                       : "r"(peer[q] + static_cast<uint32_t>(r * kAttnPartPitch + c) * 4u) : "memory");
      }
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (q < p.splits) x[0].x += x[q].x, x[0].y += x[q].y, x[0].z += x[q].z, x[0].w += x[q].w;
      store_item(r, c, x[0]);
    }
    __syncwarp();
    cluster_sync_all();  // #3: nobody leaves while a peer may still read its shared memory
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512u);
  }
}

}  // namespace rk
