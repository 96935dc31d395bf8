// Rotary position embedding of fresh query / key rows fused with the key / value cache update.
//
// What the flow-matching loop does between the q/k/v projection and the attention of every layer:
// rotate q and k (apply_rotary_pos_emb, models/pi05/modeling_gemma.py:178-209), bring q into
// [batch, heads, tokens, dim] order, and append the rotated keys and the values behind the cached
// prefix (the reference's fused form: fused_cache_update_rope_bf16,
// blackwell/csrc/fp4_cutlass_linear.cu:478-588).  As a chain of tensor ops this is about fourteen
// launches per layer; here it is one.  The cache buffers are preallocated for prefix + tokens rows
// and already hold the prefix, so only the new rows are written.
//
// Arithmetic (identical to bf16 tensor ops and to the reference's rope_element,
// fp4_cutlass_linear.cu:96-126): out = bf16( bf16(x * cos) + bf16(r * sin) ), r = -x[j + d/2] for
// j < d/2 and x[j - d/2] otherwise; three roundings to bf16, fp32 in between.
//
// One warp per (row, rotated head): lane l handles the eight elements [8 l, 8 l + 8) of the head and of its
// rotation partner (16-byte loads and stores); head_dim is a multiple of 16, at most 512.  Values go by tiles of
// 32 rows.  Bound by latency: one trip to memory and back behind the projection.  Indexes are 32-bit (the 64-bit
// divisions took longer than the rotation) and computed before the wait for the projection, and the transposed
// values are written along the keys: a layer of the action chunk is 2.1 us shorter for it with eight environments (400
// rows; the kernel took 4.4) and 0.7 with one.

#include <cuda_bf16.h>

#include "rk_common.cuh"
#include "rk_host.h"

namespace rk {
namespace {

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const uint32_t l = __bfloat16_as_ushort(__float2bfloat16_rn(lo));
  const uint32_t h = __bfloat16_as_ushort(__float2bfloat16_rn(hi));
  return l | (h << 16);
}

// eight rotated elements: x and partner are the raw words, `negate` says whether the partner enters negated
__device__ __forceinline__ uint4 rotate8(const uint4& x, const uint4& partner, const uint4& c, const uint4& s, bool negate) {
  const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, pw[4] = {partner.x, partner.y, partner.z, partner.w};
  const uint32_t cw[4] = {c.x, c.y, c.z, c.w}, sw[4] = {s.x, s.y, s.z, s.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float sign = negate ? -1.0f : 1.0f;
    const float a0 = round_bf16(__fmul_rn(bf16_lo(xw[i]), bf16_lo(cw[i])));
    const float a1 = round_bf16(__fmul_rn(bf16_hi(xw[i]), bf16_hi(cw[i])));
    const float b0 = round_bf16(__fmul_rn(sign * bf16_lo(pw[i]), bf16_lo(sw[i])));
    const float b1 = round_bf16(__fmul_rn(sign * bf16_hi(pw[i]), bf16_hi(sw[i])));
    o[i] = pack2(__fadd_rn(a0, b0), __fadd_rn(a1, b1));
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

struct RopeParams {
  const __nv_bfloat16 *q, *k, *v;        // rows of [heads * dim], [kv_heads * dim], [kv_heads * dim]
  long long q_stride, k_stride, v_stride;  // row strides in elements
  const __nv_bfloat16 *cos, *sin;        // [batch, tokens, dim]
  __nv_bfloat16 *q_out;                  // [batch, heads, tokens, dim], or [batch, tokens, heads, dim] (token_major)
  __nv_bfloat16 *k_all, *v_all;          // [batch, kv_heads, cache_rows, dim]
  __nv_bfloat16 *vt_all;                 // optional transposed values [batch, kv_heads, dim, vt_pitch]
  long long vt_pitch;
  int batch, tokens, heads, kv_heads, dim, cache_rows, prefix, token_major;
};

// Values: a CTA takes kRopeTokens rows of one head (one quarter of its columns), copies them and, through shared memory,
// writes them transposed with the lanes along the keys: a store of a warp covers 64 contiguous bytes.  With the eight values of
// a row stored one by one down a column every store of a warp touched 32 sectors.
constexpr int kRopeWarps = 8, kRopeTokens = 32;
constexpr int kRopeTile = kRopeTokens * (128 + 2);  // elements; also seven rows of the widest head (512 + 2)

__device__ __forceinline__ void append_values(const RopeParams& p, unsigned job, int parts, __nv_bfloat16* tile) {
  const unsigned token_tiles = (p.tokens + kRopeTokens - 1) / kRopeTokens;
  const unsigned plane = job / (token_tiles * parts), rest = job - plane * (token_tiles * parts);  // plane = batch * kv_heads + head
  const int token0 = static_cast<int>(rest / parts) * kRopeTokens, part = static_cast<int>(rest % parts);
  const unsigned b = plane / static_cast<unsigned>(p.kv_heads);
  const int head = static_cast<int>(plane - b * p.kv_heads);
  const int per = (p.dim / 8 + parts - 1) / parts;  // 16-byte vectors of a row that this CTA takes
  const int vec0 = part * per, vecs = min(per, p.dim / 8 - vec0);
  if (vecs <= 0) return;
  const int rows = min(kRopeTokens, p.tokens - token0);
  const __nv_bfloat16* const src = p.v + (static_cast<long long>(b) * p.tokens + token0) * p.v_stride + head * p.dim + vec0 * 8;
  __nv_bfloat16* const dst = p.v_all + (static_cast<long long>(plane) * p.cache_rows + p.prefix + token0) * p.dim + vec0 * 8;
  const int pitch = vecs * 8 + 2;  // an odd number of words: the lanes of a column read 32 banks
  for (int i = threadIdx.x; i < rows * vecs; i += kRopeWarps * 32) {
    const int r = i / vecs, c = (i - r * vecs) * 8;
    const uint4 x = *reinterpret_cast<const uint4*>(src + r * p.v_stride + c);
    *reinterpret_cast<uint4*>(dst + static_cast<long long>(r) * p.dim + c) = x;
    uint32_t* const t = reinterpret_cast<uint32_t*>(tile + r * pitch + c);
    t[0] = x.x, t[1] = x.y, t[2] = x.z, t[3] = x.w;
  }
  if (p.vt_all == nullptr) return;  // the whole block
  __syncthreads();
  const int lane = threadIdx.x & 31;
  if (lane >= rows) return;
  unsigned short* const out =
      reinterpret_cast<unsigned short*>(p.vt_all) + (static_cast<long long>(plane) * p.dim + vec0 * 8) * p.vt_pitch + p.prefix + token0 + lane;
#pragma unroll 4
  for (int c = (threadIdx.x >> 5) * 2; c < vecs * 8; c += kRopeWarps * 2) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(tile + lane * pitch + c);
    out[c * p.vt_pitch] = static_cast<unsigned short>(w & 0xFFFFu);
    out[(c + 1) * p.vt_pitch] = static_cast<unsigned short>(w >> 16);
  }
}

// The first `value_blocks` CTAs append values; in the others a warp rotates one query or key head of a row.
__global__ void __launch_bounds__(kRopeWarps * 32)
rope_cache_update_kernel(const RopeParams p, unsigned value_blocks, int parts) {
  __shared__ __align__(16) __nv_bfloat16 tile[kRopeTile];
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  if (blockIdx.x < value_blocks) {
    pdl_wait();
    append_values(p, blockIdx.x, parts, tile);
    return;
  }
  const int lane = threadIdx.x & 31;
  const unsigned units = p.heads + p.kv_heads;  // per row: query heads, key heads
  const unsigned job = (blockIdx.x - value_blocks) * kRopeWarps + (threadIdx.x >> 5);  // at most 2^31 of them
  const unsigned row = job / units;                                                    // batch * tokens + token
  const int unit = static_cast<int>(job - row * units);
  const unsigned b = row / static_cast<unsigned>(p.tokens);
  const int token = static_cast<int>(row - b * p.tokens);
  const int half = p.dim >> 1;
  const bool is_q = unit < p.heads;
  const int head = is_q ? unit : unit - p.heads;
  const __nv_bfloat16* const src = (is_q ? p.q + row * p.q_stride : p.k + row * p.k_stride) + head * p.dim;
  const __nv_bfloat16* const cs = p.cos + static_cast<long long>(row) * p.dim;
  const __nv_bfloat16* const sn = p.sin + static_cast<long long>(row) * p.dim;
  __nv_bfloat16* const dst =
      is_q ? p.q_out + (p.token_major ? (static_cast<long long>(row) * p.heads + head) * p.dim
                                      : ((static_cast<long long>(b) * p.heads + head) * p.tokens + token) * p.dim)
           : p.k_all + ((static_cast<long long>(b) * p.kv_heads + head) * p.cache_rows + p.prefix + token) * p.dim;
  pdl_wait();
  if (b >= static_cast<unsigned>(p.batch)) return;
  for (int j = lane * 8; j < p.dim; j += 256) {
    const int jp = j < half ? j + half : j - half;
    const uint4 x = *reinterpret_cast<const uint4*>(src + j);
    const uint4 partner = *reinterpret_cast<const uint4*>(src + jp);
    const uint4 c = *reinterpret_cast<const uint4*>(cs + j);
    const uint4 s = *reinterpret_cast<const uint4*>(sn + j);
    *reinterpret_cast<uint4*>(dst + j) = rotate8(x, partner, c, s, j < half);
  }
}

// The cached prefix into one chunk's working caches: keys and values copied row by row, values also transposed
// (columns from `prefix` to the pitch zeroed).  A CTA takes 64 rows of one plane; blockIdx.z = 0 keys, 1 values, whose
// tile passes through shared memory once.  Bound by HBM: every byte is read once and written once (values twice); as four
// tensor-op copies and a fill, whose transposing one stores two bytes at a time, the caches of eight environments (18 layers,
// 816 keys) took 350 us.
constexpr int kFillRows = 64, kFillDim = 256, kFillThreads = 256;
constexpr int kFillPitch = kFillDim + 2;  // elements between two rows of the tile: spreads eight rows over the banks

struct FillParams {
  const __nv_bfloat16 *k, *v;              // [planes, prefix, 256]
  __nv_bfloat16 *k_all, *v_all, *vt_all;   // [planes, cache_rows, 256] twice, [planes, 256, vt_pitch]
  int prefix, cache_rows, vt_pitch;
};

__global__ void __launch_bounds__(kFillThreads)
kv_prefix_fill_kernel(const FillParams p) {
  __shared__ __align__(16) __nv_bfloat16 tile[kFillRows * kFillPitch];
  pdl_launch_dependents();  // every thread, before any return: see launch_pdl
  pdl_wait();
  const int row0 = blockIdx.x * kFillRows;
  const long long plane = blockIdx.y;
  const bool values = blockIdx.z != 0;
  const __nv_bfloat16* const src = (values ? p.v : p.k) + plane * p.prefix * kFillDim;
  __nv_bfloat16* const dst = (values ? p.v_all : p.k_all) + plane * p.cache_rows * kFillDim;
  constexpr int kVecs = kFillRows * kFillDim / 8 / kFillThreads;  // 16-byte vectors per thread
  uint4 x[kVecs];
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int at = i * kFillThreads + threadIdx.x, row = row0 + (at >> 5);
    x[i] = row < p.prefix ? __ldcs(reinterpret_cast<const uint4*>(src + static_cast<long long>(row) * kFillDim) + (at & 31)) : make_uint4(0u, 0u, 0u, 0u);
  }
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int at = i * kFillThreads + threadIdx.x, row = row0 + (at >> 5);
    if (row < p.prefix) *(reinterpret_cast<uint4*>(dst + static_cast<long long>(row) * kFillDim) + (at & 31)) = x[i];
    if (values) {
      uint32_t* const t = reinterpret_cast<uint32_t*>(tile + (at >> 5) * kFillPitch + (at & 31) * 8);
      t[0] = x[i].x, t[1] = x[i].y, t[2] = x[i].z, t[3] = x[i].w;
    }
  }
  if (!values) return;
  __syncthreads();
  // eight lanes write 64 keys (128 bytes) of a row of the transposed cache; a thread takes two rows, eight keys of each
  __nv_bfloat16* const out = p.vt_all + plane * kFillDim * p.vt_pitch + row0;
#pragma unroll
  for (int i = 0; i < kFillRows / 8 * kFillDim / 2 / kFillThreads; ++i) {
    const int at = i * kFillThreads + threadIdx.x, g = at & 7, pair = at >> 3;
    if (row0 + g * 8 >= p.vt_pitch) continue;  // the pitch is a multiple of eight
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const uint32_t*>(tile + (g * 8 + j) * kFillPitch + pair * 2);
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lo[j] = __byte_perm(w[2 * j], w[2 * j + 1], 0x5410);
      hi[j] = __byte_perm(w[2 * j], w[2 * j + 1], 0x7632);
    }
    *reinterpret_cast<uint4*>(out + static_cast<long long>(pair * 2) * p.vt_pitch + g * 8) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    *reinterpret_cast<uint4*>(out + static_cast<long long>(pair * 2 + 1) * p.vt_pitch + g * 8) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  }
}

}  // namespace
}  // namespace rk

static int rope_cache_update_impl(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                                  int64_t v_stride, const void* cos, const void* sin, int64_t batch, int64_t tokens,
                                  int64_t heads, int64_t kv_heads, int64_t head_dim, void* q_out, int q_token_major,
                                  void* k_cache, void* v_cache, int64_t cache_rows, int64_t prefix, void* vt_cache,
                                  int64_t vt_pitch, void* stream, const char* who) {
  using namespace rk;
  if (vt_cache != nullptr && (vt_pitch < prefix + tokens || (reinterpret_cast<uintptr_t>(vt_cache) & 1u)))
    return fail(RK_EINVAL, "%s: the transposed value cache needs a pitch of at least prefix + tokens", who);
  if (!q || !k || !v || !cos || !sin || !q_out || !k_cache || !v_cache) return fail(RK_EINVAL, "%s: null pointer", who);
  if (batch < 1 || tokens < 1 || heads < 1 || kv_heads < 1) return fail(RK_EINVAL, "%s: empty problem", who);
  if (head_dim < 16 || head_dim % 16 != 0 || head_dim > 512)
    return fail(RK_EINVAL, "%s: head_dim must be a multiple of 16 up to 512", who);
  if (prefix < 0 || prefix + tokens > cache_rows) return fail(RK_EINVAL, "%s: the cache holds %lld rows, %lld + %lld needed", who,
                                                           static_cast<long long>(cache_rows), static_cast<long long>(prefix),
                                                           static_cast<long long>(tokens));
  if (q_stride % 8 || k_stride % 8 || v_stride % 8 || q_stride < heads * head_dim || k_stride < kv_heads * head_dim ||
      v_stride < kv_heads * head_dim)
    return fail(RK_EINVAL, "%s: row strides must cover a row and be multiples of 8 elements", who);
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(cos) || !aligned16(sin) || !aligned16(q_out) ||
      !aligned16(k_cache) || !aligned16(v_cache))
    return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  if (batch * tokens * (heads + 2 * kv_heads) > (1ll << 31)) return fail(RK_EUNSUPPORTED, "%s: problem too large", who);
  RopeParams p{};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.q_stride = q_stride;
  p.k_stride = k_stride;
  p.v_stride = v_stride;
  p.cos = static_cast<const __nv_bfloat16*>(cos);
  p.sin = static_cast<const __nv_bfloat16*>(sin);
  p.q_out = static_cast<__nv_bfloat16*>(q_out);
  p.k_all = static_cast<__nv_bfloat16*>(k_cache);
  p.v_all = static_cast<__nv_bfloat16*>(v_cache);
  p.vt_all = static_cast<__nv_bfloat16*>(vt_cache);
  p.vt_pitch = vt_pitch;
  p.batch = static_cast<int>(batch);
  p.tokens = static_cast<int>(tokens);
  p.heads = static_cast<int>(heads);
  p.kv_heads = static_cast<int>(kv_heads);
  p.dim = static_cast<int>(head_dim);
  p.cache_rows = static_cast<int>(cache_rows);
  p.prefix = static_cast<int>(prefix);
  p.token_major = q_token_major ? 1 : 0;
  const int parts = tokens >= 8 ? 4 : 1;  // a few rows are not worth four CTAs
  const long long value_blocks = batch * kv_heads * ((tokens + kRopeTokens - 1) / kRopeTokens) * parts;
  const long long rotate_blocks = (batch * tokens * (heads + kv_heads) + kRopeWarps - 1) / kRopeWarps;
  launch_pdl(rope_cache_update_kernel, static_cast<unsigned>(value_blocks + rotate_blocks), kRopeWarps * 32, as_stream(stream), p,
             static_cast<unsigned>(value_blocks), parts);
  return check_launch(who);
}


extern "C" int rk_rope_cache_update(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                                    int64_t v_stride, const void* cos, const void* sin, int64_t batch, int64_t tokens,
                                    int64_t heads, int64_t kv_heads, int64_t head_dim, void* q_out, int q_token_major,
                                    void* k_cache, void* v_cache, int64_t cache_rows, int64_t prefix, void* stream) {
  return rope_cache_update_impl(q, q_stride, k, k_stride, v, v_stride, cos, sin, batch, tokens, heads, kv_heads, head_dim,
                                q_out, q_token_major, k_cache, v_cache, cache_rows, prefix, nullptr, 0, stream,
                                "rk_rope_cache_update");
}

extern "C" int rk_rope_cache_update_vt(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                                       int64_t v_stride, const void* cos, const void* sin, int64_t batch, int64_t tokens,
                                       int64_t heads, int64_t kv_heads, int64_t head_dim, void* q_out, int q_token_major,
                                       void* k_cache, void* v_cache, int64_t cache_rows, int64_t prefix, void* vt_cache,
                                       int64_t vt_pitch, void* stream) {
  if (!vt_cache) return rk::fail(RK_EINVAL, "rk_rope_cache_update_vt: null transposed cache");
  return rope_cache_update_impl(q, q_stride, k, k_stride, v, v_stride, cos, sin, batch, tokens, heads, kv_heads, head_dim,
                                q_out, q_token_major, k_cache, v_cache, cache_rows, prefix, vt_cache, vt_pitch, stream,
                                "rk_rope_cache_update_vt");
}

extern "C" int rk_kv_prefix_fill(const void* k, const void* v, int64_t planes, int64_t prefix, int64_t head_dim, void* k_cache,
                                 void* v_cache, int64_t cache_rows, void* vt_cache, int64_t vt_pitch, void* stream) {
  using namespace rk;
  const char* who = "rk_kv_prefix_fill";
  if (!k || !v || !k_cache || !v_cache || !vt_cache) return fail(RK_EINVAL, "%s: null pointer", who);
  if (head_dim != kFillDim) return fail(RK_EUNSUPPORTED, "%s: head_dim must be %d", who, kFillDim);
  if (planes < 1 || planes > 65535 || prefix < 1 || prefix > (1 << 24)) return fail(RK_EINVAL, "%s: bad planes / prefix", who);
  if (cache_rows < prefix || cache_rows > (1 << 24) || vt_pitch < prefix || vt_pitch % 8 != 0 || vt_pitch > (1 << 24))
    return fail(RK_EINVAL, "%s: the caches must hold the prefix and vt_pitch be a multiple of 8", who);
  if (!aligned16(k) || !aligned16(v) || !aligned16(k_cache) || !aligned16(v_cache) || !aligned16(vt_cache))
    return fail(RK_EINVAL, "%s: pointers must be 16-byte aligned", who);
  FillParams p{};
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.k_all = static_cast<__nv_bfloat16*>(k_cache);
  p.v_all = static_cast<__nv_bfloat16*>(v_cache);
  p.vt_all = static_cast<__nv_bfloat16*>(vt_cache);
  p.prefix = static_cast<int>(prefix);
  p.cache_rows = static_cast<int>(cache_rows);
  p.vt_pitch = static_cast<int>(vt_pitch);
  const unsigned tiles = static_cast<unsigned>((vt_pitch + kFillRows - 1) / kFillRows);
  launch_pdl(kv_prefix_fill_kernel, dim3(tiles, static_cast<unsigned>(planes), 2), dim3(kFillThreads), as_stream(stream), p);
  return check_launch(who);
}
