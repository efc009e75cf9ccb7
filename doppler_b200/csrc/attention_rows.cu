// Attention of several query rows in f32 arithmetic, query-tiled: f16 or f32 caches, key and value sizes up to 256 in steps of
// four, any GQA ratio, every mask of attn_range.  For f32 caches and for f16 heads that are not 64 or 128 values (those have kernels of
// their own: attention_prefill.cu, attention_tc.cu, attn_split_kernel) or whose values are not as long as their keys.
//
// A block holds 32 (position, head) rows of one KV head and walks the keys in tiles of 64, so a key is read once for 32 rows
// and not once for each (or for the four heads of a position).  S = Q K^T and O += P V are register tiles of 4 rows x 4 keys and
// 4 rows x V / 16 values a thread, fed by 16-byte reads of shared memory: 12 wavefronts for 16 cycles of multiply-adds in S,
// 20 for 32 in P V.  K and V take turns in one buffer, so that two blocks of 255 registers a thread share an SM at every size
// and one computes while the other loads.  The eight rows of a warp meet only that warp, so P needs no block-wide barrier.
// Bound: multiply-adds 40 % of the cycles (packed, two cycles each), the rest latency of shared and global loads with two
// warps a scheduler.  1024 tokens, 32 heads of 256 over 8: 0.88 ms; the kernel that goes row by row re-reads a key for every
// row and head and takes 2.8.
// All sums are f32, in short chains: a logit is a tree of chains of 8 products, the values are added 16 keys at a time; with one
// chain over the size and one over the keys the error against 64 bits was 1.3 to 1.9 times that of the row-by-row kernel
// (which sums over 32 lanes and 4 warps), with these it is 0.6 to 1.0 times.
#include "attn_out.cuh"
#include "common.h"
#include "pdl.cuh"

#include <cfloat>
#include <climits>
#include <cstdlib>
#include <type_traits>

#define AR_THREADS 128
#define AR_ROWS 32
#define AR_KEYS 64

template <int DP> constexpr size_t ar_smem() { return sizeof(float) * ((size_t)(AR_ROWS + AR_KEYS) * (DP + 4) + AR_ROWS * (AR_KEYS + 4)); }

__device__ __forceinline__ float4 ar_load(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float4 ar_load(const __half *p) {
  const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float2 ar_fma(float2 a, float2 b, float2 c) {
  float2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(*reinterpret_cast<unsigned long long *>(&r)) : "l"(*reinterpret_cast<const unsigned long long *>(&a)),
      "l"(*reinterpret_cast<const unsigned long long *>(&b)), "l"(*reinterpret_cast<const unsigned long long *>(&c)));
  return r;
}

__device__ __forceinline__ float2 ar_mul(float2 a, float2 b) {
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(*reinterpret_cast<unsigned long long *>(&r)) : "l"(*reinterpret_cast<const unsigned long long *>(&a)),
      "l"(*reinterpret_cast<const unsigned long long *>(&b)));
  return r;
}
__device__ __forceinline__ float2 ar_add(float2 a, float2 b) {
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(*reinterpret_cast<unsigned long long *>(&r)) : "l"(*reinterpret_cast<const unsigned long long *>(&a)),
      "l"(*reinterpret_cast<const unsigned long long *>(&b)));
  return r;
}

// 64 keys (or values) of `width` elements from row `key0` on -> shared rows of DP + 4 floats; zeros outside [0, keys) and behind
// width.  check: returns whether one of the thread's elements is not finite.
template <int DP, typename KT>
__device__ __forceinline__ bool ar_tile(float *__restrict__ dst, const KT *__restrict__ src, size_t stride, int key0, int keys, int width, bool check = false) {
  unsigned top = 0;
  constexpr int PER = AR_KEYS * (DP / 4) / AR_THREADS, CHUNK = 8;
#pragma unroll
  for (int c = 0; c < PER; c += CHUNK) {
    float4 v[CHUNK];
#pragma unroll
    for (int i = 0; i < CHUNK; i++) {
      const int e = (c + i) * AR_THREADS + (int)threadIdx.x, row = e / (DP / 4), d = e % (DP / 4) * 4;
      v[i] = key0 + row < keys && d < width ? ar_load(src + (size_t)(key0 + row) * stride + d) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int i = 0; i < CHUNK; i++) {
      const int e = (c + i) * AR_THREADS + (int)threadIdx.x;
      *reinterpret_cast<float4 *>(dst + (e / (DP / 4)) * (DP + 4) + e % (DP / 4) * 4) = v[i];
    }
    if (check)
#pragma unroll
      for (int i = 0; i < CHUNK; i++)
        top = max(max(top, max(__float_as_uint(v[i].x) & 0x7fffffffu, __float_as_uint(v[i].y) & 0x7fffffffu)),
                  max(__float_as_uint(v[i].z) & 0x7fffffffu, __float_as_uint(v[i].w) & 0x7fffffffu));
  }
  return top >= 0x7f800000u;
}

// grid: (tiles of 32 / gt positions x splits, KV heads x groups of gt heads, sequences); 2^gt_log2 = gt heads of one KV head share a block
template <int DP, typename KT>
__global__ void __launch_bounds__(AR_THREADS, 2) attn_rows_kernel(dpk_attn_params p, int gt_log2, float *__restrict__ part, int splits) {
  pdl_launch();
  pdl_wait();
  extern __shared__ float4 ar_shared[];
  float *const sm_q = reinterpret_cast<float *>(ar_shared), *const sm_kv = sm_q + AR_ROWS * (DP + 4), *const sm_p = sm_kv + AR_KEYS * (DP + 4);
  const int D = p.head_dim, V = p.v_dim ? p.v_dim : D;
  const int tid = threadIdx.x, lane = tid & 31, kg = tid & 15, rg = tid >> 4;
  const int gt = 1 << gt_log2, G = p.num_heads / p.num_kv_heads, groups = G >> gt_log2, positions = AR_ROWS >> gt_log2;
  const int kvh = blockIdx.y / groups, h0 = kvh * G + blockIdx.y % groups * gt;
  const int b = blockIdx.z, split = blockIdx.x % splits;
  const int tile = (int)(gridDim.x / splits) - 1 - (int)blockIdx.x / splits;  // the rows that see the most keys first
  const int qi0 = tile * positions;
  const int kv_len = p.kv_lens ? min(max(p.kv_lens[b], 0), p.kv_len) : p.kv_len;
  // every lane: the keys of row `lane` of the block, for the block's range; then those of its own four
  auto range = [&](int r) {
    const int qi = qi0 + (r >> gt_log2);
    AttnRange a = {0, 0};
    if (qi < p.seq_len) a = attn_range(p, kv_len, qi);
    return a;
  };
  const AttnRange mine = range(lane);
  const int lo_all = __reduce_min_sync(0xffffffffu, mine.lo < mine.hi ? mine.lo : INT_MAX);
  const int hi_all = __reduce_max_sync(0xffffffffu, mine.lo < mine.hi ? mine.hi : 0);
  const int lo_last = __reduce_max_sync(0xffffffffu, mine.lo), hi_first = __reduce_min_sync(0xffffffffu, mine.hi);  // keys all rows see
  int k_begin = lo_all < hi_all ? lo_all : 0, k_end = lo_all < hi_all ? hi_all : 0;
  if (splits > 1) {
    const int per = ((k_end - k_begin + splits - 1) / splits + AR_KEYS - 1) / AR_KEYS * AR_KEYS;
    k_begin += split * per;
    k_end = min(k_end, k_begin + per);
  }
  int lo[4], hi[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const AttnRange a = range(rg * 4 + i);
    lo[i] = a.lo; hi[i] = a.hi;
  }
#pragma unroll
  for (int c = 0; c < AR_ROWS * (DP / 4) / AR_THREADS; c += 4) {
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int e = (c + i) * AR_THREADS + tid, r = e / (DP / 4), d = e % (DP / 4) * 4, qi = qi0 + (r >> gt_log2);
      v[i] = qi < p.seq_len && d < D ? ar_load(p.q + (((size_t)b * p.seq_len + qi) * p.num_heads + h0 + (r & (gt - 1))) * D + d) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int e = (c + i) * AR_THREADS + tid;
      *reinterpret_cast<float4 *>(sm_q + (e / (DP / 4)) * (DP + 4) + e % (DP / 4) * 4) = make_float4(v[i].x * p.scale, v[i].y * p.scale, v[i].z * p.scale, v[i].w * p.scale);
    }
  }
  const size_t k_stride = (size_t)p.num_kv_heads * D, v_stride = p.v_row_stride ? (size_t)p.v_row_stride : (size_t)p.num_kv_heads * V;
  const KT *kb = reinterpret_cast<const KT *>(p.k) + (size_t)b * p.kv_batch_stride + (size_t)kvh * D;
  const KT *vb = reinterpret_cast<const KT *>(p.v) + (size_t)b * (p.v_batch_stride ? p.v_batch_stride : p.kv_batch_stride) + (size_t)kvh * V;
  constexpr int NV = DP / 64;  // groups of four values a thread holds of each row
  float2 o[4][NV][2];
  float m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    m[i] = -FLT_MAX; l[i] = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; j++) o[i][j][0] = o[i][j][1] = make_float2(0.0f, 0.0f);
  }
  const float LOG2E = 1.4426950408889634f;
  for (int k0 = k_begin; k0 < k_end; k0 += AR_KEYS) {
    __syncthreads();  // the values of the tile before are used up
    ar_tile<DP>(sm_kv, kb, k_stride, k0, k_end, D);
    __syncthreads();
    float2 acc[4][4];
#pragma unroll 1
    for (int d64 = 0; d64 < DP; d64 += 64) {
      float2 mid[4][4];
#pragma unroll
      for (int d16 = 0; d16 < 64; d16 += 16) {
        float2 sum[4][4];
#pragma unroll
        for (int d = 0; d < 16; d += 4) {
          float4 q[4], k[4];
#pragma unroll
          for (int i = 0; i < 4; i++) q[i] = *reinterpret_cast<const float4 *>(sm_q + (rg * 4 + i) * (DP + 4) + d64 + d16 + d);
#pragma unroll
          for (int j = 0; j < 4; j++) k[j] = *reinterpret_cast<const float4 *>(sm_kv + (kg + 16 * j) * (DP + 4) + d64 + d16 + d);
#pragma unroll
          for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const float2 q0 = make_float2(q[i].x, q[i].y), k0 = make_float2(k[j].x, k[j].y);
              sum[i][j] = d == 0 ? ar_mul(q0, k0) : ar_fma(q0, k0, sum[i][j]);
              sum[i][j] = ar_fma(make_float2(q[i].z, q[i].w), make_float2(k[j].z, k[j].w), sum[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) mid[i][j] = d16 == 0 ? sum[i][j] : ar_add(mid[i][j], sum[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = d64 == 0 ? mid[i][j] : ar_add(acc[i][j], mid[i][j]);
    }
    // this tile's keys that row i sees: [from[i], to[i]) of its 64
    float shrink[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int from = lo[i] - k0, to = min(hi[i], k_end) - k0;
      float a[4], top = m[i];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        a[j] = acc[i][j].x + acc[i][j].y;
        if (p.softcap > 0.0f) a[j] = tanhf(a[j] / p.softcap) * p.softcap;
        a[j] *= LOG2E;
        const int key = kg + 16 * j;
        if (key >= from && key < to) top = fmaxf(top, a[j]);
      }
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, s));
      shrink[i] = exp2f(m[i] - top);
      m[i] = top;
      l[i] *= shrink[i];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int key = kg + 16 * j;
        const float pr = key >= from && key < to ? exp2f(a[j] - top) : 0.0f;
        l[i] += pr;
        sm_p[(rg * 4 + i) * (AR_KEYS + 4) + key] = pr;
      }
    }
    const bool whole = k0 >= lo_last && k0 + AR_KEYS <= min(hi_first, k_end);
    __syncthreads();  // the keys are used up
    const bool strange = ar_tile<DP>(sm_kv, vb, v_stride, k0, k_end, V, !whole);
    const bool careful = __syncthreads_or(strange);
    if (__any_sync(0xffffffffu, shrink[0] != 1.0f || shrink[1] != 1.0f || shrink[2] != 1.0f || shrink[3] != 1.0f)) {
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < NV; j++)
#pragma unroll
          for (int e = 0; e < 2; e++) o[i][j][e] = ar_mul(o[i][j][e], make_float2(shrink[i], shrink[i]));
    }
    // 16 keys at a time, each a chain of its own; groups that none of the warp's rows sees are passed over
    const int from_w = __reduce_min_sync(0xffffffffu, min(min(lo[0], lo[1]), min(lo[2], lo[3]))) - k0;
    const int to_w = __reduce_max_sync(0xffffffffu, max(max(hi[0], hi[1]), max(hi[2], hi[3]))) - k0;
#pragma unroll 1
    for (int k16 = 0; k16 < AR_KEYS; k16 += 16) {
      if (k16 >= to_w || k16 + 16 <= from_w) continue;
      float2 t[4][NV][2];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < NV; j++) t[i][j][0] = t[i][j][1] = make_float2(0.0f, 0.0f);
      auto add = [&](auto each) {
#pragma unroll 1
      for (int key = k16; key < k16 + 16; key += 4) {
        float4 pr[4];
#pragma unroll
        for (int i = 0; i < 4; i++) pr[i] = *reinterpret_cast<const float4 *>(sm_p + (rg * 4 + i) * (AR_KEYS + 4) + key);
#pragma unroll
        for (int s = 0; s < 4; s++) {
          float4 v[NV];
#pragma unroll
          for (int j = 0; j < NV; j++) v[j] = *reinterpret_cast<const float4 *>(sm_kv + (key + s) * (DP + 4) + kg * 4 + 64 * j);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            if (decltype(each)::value && (k0 + key + s < lo[i] || k0 + key + s >= hi[i])) continue;  // (0 * infinity)
            const float w = s == 0 ? pr[i].x : s == 1 ? pr[i].y : s == 2 ? pr[i].z : pr[i].w;
#pragma unroll
            for (int j = 0; j < NV; j++) {
              t[i][j][0] = ar_fma(make_float2(w, w), make_float2(v[j].x, v[j].y), t[i][j][0]);
              t[i][j][1] = ar_fma(make_float2(w, w), make_float2(v[j].z, v[j].w), t[i][j][1]);
            }
          }
        }
      }
      };
      if (careful) add(std::true_type());
      else add(std::false_type());
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < NV; j++)
#pragma unroll
          for (int e = 0; e < 2; e++) o[i][j][e] = ar_add(o[i][j][e], t[i][j][e]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], s);
    const int r = rg * 4 + i, qi = qi0 + (r >> gt_log2), h = h0 + (r & (gt - 1));
    if (qi >= p.seq_len) continue;
    const size_t z = (size_t)b * p.seq_len + qi;
    float *pp = splits > 1 ? part + ((z * p.num_heads + h) * splits + split) * (V + 2) : nullptr;
#pragma unroll
    for (int j = 0; j < NV; j++) {
      const float v[4] = {o[i][j][0].x, o[i][j][0].y, o[i][j][1].x, o[i][j][1].y};
      const int d = kg * 4 + 64 * j;
      if (d >= V) continue;
#pragma unroll
      for (int e = 0; e < 4; e++) {
        if (pp) pp[d + e] = v[e];
        else attn_store(p, z, h, V, d + e, l[i] > 0.0f ? v[e] / l[i] : 0.0f);
      }
    }
    if (pp && kg == 0) { pp[V] = m[i]; pp[V + 1] = l[i]; }
  }
}

static int rows_heads(const dpk_attn_params &p) {  // heads of a KV head that share a block: the largest power of two up to 8 that divides their number
  const int G = p.num_heads / p.num_kv_heads;
  return G % 8 == 0 ? 8 : G % 4 == 0 ? 4 : G % 2 == 0 ? 2 : 1;
}
static long rows_blocks(const dpk_attn_params &p) {
  const int gt = rows_heads(p), positions = AR_ROWS / gt;
  return (long)p.batch * (p.num_heads / gt) * ((p.seq_len + positions - 1) / positions);
}

// shapes and alignments this kernel reads
static bool rows_shape(const dpk_attn_params &p) {
  if (p.seq_len < 2 || p.k2 || p.spans || p.fuse.qkv || p.num_kv_heads <= 0 || p.num_heads % p.num_kv_heads) return false;
  const int V = p.v_dim ? p.v_dim : p.head_dim;
  if (p.head_dim > 256 || V > 256 || p.head_dim % 4 || V % 4 || p.kv_batch_stride % 4 || p.v_batch_stride % 4 || p.v_row_stride % 4) return false;
  const uintptr_t kv = p.kv_f32 ? 15 : 7;
  return !(((uintptr_t)p.k | (uintptr_t)p.v) & kv) && !((uintptr_t)p.q & 15);
}

// three blocks for every SM, of two tiles of keys at least
int dpk_attention_rows_splits(dp_ctx *ctx, const dpk_attn_params &p) {
  const long keys = p.chunk > 0 && p.chunk < p.kv_len ? p.chunk : p.kv_len;
  const long blocks = rows_blocks(p), want = (3L * ctx->sm_count + blocks - 1) / blocks, most = (keys + 2 * AR_KEYS - 1) / (2 * AR_KEYS);
  const long s = want < most ? want : most;
  return (int)(s < 1 ? 1 : s > 32 ? 32 : s);
}

// Taken from 200 000 (row, head, key) triples on; below, a block of every row and head of its own is done before one of these
// has been through its first tiles (cold code, a load behind every barrier).  us, the kernel that goes row by row -> this one:
//   f16 heads of 256, triples: 61 000 47 -> 58, 120 000 46 -> 54, 160 000 56 -> 60, 245 000 146 -> 63, 256 000 96 -> 62,
//     410 000 82 -> 56, 2 000 000 397 -> 167, 67 000 000 10 940 -> 2 940
//   f16 heads of 32 and 48, 220 000: 25 to 48 -> 15 to 27; of 96: 29 to 49 -> 25 to 37 (one KV head of 96 without a mask 25 -> 27)
//   f32 heads of 128: 58 000 16 -> 31, 116 000 25 -> 28, 230 000 38 -> 32, 500 000 72 -> 43, 3 900 000 430 -> 142
bool dpk_attention_rows_eligible(const dpk_attn_params &p) {
  if (!rows_shape(p)) return false;
  long keys = p.kv_len;
  auto at_most = [&](long n) { keys = n < keys ? (n > 0 ? n : 0) : keys; };
  if (p.causal) at_most((long)p.start_pos - p.kv_start + (p.seq_len + 1) / 2);
  if (p.sliding_window > 0) at_most(p.sliding_window);
  if (p.chunk > 0) at_most(p.causal ? (p.chunk + 1) / 2 : p.chunk);
  return (long)p.batch * p.seq_len * p.num_heads * keys >= 200000;
}
// with `splits` parts (a caller without room for more): half of the SMs have a block (250 rows of 16 f32 heads, 128 blocks: 43 us, row by row 72)
bool dpk_attention_rows_fills(dp_ctx *ctx, const dpk_attn_params &p, int splits) {
  return splits >= dpk_attention_rows_splits(ctx, p) || rows_blocks(p) * splits * 2 >= ctx->sm_count;
}

template <int DP>
static dp_status launch_rows(dp_ctx *ctx, const dpk_attn_params &p, float *scratch, int splits) {
  const int gt = rows_heads(p), positions = AR_ROWS / gt;
  constexpr size_t smem = ar_smem<DP>();
  static dp_per_device_once attr;
  if (attr.pending(ctx->device)) {
    DP_CUDA(ctx, cudaFuncSetAttribute((attn_rows_kernel<DP, float>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    DP_CUDA(ctx, cudaFuncSetAttribute((attn_rows_kernel<DP, __half>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr.done(ctx->device);
  }
  dim3 grid((p.seq_len + positions - 1) / positions * splits, p.num_heads / gt, p.batch);
  if (p.kv_f32) DP_LAUNCH(ctx, (attn_rows_kernel<DP, float>), grid, AR_THREADS, smem, p, gt == 8 ? 3 : gt == 4 ? 2 : gt == 2 ? 1 : 0, scratch, splits);
  else DP_LAUNCH(ctx, (attn_rows_kernel<DP, __half>), grid, AR_THREADS, smem, p, gt == 8 ? 3 : gt == 4 ? 2 : gt == 2 ? 1 : 0, scratch, splits);
  return DP_OK;
}

dp_status dpk_attention_rows(dp_ctx *ctx, const dpk_attn_params &p, float *scratch, int splits) {
  const int most = p.head_dim > p.v_dim ? p.head_dim : p.v_dim;
  if (most <= 64) return launch_rows<64>(ctx, p, scratch, splits);
  if (most <= 128) return launch_rows<128>(ctx, p, scratch, splits);
  return launch_rows<256>(ctx, p, scratch, splits);
}
