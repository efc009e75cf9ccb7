// Products of several rows with bf16 weights: C [M, N] = A [M, K] W [N, K]^T, f32 accumulation and output.
//
// gemm_bf16_tc_kernel (bf16 activations): tcgen05 with both operands brought in by TMA.  The weights are the MMA's M
// side (128 output features), the activation rows its N side (16..256 of them, chosen at run time), so that few rows
// cost little and a row of TMEM lanes is a run of consecutive features: the epilogue stores 128 contiguous bytes per
// warp and activation row without staging.  Persistent: one CTA per SM walks the tiles; four roles (TMA, MMA issue,
// TMEM, four epilogue warps) with two accumulators in tensor memory, so the next tile's products run under this
// tile's stores.  K tails and rows beyond M or N are zero filled by TMA.  Every wait is bounded.
//
// Bound by what the SMs fetch from L2 (a tile of 128 x 256 takes 48 KB per K step of 512 cycles of MMAs): with PAIR a
// cluster of two CTAs owns 256 features (cta_group::2) and each brings its 128 weight rows and half of the activation rows,
// 32 KB.  The products of a prompt of 2048 tokens (the ten of four 4096-wide Fenorax layers): 1777 us with the MMAs out of a
// branch of one lane, 1575 from a converged warp (umma.cuh), 1452 in pairs; of 1500 tokens (22 of four Virolorn layers) 1753, 1483, 1436;
// of 40 tokens at width 1024 129 -> 97.  (Pairs then had widths in steps of 16, 240 and 176 here; with steps of 32, 256 and 192, whole
// prompts take the same.)
//
// dpk_gemm_f16_tc: the same kernel with f16 operands and an f16 result.
//
// Optional decay: exp(-rate softplus(c + bias)) of every product is stored instead of the product.
// Optional gated activation: weight rows in groups of sixteen (eight gate rows, then their eight up rows) and
// g' sigmoid(slope g') (u' + shift) with g' = min(g, limit), u' = clamp(u, +-limit) stored in A's type.
#include "layers.h"
#include "decay.cuh"
#include "pdl.cuh"
#include "tiles.h"
#include "umma.cuh"

#include <cstring>

using namespace umma;

namespace {

struct GluArgs {
  void *dst;
  int stride;
  float limit, slope, shift;
};

// for a result that is stored as bf16
__device__ __forceinline__ float glu_act_fast(float g, float u, const GluArgs &a) {
  if (a.limit > 0.0f) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
  }
  return __fdividef(g, 1.0f + __expf(-a.slope * g)) * (u + a.shift);
}

constexpr int BT_THREADS = 256, BT_MAX_STAGES = 8;
constexpr uint32_t BT_W_TILE = 128u * 128u;  // 128 weight rows x 64 bf16

struct TcArgs {
  float *C;
  __half *C16;   // f16 operands and result (rows of c_stride elements)
  int M, N, K, bn, stages, tiles_n, tiles_m, tmem_cols, c_stride;
  GluArgs glu;
  DecayOut decay;
};

__device__ __forceinline__ uint32_t idesc_16(int M, int N, bool f16) {  // D = f32, A = B = bf16 or f16, both K-major
  return (1u << 4) | (f16 ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

template <bool PAIR>
__global__ void __launch_bounds__(BT_THREADS, 1) gemm_bf16_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                                                                     const TcArgs a, int *__restrict__ err) {
  extern __shared__ uint8_t bt_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(bt_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bars[2 * BT_MAX_STAGES + 4];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const int owner = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, owners = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int S = a.stages, rows = PAIR ? a.bn / 2 : a.bn, features = PAIR ? 256 : 128;  // activation rows of this CTA, features of a tile
  const uint32_t stage_bytes = BT_W_TILE + (uint32_t)rows * 128u;
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty = [&](int s) { return bar0 + 8u * (uint32_t)(BT_MAX_STAGES + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (uint32_t)(2 * BT_MAX_STAGES + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * BT_MAX_STAGES + 2 + b); };
  const int tiles = a.tiles_n * a.tiles_m, ksteps = (a.K + BK - 1) / BK;

  if constexpr (!PAIR) pdl_launch();  // (a launch of clusters is not made programmatic)
  pdl_wait();
  if (tid == 0) {
    for (int s = 0; s < S; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), PAIR ? 8 : 4); }
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 2) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)a.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)a.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(&tmem_slot), 0);

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0, round = 0;
      int s = 0;
      bool ok = true;
      for (int tile = owner; tile < tiles && ok; tile += owners) {
        const int n0 = (tile / a.tiles_m) * features + (int)rank * 128, m0 = (tile % a.tiles_m) * a.bn + (int)rank * rows;
        for (int k = 0; k < ksteps; k++, it++) {
          if (round > 0 && !mbar_wait_bounded(empty(s), (round - 1u) & 1u, abort_flag)) { ok = false; break; }
          const uint32_t dst = smem_u32(smem) + (uint32_t)s * stage_bytes;
          if constexpr (PAIR) {  // both CTAs' bytes are counted on CTA 0's barrier
            if (rank == 0) mbar_expect_tx(full(s), 2u * stage_bytes);
            const uint32_t there = mapa_shared(full(s), 0u);
            tma_load_2d_2sm(dst, &tmap_w, k * BK, n0, there);
            tma_load_2d_2sm(dst + BT_W_TILE, &tmap_a, k * BK, m0, there);
          } else {
            mbar_expect_tx(full(s), stage_bytes);
            tma_load_2d(dst, &tmap_w, k * BK, n0, full(s));
            tma_load_2d(dst + BT_W_TILE, &tmap_a, k * BK, m0, full(s));
          }
          if (++s == S) { s = 0; round++; }
        }
      }
      // no copy may still be in flight when the CTA ends, also where a wait gave up
      const uint32_t held = it < (uint32_t)S ? it : (uint32_t)S;
      for (uint32_t i = it - held; i < it && rank == 0; i++)
        for (uint32_t poll = 0; poll < (1u << 20) && !mbar_try_wait(full((int)(i % (uint32_t)S)), (i / (uint32_t)S) & 1u); poll++) {}
    }
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t idesc = idesc_16(features, a.bn, a.C16 != nullptr);
      const uint64_t first = umma_desc_sw128(smem_u32(smem));
      uint32_t n = 0, round = 0;
      int s = 0;
      bool ok = true;
      for (int tile = owner; tile < tiles && ok; tile += owners, n++) {
        const int b = (int)(n & 1u);
        if (n >= 2 && !mbar_wait_warp(acc_empty(b), ((n >> 1) - 1u) & 1u, abort_flag)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + (uint32_t)(b * a.bn);
        for (int k = 0; k < ksteps; k++) {
          if (!mbar_wait_warp(full(s), round & 1u, abort_flag)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t w = first + (uint64_t)((uint32_t)s * (stage_bytes >> 4));
          umma_step_warp<PAIR>(acc, w, w + (BT_W_TILE >> 4), idesc, k);
          umma_commit_warp<PAIR>(empty(s));
          if (++s == S) { s = 0; round++; }
        }
        if (ok) umma_commit_warp<PAIR>(acc_full(b));
      }
    }
  } else if (warp >= 4) {
    const int quad = warp & 3;
    const uint32_t acc_empty0 = PAIR ? mapa_shared(acc_empty(0), 0u) : 0u;
    uint32_t n = 0;
    for (int tile = owner; tile < tiles; tile += owners, n++) {
      const int b = (int)(n & 1u);
      const int n0 = (tile / a.tiles_m) * features + (int)rank * 128, m0 = (tile % a.tiles_m) * a.bn;
      const bool ready = mbar_wait_bounded(acc_full(b), (n >> 1) & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ready)) break;  // tcgen05.ld is warp-wide: together or not at all
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int f = n0 + quad * 32 + lane;
      const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(b * a.bn);
      for (int c0 = 0; c0 < a.bn; c0 += 16) {
        if (m0 + c0 >= a.M) break;  // (uniform) no such activation rows
        uint32_t r[16];
        __syncwarp();  // (lanes store by themselves; tensor memory is read by the whole warp)
        tmem_ld16(taddr + (uint32_t)c0, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (a.glu.dst) {
          // a gate row and its up row are eight lanes apart: the gate's lane takes the even activation rows of the pair,
          // the other lane the odd ones
          const bool is_up = lane & 8;
          __nv_bfloat16 *dst = reinterpret_cast<__nv_bfloat16 *>(a.glu.dst) + (f >> 4) * 8 + (f & 7);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(is_up ? r[i] : r[i + 1]), 8);
            const float gv = is_up ? got : __uint_as_float(r[i]), uv = is_up ? __uint_as_float(r[i + 1]) : got;
            const int row = m0 + c0 + i + (is_up ? 1 : 0);
            if (f < a.N && row < a.M) dst[(size_t)row * a.glu.stride] = __float2bfloat16_rn(glu_act_fast(gv, uv, a.glu));
          }
        } else if (a.C16) {
          if (f < a.N) {
            __half *dst = a.C16 + (size_t)(m0 + c0) * a.c_stride + f;
#pragma unroll
            for (int i = 0; i < 16; i++)
              if (m0 + c0 + i < a.M) dst[(size_t)i * a.c_stride] = __float2half_rn(__uint_as_float(r[i]));
          }
        } else if (f < a.N) {
          if (a.decay.rate) {
            const float rate = a.decay.rate[f], bias = a.decay.bias[f];
#pragma unroll 4
            for (int i = 0; i < 16; i++) r[i] = __float_as_uint(decay_of(__uint_as_float(r[i]), rate, bias));
          }
          float *dst = a.C + (size_t)(m0 + c0) * a.N + f;
#pragma unroll
          for (int i = 0; i < 16; i++)
            if (m0 + c0 + i < a.M) dst[(size_t)i * a.N] = __uint_as_float(r[i]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(acc_empty0 + 8u * (uint32_t)b) : "memory");
        else mbar_arrive(acc_empty(b));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (PAIR) {
    cluster_sync_all();  // neither CTA frees tensor memory or leaves while the peer still uses the pair's resources
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols) : "memory");
  } else {
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols) : "memory");
  }
  if (abort_word && tid == 0) atomicExch(err, 2);
}

GluArgs glu_args(const GluOut *g) {
  GluArgs a = {nullptr, 0, 0.0f, 0.0f, 0.0f};
  if (g) { a.dst = g->dst; a.stride = g->stride; a.limit = g->limit; a.slope = g->slope; a.shift = g->shift; }
  return a;
}

// shape, strides and outputs are in `a`; the rest is chosen here
dp_status launch_tc(dp_ctx *ctx, const void *W, int w_stride, const void *A, int a_stride, TcArgs a) {
  const int M = a.M, N = a.N, K = a.K;
  DP_CHECK(ctx, w_stride % 8 == 0 && a_stride % 8 == 0 && K <= w_stride && K <= a_stride && M > 0 && N > 0 && K > 0, "gemm (bf16): bad shape or stride");
  EncodeTiledFn encode = get_encode();
  if (!encode) return dp_fail(ctx, DP_ERR_CUDA, "gemm (bf16): cuTensorMapEncodeTiled is not available");
  // (in a decode step's graph kernels launch their dependents early; those keep to launches without clusters)
  const TilePick pick = pick_tile(ctx->sm_count, M, N, (K + BK - 1) / BK, !ctx->pdl && ctx->sm_count >= 2);
  a.bn = pick.bn;
  a.tiles_n = (N + (pick.pair ? 255 : 127)) / (pick.pair ? 256 : 128);
  a.tiles_m = (M + a.bn - 1) / a.bn;
  const int rows = pick.pair ? a.bn / 2 : a.bn;
  const uint32_t stage_bytes = BT_W_TILE + (uint32_t)rows * 128u;
  const size_t budget = ctx->smem_optin - 2048;
  int stages = (int)((budget - 1024) / stage_bytes);
  if (stages > BT_MAX_STAGES) stages = BT_MAX_STAGES;
  a.stages = stages;
  a.tmem_cols = 32;
  while (a.tmem_cols < 2 * a.bn) a.tmem_cols *= 2;
  const CUtensorMapDataType type = a.C16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tw, ta;
  const cuuint32_t estr[2] = {1, 1};
  const cuuint64_t wd[2] = {(cuuint64_t)K, (cuuint64_t)N}, ad[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t ws[1] = {(cuuint64_t)w_stride * 2}, as[1] = {(cuuint64_t)a_stride * 2};
  const cuuint32_t wb[2] = {BK, 128}, ab[2] = {BK, (cuuint32_t)rows};
  CUresult r = encode(&tw, type, 2, (void *)W, wd, ws, wb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS)
    r = encode(&ta, type, 2, (void *)A, ad, as, ab, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return dp_fail(ctx, DP_ERR_CUDA, "gemm (bf16): cuTensorMapEncodeTiled failed (%d) for [%d,%d] x [%d,%d]", (int)r, M, K, N, K);
  const size_t smem = (size_t)stages * stage_bytes + 1024;
  const int tiles = a.tiles_n * a.tiles_m;
  if (!pick.pair) {
    static dp_per_device_once attr;
    if (attr.pending(ctx->device)) {
      DP_CUDA(ctx, cudaFuncSetAttribute(gemm_bf16_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
      attr.done(ctx->device);
    }
    DP_LAUNCH(ctx, gemm_bf16_tc_kernel<false>, tiles < ctx->sm_count ? tiles : ctx->sm_count, BT_THREADS, smem, tw, ta, a, ctx->dev_status);
    return DP_OK;
  }
  static dp_per_device_once attr;
  if (attr.pending(ctx->device)) {
    DP_CUDA(ctx, cudaFuncSetAttribute(gemm_bf16_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
    attr.done(ctx->device);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (unsigned)(tiles < ctx->sm_count / 2 ? tiles : ctx->sm_count / 2));
  cfg.blockDim = dim3(BT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute cluster[1];
  cluster[0].id = cudaLaunchAttributeClusterDimension;
  cluster[0].val.clusterDim.x = 2;
  cluster[0].val.clusterDim.y = 1;
  cluster[0].val.clusterDim.z = 1;
  cfg.attrs = cluster;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_bf16_tc_kernel<true>, tw, ta, a, ctx->dev_status);
  ctx->launches++;
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return dp_fail(ctx, DP_ERR_CUDA, "launch of gemm_bf16_tc_kernel failed: %s", cudaGetErrorString(e));
  return DP_OK;
}

}  // namespace

dp_status dpk_gemm_bf16_tc(dp_ctx *ctx, const __nv_bfloat16 *W, int w_stride, const __nv_bfloat16 *A, int a_stride, float *C, int M, int N, int K,
                           const GluOut *glu, const DecayOut *decay) {
  DP_CHECK(ctx, !glu || N % 16 == 0, "gemm (bf16): gate and up rows come in groups of sixteen");
  TcArgs a = {};
  a.C = C; a.M = M; a.N = N; a.K = K;
  a.glu = glu_args(glu);
  if (decay) a.decay = *decay;
  return launch_tc(ctx, W, w_stride, A, a_stride, a);
}

dp_status dpk_gemm_f16_tc(dp_ctx *ctx, const __half *W, int w_stride, const __half *A, int a_stride, __half *C, int c_stride, int M, int N, int K) {
  TcArgs a = {};
  a.C16 = C; a.c_stride = c_stride; a.M = M; a.N = N; a.K = K;
  return launch_tc(ctx, W, w_stride, A, a_stride, a);
}
