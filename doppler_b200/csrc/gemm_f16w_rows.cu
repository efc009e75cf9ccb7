// Dense f16 weights times several activation rows: the LM head of a batched decode step (reference: the tied-embedding logits
// matmul, src/inference/pipelines/text/logits/gpu.js:245, which runs matmul_f16w_f32a.wgsl for 'ehf16' heads).
//
// HBM-bound: the weights (1.24 GB for a 151936 x 4096 head) are streamed once for up to 128 rows.  They are the MMA's M side
// (tcgen05.mma kind::f16, D in tensor memory), straight from memory by TMA.  The activation rows are its N side: f32 rows are
// split beforehand into an f16 half and its rounding residue, both scaled per row by a power of two (scale_cast_rows in
// gemm_q4k_tc.cu), so that hi + lo carries about 22 bits and the product is the f32 one to f32 accuracy.  Both halves lie one
// behind the other in a stage and are one MMA of twice the columns; their sums meet in the epilogue, in f32.
//
// Persistent, one CTA per SM.  The rows of a tile are what divides N evenly over the SMs, one MMA tile of up to 128 or two that
// share the activations (their bytes cross from L2 once for up to 256 weight rows), packed in the ring as they are: an MMA reads
// 128 rows whatever the tile holds, what lies behind it lands in lanes that nobody reads.  At 32000 x 4096 and 64 rows a stage of
// 44 KB holds 28 KB of weights, four of them keep 16 MB in flight.  The ring's first stages of weights are asked for before the wait for
// the kernel in front.  f32 rows with their split, us (the kernel of mma.sync fragments this replaces, whose shared-memory reads
// and tensor pipe took as long as its weights; the weights at 6.45 TB/s): 2 x 32000 x 4096 50 (68; 41), 64 x 32000 x 4096 57 (138; 41), 96 rows
// 62 (221; 41), 64 x 151936 x 4096 218 (563; 193), 64 x 3072 x 1024 17 (29), 2 x 256 x 256 12 (12).  hi and lo in sums of their own
// halve the error of f32 rows: 4.9e-6 of the result at K = 4096 (9.7e-6).  Two sets of accumulators, so that the stores of a tile run beside the next one's products.
#include "common.h"
#include "pdl.cuh"
#include "umma.cuh"

using namespace umma;

namespace {

constexpr int FR_EPI = 8;                       // storing warps: two per quarter of the lanes
constexpr int FR_THREADS = (4 + FR_EPI) * 32;
constexpr int FR_STAGES = 12;
constexpr int FR_BATCH = 128;                   // most activation rows of a launch

struct RowsArgs {
  void *C;
  const float *row_scale;
  float alpha;
  int M, m_base, N, K;
  int n, planes;                                // activation rows of a stage (a multiple of 16); hi alone or hi and lo
  int rows, halves, tiles, stages, tmem_cols;   // weight rows of an MMA, MMAs that share the activations
};

template <typename OutT>
__global__ void __launch_bounds__(FR_THREADS, 1) gemm_f16w_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                                                                       const RowsArgs a, int *__restrict__ err) {
  extern __shared__ uint8_t fr_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(fr_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bars[2 * FR_STAGES + 4];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int S = a.stages, cols = a.planes * a.n, tile_rows = a.rows * a.halves, ksteps = a.K / BK;
  const uint32_t w_bytes = (uint32_t)a.rows * 128u, x_off = w_bytes * (uint32_t)a.halves, stage_bytes = x_off + (uint32_t)cols * 128u;
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty = [&](int s) { return bar0 + 8u * (uint32_t)(FR_STAGES + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (uint32_t)(2 * FR_STAGES + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (uint32_t)(2 * FR_STAGES + 2 + b); };

  pdl_launch();
  if (tid == 0) {
    for (int s = 0; s < S; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), FR_EPI); }
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)a.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(&tmem_slot), 0);

  if (warp == 0) {
    if (lane == 0) {
      const int total = ((a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * ksteps;  // K steps of this CTA
      auto weights = [&](int s, int n0, int k) {
        const uint32_t dst = smem_u32(smem) + (uint32_t)s * stage_bytes;
        mbar_expect_tx(full(s), stage_bytes);
        tma_load_2d(dst, &tmap_w, k * BK, n0, full(s));
        if (a.halves == 2) tma_load_2d(dst + w_bytes, &tmap_w, k * BK, n0 + a.rows, full(s));
      };
      auto activations = [&](int s, int k) {
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                         smem_u32(smem) + (uint32_t)s * stage_bytes + x_off),
                     "l"(&tmap_a), "r"(k * BK), "r"(a.m_base), "r"(0), "r"(full(s))
                     : "memory");
      };
      const int step = (int)gridDim.x * tile_rows, first = total < S ? total : S;
      int n0 = (int)blockIdx.x * tile_rows, k = 0, it = 0;
      for (; it < first; it++) {
        weights(it, n0, k);
        if (++k == ksteps) { k = 0; n0 += step; }
      }
      pdl_wait();
      for (int i = 0, ki = 0; i < first; i++) {
        activations(i, ki);
        if (++ki == ksteps) ki = 0;
      }
      int s = 0;
      uint32_t round = 0;
      for (; it < total; it++) {
        if (!mbar_wait_bounded(empty(s), round & 1u, abort_flag)) break;
        weights(s, n0, k);
        activations(s, k);
        if (++k == ksteps) { k = 0; n0 += step; }
        if (++s == S) { s = 0; round++; }
      }
      // no copy may still be in flight when the CTA ends, also where a wait gave up
      for (int i = it < S ? 0 : it - S; i < it; i++)
        for (uint32_t poll = 0; poll < (1u << 20) && !mbar_try_wait(full(i % S), (uint32_t)(i / S) & 1u); poll++) {}
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_f16(128, cols);
    const uint64_t first = umma_desc_sw128(smem_u32(smem));
    uint32_t n = 0, round = 0;
    int s = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < a.tiles && ok; tile += gridDim.x, n++) {
      const int b = (int)(n & 1u);
      if (n >= 2 && !mbar_wait_warp(acc_empty(b), ((n >> 1) - 1u) & 1u, abort_flag)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + (uint32_t)(b * a.halves * cols);
      for (int k = 0; k < ksteps; k++) {
        if (!mbar_wait_warp(full(s), round & 1u, abort_flag)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t w = first + (uint64_t)((uint32_t)s * (stage_bytes >> 4)), x = w + (x_off >> 4);
        umma_step_warp<false>(acc, w, x, idesc, k);
        if (a.halves == 2) umma_step_warp<false>(acc + (uint32_t)cols, w + (w_bytes >> 4), x, idesc, k);
        umma_commit_warp<false>(empty(s));
        if (++s == S) { s = 0; round++; }
      }
      if (ok) umma_commit_warp<false>(acc_full(b));
    }
  } else if (warp >= 4) {
    const int quad = warp & 3, which = (warp - 4) >> 2, chunks = a.n / 16, row = quad * 32 + lane;
    pdl_wait();  // (the scales, and C)
    uint32_t n = 0;
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, n++) {
      const int b = (int)(n & 1u);
      const bool ready = mbar_wait_bounded(acc_full(b), (n >> 1) & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ready)) break;  // tcgen05.ld is warp-wide: together or not at all
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int u = which; u < a.halves * chunks; u += 2) {
        const int h = u / chunks, c0 = (u - h * chunks) * 16, f = tile * tile_rows + h * a.rows + row;
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((b * a.halves + h) * cols + c0);
        uint32_t hi[16], lo[16];
        __syncwarp();  // (lanes without a row skip the stores below; tensor memory is read by the whole warp)
        tmem_ld16(taddr, hi);
        if (a.planes == 2) tmem_ld16(taddr + (uint32_t)a.n, lo);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row < a.rows && f < a.N) {
#pragma unroll
          for (int i = 0; i < 16; i++) {
            const int m = a.m_base + c0 + i;
            if (m < a.M) {
              const float v = (a.planes == 2 ? __uint_as_float(hi[i]) + __uint_as_float(lo[i]) : __uint_as_float(hi[i])) * a.alpha * (a.row_scale ? __ldg(a.row_scale + m) : 1.0f);
              if constexpr (sizeof(OutT) == 4) reinterpret_cast<float *>(a.C)[(size_t)m * a.N + f] = v;
              else reinterpret_cast<__half *>(a.C)[(size_t)m * a.N + f] = __float2half_rn(v);
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(b));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols) : "memory");
  if (abort_word && tid == 0) atomicExch(err, 2);
}

// x: [planes][M][K], `plane` elements apart
template <typename OutT>
dp_status launch_rows(dp_ctx *ctx, const __half *W, const __half *x, size_t plane, RowsArgs a) {
  EncodeTiledFn encode = get_encode();
  if (!encode) return dp_fail(ctx, DP_ERR_CUDA, "matmul (f16 weights, rows): cuTensorMapEncodeTiled is not available");
  static dp_per_device_once attr;
  const size_t budget = ctx->smem_optin - 2048;
  if (attr.pending(ctx->device)) {
    DP_CUDA(ctx, cudaFuncSetAttribute(gemm_f16w_rows_kernel<OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
    attr.done(ctx->device);
  }
  const cuuint32_t estr[3] = {1, 1, 1};
  for (a.m_base = 0; a.m_base < a.M; a.m_base += FR_BATCH) {
    const int mb = a.M - a.m_base < FR_BATCH ? a.M - a.m_base : FR_BATCH;
    a.n = (mb + 15) / 16 * 16;
    // both halves' accumulators and a second set of them in 512 columns
    const int cols = a.planes * a.n, most = 4 * cols <= 512 ? 256 : 128, per_round = ctx->sm_count * most;
    const int share = (a.N + ctx->sm_count * ((a.N + per_round - 1) / per_round) - 1) / (ctx->sm_count * ((a.N + per_round - 1) / per_round));
    a.halves = share > 128 ? 2 : 1;
    a.rows = ((share + a.halves - 1) / a.halves + 7) / 8 * 8;
    a.tiles = (a.N + a.rows * a.halves - 1) / (a.rows * a.halves);
    const size_t stage_bytes = (size_t)a.rows * a.halves * 128 + (size_t)cols * 128;
    a.stages = (int)((budget - 1024 - 128 * 128) / stage_bytes);  // an MMA reads 128 rows also of the last stage's few
    if (a.stages > FR_STAGES) a.stages = FR_STAGES;
    a.tmem_cols = 32;
    while (a.tmem_cols < 2 * a.halves * cols) a.tmem_cols *= 2;
    CUtensorMap tw, ta;
    const cuuint64_t wd[2] = {(cuuint64_t)a.K, (cuuint64_t)a.N}, ad[3] = {(cuuint64_t)a.K, (cuuint64_t)a.M, (cuuint64_t)a.planes};
    const cuuint64_t ws[1] = {(cuuint64_t)a.K * 2}, as[2] = {(cuuint64_t)a.K * 2, (cuuint64_t)plane * 2};
    const cuuint32_t wb[2] = {BK, (cuuint32_t)a.rows}, ab[3] = {BK, (cuuint32_t)a.n, (cuuint32_t)a.planes};
    CUresult r = encode(&tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void *)W, wd, ws, wb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS)
      r = encode(&ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void *)x, ad, as, ab, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return dp_fail(ctx, DP_ERR_CUDA, "matmul (f16 weights, rows): cuTensorMapEncodeTiled failed (%d) for [%d,%d] x [%d,%d]", (int)r, a.M, a.K, a.N, a.K);
    DP_LAUNCH(ctx, gemm_f16w_rows_kernel<OutT>, a.tiles < ctx->sm_count ? a.tiles : ctx->sm_count, FR_THREADS, a.stages * stage_bytes + 1024 + 128 * 128, tw, ta, a,
              ctx->dev_status);
  }
  return DP_OK;
}

}  // namespace

// C[M, N] = alpha * A[M, K] . W[N, K]^T for f16 weights and M >= 2.  f32 activations are multiplied in to f32 accuracy (two f16
// halves per element), f16 activations as they are.  *handled stays false for shapes the kernel does not take (K not a multiple
// of 64, operands off 16-byte boundaries).
dp_status dpk_gemm_f16w_rows(dp_ctx *ctx, const __half *W, const void *A, dp_dtype a_dtype, void *C, dp_dtype c_dtype, int M, int N, int K,
                             float alpha, bool *handled) {
  *handled = false;
  if (M < 2 || K < BK || K % BK || N < 1) return DP_OK;
  if ((c_dtype != DP_F32 && c_dtype != DP_F16) || (a_dtype != DP_F32 && a_dtype != DP_F16)) return DP_OK;
  if (((uintptr_t)W & 15) || (a_dtype == DP_F16 && ((uintptr_t)A & 15))) return DP_OK;
  RowsArgs a = {};
  a.C = C; a.alpha = alpha; a.M = M; a.N = N; a.K = K;
  const __half *x = (const __half *)A;
  size_t plane = (size_t)M * K;
  a.planes = 1;
  if (a_dtype == DP_F32) {
    const size_t a_bytes = ((size_t)M * K * 2 + 255) / 256 * 256;
    DP_TRY(dp_scratch(ctx, &ctx->gemm_scratch, 2 * a_bytes + (size_t)M * 4, "matmul_a_f16"));
    char *base = (char *)ctx->gemm_scratch->dptr;
    __half *hi = (__half *)base, *lo = (__half *)(base + a_bytes);
    float *scales = (float *)(base + 2 * a_bytes);
    DP_TRY(dpk_scale_cast_rows(ctx, (const float *)A, hi, lo, scales, M, K));
    x = hi; plane = a_bytes / 2; a.planes = 2; a.row_scale = scales;
  }
  DP_TRY(c_dtype == DP_F32 ? launch_rows<float>(ctx, W, x, plane, a) : launch_rows<__half>(ctx, W, x, plane, a));
  *handled = true;
  return DP_OK;
}
