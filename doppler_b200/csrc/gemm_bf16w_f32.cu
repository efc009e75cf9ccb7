// Products of several f32 rows with bf16 weights, the 32-bit mode of the decoders described layer by layer:
// C [M, N] = A [M, K] W [N, K]^T to f32 accuracy on the tensor cores.
//
// A value of f32 is the sum of three bf16 numbers (its 24 bits cut in eights), and a product of two bf16 numbers is exact
// in f32, so three bf16 products per weight give the f32 products.  What the tensor core adds up is kept short: the twelve
// MMAs of one 64-wide K step (the small terms first) go into an accumulator of their own, one of four in tensor memory,
// and eight warps add it to f32 registers while the next steps are multiplied.  Against 64-bit results a decoder's logits are
// off by 2.8e-7; with a chain of f32 FMAs for every product they were off by 1.0e-6.
//
// Bound: the tensor pipe in long products (three times the bf16 work), the tiles' fixed cost in short ones.  The weights
// are the MMA's M side (128 rows), the activation rows its N side (32..128, chosen so that the tiles fill whole waves); a
// stage of the ring holds the weight tile once and the three terms of the activations.  Persistent, one CTA per SM.  The
// products of a 700-token prompt (width 1024, 4 layers) average 41 us and 4 us for the terms; the prompt and four tokens
// behind it took 5.97 ms with CUDA-core FMAs, 3.29 with these products, and take 2.94 ms now.
// Every wait is bounded.
//
// Optional decay and gated activation as in gemm_bf16.cu, the activation stored as f32.
#include "layers.h"
#include "decay.cuh"
#include "pdl.cuh"
#include "umma.cuh"

using namespace umma;

namespace {

constexpr int FX_EPI = 8;                       // draining warps: two per quarter of the lanes
constexpr int FX_THREADS = (4 + FX_EPI) * 32;
constexpr int FX_BUFS = 4;                      // accumulators, also the ring of "K step multiplied" barriers
constexpr int FX_BN = 128;                      // most activation rows of a tile
constexpr uint32_t FX_W_TILE = 128u * 128u;     // 128 weight rows x 64 bf16

struct F32Args {
  float *C;
  int M, N, K, bn, stages, tiles_n, tiles_m, tmem_cols;
  GluOut glu;
  DecayOut decay;
};

__device__ __forceinline__ float glu_f32(float g, float u, const GluOut &a) {
  if (a.limit > 0.0f) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
  }
  return g * (1.0f / (1.0f + expf(-a.slope * g))) * (u + a.shift);
}

// rows of A -> three planes [M][kp] of bf16 that add up to it (zeros beyond K); an infinity or NaN is the first term alone
__global__ void __launch_bounds__(256) split_bf16x3_kernel(const float *__restrict__ A, int a_stride, __nv_bfloat16 *__restrict__ out, size_t plane, int M, int K, int kp) {
  pdl_launch();
  pdl_wait();
  const int pairs = kp / 2;
  const long total = (long)M * pairs;
  for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long)gridDim.x * 256) {
    const int r = (int)(i / pairs), c = (int)(i - (long)r * pairs) * 2;
    uint32_t t[3] = {0u, 0u, 0u};
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const float v = c + j < K ? A[(size_t)r * a_stride + c + j] : 0.0f;
      uint32_t b[3];
      if (isfinite(v)) {
        b[0] = __float_as_uint(v) & 0xffff0000u;
        const float r1 = v - __uint_as_float(b[0]);
        b[1] = __float_as_uint(r1) & 0xffff0000u;
        b[2] = __float_as_uint(r1 - __uint_as_float(b[1]));  // eight bits are left
      } else {
        b[0] = isnan(v) ? 0x7fc00000u : __float_as_uint(v);
        b[1] = b[2] = 0u;
      }
#pragma unroll
      for (int k = 0; k < 3; k++) t[k] |= (b[k] >> 16) << (16 * j);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) *reinterpret_cast<uint32_t *>(out + (size_t)k * plane + (size_t)r * kp + c) = t[k];
  }
}

__global__ void __launch_bounds__(FX_THREADS, 1) gemm_bf16w_f32_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                                                                          const F32Args a, int *__restrict__ err) {
  extern __shared__ uint8_t fx_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(fx_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bars[FX_BUFS * 3];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t S = (uint32_t)a.stages, x_tile = (uint32_t)a.bn * 128u, stage_bytes = FX_W_TILE + 3u * x_tile;
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](uint32_t s) { return bar0 + 8u * s; };                       // stages <= FX_BUFS
  auto done = [&](uint32_t b) { return bar0 + 8u * (FX_BUFS + b); };           // K step it: ring of FX_BUFS
  auto drained = [&](uint32_t b) { return bar0 + 8u * (2 * FX_BUFS + b); };
  const int tiles = a.tiles_n * a.tiles_m, ksteps = (a.K + BK - 1) / BK;

  pdl_launch();
  pdl_wait();
  if (tid == 0) {
    for (uint32_t b = 0; b < FX_BUFS; b++) { mbar_init(full(b), 1); mbar_init(done(b), 1); mbar_init(drained(b), FX_EPI); }
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
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int n0 = (tile / a.tiles_m) * 128, m0 = (tile % a.tiles_m) * a.bn;
        for (int k = 0; k < ksteps; k++, it++) {
          const uint32_t s = it % S, before = it - S;  // the step that used this stage last
          if (it >= S && !mbar_wait_bounded(done(before % FX_BUFS), (before / FX_BUFS) & 1u, abort_flag)) { ok = false; break; }
          mbar_expect_tx(full(s), stage_bytes);
          const uint32_t dst = smem_u32(smem) + s * stage_bytes;
          tma_load_2d(dst, &tmap_w, k * BK, n0, full(s));
          asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst + FX_W_TILE),
                       "l"(&tmap_a), "r"(k * BK), "r"(m0), "r"(0), "r"(full(s))  // all three terms
                       : "memory");
        }
      }
      // no copy may still be in flight when the CTA ends, also where a wait gave up
      const uint32_t held = it < S ? it : S;
      for (uint32_t i = it - held; i < it; i++)
        for (uint32_t poll = 0; poll < (1u << 20) && !mbar_try_wait(full(i % S), (i / S) & 1u); poll++) {}
    }
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.bn >> 3) << 17) | (128u >> 4 << 24);  // D = f32, A = B = bf16, K-major
    const uint64_t first = umma_desc_sw128(smem_u32(smem));
    uint32_t it = 0, s = 0, round = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      for (int k = 0; k < ksteps; k++, it++) {
        const uint32_t b = it % FX_BUFS;
        if (it >= FX_BUFS && !mbar_wait_warp(drained(b), ((it / FX_BUFS) - 1u) & 1u, abort_flag)) { ok = false; break; }
        if (!mbar_wait_warp(full(s), round & 1u, abort_flag)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t w = first + (uint64_t)(s * (stage_bytes >> 4)), x = w + (FX_W_TILE >> 4);
        const uint32_t acc = tmem + b * (uint32_t)a.bn;
        umma_step_warp<false>(acc, w, x + 2u * (x_tile >> 4), idesc, 0u);
        umma_step_warp<false>(acc, w, x + (x_tile >> 4), idesc, 1u);
        umma_step_warp<false>(acc, w, x, idesc, 1u);
        umma_commit_warp<false>(done(b));  // the stage is free, the step's sums are complete
        if (++s == S) { s = 0; round++; }
      }
    }
  } else if (warp >= 4) {
    const int quad = warp & 3, half = (warp - 4) >> 2, cw = a.bn / 2;  // this warp's columns: half * cw ..
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const int n0 = (tile / a.tiles_m) * 128, m0 = (tile % a.tiles_m) * a.bn + half * cw;
      float sum[FX_BN / 2];
#pragma unroll
      for (int i = 0; i < FX_BN / 2; i++) sum[i] = 0.0f;
      for (int k = 0; k < ksteps; k++, it++) {
        const uint32_t b = it % FX_BUFS;
        const bool ready = mbar_wait_bounded(done(b), (it / FX_BUFS) & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, ready)) { ok = false; break; }  // tcgen05.ld is warp-wide: together or not at all
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + b * (uint32_t)a.bn + (uint32_t)(half * cw);
#pragma unroll
        for (int c = 0; c < FX_BN / 32; c++) {
          if (c * 16 < cw) {  // (uniform)
            uint32_t r[16];
            tmem_ld16(taddr + (uint32_t)(c * 16), r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; i++) sum[c * 16 + i] += __uint_as_float(r[i]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(drained(b));
      }
      if (!ok) break;
      const int f = n0 + quad * 32 + lane;
      const bool is_up = lane & 8;
      float rate = 0.0f, bias = 0.0f;
      if (a.decay.rate && f < a.N) { rate = a.decay.rate[f]; bias = a.decay.bias[f]; }
#pragma unroll
      for (int i = 0; i < FX_BN / 2; i += 2) {
        if (i >= cw || m0 + i >= a.M) continue;  // (uniform)
        if (a.glu.dst) {
          // a gate row and its up row are eight lanes apart: the gate's lane takes the even activation rows, the other the odd
          const float got = __shfl_xor_sync(0xffffffffu, is_up ? sum[i] : sum[i + 1], 8);
          const float gv = is_up ? got : sum[i], uv = is_up ? sum[i + 1] : got;
          const int row = m0 + i + (is_up ? 1 : 0);
          if (f < a.N && row < a.M) reinterpret_cast<float *>(a.glu.dst)[(size_t)row * a.glu.stride + (f >> 4) * 8 + (f & 7)] = glu_f32(gv, uv, a.glu);
        } else if (f < a.N) {
#pragma unroll
          for (int j = 0; j < 2; j++)
            if (m0 + i + j < a.M) a.C[(size_t)(m0 + i + j) * a.N + f] = a.decay.rate ? decay_of(sum[i + j], rate, bias) : sum[i + j];
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols) : "memory");
  if (abort_word && tid == 0) atomicExch(err, 2);
}

}  // namespace

dp_status dpk_gemm_bf16w_f32(dp_ctx *ctx, const __nv_bfloat16 *W, int w_stride, const float *A, int a_stride, float *C, int M, int N, int K, const GluOut *glu,
                             const DecayOut *decay) {
  DP_CHECK(ctx, M > 0 && N > 0 && K > 0 && w_stride % 8 == 0 && K <= w_stride && K <= a_stride, "gemm (bf16 weights, f32): bad shape");
  DP_CHECK(ctx, !glu || N % 16 == 0, "gemm (bf16): gate and up rows come in groups of sixteen");
  EncodeTiledFn encode = get_encode();
  if (!encode) return dp_fail(ctx, DP_ERR_CUDA, "gemm (bf16 weights, f32): cuTensorMapEncodeTiled is not available");
  // the three terms of the activations: one scratch of the context, reused in stream order
  const int kp = (K + 7) / 8 * 8;
  const size_t plane = ((size_t)M * kp + 63) / 64 * 64;
  DP_TRY(dp_scratch(ctx, &ctx->gemm_scratch, 3 * plane * 2, "matmul_a_bf16x3"));
  __nv_bfloat16 *terms = (__nv_bfloat16 *)ctx->gemm_scratch->dptr;
  {
    size_t grid = ((size_t)M * (kp / 2) + 255) / 256;
    if (grid > (size_t)ctx->sm_count * 16) grid = (size_t)ctx->sm_count * 16;
    DP_LAUNCH(ctx, split_bf16x3_kernel, (unsigned)grid, 256, 0, A, a_stride, terms, plane, M, K, kp);
  }
  F32Args a = {};
  a.C = C; a.M = M; a.N = N; a.K = K;
  if (glu) a.glu = *glu;
  if (decay) a.decay = *decay;
  a.tiles_n = (N + 127) / 128;
  double best = -1.0;
  for (int bn = 32; bn <= FX_BN; bn += 32) {  // the width with the least (waves x (products of a tile + its fixed cost))
    const long tiles = (long)a.tiles_n * ((M + bn - 1) / bn), waves = (tiles + ctx->sm_count - 1) / ctx->sm_count;
    const double cost = (double)waves * ((bn < 64 ? 64 : bn) + 16);  // narrow tiles are paced by the weight operand's shared-memory reads
    if (best < 0 || cost < best) { best = cost; a.bn = bn; }
  }
  a.tiles_m = (M + a.bn - 1) / a.bn;
  const uint32_t stage_bytes = FX_W_TILE + 3u * (uint32_t)a.bn * 128u;
  const size_t budget = ctx->smem_optin - 2048;
  a.stages = (int)((budget - 1024) / stage_bytes);
  if (a.stages > FX_BUFS) a.stages = FX_BUFS;
  a.tmem_cols = FX_BUFS * a.bn <= 128 ? 128 : FX_BUFS * a.bn <= 256 ? 256 : 512;
  CUtensorMap tw, ta;
  const cuuint32_t estr[3] = {1, 1, 1};
  const cuuint64_t wd[2] = {(cuuint64_t)K, (cuuint64_t)N}, ad[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
  const cuuint64_t ws[1] = {(cuuint64_t)w_stride * 2}, as[2] = {(cuuint64_t)kp * 2, (cuuint64_t)plane * 2};
  const cuuint32_t wb[2] = {BK, 128}, ab[3] = {BK, (cuuint32_t)a.bn, 3};
  CUresult r = encode(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)W, wd, ws, wb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS)
    r = encode(&ta, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void *)terms, ad, as, ab, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return dp_fail(ctx, DP_ERR_CUDA, "gemm (bf16 weights, f32): cuTensorMapEncodeTiled failed (%d) for [%d,%d] x [%d,%d]", (int)r, M, K, N, K);
  static dp_per_device_once attr;
  if (attr.pending(ctx->device)) {
    DP_CUDA(ctx, cudaFuncSetAttribute(gemm_bf16w_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
    attr.done(ctx->device);
  }
  const int tiles = a.tiles_n * a.tiles_m, grid = tiles < ctx->sm_count ? tiles : ctx->sm_count;
  DP_LAUNCH(ctx, gemm_bf16w_f32_tc_kernel, grid, FX_THREADS, (size_t)a.stages * stage_bytes + 1024, tw, ta, a, ctx->dev_status);
  return DP_OK;
}
