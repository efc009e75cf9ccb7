// The tied head of a decoder described layer by layer for several rows of a portion: logits [R, N] = norm(rows) W^T, bf16
// weights, f32 results, 2..32 rows per launch (scoring a prompt: the logits of many of its places).
//
// HBM-bound: the table (262 MB at 32000 x 4096) is streamed once for all rows, where the one-row kernel streams it once per
// row.  32 rows at 32000 x 4096: 103 us; with that kernel 32 x 42 us and as many copies to the host between them.  A CTA of
// eight warps owns 128 table rows; the weights are the A operand of mma.sync m16n8k16 straight from global memory (16-byte
// loads; K is permuted to fit them: a lane's eight values at 32 c + 8 t feed two MMAs, four as its k of the first, four of
// the second, the B fragments likewise).  The normed rows enter as three bf16 terms that add up to their
// 24 bits, so every product is the f32 one; the products of a 64-wide slice of K are summed in a fragment of their own and
// added to the result with f32 additions, so that the tensor core's accumulation is never longer than twelve steps.
#include "layers.h"
#include "model.h"
#include "pdl.cuh"

namespace {

constexpr int HR_ROWS = DP_WANTED_ROWS;  // rows per launch
constexpr int HR_TILE = 128;             // table rows per CTA
constexpr int HR_KS = 64;                // K slice per stage
constexpr int HR_PITCH = HR_KS * 2 + 64; // bytes per staged row: 128 data + 64 pad (conflict-free 16-byte reads)

struct RowList {
  int at[HR_ROWS];
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// one block per wanted row: grouped RMSNorm, then the three bf16 terms of every value, planes [3][padded rows][K];
// blocks beyond R write the zero rows that fill the last group of eight
__global__ void __launch_bounds__(256) head_prep_kernel(const float *__restrict__ h, int h_stride, const RowList rows, int R, const GroupNorm n, int K,
                                                        __nv_bfloat16 *__restrict__ planes, size_t plane) {
  __shared__ float part[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gs = K / n.groups;
  __nv_bfloat16 *out = planes + (size_t)blockIdx.x * K;
  if ((int)blockIdx.x >= R) {
    for (int i = tid; i < K; i += 256)
      for (int j = 0; j < 3; j++) out[(size_t)j * plane + i] = __float2bfloat16_rn(0.0f);
    return;
  }
  const float *x = h + (size_t)rows.at[blockIdx.x] * h_stride;
  for (int g = 0; g < n.groups; g++) {
    float ss = 0.0f;
    for (int i = g * gs + tid; i < (g + 1) * gs; i += 256) ss = fmaf(x[i], x[i], ss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; w++) total += part[w];
    __syncthreads();
    const float inv = 1.0f / sqrtf(total / (float)gs + n.eps);
    for (int i = g * gs + tid; i < (g + 1) * gs; i += 256) {
      const float v = x[i] * inv * __bfloat162float(n.w[i]);
      const __nv_bfloat16 hi = __float2bfloat16_rn(v);
      const float r = isfinite(v) ? v - __bfloat162float(hi) : 0.0f;
      const __nv_bfloat16 mid = __float2bfloat16_rn(r);
      out[i] = hi;
      out[plane + i] = mid;
      out[2 * plane + i] = __float2bfloat16_rn(r - __bfloat162float(mid));
    }
  }
}

// NT: groups of eight rows
template <int NT>
__global__ void __launch_bounds__(256, 2) head_rows_kernel(const __nv_bfloat16 *__restrict__ W, int w_stride, const __nv_bfloat16 *__restrict__ planes, size_t plane,
                                                           float *__restrict__ C, int R, int N, int K) {
  extern __shared__ __align__(16) unsigned char hr_smem[];
  constexpr int ROWS = NT * 8, ARR = ROWS * HR_PITCH, STAGE = 3 * ARR;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int row0 = blockIdx.x * HR_TILE + warp * 16;
  const uint4 *wa = reinterpret_cast<const uint4 *>(W + (size_t)min(row0 + g, N - 1) * w_stride) + t;
  const uint4 *wb = reinterpret_cast<const uint4 *>(W + (size_t)min(row0 + g + 8, N - 1) * w_stride) + t;
  const int slices = K / HR_KS;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(hr_smem);

  auto stage_load = [&](int s) {
    const uint32_t dst = base + (uint32_t)(s & 1) * STAGE;
#pragma unroll
    for (int p = tid; p < 3 * ROWS * 8; p += 256) {
      const int arr = p / (ROWS * 8), rem = p % (ROWS * 8), r = rem >> 3, c = rem & 7;
      cp_async16(dst + arr * ARR + r * HR_PITCH + c * 16, planes + (size_t)arr * plane + (size_t)r * K + (size_t)s * HR_KS + c * 8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
  uint4 curA[2], curB[2], nxtA[2], nxtB[2];
  curA[0] = __ldg(wa); curB[0] = __ldg(wb);
  curA[1] = __ldg(wa + 4); curB[1] = __ldg(wb + 4);
  stage_load(0);
  for (int s = 0; s < slices; s++) {
    if (s + 1 < slices) {
      stage_load(s + 1);  // (this stage was last read in iteration s - 1, which ended with a barrier)
      const uint4 *na = wa + (size_t)(s + 1) * 8, *nb = wb + (size_t)(s + 1) * 8;
      nxtA[0] = __ldg(na); nxtB[0] = __ldg(nb);
      nxtA[1] = __ldg(na + 4); nxtB[1] = __ldg(nb + 4);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const unsigned char *st = hr_smem + (s & 1) * STAGE;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int arr = 2; arr >= 0; arr--) {  // the small terms first
#pragma unroll
        for (int hf = 0; hf < 2; hf++) {
          const uint4 b = *reinterpret_cast<const uint4 *>(st + arr * ARR + (nt * 8 + g) * HR_PITCH + hf * 64 + t * 16);
          mma_bf16(sum, curA[hf].x, curB[hf].x, curA[hf].y, curB[hf].y, b.x, b.y);
          mma_bf16(sum, curA[hf].z, curB[hf].z, curA[hf].w, curB[hf].w, b.z, b.w);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j++) acc[nt][j] += sum[j];
    }
    __syncthreads();
    curA[0] = nxtA[0]; curA[1] = nxtA[1];
    curB[0] = nxtB[0]; curB[1] = nxtB[1];
  }
#pragma unroll
  for (int nt = 0; nt < NT; nt++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int m = nt * 8 + 2 * t + (j & 1), row = row0 + g + (j >> 1) * 8;
      if (m < R && row < N) C[(size_t)m * N + row] = acc[nt][j];
    }
}

template <int NT>
dp_status launch_head(dp_ctx *ctx, const __nv_bfloat16 *W, int w_stride, const __nv_bfloat16 *planes, size_t plane, float *C, int R, int N, int K) {
  constexpr size_t smem = (size_t)2 * 3 * NT * 8 * HR_PITCH;
  static_assert(smem <= 48 * 1024, "stages exceed the default shared memory");
  DP_LAUNCH(ctx, head_rows_kernel<NT>, (unsigned)((N + HR_TILE - 1) / HR_TILE), 256, smem, W, w_stride, planes, plane, C, R, N, K);
  return DP_OK;
}

}  // namespace

bool dpk_head_rows_ok(int K) { return K % HR_KS == 0; }
size_t dpk_head_rows_scratch(int K) { return (size_t)3 * HR_ROWS * K * 2; }

// logits [R, N] of the rows h + at[i] * h_stride, R <= DP_WANTED_ROWS; scratch of dpk_head_rows_scratch bytes.
// The table's rows are w_stride elements apart (multiple of 8).
dp_status dpk_head_rows(dp_ctx *ctx, const float *h, int h_stride, const int *at, int R, const GroupNorm &n, const __nv_bfloat16 *W, int w_stride, void *scratch,
                        float *C, int N, int K) {
  DP_CHECK(ctx, R > 0 && R <= HR_ROWS && dpk_head_rows_ok(K) && w_stride % 8 == 0, "head: %d rows of %d values", R, K);
  RowList list = {};
  for (int i = 0; i < R; i++) list.at[i] = at[i];
  const int nt = R <= 8 ? 1 : R <= 16 ? 2 : 4;
  const size_t plane = (size_t)nt * 8 * K;
  __nv_bfloat16 *planes = (__nv_bfloat16 *)scratch;
  DP_LAUNCH(ctx, head_prep_kernel, (unsigned)(nt * 8), 256, 0, h, h_stride, list, R, n, K, planes, plane);
  if (nt == 1) return launch_head<1>(ctx, W, w_stride, planes, plane, C, R, N, K);
  if (nt == 2) return launch_head<2>(ctx, W, w_stride, planes, plane, C, R, N, K);
  return launch_head<4>(ctx, W, w_stride, planes, plane, C, R, N, K);
}
