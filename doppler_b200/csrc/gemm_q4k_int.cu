// Q4_K GEMM of many activation rows on the 5th-generation tensor cores with INTEGER weight tiles (the weights exact).
//
//   C[M, N] = alpha * A[M, K] . W[N, K]^T,  w = d * (sc * q) - dmin * m  per 256-weight super-block / 32-weight sub-block
//
// sc * q <= 945 is exact in f16, so for every super-block the tensor core multiplies the integer tile
//
//   P[n, m] = sum over the 256 k of (sc * q)[n, k] * x[m, k]
//
// and d is applied once per super-block when P is read back from tensor memory and added to f32 registers.  One product
// per K step for f16 activations and two for f32 ones (x * 2^-e = hi + lo, both f16) give the result to f32 accuracy, where
// tiles of dequantised weights (an f16 value and its residue) need two and three.  No weight is rounded, and the tensor
// core never adds up more than one super-block: the error against 64 bits is 9e-7 where those tiles are off by 4e-6 to 4e-5.
//
// The min term  sum over sub-blocks of  -(dmin * m)[n, s] * xsum[m, s]  is a small product of its own, with K / 32 instead
// of K: at the start of a tile up to ten super-blocks at a time share one 256-wide "sum unit" whose columns are
// [ hi | lo | hi ] parts of dmin * m against [ hi | hi | lo ] parts of the sub-block sums (f16 pairs; dmin scaled by a power
// of two per weight row, the sums by one per activation row, both undone on read-back).  hi + lo holds all 17 bits of
// dmin * m; 22 bits of the sums.
//
// The tensor core cuts off what falls below its accumulator's last bit, so that products added while the accumulator is
// small cost no accuracy.  f32 rows have two orders of their products: lo and hi in turn for every K slice, or (lo_first) the lo
// products of the whole super-block before its hi products, which waits for both of its groups first.  Error against 64 bits,
// random normal rows, K 1024 to 12288: 9.3e-7 in turn, 4.6e-7 to 5.1e-7 lo first (f32 FMAs: 5.7e-7 at K = 1024, 1.9e-6 at
// 11111; gemm_q4k_tc_rows.cu: 5.2e-7 to 5.4e-7; dequantised tiles: 3.7e-6 to 2.2e-5).  us in turn -> lo first: 128 x 6144 x 4096
// 44.1 -> 45.7, 256 x 24576 x 4096 137 -> 144, 512 x 6144 x 4096 (192-wide tiles, a ring of two weight groups) 69 -> 79.  Lo
// first therefore where calls would otherwise lose accuracy: shapes no tile divides, which f32 FMAs multiplied, and rows of
// several prompts, which one by one go through gemm_q4k_tc_rows.cu.  The small products of a sum unit come first from seven
// super-blocks on (K = 12288: 6.3e-7 -> 5.3e-7); up to six, what is cut off there and in the super-blocks cancels in part
// (four: 4.6e-7, with the small ones first 5.1e-7), and so it does at any number where lo and hi take turns (9.2e-7, 1.08e-6).
//
// A cluster of two CTAs owns 256 weight rows x bn activation rows (cta_group::2, M = 256: CTA r holds 128 weight rows and
// their 128 lanes of the result, and half of the activation tile).  Sharing the activation tile halves its L2 and
// shared-memory traffic.  The weight tiles are the A operand in TENSOR MEMORY: out of shared memory every MMA would read
// its 4 KB slice once more, beside the activations' copies and the builders' stores (512 x 12288 x 4096 with f16 rows:
// 116 -> 109 us).  Two accumulators of up to 192 columns leave room for two to four groups of weights; a super-block is read
// back while the next one is multiplied.  Clusters walk the (tile, part of K) items persistently; bn is chosen so that the
// items fill whole waves of clusters.
//
// Roles per CTA (registers are moved to the draining warps with setmaxnreg): warp 0 TMA of activations, warps 1 and 2 MMA
// issue (CTA 0; warp 1 of CTA 1 relays its builders' barrier), warp 3 TMA of packed super-blocks, eight warps build weight
// tiles out of them (a thread one weight row, a warp one of the two K steps), eight drain (a lane quarter and half of the
// columns per warp, up to 96 sums per thread).  A ring group is two 64-wide K steps; one commit per group frees activation
// and weight stages and, on a unit's second group, hands the accumulator to the drains.  What bounds it: the tensor pipe is
// active 57 % of the time (1024 x 24576 x 4096, f32 rows); the rest is the hand-over of accumulators between MMAs and
// drains and the stores at the end of a tile.  Every wait is bounded; on give-up the CTA raises the status word and still
// frees its tensor memory.
#include "common.h"
#include "mbar.cuh"
#include "pdl.cuh"
#include "q4k.cuh"
#include "umma.cuh"

namespace {

using namespace umma;

constexpr int QI_ROWS = 128;       // weight rows per CTA
constexpr int QI_BN = 192;         // most activation rows of a tile
constexpr int QI_SUMS = 10;        // super-blocks of a sum unit: 3 * 8 * 10 = 240 of its 256 columns
constexpr int QI_SUMS_LO_FIRST = 8, QI_SUMS_LONG = 6;  // ... lo first; and where a part is longer than 24 (more f32 additions)
constexpr int QI_BUILDERS = 8, QI_DRAINERS = 8;
constexpr int QI_THREADS = (4 + QI_BUILDERS + QI_DRAINERS) * 32;
constexpr int QI_RING = 4;         // most stages of a ring; also the rings of barriers that go by group
constexpr int QI_SCALES = 8;       // units whose row scales are kept (a drain is at most two units behind the builders' ring)

struct IntPlan {
  int bpr, parts, pb, npu;         // super-blocks of a row; parts of K; super-blocks and sum units of a part
  int bn, tiles_n, tiles_m, items;
  int sa, sb, sp;                  // stages: groups of activations, groups of weight tiles (tensor memory), packed super-blocks
};

__host__ __device__ __forceinline__ int qi_sum_begin(const IntPlan &p, int u) { return u * p.pb / p.npu; }
// places (eighths of columns) of the products of a sum unit of nsb super-blocks: [hi hi], [lo hi], [hi lo] of weights and sums
struct QiSumOrder {
  int hh, lh, hl;
};
constexpr QiSumOrder qi_sums_in_turn(int nsb) { return QiSumOrder{0, nsb, 2 * nsb}; }
constexpr QiSumOrder qi_sums_lo_first(int nsb) { return nsb < 7 ? qi_sums_in_turn(nsb) : QiSumOrder{2 * nsb, 0, nsb}; }

constexpr uint32_t QI_P_STAGE = QI_ROWS * Q4K_BLOCK_BYTES;  // packed super-blocks of the CTA's weight rows
constexpr uint32_t QI_W_COLS = 64;                          // tensor-memory columns of a weight group: 128 K, two f16 each
__host__ __device__ __forceinline__ uint32_t qi_x_tile(const IntPlan &p) { return (uint32_t)(p.bn / 2) * 128u; }
__host__ __device__ __forceinline__ uint32_t qi_x_stage(const IntPlan &p, bool lo) { return qi_x_tile(p) * (lo ? 4u : 2u); }
__host__ __device__ __forceinline__ uint32_t qi_rings(const IntPlan &p, bool lo) { return (uint32_t)p.sa * qi_x_stage(p, lo) + (uint32_t)p.sp * QI_P_STAGE; }

struct QiRing {  // a place in a ring of n stages and how often the ring has gone round
  uint32_t i = 0, uses = 0;
  __device__ __forceinline__ void next(int n) {
    if (++i == (uint32_t)n) { i = 0; uses++; }
  }
};

__device__ __forceinline__ uint32_t qi_hfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t qi_hmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t qi_hsub2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// e with 2^e <= |dmin| < 2^(e + 1) for the largest |dmin| of a weight row in a sum unit: times 2^(8 - e) the products stay below 2^15
__device__ __forceinline__ int qi_exponent(float most) {
  const int e = (int)((__float_as_uint(most) >> 23) & 0xffu) - 127;
  return max(-100, min(100, e));
}
__device__ __forceinline__ float qi_pow2(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

// arrive on a barrier of the pair's other CTA.  (With a release at cluster scope the arrive costs a thousand cycles, in the
// drains' path to the next super-block.  Nothing that generic loads read goes this way: tensor memory is ordered by
// tcgen05.wait and the tcgen05 fences, and the row scales have barriers of their own inside each CTA.)
__device__ __forceinline__ void qi_arrive_remote(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// MMA of the pair with the A operand in tensor memory
__device__ __forceinline__ void qi_umma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void qi_tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void qi_tmem_st4(uint32_t taddr, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}

struct IntOut {
  float alpha;
  const float *row_scale;  // per activation row, or null
  const float *sum_scale;  // per activation row: undoes the scale of its sub-block sums, or null
  const float *residual;   // added to the result (f32, may be the output itself), or null
  int silu;                // f32 output: weight rows are gate|up pairs (groups of sixteen); store silu(gate) * up, N / 2 columns
};

// F32: f16 activations (0), f32 activations with lo and hi products in turn (1) or the lo products first (2)
template <int F32, typename OutT>
__global__ void __launch_bounds__(QI_THREADS, 1) gemm_q4k_int_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_lo,
                                                                     const __grid_constant__ CUtensorMap tmap_s, const __grid_constant__ CUtensorMap tmap_w,
                                                                     const uint8_t *__restrict__ W, OutT *C, int M, int N, IntPlan p, IntOut o,
                                                                     int *__restrict__ err) {
  constexpr bool LO = F32 > 0;
  extern __shared__ uint8_t qi_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(qi_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bar_words[5 * QI_RING + 2];
  __shared__ float row_scales[QI_SCALES][QI_ROWS];  // what a unit's product is multiplied by on read-back: d, or the sum unit's power of two
  __shared__ uint32_t tmem_word;
  __shared__ int abort_word;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = cluster_ctarank();
  const int cluster = (int)(blockIdx.x >> 1), clusters = (int)(gridDim.x >> 1);
  const int hb = p.bn / 2, units = p.npu + p.pb;
  const uint32_t x_tile = qi_x_tile(p), x_step = x_tile * (LO ? 2u : 1u), x_stage = 2u * x_step;
  uint8_t *ring_p = smem + (uint32_t)p.sa * x_stage;
  volatile int *abort_flag = &abort_word;
  const uint32_t bars = smem_u32(bar_words);
  // One barrier says that a group's activations and weights are there (a wait costs the MMA lane two hundred cycles).  It
  // goes by group like "multiplied", not by stage: a group is loaded or built only after the one `ring depth` before it has
  // been multiplied, so neither barrier is used again too early.
  auto full = [&](uint32_t g) { return bars + 8u * (g & (QI_RING - 1)); };
  auto done = [&](uint32_t g) { return bars + 8u * (QI_RING + (g & (QI_RING - 1))); };
  auto parity = [&](uint32_t g) { return (g / QI_RING) & 1u; };
  auto full_p = [&](uint32_t s) { return bars + 8u * (2 * QI_RING + s); };
  auto free_p = [&](uint32_t s) { return bars + 8u * (3 * QI_RING + s); };
  // The row scales of unit n are written: builders to drains of the same CTA (by way of "full", the MMAs and "multiplied" they
  // would leave the CTA and come back through arrives that order nothing there).  The ring is long enough: a builder reaches
  // unit n + 4 only after unit n + 2 has been started, and that after every drain has handed back unit n.
  auto scaled = [&](uint32_t n) { return bars + 8u * (4 * QI_RING + (n & (QI_RING - 1))); };
  auto empty = [&](uint32_t b) { return bars + 8u * (5 * QI_RING + b); };
  // item -> tile and part: neighbouring clusters share the weight rows
  auto tile_n_of = [&](int item) { return item / (p.tiles_m * p.parts); };
  auto tile_m_of = [&](int item) { return item % p.tiles_m; };
  auto part_of = [&](int item) { return (item / p.tiles_m) % p.parts; };
  // unit -> super-block: every item starts at its own place, so that clusters do not ask L2 for the same lines at once
  auto block_of = [&](int item, int u) { return part_of(item) * p.pb + (u - p.npu + item) % p.pb; };

  // No early launch of dependents here: in decode steps of 65 to 256 sequences the next kernel was seen to read rows that this one
  // (a launch of clusters without the programmatic attribute) had not stored yet, its own wait notwithstanding.  It now
  // starts when this kernel is complete.
  pdl_wait();
  if (tid == 0) {
    for (uint32_t s = 0; s < QI_RING; s++) {
      // CTA 0: the activation copies' expected bytes, its builders, the relay of CTA 1; CTA 1: its builders
      mbar_init(full(s), rank == 0 ? QI_BUILDERS + 2 : QI_BUILDERS);
      mbar_init(done(s), 1);
      mbar_init(full_p(s), 1);
      mbar_init(free_p(s), QI_BUILDERS);
      mbar_init(scaled(s), QI_BUILDERS / 2);
    }
    for (uint32_t b = 0; b < 2; b++) mbar_init(empty(b), 2 * QI_DRAINERS);  // CTA 0's: the drains of both CTAs
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_word)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // columns: two accumulators, then the weight groups
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_word), tmem_w = tmem + 2u * (uint32_t)p.bn;

  // 4 warps x 40 (lo first: 48) + 8 x 72 + 8 x 144 registers, of what the launch holds (20 warps x 96)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F32 == 2 ? 48 : 40));
    if (warp == 0 && lane == 0) {
      // ---------------- activation tiles: this CTA's half of the rows ----------------
      uint32_t g = 0;
      QiRing r;
      bool ok = true;
      for (int item = cluster; item < p.items && ok; item += clusters) {
        const int row0 = tile_m_of(item) * p.bn + (int)rank * hb, part = part_of(item);
        for (int u = 0; u < units && ok; u++) {
          const bool sums = u < p.npu;
          const int x0 = sums ? (part * p.npu + u) * 256 : block_of(item, u) * 256;
          for (int h = 0; h < 2; h++, g++, r.next(p.sa)) {
            const uint32_t before = g - (uint32_t)p.sa;  // the group that used this stage last
            if (r.uses && !mbar_wait_bounded(done(before), parity(before), abort_flag)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(full(g), 2u * 2u * x_tile * (LO && !sums ? 2u : 1u));  // both CTAs' bytes
            const uint32_t dst = smem_u32(smem) + r.i * x_stage, bar0 = mapa_shared(full(g), 0u);
            for (int j = 0; j < 2; j++) {
              const int x = x0 + (h * 2 + j) * BK;
              tma_load_2d_2sm(dst + (uint32_t)j * x_step, sums ? &tmap_s : &tmap_x, x, row0, bar0);
              if (LO && !sums) tma_load_2d_2sm(dst + (uint32_t)j * x_step + x_tile, &tmap_lo, x, row0, bar0);
            }
          }
        }
      }
      // no copy of the pair may still be in flight at the end, also where a wait gave up (the builders' arrivals are missing then)
      if (rank == 0 && g > 0)
        for (uint32_t poll = 0; poll < (1u << 16) && !mbar_try_wait(full(g - 1), parity(g - 1)); poll++) {}
    } else if (warp == 3 && lane == 0) {
      // ---------------- packed super-blocks of this CTA's weight rows ----------------
      QiRing r;
      uint32_t n = 0;
      bool ok = true;
      for (int item = cluster; item < p.items && ok; item += clusters)
        for (int u = p.npu; u < units; u++, n++, r.next(p.sp)) {
          if (r.uses && !mbar_wait_bounded(free_p(r.i), (r.uses - 1u) & 1u, abort_flag)) { ok = false; break; }
          mbar_expect_tx(full_p(r.i), QI_P_STAGE);
          tma_load_2d(smem_u32(ring_p) + r.i * QI_P_STAGE, &tmap_w, block_of(item, u) * Q4K_BLOCK_BYTES, tile_n_of(item) * 256 + (int)rank * QI_ROWS, full_p(r.i));
        }
      const uint32_t held = n < (uint32_t)p.sp ? n : (uint32_t)p.sp;
      for (uint32_t i = n - held; i < n; i++)
        for (uint32_t poll = 0; poll < (1u << 20) && !mbar_try_wait(full_p(i % (uint32_t)p.sp), (i / (uint32_t)p.sp) & 1u); poll++) {}
    } else if (warp == 1 && lane == 0 && rank == 1) {
      // ---------------- CTA 1: its half of a weight group is written ----------------
      const uint32_t full0 = mapa_shared(full(0), 0u);
      uint32_t g = 0;
      bool ok = true;
      for (int item = cluster; item < p.items && ok; item += clusters)
        for (int u = 0; u < 2 * units; u++, g++) {
          if (!mbar_wait_bounded(full(g), parity(g), abort_flag)) { ok = false; break; }
          qi_arrive_remote(full0 + 8u * (g & (QI_RING - 1)));
        }
    } else if ((warp == 1 || warp == 2) && lane == 0 && rank == 0) {
      // ---------------- MMA issue for the pair: warp 1 the even units, warp 2 the odd ones, each into its own accumulator ----------------
      // The queue in front of the tensor cores is short: a lane that issues everything leaves them idle while it waits for the
      // next group's barrier.  Two lanes: one waits while the other's MMAs run (4960 -> 3970 cycles per super-block of a tile of
      // 160 f32 rows).  Made to strictly take turns they were slower: the hand-over is one more wait.
      const uint32_t idesc = umma_idesc_f16(256, p.bn), to_step = x_step >> 4, to_lo = x_tile >> 4;
      const int mine = warp - 1, total = units * (cluster < p.items ? (p.items - 1 - cluster) / clusters + 1 : 0);
      const uint32_t acc = tmem + (uint32_t)(mine * p.bn);
      QiRing rx, rw;
      if (mine == 1)
        for (int i = 0; i < 2; i++) { rx.next(p.sa); rw.next(p.sb); }
      bool ok = true;
      int u = mine;  // unit of the item
      for (int n = mine; n < total && ok; n += 2) {
        if (n >= 2 && !mbar_wait_bounded(empty((uint32_t)mine), (uint32_t)((n >> 1) - 1) & 1u, abort_flag)) break;
        const bool sums = u < p.npu;
        // K slices of sixteen: a sum unit's columns are three for every sub-block
        const int slices = sums ? (3 * (qi_sum_begin(p, u + 1) - qi_sum_begin(p, u)) + 1) / 2 : 16;
        if (F32 == 2 && !sums) {
          uint32_t w0[2];
          uint64_t x0[2];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const uint32_t g = 2u * (uint32_t)n + (uint32_t)h;
            if (!mbar_wait_bounded(full(g), parity(g), abort_flag)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            w0[h] = tmem_w + rw.i * QI_W_COLS;
            x0[h] = umma_desc_sw128(smem_u32(smem) + rx.i * x_stage);
#pragma unroll
            for (int k = 0; k < 8; k++) qi_umma(acc, w0[h] + 8u * k, x0[h] + to_lo + (k >> 2) * to_step + 2 * (k & 3), idesc, h == 0 && k == 0 ? 0u : 1u);
            rx.next(p.sa);
            rw.next(p.sb);
          }
          if (!ok) break;
#pragma unroll
          for (int h = 0; h < 2; h++) {
#pragma unroll
            for (int k = 0; k < 8; k++) qi_umma(acc, w0[h] + 8u * k, x0[h] + (k >> 2) * to_step + 2 * (k & 3), idesc, 1u);
            umma_commit_2sm(done(2u * (uint32_t)n + (uint32_t)h));
          }
        } else {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint32_t g = 2u * (uint32_t)n + (uint32_t)h;
          if (!mbar_wait_bounded(full(g), parity(g), abort_flag)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t w0 = tmem_w + rw.i * QI_W_COLS;  // a slice of sixteen K: eight columns
          const uint64_t x0 = umma_desc_sw128(smem_u32(smem) + rx.i * x_stage);
          if (!sums) {
#pragma unroll
            for (int k = 0; k < 8; k++) {  // descriptors differ by constants: an MMA must cost its lane a few instructions
              const uint64_t x = x0 + (k >> 2) * to_step + 2 * (k & 3);
              qi_umma(acc, w0 + 8u * k, x, idesc, h == 0 && k == 0 ? 0u : 1u);
              if constexpr (LO) qi_umma(acc, w0 + 8u * k, x + to_lo, idesc, 1u);
            }
          } else {
            for (int k = 0; k < 8 && h * 8 + k < slices; k++) qi_umma(acc, w0 + 8u * k, x0 + (k >> 2) * to_step + 2 * (k & 3), idesc, h == 0 && k == 0 ? 0u : 1u);
          }
          umma_commit_2sm(done(g));
          rx.next(p.sa);
          rw.next(p.sb);
        }
        }
        for (int i = 0; i < 2; i++) { rx.next(p.sa); rw.next(p.sb); }  // the other lane's unit
        u += 2;
        if (u >= units) u -= units;
      }
    }
  } else if (warp < 4 + QI_BUILDERS) {
    // ---------------- weight tiles into tensor memory: a thread one row, warps 0..3 the first K step of a group, 4..7 the second ----------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    const int quad = warp & 3, step = (warp - 4) >> 2, row = quad * 32 + lane;
    const uint32_t lanes = tmem_w + ((uint32_t)(quad * 32) << 16);
    constexpr uint32_t Y64 = 0x64646464u, K1024 = 0x64006400u, KM1024 = 0xE400E400u;
    uint32_t g = 0;
    QiRing rw, rp;
    bool ok = true;
    auto stage_free = [&](uint32_t gg) {
      bool fr = true;
      if (gg >= (uint32_t)p.sb) fr = mbar_wait_bounded(done(gg - (uint32_t)p.sb), parity(gg - (uint32_t)p.sb), abort_flag);
      return __all_sync(0xffffffffu, fr) != 0;
    };
    // the stores of this warp are in tensor memory: tell the MMA warps
    auto written = [&]() {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
    };
    for (int item = cluster; item < p.items && ok; item += clusters) {
      // ---- sum units: warps 0..3 the even super-blocks, 4..7 the odd ones ----
      for (int u = 0; u < p.npu; u++) {
        const int b0 = qi_sum_begin(p, u), nsb = qi_sum_begin(p, u + 1) - b0;
        const int n = min(tile_n_of(item) * 256 + (int)rank * QI_ROWS + row, N - 1);  // rows beyond N are not stored
        const uint32_t *src = reinterpret_cast<const uint32_t *>(W) + ((size_t)n * p.bpr + part_of(item) * p.pb + b0) * Q4K_BLOCK_WORDS;
        uint4 hd[QI_SUMS / 2];
        float most = 0.0f;
#pragma unroll
        for (int i = 0; i < QI_SUMS / 2; i++) {
          const int k = 2 * i + step, other = 2 * i + 1 - step;
          hd[i] = make_uint4(0u, 0u, 0u, 0u);
          if (k < nsb) hd[i] = __ldg(reinterpret_cast<const uint4 *>(src + k * Q4K_BLOCK_WORDS));
          if (other < nsb) most = fmaxf(most, fabsf(q4k_d_dmin(__ldg(src + other * Q4K_BLOCK_WORDS)).y));
        }
#pragma unroll
        for (int i = 0; i < QI_SUMS / 2; i++) most = fmaxf(most, fabsf(q4k_d_dmin(hd[i].x).y));
        const float scale = qi_pow2(8 - qi_exponent(most));
        if (!stage_free(g) || !stage_free(g + 1)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t s0 = rw.i;
        rw.next(p.sb);
        const uint32_t s1 = rw.i;
        rw.next(p.sb);
        if (step == 0) row_scales[(g >> 1) % QI_SCALES][row] = -64.0f * qi_pow2(qi_exponent(most) - 8);  // (the sums are stored divided by 64)
        const QiSumOrder at = F32 == 2 ? qi_sums_lo_first(nsb) : qi_sums_in_turn(nsb);
        // eight values of a super-block, four columns: place c of the unit's 32
        auto put = [&](int c, const uint32_t (&v)[4]) { qi_tmem_st4(lanes + (c < 16 ? s0 : s1) * QI_W_COLS + (uint32_t)(c & 15) * 4u, v); };
#pragma unroll
        for (int i = 0; i < QI_SUMS / 2; i++) {
          const int k = 2 * i + step;
          if (k < nsb) {  // (uniform)
            const Q4KScales sc = q4k_unpack_scales(hd[i].y, hd[i].z, hd[i].w);
            const __half2 dm2 = __float2half2_rn(q4k_d_dmin(hd[i].x).y * scale);
            const uint32_t dm = *reinterpret_cast<const uint32_t *>(&dm2);
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const uint32_t m = qi_hsub2(__byte_perm(j < 2 ? sc.mn03 : sc.mn47, Y64, (j & 1) ? 0x4342u : 0x4140u), K1024);
              hi[j] = qi_hmul2(dm, m);
              lo[j] = qi_hfma2(dm, m, hi[j] ^ 0x80008000u);  // exactly what the rounding dropped
            }
            put(at.hh + k, hi);
            put(at.lh + k, lo);
            put(at.hl + k, hi);
          }
        }
        if ((nsb & 1) && step == 0) {  // the other half of the last K slice
          const uint32_t zero[4] = {0u, 0u, 0u, 0u};
          put(3 * nsb, zero);
        }
        written();
        if (lane == 0) {
          if (step == 0) mbar_arrive(scaled(g >> 1));
          mbar_arrive(full(g));
          mbar_arrive(full(g + 1));
        }
        g += 2;
      }
      // ---- super-blocks ----
      for (int u = 0; u < p.pb && ok; u++, rp.next(p.sp)) {
        const bool here = mbar_wait_bounded(full_p(rp.i), rp.uses & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, here)) { ok = false; break; }
        const uint8_t *blk = ring_p + rp.i * QI_P_STAGE + (uint32_t)row * Q4K_BLOCK_BYTES;
        const uint4 hd = *reinterpret_cast<const uint4 *>(blk);
        if (step == 0) row_scales[(g >> 1) % QI_SCALES][row] = q4k_d_dmin(hd.x).x;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint4 qa = *reinterpret_cast<const uint4 *>(blk + 16 + 32 * (2 * h + step)), qb = *reinterpret_cast<const uint4 *>(blk + 32 + 32 * (2 * h + step));
          // the four scale codes of this half of the super-block; this K step's two as f16 pairs, and -1024 * code
          const uint32_t cw = (h == 0 ? hd.y & 0x3f3f3f3fu : (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u)) >> (16 * step);
          const uint32_t sca = qi_hsub2(__byte_perm(cw, Y64, 0x4040u), K1024), scb = qi_hsub2(__byte_perm(cw, Y64, 0x4141u), K1024);
          const uint32_t nega = qi_hmul2(sca, KM1024), negb = qi_hmul2(scb, KM1024);
          if (!stage_free(g)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t at = lanes + rw.i * QI_W_COLS + (uint32_t)step * 32u;
          const uint32_t q[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
          uint32_t v[16];
#pragma unroll
          for (int i = 0; i < 8; i++) {  // byte -> f16 1024 + q with one permute; (1024 + q) * sc - 1024 * sc = sc * q exactly
            const uint32_t t = q[i] & 0x0f0f0f0fu;
            v[2 * i] = qi_hfma2(__byte_perm(t, Y64, 0x4140u), sca, nega);
            v[2 * i + 1] = qi_hfma2(__byte_perm(t, Y64, 0x4342u), sca, nega);
          }
          qi_tmem_st16(at, v);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const uint32_t t = (q[i] >> 4) & 0x0f0f0f0fu;
            v[2 * i] = qi_hfma2(__byte_perm(t, Y64, 0x4140u), scb, negb);
            v[2 * i + 1] = qi_hfma2(__byte_perm(t, Y64, 0x4342u), scb, negb);
          }
          qi_tmem_st16(at + 16u, v);
          written();
          if (lane == 0) {
            if (h == 0 && step == 0) mbar_arrive(scaled(g >> 1));
            mbar_arrive(full(g));
            if (h == 1) mbar_arrive(free_p(rp.i));
          }
          rw.next(p.sb);
          g++;
        }
      }
    }
  } else {
    // ---------------- tensor memory -> d * P (and the sum units) -> f32 sums -> C ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    const int quad = warp & 3, half = (warp - 4 - QI_BUILDERS) >> 2, cw = p.bn / 2;  // this warp's columns: half * cw ..
    const uint32_t empty0 = mapa_shared(empty(0), 0u);
    uint32_t n = 0;
    bool ok = true;
    for (int item = cluster; item < p.items && ok; item += clusters) {
      const int f = tile_n_of(item) * 256 + (int)rank * QI_ROWS + quad * 32 + lane, m0 = tile_m_of(item) * p.bn + half * cw;
      float acc[QI_BN / 2];
#pragma unroll
      for (int i = 0; i < QI_BN / 2; i++) acc[i] = 0.0f;
      for (int u = 0; u < units; u++, n++) {
        const uint32_t g = 2u * n + 1u, b = n & 1u;
        const bool ready = mbar_wait_bounded(scaled(n), parity(n), abort_flag) && mbar_wait_bounded(done(g), parity(g), abort_flag);
        if (!__all_sync(0xffffffffu, ready)) { ok = false; break; }  // tcgen05.ld is warp-wide: together or not at all
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float scale = row_scales[n % QI_SCALES][quad * 32 + lane];
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + b * (uint32_t)p.bn + (uint32_t)(half * cw);
#pragma unroll
        for (int c = 0; c < QI_BN / 64; c++) {
          if (c * 32 < cw) {  // (uniform; where cw is an odd number of sixteens the last sixteen columns are read and not stored)
            uint32_t r[32];
            tmem_ld32(taddr + (uint32_t)(c * 32), r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 32; i++) acc[c * 32 + i] = fmaf(scale, __uint_as_float(r[i]), acc[c * 32 + i]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) qi_arrive_remote(empty0 + 8u * b);
        if (o.sum_scale && u == p.npu - 1) {
#pragma unroll
          for (int c = 0; c < QI_BN / 64; c++) {
            const int m = m0 + 32 * c + lane;
            const float mine = m < M && 32 * c < cw ? __ldg(o.sum_scale + m) : 0.0f;
#pragma unroll
            for (int i = 0; i < 32; i++) acc[32 * c + i] *= __shfl_sync(0xffffffffu, mine, i);
          }
        }
      }
      if (!ok) break;
      // A warp stores 32 consecutive features of an activation row at a time.  The code of eight rows is run over and over
      // while the sums move down eight registers: unrolled over all columns it was run once per tile straight out of
      // instruction cache misses (33 thousand cycles per tile).
      OutT *dst = C + (p.parts > 1 ? (size_t)part_of(item) * (size_t)M * (size_t)N : (size_t)0);
      const bool is_up = lane & 8;
      auto scale_at = [&](int c) {  // lane i: the scale of row c + i
        const int m = m0 + c + (lane & 7);
        return o.row_scale ? (m < M ? o.alpha * __ldg(o.row_scale + m) : 0.0f) : o.alpha;
      };
      float mine = scale_at(0);
#pragma unroll 1
      for (int c = 0; c < cw && m0 + c < M; c += 8) {
        const float next = scale_at(c + 8);
        if constexpr (sizeof(OutT) == 4) {
          if (o.silu) {
            // a gate row and its up row are eight lanes apart: the gate's lane takes the even activation rows, the other the odd
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
              const float v0 = acc[i] * __shfl_sync(0xffffffffu, mine, i), v1 = acc[i + 1] * __shfl_sync(0xffffffffu, mine, i + 1);
              const float got = __shfl_xor_sync(0xffffffffu, is_up ? v0 : v1, 8);
              const float gv = is_up ? got : v0, uv = is_up ? v1 : got;
              const int m = m0 + c + i + (is_up ? 1 : 0);
              const float cl = fminf(fmaxf(gv, -15.0f), 15.0f);  // silu.wgsl:30-37,98-104
              if (f < N && m < M) dst[(size_t)m * (size_t)(N / 2) + (size_t)((f >> 4) * 8 + (f & 7))] = (gv * (1.0f / (1.0f + expf(-cl)))) * uv;
            }
          } else {
            float res[8];
#pragma unroll
            for (int i = 0; i < 8; i++) res[i] = o.residual && f < N && m0 + c + i < M ? o.residual[(size_t)(m0 + c + i) * N + f] : 0.0f;
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const float v = acc[i] * __shfl_sync(0xffffffffu, mine, i) + res[i];
              if (f < N && m0 + c + i < M) dst[(size_t)(m0 + c + i) * N + f] = v;
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const float v = acc[i] * __shfl_sync(0xffffffffu, mine, i);
            if (f < N && m0 + c + i < M) dst[(size_t)(m0 + c + i) * N + f] = __float2half_rn(v);
          }
        }
#pragma unroll
        for (int i = 0; i + 8 < QI_BN / 2; i++) acc[i] = acc[i + 8];
        mine = next;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();  // neither CTA frees tensor memory or leaves while the peer still uses the pair's resources
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  if (*abort_flag && tid == 0) atomicExch(err, 2);
}

// ---- activation rows: f16 halves, scales and sub-block sums ----
// Where a sub-block's sum goes: its unit's three places, eight columns per super-block
template <bool LO_FIRST>
__device__ __forceinline__ void qi_put_sum(__half *sums_row, const IntPlan &p, int s, float v) {
  const int sb = s >> 3, part = sb / p.pb, k = sb - part * p.pb;
  const int u = ((k + 1) * p.npu - 1) / p.pb, b0 = qi_sum_begin(p, u), nsb = qi_sum_begin(p, u + 1) - b0;
  const QiSumOrder to = LO_FIRST ? qi_sums_lo_first(nsb) : qi_sums_in_turn(nsb);
  __half *at = sums_row + (size_t)(part * p.npu + u) * 256 + (s & 7);
  const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi));
  at[(to.hh + k - b0) * 8] = hi;
  at[(to.lh + k - b0) * 8] = hi;
  at[(to.hl + k - b0) * 8] = lo;
  if ((nsb & 1) && k == b0) at[3 * nsb * 8] = __float2half_rn(0.0f);  // pairs with the weights' zero place
}

__device__ __forceinline__ int qi_row_exponent(float mx) {  // exponent that brings the row's maximum into [2^13, 2^14)
  int e = 0;                                                // (0 for an all-zero or non-finite row)
  if (mx > 0.0f && mx < __int_as_float(0x7f800000)) e = (int)((__float_as_uint(mx) >> 23) & 0xffu) - 127 - 13;
  return max(-100, min(100, e));
}

// A row that f16 halves do not hold: an infinity in it (infinity minus infinity would be its residue), or a largest value that
// the exponent brings near the ends of f32's range, where the scale or its product with alpha would lose bits.  Where `guard`
// is set (shapes that f32 FMAs multiplied before) such a row's scale is NaN, and dpk_gemm_q4k_simt computes the row afterwards.
constexpr int QI_EXP_MOST = 60;
__device__ __forceinline__ float qi_row_scale(float mx, int e, int guard) {
  const bool special = mx == __int_as_float(0x7f800000) || e > QI_EXP_MOST || e < -QI_EXP_MOST;
  return guard && special ? __int_as_float(0x7fc00000) : qi_pow2(e);
}

__device__ __forceinline__ float qi_block_max(float v, float *sh) {  // eight warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = sh[0];
#pragma unroll
  for (int w = 1; w < 8; w++) t = fmaxf(t, sh[w]);
  return t;
}

// One block per row, any K and alignment.  f32 rows: scaled by a power of two and split, x * 2^-e = hi + lo (rows of kp
// halves, zeros beyond K), row_scale = 2^e.  f16 rows: left as they are (copied to hi where hi is given), the sums alone
// are scaled, sum_scale = 2^e.  The sums are divided by 64 on top.
template <typename AT, bool LO_FIRST>
__global__ void __launch_bounds__(256) int_rows_kernel(const AT *__restrict__ in, __half *__restrict__ hi, __half *__restrict__ lo, float *__restrict__ scale,
                                                       __half *__restrict__ sums, int K, int kp, const IntPlan p, int guard) {
  pdl_launch();
  pdl_wait();
  __shared__ float sh[8];
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const AT *x = in + (size_t)row * K;
  float mx = 0.0f;
  for (int i = threadIdx.x; i < K; i += 256) mx = fmaxf(mx, fabsf((float)x[i]));
  mx = qi_block_max(mx, sh);
  const int e = qi_row_exponent(mx);
  const float down = qi_pow2(-e);
  if (threadIdx.x == 0) scale[row] = qi_row_scale(mx, e, guard);
  for (int s = warp; s < p.bpr * 8; s += 8) {
    const int i = s * 32 + lane;
    const float v = i < K ? (float)x[i] : 0.0f;
    float t = v * down;
    if (i < kp) {
      if constexpr (sizeof(AT) == 4) {
        const __half h = __float2half_rn(t);
        hi[(size_t)row * kp + i] = h;
        lo[(size_t)row * kp + i] = __float2half_rn(t - __half2float(h));
      } else if (hi) {
        hi[(size_t)row * kp + i] = __float2half_rn(v);
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
    if (lane == 0) qi_put_sum<LO_FIRST>(sums + (size_t)row * ((size_t)p.parts * p.npu * 256), p, s, t * 0.015625f);
  }
}

// The same for f32 rows with the row in registers (K % 32 == 0, K <= 1024 * NV, 16-byte aligned): one pass, 16-byte loads.
// With norm_w the row is RMS-normalised first (rmsnorm.wgsl:119-187), element for element and reduction step for
// reduction step as rmsnorm_vec_kernel (small_ops.cu) does it for rows of 1024..4096 values.
template <int NV, bool LO_FIRST>
__global__ void __launch_bounds__(256) int_rows_vec_kernel(const float *__restrict__ in, __half *__restrict__ hi, __half *__restrict__ lo, float *__restrict__ scale,
                                                           __half *__restrict__ sums, int K, const IntPlan p, const float *__restrict__ norm_w, float eps, int guard) {
  pdl_launch();
  pdl_wait();
  __shared__ float sh[8], shn[8];
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n4 = K >> 2;
  const size_t base = (size_t)row * K;
  float4 v[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int idx = threadIdx.x + i * 256;
    v[i] = idx < n4 ? *reinterpret_cast<const float4 *>(in + base + 4 * idx) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  if (norm_w) {
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; i++) ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    if (lane == 0) shn[warp] = ss;
    __syncthreads();
    float total = lane < 8 ? shn[lane] : 0.0f;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
    const float inv_rms = 1.0f / sqrtf(total / (float)K + eps);
#pragma unroll
    for (int i = 0; i < NV; i++) {
      const int idx = threadIdx.x + i * 256;
      if (idx < n4) {
        const float4 w = *reinterpret_cast<const float4 *>(norm_w + 4 * idx);
        v[i].x = v[i].x * inv_rms * w.x; v[i].y = v[i].y * inv_rms * w.y; v[i].z = v[i].z * inv_rms * w.z; v[i].w = v[i].w * inv_rms * w.w;
      }
    }
  }
  float mx = 0.0f;
#pragma unroll
  for (int i = 0; i < NV; i++) mx = fmaxf(fmaxf(mx, fmaxf(fabsf(v[i].x), fabsf(v[i].y))), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
  mx = qi_block_max(mx, sh);
  const int e = qi_row_exponent(mx);
  const float down = qi_pow2(-e);
  if (threadIdx.x == 0) scale[row] = qi_row_scale(mx, e, guard);
  __half *sums_row = sums + (size_t)row * ((size_t)p.parts * p.npu * 256);
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int idx = threadIdx.x + i * 256;
    const float s0 = v[i].x * down, s1 = v[i].y * down, s2 = v[i].z * down, s3 = v[i].w * down;
    float t = (s0 + s1) + (s2 + s3);  // eight consecutive threads hold a sub-block
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    if (idx >= n4) continue;
    const __half2 h01 = __floats2half2_rn(s0, s1), h23 = __floats2half2_rn(s2, s3);
    const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
    const __half2 l01 = __floats2half2_rn(s0 - f01.x, s1 - f01.y), l23 = __floats2half2_rn(s2 - f23.x, s3 - f23.y);
    *reinterpret_cast<uint2 *>(hi + base + 4 * idx) = make_uint2(*reinterpret_cast<const uint32_t *>(&h01), *reinterpret_cast<const uint32_t *>(&h23));
    *reinterpret_cast<uint2 *>(lo + base + 4 * idx) = make_uint2(*reinterpret_cast<const uint32_t *>(&l01), *reinterpret_cast<const uint32_t *>(&l23));
    if ((threadIdx.x & 7) == 0) qi_put_sum<LO_FIRST>(sums_row, p, idx >> 3, t * 0.015625f);
  }
  // (sub-blocks beyond a K that is no multiple of 256)
  for (int s = (K >> 5) + (int)threadIdx.x; s < p.bpr * 8; s += 256) qi_put_sum<LO_FIRST>(sums_row, p, s, 0.0f);
}

// C = sum of the parts of a K-split launch, in a fixed order (+ residual, which may be C itself)
template <typename OutT>
__global__ void __launch_bounds__(256) int_reduce_kernel(const float *__restrict__ parts, OutT *C, size_t n, int splits, const float *residual) {
  pdl_launch();
  pdl_wait();
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
    float acc = parts[i];
    for (int z = 1; z < splits; z++) acc += parts[(size_t)z * n + i];
    if (residual) acc += residual[i];
    if constexpr (sizeof(OutT) == 4) C[i] = acc;
    else C[i] = __float2half_rn(acc);
  }
}

// shared memory a plan's rings may take: what a launch may ask for, less alignment, barriers and row scales
size_t qi_ring_budget(const dp_ctx *ctx) { return ctx->smem_optin - 1024 - 8192; }

// Tile width and parts of K with the least estimated time, in cycles: an MMA of sixteen K takes half a cycle per activation
// row, a super-block no less than what builders and drains need; an item has a fixed cost (fill, store); a K split is paid
// for with the traffic of its parts.
IntPlan qi_plan(dp_ctx *ctx, int M, int N, int K, bool lo, bool lo_first, bool may_split) {
  IntPlan best = {};
  double best_cost = -1.0;
  const int clusters = ctx->sm_count / 2, bpr = (K + QK_K - 1) / QK_K, tiles_n = (N + 255) / 256;
  const size_t budget = qi_ring_budget(ctx);
  for (int parts = 1; parts <= (may_split ? 8 : 1); parts++) {
    if (bpr % parts || (parts > 1 && bpr / parts < 2)) continue;
    for (int bn = 32; bn <= QI_BN; bn += 32) {
      IntPlan p;
      p.bpr = bpr; p.parts = parts; p.pb = bpr / parts;       const int most = !lo_first ? QI_SUMS : p.pb > 24 ? QI_SUMS_LONG : QI_SUMS_LO_FIRST;
      p.npu = (p.pb + most - 1) / most;
      p.bn = bn; p.tiles_n = tiles_n; p.tiles_m = (M + bn - 1) / bn;
      p.items = p.tiles_n * p.tiles_m * parts;
      // tensor memory beside the accumulators; shared memory: activation groups first, then packed blocks
      p.sb = (512 - 2 * bn) / (int)QI_W_COLS;
      if (p.sb > QI_RING) p.sb = QI_RING;
      p.sa = 2; p.sp = 2;
      if (qi_rings(p, lo) > budget) continue;
      for (int *stages : {&p.sa, &p.sp})
        while (*stages < QI_RING) {
          ++*stages;
          if (qi_rings(p, lo) > budget) { --*stages; break; }
        }
      const double mma = 16.0 * (bn < 96 ? 56.0 : 0.5 * bn + 8.0), unit = lo ? 2.0 * mma : mma;
      const double item = p.pb * (unit < 1600.0 ? 1600.0 : unit) + p.npu * (mma < 2500.0 ? 2500.0 : mma) + 3000.0 + 10.0 * bn;
      const double waves = (double)((p.items + clusters - 1) / clusters);
      const double cost = waves * item + (parts > 1 ? 4000.0 + 4.0 * (double)M * N * (2 * parts + 1) / 3000.0 : 0.0);
      if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = p; }
    }
  }
  return best;
}

template <int F32, typename OutT>
dp_status launch_int(dp_ctx *ctx, const CUtensorMap *tm, const uint8_t *W, OutT *C, int M, int N, const IntPlan &p, const IntOut &o) {
  const size_t smem = qi_rings(p, F32 > 0) + 1024;
  auto kernel = gemm_q4k_int_kernel<F32, OutT>;
  // once, to the most any plan takes: set to each launch's own size, a small one lowered it under a large one that another
  // thread was about to launch
  static dp_per_device_once limit;
  if (limit.pending(ctx->device)) {
    DP_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(qi_ring_budget(ctx) + 1024)));
    limit.done(ctx->device);
  }
  const int clusters = ctx->sm_count / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (unsigned)(p.items < clusters ? p.items : clusters));
  cfg.blockDim = dim3(QI_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tm[0], tm[1], tm[2], tm[3], W, C, M, N, p, o, ctx->dev_status);
  ctx->launches++;
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return dp_fail(ctx, DP_ERR_CUDA, "launch of gemm_q4k_int_kernel failed: %s", cudaGetErrorString(e));
  return DP_OK;
}

}  // namespace

// A: f32 (multiplied in as two f16 halves) or f16 activations, the weights exact; C f32 or f16 (f16: from f16 activations only).
// Any N and K.  fuse (optional, f32): see dpk_tc_fuse; norm_w only for the rows int_rows_vec_kernel takes.
dp_status dpk_gemm_q4k_int(dp_ctx *ctx, const uint8_t *W, const void *A, dp_dtype a_dtype, void *C, dp_dtype c_dtype, int M, int N, int K, float alpha, bool *handled,
                           dpk_tc_fuse *fuse) {
  *handled = false;
  const bool f32a = a_dtype == DP_F32;
  if (M < 1 || !ctx->dev_status || ctx->sm_count < 2 || (!f32a && a_dtype != DP_F16) || (c_dtype != DP_F32 && (c_dtype != DP_F16 || f32a))) return DP_OK;
  EncodeTiledFn encode = get_encode();
  if (!encode) return DP_OK;
  const float *norm_w = fuse ? fuse->norm_w : nullptr;
  const bool vec = f32a && K % 32 == 0 && K <= 16384 && ((uintptr_t)A & 15) == 0;
  // (rows that are computed apart need the rows themselves, and no output that holds something else already)
  const int guard = K % QK_K != 0 || N % 128 != 0;
  if (norm_w && (guard || !(vec && K >= 1024 && K <= 4096 && ((uintptr_t)norm_w & 15) == 0))) return DP_OK;
  const bool silu = !guard && fuse && fuse->silu_dst && c_dtype == DP_F32 && N % 16 == 0;
  const bool lo_first = f32a && (guard || (fuse && fuse->exact_weights));
  const IntPlan p = qi_plan(ctx, M, N, K, f32a, lo_first, !silu);

  const int kp = (K + 7) / 8 * 8;
  const bool copy = f32a || K % 8 || ((uintptr_t)A & 15);  // f16 rows that TMA can read stay where they are
  const size_t a_bytes = copy ? ((size_t)M * kp * 2 + 255) / 256 * 256 : 0;
  const size_t sum_cols = (size_t)p.parts * p.npu * 256, s_bytes = ((size_t)M * sum_cols * 2 + 255) / 256 * 256;
  dp_status st = dp_scratch(ctx, &ctx->gemm_scratch, a_bytes * (f32a ? 2 : 1) + s_bytes + (size_t)M * 4, "matmul_a_f16");
  if (st == DP_OK && p.parts > 1) st = dp_scratch(ctx, &ctx->gemm_split_scratch, (size_t)p.parts * M * N * 4, "matmul_k_split_parts");
  if (st == DP_ERR_OOM && guard) return DP_OK;  // no memory for the pass over the rows: the CUDA cores need none
  DP_TRY(st);
  char *base = (char *)ctx->gemm_scratch->dptr;
  __half *hi = (__half *)base, *lo = (__half *)(base + a_bytes), *sums = (__half *)(base + a_bytes * (f32a ? 2 : 1));
  float *scale = (float *)((char *)sums + s_bytes);
  const float eps = fuse ? fuse->eps : 0.0f;
  if (vec) {
    const float *a = (const float *)A;
    auto rows = K <= 1024    ? (lo_first ? int_rows_vec_kernel<1, true> : int_rows_vec_kernel<1, false>)
                : K <= 4096  ? (lo_first ? int_rows_vec_kernel<4, true> : int_rows_vec_kernel<4, false>)
                : K <= 12288 ? (lo_first ? int_rows_vec_kernel<12, true> : int_rows_vec_kernel<12, false>)
                             : (lo_first ? int_rows_vec_kernel<16, true> : int_rows_vec_kernel<16, false>);
    DP_LAUNCH(ctx, rows, (unsigned)M, 256, 0, a, hi, lo, scale, sums, K, p, norm_w, eps, guard);
  } else if (f32a) {
    auto rows = lo_first ? int_rows_kernel<float, true> : int_rows_kernel<float, false>;
    DP_LAUNCH(ctx, rows, (unsigned)M, 256, 0, (const float *)A, hi, lo, scale, sums, K, kp, p, guard);
  } else {
    DP_LAUNCH(ctx, (int_rows_kernel<__half, false>), (unsigned)M, 256, 0, (const __half *)A, copy ? hi : (__half *)nullptr, (__half *)nullptr, scale, sums, K, kp, p, guard);
    if (!copy) hi = (__half *)A;
  }

  CUtensorMap tm[4];
  const cuuint32_t box[2] = {BK, (cuuint32_t)(p.bn / 2)}, estr[2] = {1, 1};
  for (int i = 0; i < 3; i++) {
    const cuuint64_t dims[2] = {i == 2 ? (cuuint64_t)sum_cols : (cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {i == 2 ? (cuuint64_t)sum_cols * 2 : (cuuint64_t)kp * 2};
    void *ptr = i == 0 ? (void *)hi : i == 1 ? (void *)(f32a ? lo : hi) : (void *)sums;
    const CUresult r = encode(&tm[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return dp_fail(ctx, DP_ERR_CUDA, "matmul: cuTensorMapEncodeTiled failed (%d) for A[%d,%d]", (int)r, M, K);
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)p.bpr * Q4K_BLOCK_BYTES, (cuuint64_t)N}, strides[1] = {(cuuint64_t)p.bpr * Q4K_BLOCK_BYTES};
    const cuuint32_t wbox[2] = {Q4K_BLOCK_BYTES, QI_ROWS};
    const CUresult r = encode(&tm[3], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)W, dims, strides, wbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return dp_fail(ctx, DP_ERR_CUDA, "matmul: cuTensorMapEncodeTiled failed (%d) for W[%d,%d]", (int)r, N, K);
  }

  IntOut o = {alpha, f32a ? scale : nullptr, f32a ? nullptr : scale, nullptr, silu ? 1 : 0};
  void *dst = silu ? (void *)fuse->silu_dst : C, *final_dst = C;
  const float *residual = nullptr;
  if (!guard && fuse && fuse->residual && fuse->residual_out && c_dtype == DP_F32 && !silu) {
    residual = fuse->residual;
    final_dst = dst = fuse->residual_out;
    fuse->residual_done = true;
  }
  if (silu) fuse->silu_done = true;
  if (p.parts > 1) {
    dst = ctx->gemm_split_scratch->dptr;
  } else {
    o.residual = residual;
  }
  if (f32a && lo_first) st = launch_int<2, float>(ctx, tm, W, (float *)dst, M, N, p, o);
  else if (f32a) st = launch_int<1, float>(ctx, tm, W, (float *)dst, M, N, p, o);
  else if (c_dtype == DP_F32 || p.parts > 1) st = launch_int<0, float>(ctx, tm, W, (float *)dst, M, N, p, o);
  else st = launch_int<0, __half>(ctx, tm, W, (__half *)dst, M, N, p, o);
  DP_TRY(st);
  if (p.parts > 1) {
    const size_t n = (size_t)M * N;
    size_t grid = (n + 255) / 256;
    if (grid > (size_t)ctx->sm_count * 8) grid = (size_t)ctx->sm_count * 8;
    const float *parts = (const float *)dst;
    if (c_dtype == DP_F32) DP_LAUNCH(ctx, int_reduce_kernel<float>, (unsigned)grid, 256, 0, parts, (float *)final_dst, n, p.parts, residual);
    else DP_LAUNCH(ctx, int_reduce_kernel<__half>, (unsigned)grid, 256, 0, parts, (__half *)final_dst, n, p.parts, residual);
  }
  if (guard) {  // its launch prepared while the kernel before it runs: it has nothing to do as a rule
    const bool pdl = ctx->pdl;
    ctx->pdl = true;
    st = dpk_gemm_q4k_simt(ctx, W, A, a_dtype, C, c_dtype, M, N, K, alpha, scale);
    ctx->pdl = pdl;
    DP_TRY(st);
  }
  *handled = true;
  return DP_OK;
}
