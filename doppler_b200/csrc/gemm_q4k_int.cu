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
// of K: at the start of a tile up to eight super-blocks at a time share one 256-wide "sum unit" of three products, [hi hi],
// [lo hi] and [hi lo] parts of dmin * m and of the sub-block sums (f16 pairs; dmin scaled by a power of two per weight row, the
// sums by one per activation row, both undone on read-back).  hi + lo holds all 17 bits of dmin * m; 22 bits of the sums.
//
// The tensor core cuts off what falls below its accumulator's last bit, so that products added while the accumulator is
// small cost no accuracy.  f32 rows have two orders of their products: lo and hi in turn for every K slice, or (lo_first) the lo
// products of the whole super-block before its hi products, which waits for all of its groups first.  Error against 64 bits,
// random normal rows, K 1024 to 12288: 9.3e-7 in turn, 4.6e-7 to 5.1e-7 lo first (f32 FMAs: 5.7e-7 at K = 1024, 1.9e-6 at
// 11111; tiles of dequantised weights: 3.7e-6 to 2.2e-5).  Lo first where calls would otherwise lose accuracy against the kernels
// that ran them before: shapes no tile divides, which f32 FMAs multiplied, up to 64 rows, and rows of several prompts, which
// have it one by one.  The small products of a sum unit come first from seven super-blocks on (K = 12288: 6.3e-7 -> 5.3e-7); up to
// six, what is cut off there and in the super-blocks cancels in part (four: 4.6e-7, with the small ones first 5.1e-7), and so it
// does at any number where lo and hi take turns (9.2e-7, 1.08e-6).
//
// A cluster of two CTAs owns 256 weight rows x bn activation rows (cta_group::2, M = 256: CTA r holds 128 weight rows and
// their 128 lanes of the result, and half of the activation tile).  Sharing the activation tile halves its L2 and
// shared-memory traffic.  The weight tiles are the A operand in TENSOR MEMORY: out of shared memory every MMA would read
// its 4 KB slice once more, beside the activations' copies.  Two to four accumulators, and in what tensor memory they leave four
// to eight groups of weights, a 64-wide K step each (four groups of 64 instead of two of 128 beside two accumulators of 192 columns:
// 92 -> 87 us for 512 f16 rows x [12288, 4096]; with two, a group's builders had one group's MMAs to hide behind).  Clusters walk
// the (tile, part of K) items persistently; bn is chosen so that the items fill whole waves of clusters.
//
// Roles per CTA (registers are moved to the draining warps with setmaxnreg): warp 0 TMA of activations, two K steps a copy;
// warps 1 and 2 MMA issue (CTA 0), a unit (super-block) each in turn; warp 3 TMA of packed super-blocks; sixteen warps build
// weight tiles out of them, eight drain (a lane quarter and half of the columns per warp, up to 96 sums per thread).  The SM's
// four schedulers are what is short: with 28 warps an instruction of a warp that waits for its own results takes some ten
// cycles, so every role's serial chain was cut until none of them paced the MMAs.  512 f16 rows x [12288, 4096], us: 86 with eight
// building warps and MMAs out of a branch of one lane; issued by a converged warp (umma.cuh), activations by one copy per
// two K steps instead of four 70; two K steps of every other unit per building warp, f32x2 sums, no spilled sums 63; headers of
// sum units by cp.async instead of TMA boxes of sixteen bytes, pointers instead of products in the store code 61.  64 f32 rows
// x [24576, 4096] 78 -> 52, 2048 f32 rows 738 -> 582 (0.71 of the measured burst executed in two products; the power limit holds the
// clock at 1.5 GHz there).  What bounds it now: few rows, the builders (a super-block takes them 0.9 us); many, the MMAs and
// the power limit.  Every wait is bounded; on give-up the CTA raises the status word and still frees its tensor memory.
#include "common.h"
#include "mbar.cuh"
#include "pdl.cuh"
#include "q4k.cuh"
#include "umma.cuh"

namespace {

using namespace umma;

constexpr int QI_ROWS = 128;       // weight rows per CTA
constexpr int QI_BN = 192;         // most activation rows of a tile
constexpr int QI_SUMS = 8, QI_SUMS_LONG = 6;  // most super-blocks of a sum unit; ... lo first, where a part is longer than 24 (more f32 additions)
constexpr int QI_BUILDERS = 16, QI_DRAINERS = 8;
constexpr int QI_THREADS = (4 + QI_BUILDERS + QI_DRAINERS) * 32;
constexpr int QI_RING = 8;         // most stages of the ring of weight groups
constexpr int QI_PAIRS = 8;        // ... of pairs of K steps of activations
constexpr int QI_PACKED = 4;       // ... of packed super-blocks
constexpr int QI_ACCS = 4;         // most accumulators
constexpr int QI_BARS = 16;        // the rings of barriers that go by group, see `full`
constexpr int QI_STORE = 32;       // rows that are stored by one run of the store code
constexpr int QI_SCALES = 8;       // units whose row scales are kept (a drain is at most two units behind the builders' ring)

struct IntPlan {
  int bpr, parts, pb, npu;         // super-blocks of a row; parts of K; super-blocks and sum units of a part
  int bn, tiles_n, tiles_m, items;
  int na;                          // accumulators
  int sa, sb, sp;                  // stages: pairs of K steps of activations, groups of weight tiles (tensor memory), packed super-blocks
};

__host__ __device__ __forceinline__ int qi_sum_begin(const IntPlan &p, int u) { return u * p.pb / p.npu; }
// Columns of a sum unit: each half of the 256 holds the three products of about half of the unit's super-blocks, so that a
// building warp computes both parts of a minimum once: eight columns a super-block, a product's padded with zeros to whole K
// slices.  The first half takes an even number of super-blocks: every slice is one more addition that the tensor core truncates.
__host__ __device__ __forceinline__ int qi_sum_first(int nsb) { return nsb < 2 ? nsb : (nsb + 3) / 4 * 2; }  // super-blocks of the first half
__host__ __device__ __forceinline__ int qi_sum_slices(int count) { return (count + 1) >> 1; }  // K slices of a product of a half
// products: [hi hi], [lo hi], [hi lo] of weights and sums
constexpr int QI_HH = 0, QI_LH = 1, QI_HL = 2;

constexpr uint32_t QI_P_STAGE = QI_ROWS * Q4K_BLOCK_BYTES;  // packed super-blocks of the CTA's weight rows, or the headers of a sum unit
static_assert(QI_SUMS * 16 <= Q4K_BLOCK_BYTES, "the headers of a sum unit take the place of one super-block a row");
constexpr uint32_t QI_W_COLS = 32;                          // tensor-memory columns of a weight group: a K step of 64, two f16 each
__host__ __device__ __forceinline__ uint32_t qi_x_tile(const IntPlan &p) { return (uint32_t)(p.bn / 2) * 128u; }
__host__ __device__ __forceinline__ uint32_t qi_x_stage(const IntPlan &p, bool lo) { return qi_x_tile(p) * (lo ? 4u : 2u); }
__host__ __device__ __forceinline__ uint32_t qi_rings(const IntPlan &p, bool lo) { return (uint32_t)p.sa * qi_x_stage(p, lo) + (uint32_t)p.sp * QI_P_STAGE; }

typedef unsigned long long qi_f2;  // two f32
__device__ __forceinline__ qi_f2 qi_pack(float a, float b) {
  qi_f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float qi_low(qi_f2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float qi_high(qi_f2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ qi_f2 qi_fma(qi_f2 a, qi_f2 b, qi_f2 c) {
  qi_f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ qi_f2 qi_mul(qi_f2 a, qi_f2 b) {
  qi_f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ void qi_store(float *p, float v) { *p = v; }
__device__ __forceinline__ void qi_store(__half *p, float v) { *p = __float2half_rn(v); }

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

// Four MMAs of the pair, a K step of 64, with the A operand in tensor memory, issued by a converged warp (umma.cuh)
__device__ __forceinline__ void qi_umma4(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q, t;\n .reg .b32 a1, a2, a3;\n .reg .b64 b1, b2, b3;\n setp.ne.b32 p, %4, 0;\n setp.eq.u32 t, 0, 0;\n elect.sync _|q, 0xffffffff;\n"
      " add.u32 a1, %1, 8;\n add.u32 a2, %1, 16;\n add.u32 a3, %1, 24;\n add.s64 b1, %2, 2;\n add.s64 b2, %2, 4;\n add.s64 b3, %2, 6;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], b1, %3, t;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a2], b2, %3, t;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a3], b3, %3, t;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the same, of every slice of sixteen K first the product with the tile at bdesc, then the one `to_lo` behind it
__device__ __forceinline__ void qi_umma8(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint64_t to_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q, t;\n .reg .b32 a1, a2, a3;\n .reg .b64 b1, b2, b3, c0, c1, c2, c3;\n setp.ne.b32 p, %5, 0;\n setp.eq.u32 t, 0, 0;\n elect.sync _|q, 0xffffffff;\n"
      " add.u32 a1, %1, 8;\n add.u32 a2, %1, 16;\n add.u32 a3, %1, 24;\n add.s64 b1, %2, 2;\n add.s64 b2, %2, 4;\n add.s64 b3, %2, 6;\n"
      " add.s64 c0, %2, %3;\n add.s64 c1, c0, 2;\n add.s64 c2, c0, 4;\n add.s64 c3, c0, 6;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %4, p;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], c0, %4, t;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], b1, %4, t;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], c1, %4, t;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a2], b2, %4, t;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a2], c2, %4, t;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a3], b3, %4, t;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [a3], c3, %4, t;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "l"(to_lo), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void qi_umma1(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n elect.sync _|q, 0xffffffff;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// two K steps of this CTA's activation rows: the box is (64 K, rows, parts, 2 K steps); bytes are counted on CTA 0's barrier,
// which also expects them there (`expect` > 0)
__device__ __forceinline__ void qi_load_x(uint32_t dst, const CUtensorMap *map, int row, int kstep, uint32_t bar_cluster, uint32_t bar_own, uint32_t expect) {
  asm volatile(
      "{\n .reg .pred q, e, n;\n elect.sync _|q, 0xffffffff;\n setp.ne.and.u32 e|n, %6, 0, q;\n @e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%5], %6;\n"
      " @q cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {0, %2, 0, %3}], [%4];\n}\n" ::"r"(dst),
      "l"(map), "r"(row), "r"(kstep), "r"(bar_cluster), "r"(bar_own), "r"(expect)
      : "memory");
}
__device__ __forceinline__ void qi_cp16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void qi_cp_arrive(uint32_t bar) {  // this thread's copies count as one more arrival, when they are there
  asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// waits for this thread's loads of tensor memory, those of r among them
__device__ __forceinline__ void qi_tmem_wait32(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                 "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28])
               :
               : "memory");
  asm volatile("" : "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
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
  const float *col_scale;  // per activation row: undoes the scale of the row (f32), or that of its sub-block sums (f16)
  const float *residual;   // added to the result (f32, may be the output itself), or null
  int silu;                // f32 output: weight rows are gate|up pairs (groups of sixteen); store silu(gate) * up, N / 2 columns
};

// F32: f16 activations (0), f32 activations with lo and hi products in turn (1) or the lo products first (2)
template <int F32, typename OutT>
__global__ void __launch_bounds__(QI_THREADS, 1) gemm_q4k_int_kernel(const __grid_constant__ CUtensorMap tmap_x,
                                                                     const __grid_constant__ CUtensorMap tmap_s, const __grid_constant__ CUtensorMap tmap_w,
                                                                     const uint8_t *__restrict__ W, OutT *C, int M, int N, IntPlan p, IntOut o,
                                                                     int *__restrict__ err) {
  constexpr bool LO = F32 > 0;
  extern __shared__ uint8_t qi_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(qi_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bar_words[2 * QI_BARS + 2 * QI_PACKED + QI_SCALES + QI_ACCS];
  __shared__ float row_scales[QI_SCALES][QI_ROWS];  // what a unit's product is multiplied by on read-back: d, or the sum unit's power of two
  __shared__ __align__(16) float col_scales[QI_DRAINERS][QI_BN / 2];  // of a draining warp's activation rows: alpha * row_scale, or sum_scale
  __shared__ uint32_t tmem_word;
  __shared__ int abort_word;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t rank = cluster_ctarank();
  const int cluster = (int)(blockIdx.x >> 1), clusters = (int)(gridDim.x >> 1);
  const int hb = p.bn / 2, units = p.npu + p.pb;
  const uint32_t x_tile = qi_x_tile(p), x_step = x_tile * (LO ? 2u : 1u), x_stage = 2u * x_step;  // a K step; the two of a stage
  uint8_t *ring_p = smem + (uint32_t)p.sa * x_stage;
  volatile int *abort_flag = &abort_word;
  const uint32_t bars = smem_u32(bar_words);
  // One barrier says that a group's activations and weights are there (a wait costs the MMA lane two hundred cycles).  It
  // goes by group like "multiplied", not by stage: a group is loaded or built only after the one `ring depth` before it has
  // been multiplied.  The four sets of builders are not in step, so a ring of barriers must be longer than those of the
  // stages: whoever waits for group g - 8 must see it before group g + 8 is multiplied, which needs this waiter's own group g.
  auto full = [&](uint32_t g) { return bars + 8u * (g & (QI_BARS - 1)); };
  auto done = [&](uint32_t g) { return bars + 8u * (QI_BARS + (g & (QI_BARS - 1))); };
  auto parity = [&](uint32_t g) { return (g / QI_BARS) & 1u; };
  auto full_p = [&](uint32_t s) { return bars + 8u * (2 * QI_BARS + s); };
  auto free_p = [&](uint32_t s) { return bars + 8u * (2 * QI_BARS + QI_PACKED + s); };
  // The row scales of unit n are written: builders to drains of the same CTA (by way of "full", the MMAs and "multiplied" they
  // would leave the CTA and come back through arrives that order nothing there).  The ring is long enough: a builder says so of
  // unit n only after unit n - 2 has been started, and that after every drain has handed back unit n - 2 - QI_ACCS; it writes
  // them after unit n - 3 has been started.
  auto scaled = [&](uint32_t n) { return bars + 8u * (2 * QI_BARS + 2 * QI_PACKED + (n & (QI_SCALES - 1))); };
  auto scaled_parity = [&](uint32_t n) { return (n / QI_SCALES) & 1u; };
  auto empty = [&](uint32_t b) { return bars + 8u * (2 * QI_BARS + 2 * QI_PACKED + QI_SCALES + b); };
  // how often the accumulators had been gone through before unit n, which takes accumulator n - na * rounds
  auto rounds = [&](uint32_t n) { return p.na == 3 ? __umulhi(n, 0xAAAAAAABu) >> 1 : n >> (p.na >> 1); };
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
    for (uint32_t s = 0; s < QI_BARS; s++) {
      // CTA 0's: a set of builders of either CTA, and with a pair's first group the activation copies' expected bytes
      mbar_init(full(s), 2 * QI_BUILDERS / 4 + (s & 1 ? 0 : 1));
      mbar_init(done(s), 1);
    }
    for (uint32_t s = 0; s < QI_PACKED; s++) {
      mbar_init(full_p(s), 1);
      mbar_init(free_p(s), QI_BUILDERS / 2);
    }
    for (uint32_t s = 0; s < QI_SCALES; s++) mbar_init(scaled(s), QI_BUILDERS / 4);
    for (uint32_t b = 0; b < QI_ACCS; b++) mbar_init(empty(b), 2 * QI_DRAINERS);  // CTA 0's: the drains of both CTAs
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
  // columns: the accumulators, then the weight groups
  const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(&tmem_word), 0), tmem_w = tmem + (uint32_t)(p.na * p.bn);

  // 4 warps x 24 + 16 x 48 + 8 x 144 registers: what the launch holds (28 warps x 72)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    if (warp == 0) {
      // ---------------- activation tiles: this CTA's half of the rows, two K steps a copy ----------------
      const uint32_t full0 = mapa_shared(full(0), 0u);
      uint32_t g = 0, i = 0, dst = smem_u32(smem);
      const uint32_t depth = 2u * (uint32_t)p.sa, end = dst + (uint32_t)p.sa * x_stage;
      bool ok = true;
      for (int item = cluster; item < p.items && ok; item += clusters) {
        const int row0 = tile_m_of(item) * p.bn + (int)rank * hb, part = part_of(item);
        for (int u = 0; u < units && ok; u++) {
          const bool sums = u < p.npu;
          const int step0 = sums ? (part * p.npu + u) * 4 : block_of(item, u) * 4;
          const uint32_t expect = rank == 0 ? 2u * (sums ? 2u * x_tile : x_stage) : 0u;  // both CTAs' bytes
#pragma unroll
          for (int h = 0; h < 4; h += 2, g += 2) {
            const uint32_t before = g + 1u - depth;  // the last group of the pair that used this stage last
            if (i >= (uint32_t)p.sa && !mbar_wait_warp(done(before), parity(before), abort_flag)) { ok = false; break; }
            qi_load_x(dst, sums ? &tmap_s : &tmap_x, row0, step0 + h, full0 + 8u * (g & (QI_BARS - 1)), full(g), expect);
            i++;
            dst += x_stage;
            if (dst == end) dst = smem_u32(smem);
          }
        }
      }
      // no copy of the pair may still be in flight at the end, also where a wait gave up (the builders' arrivals are missing then)
      if (rank == 0 && g > 0 && lane == 0)
        for (uint32_t poll = 0; poll < (1u << 16) && !mbar_try_wait(full(g - 2), parity(g - 2)); poll++) {}
    } else if (warp == 3) {
      // ---------------- packed super-blocks of this CTA's weight rows by TMA; for a sum unit their headers, sixteen bytes each ----------------
      // (a TMA box of sixteen bytes a row takes two thousand cycles, in which no other copy gets through)
      QiRing r;
      uint32_t n = 0;
      bool ok = true;
      for (int item = cluster; item < p.items && ok; item += clusters) {
        const int row0 = tile_n_of(item) * 256 + (int)rank * QI_ROWS;
        for (int u = 0; u < units; u++, n++, r.next(p.sp)) {
          if (r.uses && !mbar_wait_warp(free_p(r.i), (r.uses - 1u) & 1u, abort_flag)) { ok = false; break; }
          const uint32_t dst = smem_u32(ring_p) + r.i * QI_P_STAGE, bar = full_p(r.i);
          if (u < p.npu) {
            const int b0 = qi_sum_begin(p, u), nsb = qi_sum_begin(p, u + 1) - b0;
            // eight lanes a row, four rows at a time; rows beyond N are not stored
            const int k = lane & 7;
            for (int i = lane >> 3; i < QI_ROWS; i += 4)
              if (k < nsb)
                qi_cp16(dst + (uint32_t)i * Q4K_BLOCK_BYTES + 16u * k, W + ((size_t)min(row0 + i, N - 1) * p.bpr + part_of(item) * p.pb + b0 + k) * Q4K_BLOCK_BYTES);
            qi_cp_arrive(bar);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
          } else if (lane == 0) {
            mbar_expect_tx(bar, QI_P_STAGE);
            tma_load_2d(dst, &tmap_w, block_of(item, u) * Q4K_BLOCK_BYTES, row0, bar);
          }
          __syncwarp();
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      const uint32_t held = n < (uint32_t)p.sp ? n : (uint32_t)p.sp;
      for (uint32_t i = n - held; i < n && lane == 0; i++)
        for (uint32_t poll = 0; poll < (1u << 20) && !mbar_try_wait(full_p(i % (uint32_t)p.sp), (i / (uint32_t)p.sp) & 1u); poll++) {}
    } else if ((warp == 1 || warp == 2) && rank == 0) {
      // ---------------- MMA issue for the pair: warp 1 the even units, warp 2 the odd ones, each into its own accumulator ----------------
      // The queue in front of the tensor cores is short: a lane that issues everything leaves them idle while it waits for the
      // next group's barrier.  Two lanes: one waits while the other's MMAs run (4960 -> 3970 cycles per super-block of a tile of
      // 160 f32 rows).  Made to strictly take turns they were slower: the hand-over is one more wait.
      const uint32_t idesc = umma_idesc_f16(256, p.bn);
      const uint64_t to_lo = x_tile >> 4;
      const int mine = warp - 1, total = units * (cluster < p.items ? (p.items - 1 - cluster) / clusters + 1 : 0);
      const uint32_t w_end = tmem_w + (uint32_t)p.sb * QI_W_COLS;
      const uint64_t x_first = umma_desc_sw128(smem_u32(smem)), x_end = x_first + (uint64_t)((uint32_t)p.sa * x_stage >> 4);
      // the weight group and the pair of K steps a unit begins with
      uint32_t w = tmem_w;
      uint64_t x = x_first;
      auto next_w = [&](uint32_t &at) { at += QI_W_COLS; if (at == w_end) at = tmem_w; };
      auto next_x = [&](uint64_t &at) { at += x_stage >> 4; if (at == x_end) at = x_first; };
      auto skip = [&]() {
#pragma unroll
        for (int i = 0; i < 4; i++) next_w(w);
        next_x(x);
        next_x(x);
      };
      if (mine == 1) skip();
      bool ok = true;
      int u = mine;  // unit of the item
      for (int n = mine; n < total && ok; n += 2) {
        const bool sums = u < p.npu;
        const uint32_t g0 = 4u * (uint32_t)n, round = rounds((uint32_t)n), b = (uint32_t)n - (uint32_t)p.na * round, acc = tmem + b * (uint32_t)p.bn;
        // A barrier is looked at ahead of its turn: the answer takes a while, also where it has long been there.
        uint32_t seen = mbar_try_wait(full(g0), parity(g0));
        auto there = [&](uint32_t g) { return __shfl_sync(0xffffffffu, seen, 0) || mbar_wait_warp(full(g), parity(g), abort_flag); };
        if (round > 0 && !mbar_wait_warp(empty(b), (round - 1u) & 1u, abort_flag)) break;
        if (F32 == 2 && !sums) {  // lo products first
          uint32_t w2 = w;
          uint64_t x2 = x;
#pragma unroll
          for (int h = 0; h < 4; h++) {
            if (!there(g0 + h)) { ok = false; break; }
            if (h < 3) seen = mbar_try_wait(full(g0 + h + 1), parity(g0 + h + 1));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            qi_umma4(acc, w2, x2 + (h & 1) * (x_step >> 4) + to_lo, idesc, h);
            next_w(w2);
            if (h & 1) next_x(x2);
          }
          if (!ok) break;
        }
        if (sums) {
          const int nsb = qi_sum_begin(p, u + 1) - qi_sum_begin(p, u), first = qi_sum_first(nsb);
          const int slices[2] = {qi_sum_slices(first), qi_sum_slices(nsb - first)};
          uint32_t wg[4];
          uint64_t xg[4];
          for (int h = 0; h < 4 && ok; h++) {
            if (!there(g0 + h)) ok = false;
            if (h < 3) seen = mbar_try_wait(full(g0 + h + 1), parity(g0 + h + 1));
          }
          if (!ok) break;
#pragma unroll
          for (int h = 0; h < 4; h++) {
            wg[h] = w;
            xg[h] = x + (h & 1) * (x_tile >> 4);
            next_w(w);
            if (h & 1) next_x(x);
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // the small products first, or the large ones: see above
          const int large = F32 == 2 && nsb >= 7 ? 2 : 0;
          uint32_t more = 0;
#pragma unroll 1
          for (int i = 0; i < 3; i++) {
            const int product = large == 2 ? (i == 2 ? QI_HH : i + 1) : i;
#pragma unroll
            for (int half = 0; half < 2; half++)
#pragma unroll 1
              for (int k = 0; k < slices[half]; k++) {
                const int t = product * slices[half] + k;  // slice of the half
                qi_umma1(acc, (t < 4 ? wg[2 * half] : wg[2 * half + 1]) + 8u * (t & 3), (t < 4 ? xg[2 * half] : xg[2 * half + 1]) + 2 * (t & 3), idesc, more);
                more = 1;
              }
          }
#pragma unroll
          for (int h = 0; h < 4; h++) umma_commit_warp<true>(done(g0 + h));
        } else {
#pragma unroll
          for (int h = 0; h < 4; h++) {
            if (F32 != 2 && !there(g0 + h)) { ok = false; break; }
            if (F32 != 2 && h < 3) seen = mbar_try_wait(full(g0 + h + 1), parity(g0 + h + 1));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if constexpr (F32 == 1) qi_umma8(acc, w, x + (h & 1) * (x_step >> 4), to_lo, idesc, h);
            else qi_umma4(acc, w, x + (h & 1) * (x_step >> 4), idesc, F32 == 2 ? 1u : h);
            umma_commit_warp<true>(done(g0 + h));
            next_w(w);
            if (h & 1) next_x(x);
          }
        }
        skip();  // the other lane's unit
        u += 2;
        if (u >= units) u -= units;
      }
    }
  } else if (warp < 4 + QI_BUILDERS) {
    // ---------------- weight tiles into tensor memory ----------------
    // A thread one row.  Eight warps build the even units, eight the odd ones, of a unit's four K steps a warp two: a warp's time
    // goes to waits for barriers, loads and stores of its own, 1800 cycles a unit when each warp took a K step of every unit.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    const int quad = warp & 3, half = ((warp - 4) >> 2) & 1, odd = (warp - 4) >> 3, row = quad * 32 + lane;
    constexpr uint32_t Y64 = 0x64646464u, K1024 = 0x64006400u, KM1024 = 0xE400E400u, R16 = 0x2C002C00u;
    const uint32_t full0 = mapa_shared(full(0), 0u), w_size = (uint32_t)p.sb * QI_W_COLS;
    const uint32_t lanes = tmem_w + ((uint32_t)(quad * 32) << 16);
    uint32_t w = 2u * (uint32_t)half * QI_W_COLS;  // this warp's first group of the unit, in the ring
    QiRing rp;
    auto step_unit = [&]() {
      rp.next(p.sp);
      w += 4u * QI_W_COLS;
      while (w >= w_size) w -= w_size;
    };
    if (odd) step_unit();
    bool ok = true;
    auto stage_free = [&](uint32_t g) {
      bool fr = true;
      if (g >= (uint32_t)p.sb) fr = mbar_wait_bounded(done(g - (uint32_t)p.sb), parity(g - (uint32_t)p.sb), abort_flag);
      return __all_sync(0xffffffffu, fr) != 0;
    };
    // this warp's stores of a group are in tensor memory: tell the MMA warps
    auto written = [&](uint32_t g) {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (rank == 0) mbar_arrive(full(g));
        else qi_arrive_remote(full0 + 8u * (g & (QI_BARS - 1)));
      }
    };
    uint32_t n0 = 0;  // units of the items before
    for (int item = cluster; item < p.items && ok; item += clusters, n0 += (uint32_t)units) {
      for (int u = (int)((n0 ^ (uint32_t)odd) & 1u); u < units; u += 2) {
        const uint32_t n = n0 + (uint32_t)u;
        uint32_t g = 4u * n + 2u * (uint32_t)half;
        const bool here = mbar_wait_bounded(full_p(rp.i), rp.uses & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, here)) { ok = false; break; }
        const uint8_t *blk = ring_p + rp.i * QI_P_STAGE + (uint32_t)row * Q4K_BLOCK_BYTES;
        if (u < p.npu) {
          // ---- sum unit: of half of its super-blocks all three products ----
          const int nsb = qi_sum_begin(p, u + 1) - qi_sum_begin(p, u);
          float most = 0.0f;
#pragma unroll
          for (int k = 0; k < QI_SUMS; k++)
            if (k < nsb) most = fmaxf(most, fabsf(q4k_d_dmin(*reinterpret_cast<const uint32_t *>(blk + 16 * k)).y));
          const float scale = qi_pow2(8 - qi_exponent(most));
          if (half == 0) row_scales[n % QI_SCALES][row] = -64.0f * qi_pow2(qi_exponent(most) - 8);  // (the sums are stored divided by 64)
          const int k0 = half ? qi_sum_first(nsb) : 0, count = half ? nsb - k0 : qi_sum_first(nsb), wide = 2 * qi_sum_slices(count);
          if (!stage_free(g) || !stage_free(g + 1)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t w1 = w + QI_W_COLS == w_size ? 0u : w + QI_W_COLS;
          // eight values of a super-block, four columns: place c of this half's sixteen
          auto put = [&](int c, const uint32_t (&v)[4]) { qi_tmem_st4(lanes + (c & 8 ? w1 : w) + (uint32_t)(c & 7) * 4u, v); };
#pragma unroll 2
          for (int k = 0; k < wide; k++) {  // (uniform)
            uint32_t hi[4] = {0u, 0u, 0u, 0u}, lo[4] = {0u, 0u, 0u, 0u};  // zeros beyond the last super-block
            if (k < count) {
              const uint4 hd = *reinterpret_cast<const uint4 *>(blk + 16 * (k0 + k));
              const Q4KScales sc = q4k_unpack_scales(hd.y, hd.z, hd.w);
              const __half2 dm2 = __float2half2_rn(q4k_d_dmin(hd.x).y * scale);
              const uint32_t dm = *reinterpret_cast<const uint32_t *>(&dm2);
#pragma unroll
              for (int j = 0; j < 4; j++) {
                const uint32_t m = qi_hsub2(__byte_perm(j < 2 ? sc.mn03 : sc.mn47, Y64, (j & 1) ? 0x4342u : 0x4140u), K1024);
                hi[j] = qi_hmul2(dm, m);
                lo[j] = qi_hfma2(dm, m, hi[j] ^ 0x80008000u);  // exactly what the rounding dropped
              }
            }
            put(QI_HH * wide + k, hi);
            put(QI_LH * wide + k, lo);
            put(QI_HL * wide + k, hi);
          }
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(free_p(rp.i));
            if (half == 0) mbar_arrive(scaled(n));
          }
          written(g);
          written(g + 1);
          step_unit();
          step_unit();
          continue;
        }
        // ---- super-block ----
        const uint4 hd = *reinterpret_cast<const uint4 *>(blk);
        blk += 16 + 64 * half;  // this warp's two K steps: 64 weights in 32 bytes each
        // the four scale codes of this half of the super-block
        const uint32_t cw = half == 0 ? hd.y & 0x3f3f3f3fu : (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);
        if (half == 0) row_scales[n % QI_SCALES][row] = q4k_d_dmin(hd.x).x;
        uint4 qa = *reinterpret_cast<const uint4 *>(blk), qb = *reinterpret_cast<const uint4 *>(blk + 16);
#pragma unroll
        for (int h = 0; h < 2; h++, g++) {
          // The K step's two scale codes as f16 pairs (the second divided by 16), and -1024 times them.  A word of eight weights:
          // nibbles two bytes apart make a pair, so that one LOP3 makes 1024 + q (of the high nibbles 1024 + 16 q) out of it;
          // (1024 + q) * sc - 1024 * sc = sc * q exactly.  The activations are stored with the second and third of every four
          // values swapped to match.
          const uint32_t sca = qi_hsub2(__byte_perm(cw, Y64, h ? 0x4242u : 0x4040u), K1024), scb = qi_hmul2(qi_hsub2(__byte_perm(cw, Y64, h ? 0x4343u : 0x4141u), K1024), R16);
          const uint32_t nega = qi_hmul2(sca, KM1024), negb = qi_hmul2(scb, KM1024);
          const uint32_t q[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
          uint32_t v[16];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            v[2 * i] = qi_hfma2((q[i] & 0x000f000fu) | K1024, sca, nega);
            v[2 * i + 1] = qi_hfma2(((q[i] >> 8) & 0x000f000fu) | K1024, sca, nega);
          }
          if (!stage_free(g)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t at = lanes + w;
          qi_tmem_st16(at, v);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            v[2 * i] = qi_hfma2((q[i] & 0x00f000f0u) | K1024, scb, negb);
            v[2 * i + 1] = qi_hfma2(((q[i] >> 8) & 0x00f000f0u) | K1024, scb, negb);
          }
          if (h == 0) {
            qa = *reinterpret_cast<const uint4 *>(blk + 32);
            qb = *reinterpret_cast<const uint4 *>(blk + 48);
          }
          qi_tmem_st16(at + 16u, v);
          if (h == 1) {
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(free_p(rp.i));
              if (half == 0) mbar_arrive(scaled(n));
            }
          }
          written(g);
          w += QI_W_COLS;
          if (w == w_size) w = 0;
        }
        if (!ok) break;
        // (w has moved by two groups)
        w += 6u * QI_W_COLS;
        while (w >= w_size) w -= w_size;
        rp.next(p.sp);
        rp.next(p.sp);
      }
    }
  } else {
    // ---------------- tensor memory -> d * P (and the sum units) -> f32 sums -> C ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    const int drain = warp - 4 - QI_BUILDERS, quad = warp & 3, half = drain >> 2, cw = p.bn / 2;  // this warp's columns: half * cw ..
    const uint32_t empty0 = mapa_shared(empty(0), 0u);
    float *col = col_scales[drain];
    uint32_t n = 0;
    bool ok = true;
    for (int item = cluster; item < p.items && ok; item += clusters) {
      const int f = tile_n_of(item) * 256 + (int)rank * QI_ROWS + quad * 32 + lane, m0 = tile_m_of(item) * p.bn + half * cw;
      __syncwarp();  // the scales of the tile before have been read
      for (int c = lane; c < QI_BN / 2; c += 32) {
        float v = 0.0f;
        if (c < cw && m0 + c < M) v = LO ? o.alpha * __ldg(o.col_scale + m0 + c) : __ldg(o.col_scale + m0 + c);
        col[c] = v;
      }
      __syncwarp();
      qi_f2 acc[QI_BN / 4];  // two activation rows each
#pragma unroll
      for (int i = 0; i < QI_BN / 4; i++) acc[i] = 0;
      for (int u = 0; u < units; u++, n++) {
        const uint32_t g = 4u * n + 3u, b = n - (uint32_t)p.na * rounds(n);
        const bool ready = mbar_wait_bounded(scaled(n), scaled_parity(n), abort_flag) && mbar_wait_bounded(done(g), parity(g), abort_flag);
        if (!__all_sync(0xffffffffu, ready)) { ok = false; break; }  // tcgen05.ld is warp-wide: together or not at all
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + b * (uint32_t)p.bn + (uint32_t)(half * cw);
        const float scale1 = row_scales[n % QI_SCALES][quad * 32 + lane];
        const qi_f2 scale = qi_pack(scale1, scale1);
#pragma unroll
        for (int c = 0; c < QI_BN / 64; c++) {
          if (c * 32 < cw) {  // (uniform; where cw is an odd number of sixteens the last sixteen columns are read and not stored)
            uint32_t r[32];
            tmem_ld32(taddr + (uint32_t)(c * 32), r);
            qi_tmem_wait32(r);
            if (c * 32 + 32 >= cw) {  // all of it is read: hand it back
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              __syncwarp();
              if (lane == 0) qi_arrive_remote(empty0 + 8u * b);
            }
#pragma unroll
            for (int i = 0; i < 16; i++) acc[c * 16 + i] = qi_fma(scale, qi_pack(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), acc[c * 16 + i]);
          }
        }
        if (!LO && u == p.npu - 1) {
#pragma unroll
          for (int i = 0; i < QI_BN / 2; i += 4) {
            const float4 t = *reinterpret_cast<const float4 *>(col + i);
            acc[i / 2] = qi_mul(acc[i / 2], qi_pack(t.x, t.y));
            acc[i / 2 + 1] = qi_mul(acc[i / 2 + 1], qi_pack(t.z, t.w));
          }
        }
      }
      if (!ok) break;
      // A warp stores 32 consecutive features of an activation row at a time.  The code of QI_STORE rows is run over and over
      // while the sums move down as many registers: unrolled over all columns it was run once per tile straight out of
      // instruction cache misses (33 thousand cycles per tile), and eight rows at a time spent 10 to 20 thousand cycles, in
      // which the tensor cores run dry, mostly on moves and on the scales' shuffles.
      OutT *tile = C + (p.parts > 1 ? (size_t)part_of(item) * (size_t)M * (size_t)N : (size_t)0);
      const bool is_up = lane & 8, in = f < N;
      const int rows = min(cw, M - m0);
      const size_t pitch = o.silu ? (size_t)(N / 2) : (size_t)N;
      OutT *dst = tile + (size_t)m0 * pitch + (o.silu ? (size_t)((f >> 4) * 8 + (f & 7)) + (is_up ? pitch : (size_t)0) : (size_t)f);
      const float *res = o.residual ? o.residual + (size_t)m0 * pitch + f : nullptr;
#pragma unroll 1
      for (int c = 0; c < rows; c += QI_STORE) {
        const int left = rows - c;
#pragma unroll
        for (int i = 0; i < QI_STORE; i += 4) {
          if (i >= left) break;  // (uniform)
          const float4 t = LO ? *reinterpret_cast<const float4 *>(col + c + i) : make_float4(o.alpha, o.alpha, o.alpha, o.alpha);
          float v[4] = {qi_low(acc[i / 2]) * t.x, qi_high(acc[i / 2]) * t.y, qi_low(acc[i / 2 + 1]) * t.z, qi_high(acc[i / 2 + 1]) * t.w};
          const bool all = i + 4 <= left;  // (uniform)
          if (sizeof(OutT) == 4 && o.silu) {
            // a gate row and its up row are eight lanes apart: the gate's lane takes the even activation rows, the other the odd
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
              const float got = __shfl_xor_sync(0xffffffffu, is_up ? v[j] : v[j + 1], 8);
              const float gv = is_up ? got : v[j], uv = is_up ? v[j + 1] : got;
              const float cl = fminf(fmaxf(gv, -15.0f), 15.0f);  // silu.wgsl:30-37,98-104
              if (in && (all || i + j + (is_up ? 1 : 0) < left)) qi_store(dst, (gv * (1.0f / (1.0f + expf(-cl)))) * uv);
              dst += 2 * pitch;
            }
          } else {
            if (sizeof(OutT) == 4 && res) {
#pragma unroll
              for (int j = 0; j < 4; j++) {
                if (in && (all || i + j < left)) v[j] += *res;
                res += pitch;
              }
            }
            if (all) {
              if (in) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                  qi_store(dst, v[j]);
                  dst += pitch;
                }
              }
            } else if (in) {
#pragma unroll
              for (int j = 0; j < 3; j++) {
                if (i + j < left) qi_store(dst, v[j]);
                dst += pitch;
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i + QI_STORE / 2 < QI_BN / 4; i++) acc[i] = acc[i + QI_STORE / 2];
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
__device__ __forceinline__ void qi_put_sum(__half *sums_row, const IntPlan &p, int s, float v) {
  const int sb = s >> 3, part = sb / p.pb, k = sb - part * p.pb;
  const int u = ((k + 1) * p.npu - 1) / p.pb, b0 = qi_sum_begin(p, u), nsb = qi_sum_begin(p, u + 1) - b0;
  const int first = qi_sum_first(nsb), half = k - b0 >= first, count = half ? nsb - first : first, wide = 2 * qi_sum_slices(count), j = k - b0 - (half ? first : 0);
  __half *at = sums_row + (size_t)(part * p.npu + u) * 256 + half * 128 + (s & 7);
  const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi)), zero = __float2half_rn(0.0f);
  at[(QI_HH * wide + j) * 8] = hi;
  at[(QI_LH * wide + j) * 8] = hi;
  at[(QI_HL * wide + j) * 8] = lo;
  if (j == 0 && (count & 1))  // they pair with the weights' zeros
    at[(QI_HH * wide + count) * 8] = at[(QI_LH * wide + count) * 8] = at[(QI_HL * wide + count) * 8] = zero;
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

template <int WARPS = 8>
__device__ __forceinline__ float qi_block_max(float v, float *sh) {  // 8 or 32 warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = sh[WARPS == 32 ? threadIdx.x & 31 : 0];
  if constexpr (WARPS == 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, o));
  } else {
#pragma unroll
    for (int w = 1; w < WARPS; w++) t = fmaxf(t, sh[w]);
  }
  return t;
}

// One block per row, any K and alignment.  f32 rows: scaled by a power of two and split, x * 2^-e = hi + lo (rows of kp
// halves, a multiple of 64, zeros beyond K), row_scale = 2^e.  f16 rows: copied to hi as they are, the sums alone are scaled,
// sum_scale = 2^e.  Of every four values the second and the third change places, as the weight tiles have them.  The sums are divided by 64 on top.
template <typename AT>
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
      const size_t at = (size_t)row * kp + ((i & ~3) | (i & 1) << 1 | (i >> 1 & 1));
      if constexpr (sizeof(AT) == 4) {
        const __half h = __float2half_rn(t);
        hi[at] = h;
        lo[at] = __float2half_rn(t - __half2float(h));
      } else {
        hi[at] = __float2half_rn(v);
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
    if (lane == 0) qi_put_sum(sums + (size_t)row * ((size_t)p.parts * p.npu * 256), p, s, t * 0.015625f);
  }
}

// The same for f32 rows with the row in registers (K % 32 == 0, K <= 1024 * NV, 16-byte aligned): one pass, 16-byte loads.
// With norm_w the row is RMS-normalised first (rmsnorm.wgsl:119-187), element for element and reduction step for
// reduction step as rmsnorm_vec_kernel (small_ops.cu) does it for rows of 1024..4096 values, by 256 threads.  Few rows without
// a norm take 1024 threads each (the same bits): a row's loads are one wait and not twelve deep; 64 x 12288 8.6 -> 5.7 us, 64 x 4096 4.6 -> 4.1.
template <int NV, int T = 256>
__global__ void __launch_bounds__(T) int_rows_vec_kernel(const float *__restrict__ in, __half *__restrict__ hi, __half *__restrict__ lo, float *__restrict__ scale,
                                                           __half *__restrict__ sums, int K, int kp, const IntPlan p, const float *__restrict__ norm_w, float eps, int guard) {
  pdl_launch();
  pdl_wait();
  __shared__ float sh[T / 32], shn[8];
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n4 = K >> 2;
  const size_t base = (size_t)row * K, out = (size_t)row * kp;
  float4 v[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int idx = threadIdx.x + i * T;
    v[i] = idx < n4 ? *reinterpret_cast<const float4 *>(in + base + 4 * idx) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  if (T == 256 && norm_w) {
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
      const int idx = threadIdx.x + i * T;
      if (idx < n4) {
        const float4 w = *reinterpret_cast<const float4 *>(norm_w + 4 * idx);
        v[i].x = v[i].x * inv_rms * w.x; v[i].y = v[i].y * inv_rms * w.y; v[i].z = v[i].z * inv_rms * w.z; v[i].w = v[i].w * inv_rms * w.w;
      }
    }
  }
  float mx = 0.0f;
#pragma unroll
  for (int i = 0; i < NV; i++) mx = fmaxf(fmaxf(mx, fmaxf(fabsf(v[i].x), fabsf(v[i].y))), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
  mx = qi_block_max<T / 32>(mx, sh);
  const int e = qi_row_exponent(mx);
  const float down = qi_pow2(-e);
  if (threadIdx.x == 0) scale[row] = qi_row_scale(mx, e, guard);
  __half *sums_row = sums + (size_t)row * ((size_t)p.parts * p.npu * 256);
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int idx = threadIdx.x + i * T;
    const float s0 = v[i].x * down, s1 = v[i].y * down, s2 = v[i].z * down, s3 = v[i].w * down;
    float t = (s0 + s1) + (s2 + s3);  // eight consecutive threads hold a sub-block
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    if (idx >= n4) continue;
    const __half2 h01 = __floats2half2_rn(s0, s2), h23 = __floats2half2_rn(s1, s3);  // (in the order of the weight tiles)
    const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
    const __half2 l01 = __floats2half2_rn(s0 - f01.x, s2 - f01.y), l23 = __floats2half2_rn(s1 - f23.x, s3 - f23.y);
    *reinterpret_cast<uint2 *>(hi + out + 4 * idx) = make_uint2(*reinterpret_cast<const uint32_t *>(&h01), *reinterpret_cast<const uint32_t *>(&h23));
    *reinterpret_cast<uint2 *>(lo + out + 4 * idx) = make_uint2(*reinterpret_cast<const uint32_t *>(&l01), *reinterpret_cast<const uint32_t *>(&l23));
    if ((threadIdx.x & 7) == 0) qi_put_sum(sums_row, p, idx >> 3, t * 0.015625f);
  }
  if ((int)threadIdx.x < kp - K) hi[out + K + threadIdx.x] = lo[out + K + threadIdx.x] = __float2half_rn(0.0f);
  // (sub-blocks beyond a K that is no multiple of 256)
  for (int s = (K >> 5) + (int)threadIdx.x; s < p.bpr * 8; s += T) qi_put_sum(sums_row, p, s, 0.0f);
}

// The same for f16 rows (K % 32 == 0, K <= 2048 * NV, 16-byte aligned): one pass, 16-byte accesses, where int_rows_kernel reads
// two bytes at a time, twice (512 x 4096: 19 -> 5 us, 512 x 12288: 53 -> 10 us).
template <int NV>
__global__ void __launch_bounds__(256) int_rows_f16_kernel(const __half *__restrict__ in, __half *__restrict__ hi, float *__restrict__ scale, __half *__restrict__ sums, int K, int kp,
                                                           const IntPlan p, int guard) {
  pdl_launch();
  pdl_wait();
  __shared__ float sh[8];
  const int row = blockIdx.x, n8 = K >> 3;
  uint4 v[NV];
  __half2 most = __float2half2_rn(0.0f);
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int idx = threadIdx.x + i * 256;
    v[i] = idx < n8 ? __ldg(reinterpret_cast<const uint4 *>(in + (size_t)row * K) + idx) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
    for (int j = 0; j < 4; j++) most = __hmax2(most, __habs2(*reinterpret_cast<const __half2 *>(&w[j])));
  }
  const float mx = qi_block_max(fmaxf(__low2float(most), __high2float(most)), sh);
  const int e = qi_row_exponent(mx);
  const float down = qi_pow2(-e);
  if (threadIdx.x == 0) scale[row] = qi_row_scale(mx, e, guard);
  __half *sums_row = sums + (size_t)row * ((size_t)p.parts * p.npu * 256);
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int idx = threadIdx.x + i * 256;
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
    if (idx < n8)
      reinterpret_cast<uint4 *>(hi + (size_t)row * kp)[idx] = make_uint4(__byte_perm(w[0], w[1], 0x5410u), __byte_perm(w[0], w[1], 0x7632u), __byte_perm(w[2], w[3], 0x5410u), __byte_perm(w[2], w[3], 0x7632u));
    float t = 0.0f;  // four consecutive threads hold a sub-block
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[j]));
      t += f.x * down + f.y * down;
    }
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    if (idx < n8 && (threadIdx.x & 3) == 0) qi_put_sum(sums_row, p, idx >> 2, t * 0.015625f);
  }
  if ((int)threadIdx.x < kp - K) hi[(size_t)row * kp + K + threadIdx.x] = __float2half_rn(0.0f);
  for (int s = (K >> 5) + (int)threadIdx.x; s < p.bpr * 8; s += 256) qi_put_sum(sums_row, p, s, 0.0f);
}

// C = sum of the parts of a K-split launch, in a fixed order (+ residual, which may be C itself)
template <typename OutT>
__global__ void __launch_bounds__(256) int_reduce_kernel(const float *__restrict__ parts, OutT *C, size_t n, int splits, const float *residual, int wide) {
  pdl_launch();
  pdl_wait();
  auto put = [&](size_t i, float v) {
    if constexpr (sizeof(OutT) == 4) C[i] = v;
    else C[i] = __float2half_rn(v);
  };
  if (wide) {  // all parts' loads at once, 16 bytes each: one wait (64 x 4096, five parts: 3.6 us -> 2.6)
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n / 4; i += (size_t)gridDim.x * 256) {
      float4 v[8];
#pragma unroll
      for (int z = 0; z < 8; z++)
        if (z < splits) v[z] = *reinterpret_cast<const float4 *>(parts + (size_t)z * n + 4 * i);
      const float4 r = residual ? *reinterpret_cast<const float4 *>(residual + 4 * i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int z = 1; z < 8; z++)
        if (z < splits) { v[0].x += v[z].x; v[0].y += v[z].y; v[0].z += v[z].z; v[0].w += v[z].w; }
      if (residual) { v[0].x += r.x; v[0].y += r.y; v[0].z += r.z; v[0].w += r.w; }
      if constexpr (sizeof(OutT) == 4) *reinterpret_cast<float4 *>(C + 4 * i) = v[0];
      else { put(4 * i, v[0].x); put(4 * i + 1, v[0].y); put(4 * i + 2, v[0].z); put(4 * i + 3, v[0].w); }
    }
    return;
  }
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
    float acc = parts[i];
    for (int z = 1; z < splits; z++) acc += parts[(size_t)z * n + i];
    if (residual) acc += residual[i];
    put(i, acc);
  }
}

// shared memory a plan's rings may take: what a launch may ask for, less alignment, barriers and row scales
size_t qi_ring_budget(const dp_ctx *ctx) { return ctx->smem_optin - 1024 - 8192; }

// Tile width and parts of K with the least estimated time, in microseconds.  A unit takes what the builders need or what its MMAs
// do, an item a fixed cost on top (fill, stores), a K split the pass that adds its parts.  The figures are from 2048 f32 rows x
// [24576, 4096] (32 / 64 / 96 / 128 / 160 / 192 columns: 1508 / 813 / 671 / 589 / 582 / 589 us) and 1024 f16 rows x [12288, 4096] (397 /
// 221 / 173 / 138 / 127 / 113 us).
IntPlan qi_plan(dp_ctx *ctx, int M, int N, int K, bool lo, bool lo_first, bool may_split) {
  IntPlan best = {};
  double best_cost = -1.0;
  const int clusters = ctx->sm_count / 2, bpr = (K + QK_K - 1) / QK_K, tiles_n = (N + 255) / 256;
  const size_t budget = qi_ring_budget(ctx);
  for (int parts = 1; parts <= (may_split ? 8 : 1); parts++) {
    if (bpr % parts || (parts > 1 && bpr / parts < 2)) continue;
    for (int bn = 32; bn <= QI_BN; bn += 32) {
      IntPlan p;
      p.bpr = bpr; p.parts = parts; p.pb = bpr / parts;       const int most = lo_first && p.pb > 24 ? QI_SUMS_LONG : QI_SUMS;
      p.npu = (p.pb + most - 1) / most;
      p.bn = bn; p.tiles_n = tiles_n; p.tiles_m = (M + bn - 1) / bn;
      p.items = p.tiles_n * p.tiles_m * parts;
      // tensor memory beside the accumulators; shared memory: three packed blocks, then activation groups, then a packed block more
      p.na = bn <= 64 ? QI_ACCS : bn <= 128 ? 3 : 2;
      p.sb = (512 - p.na * bn) / (int)QI_W_COLS;
      if (p.sb > QI_RING) p.sb = QI_RING;
      p.sa = 2; p.sp = QI_PACKED;  // (lo first holds the two pairs of a unit)
      if (qi_rings(p, lo) > budget) p.sp = 2;  // (never odd: a set of builders goes by every second stage)
      if (qi_rings(p, lo) > budget) continue;
      while (p.sa < QI_PAIRS) {
        ++p.sa;
        if (qi_rings(p, lo) > budget) { --p.sa; break; }
      }
      const double builders = lo ? 0.9 + 0.0008 * bn : 0.88 + 0.0022 * bn, unit = lo && 0.0104 * bn > builders ? 0.0104 * bn : builders;
      const double item = (p.pb + p.npu) * unit + 1.0 + 0.02 * bn, waves = (double)((p.items + clusters - 1) / clusters);
      const double cost = waves * item + (parts > 1 ? 2.0 + 4.0 * (double)M * N * (parts + 1) / 6e6 : 0.0);
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
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tm[0], tm[1], tm[2], W, C, M, N, p, o, ctx->dev_status);
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
  const bool lo_first = f32a && (guard || M <= 64 || (fuse && fuse->exact_weights));
  IntPlan p = qi_plan(ctx, M, N, K, f32a, lo_first, !silu);
  const int kp = (K + BK - 1) / BK * BK;
  const size_t a_bytes = ((size_t)M * kp * 2 + 255) / 256 * 256;
  size_t sum_cols, s_bytes;
  auto rows_scratch = [&]() -> dp_status {
    sum_cols = (size_t)p.parts * p.npu * 256;
    s_bytes = ((size_t)M * sum_cols * 2 + 255) / 256 * 256;
    return dp_scratch(ctx, &ctx->gemm_scratch, a_bytes * (f32a ? 2 : 1) + s_bytes + (size_t)M * 4, "matmul_a_f16");
  };
  // Where memory is short: one part of K needs none for its sums, and the kernels behind this one need none for the rows.
  dp_status st = rows_scratch();
  if (st == DP_OK && p.parts > 1) {
    st = dp_scratch(ctx, &ctx->gemm_split_scratch, (size_t)p.parts * M * N * 4, "matmul_k_split_parts");
    if (st == DP_ERR_OOM) {
      p = qi_plan(ctx, M, N, K, f32a, lo_first, false);
      st = rows_scratch();
    }
  }
  if (st == DP_ERR_OOM) return DP_OK;
  DP_TRY(st);
  char *base = (char *)ctx->gemm_scratch->dptr;
  __half *hi = (__half *)base, *lo = (__half *)(base + a_bytes), *sums = (__half *)(base + a_bytes * (f32a ? 2 : 1));
  float *scale = (float *)((char *)sums + s_bytes);
  const float eps = fuse ? fuse->eps : 0.0f;
  if (vec) {
    const float *a = (const float *)A;
    const bool few = M <= ctx->sm_count && !norm_w && K > 1024;
    auto rows = K <= 1024 ? int_rows_vec_kernel<1> : K <= 4096 ? int_rows_vec_kernel<4> : K <= 12288 ? int_rows_vec_kernel<12> : int_rows_vec_kernel<16>;
    if (few) rows = K <= 4096 ? int_rows_vec_kernel<1, 1024> : K <= 12288 ? int_rows_vec_kernel<3, 1024> : int_rows_vec_kernel<4, 1024>;
    DP_LAUNCH(ctx, rows, (unsigned)M, few ? 1024 : 256, 0, a, hi, lo, scale, sums, K, kp, p, norm_w, eps, guard);
  } else if (f32a) {
    DP_LAUNCH(ctx, int_rows_kernel<float>, (unsigned)M, 256, 0, (const float *)A, hi, lo, scale, sums, K, kp, p, guard);
  } else if (K % 32 == 0 && K <= 16384 && ((uintptr_t)A & 15) == 0) {
    auto rows = K <= 2048 ? int_rows_f16_kernel<1> : K <= 4096 ? int_rows_f16_kernel<2> : K <= 8192 ? int_rows_f16_kernel<4> : int_rows_f16_kernel<8>;
    DP_LAUNCH(ctx, rows, (unsigned)M, 256, 0, (const __half *)A, hi, scale, sums, K, kp, p, guard);
  } else {
    DP_LAUNCH(ctx, int_rows_kernel<__half>, (unsigned)M, 256, 0, (const __half *)A, hi, (__half *)nullptr, scale, sums, K, kp, p, guard);
  }

  CUtensorMap tm[3];
  for (int i = 0; i < 2; i++) {  // activations (f32: both halves), sums: (K within a step, row, half, K step)
    const bool sum = i == 1;
    const cuuint64_t pitch = sum ? (cuuint64_t)sum_cols * 2 : (cuuint64_t)kp * 2, halves = f32a && !sum ? 2 : 1;
    const cuuint64_t dims[4] = {BK, (cuuint64_t)M, halves, pitch / (2 * BK)}, strides[3] = {pitch, halves == 2 ? (cuuint64_t)a_bytes : pitch, 2 * BK};
    const cuuint32_t box[4] = {BK, (cuuint32_t)(p.bn / 2), (cuuint32_t)halves, 2}, estr[4] = {1, 1, 1, 1};
    const CUresult r = encode(&tm[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, sum ? (void *)sums : (void *)hi, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return dp_fail(ctx, DP_ERR_CUDA, "matmul: cuTensorMapEncodeTiled failed (%d) for A[%d,%d]", (int)r, M, K);
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)p.bpr * Q4K_BLOCK_BYTES, (cuuint64_t)N}, strides[1] = {(cuuint64_t)p.bpr * Q4K_BLOCK_BYTES};
    const cuuint32_t wbox[2] = {Q4K_BLOCK_BYTES, QI_ROWS}, estr[2] = {1, 1};
    const CUresult r = encode(&tm[2], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)W, dims, strides, wbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return dp_fail(ctx, DP_ERR_CUDA, "matmul: cuTensorMapEncodeTiled failed (%d) for W[%d,%d]", (int)r, N, K);
  }

  IntOut o = {alpha, scale, nullptr, silu ? 1 : 0};
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
    const int wide = n % 4 == 0 && !(((uintptr_t)final_dst | (uintptr_t)residual) & 15);
    size_t grid = ((wide ? n / 4 : n) + 255) / 256;
    if (grid > (size_t)ctx->sm_count * 8) grid = (size_t)ctx->sm_count * 8;
    const float *parts = (const float *)dst;
    if (c_dtype == DP_F32) DP_LAUNCH(ctx, int_reduce_kernel<float>, (unsigned)grid, 256, 0, parts, (float *)final_dst, n, p.parts, residual, wide);
    else DP_LAUNCH(ctx, int_reduce_kernel<__half>, (unsigned)grid, 256, 0, parts, (__half *)final_dst, n, p.parts, residual, wide);
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
