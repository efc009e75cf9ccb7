// Sizes of the tensor-core kernels' output tiles, chosen on the host.
#pragma once

// An MMA of two CTAs over 16-bit operands (tcgen05.mma.cta_group::2, kind::f16) takes 32 to 256 columns in steps of 32.  One of a
// single CTA with 128 rows takes steps of 16.
constexpr int PAIR_STEP = 32;

// gemm_bf16.cu: activation rows per tile, and whether two SMs share one: the least estimated time in cycles.  A K step takes its
// MMAs (two cycles per activation row) or what it fetches from L2, at some 44 bytes a cycle and SM.
struct TilePick {
  int bn;
  bool pair;
};
inline TilePick pick_tile(int sm_count, int M, int N, int ksteps, bool may_pair) {
  TilePick best = {16, false};
  double best_cost = -1.0;
  for (int pair = 0; pair <= (may_pair ? 1 : 0); pair++) {
    const int step = pair ? PAIR_STEP : 16;
    for (int bn = step; bn <= 256; bn += step) {
      const long tiles = (long)((N + (pair ? 255 : 127)) / (pair ? 256 : 128)) * ((M + bn - 1) / bn), owners = pair ? sm_count / 2 : sm_count;
      const long waves = (tiles + owners - 1) / owners;
      const double fetch = (16384.0 + 128.0 * (pair ? bn / 2 : bn)) / 44.0, mma = 2.0 * bn;
      // (a pair's advantage counts by less than its bytes: it gains 8 % on the largest products, and loses 3 to 8 % on those of a few
      // microseconds, 301 -> 311 us for 1500 tokens at width 1024)
      const double cost = ((double)waves * (ksteps * (fetch > mma ? fetch : mma) + 1500.0) + 12.0 * bn) * (pair ? 1.3 : 1.0);
      if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = {bn, pair != 0}; }
    }
  }
  return best;
}

// gemm_q4k_tc2_kernel (gemm_q4k_tc.cu): column tiles of a grid row of 512 activation rows, the first `wide_tiles` of them `wide`
// columns, the others `narrow`: as many as fit the fewest waves of clusters that 256-wide tiles need.  Tiles of less than 128 columns
// are not taken (cols == 0).
struct PairColumns {
  int cols, wide_tiles, wide, narrow;
};
inline PairColumns pair_columns(int sm_count, int M, int N) {
  const int clusters = sm_count / 2, rows = (M + 511) / 512;
  if (N % PAIR_STEP || clusters < 1) return {0, 0, 0, 0};
  const int waves = (rows * ((N + 255) / 256) + clusters - 1) / clusters;
  int cols = waves * clusters / rows;
  if (cols > N / 96) cols = N / 96;
  if (cols < 1) return {0, 0, 0, 0};
  const int narrow = N / PAIR_STEP / cols * PAIR_STEP;
  if (narrow < 128) return {0, 0, 0, 0};
  return {cols, (N - cols * narrow) / PAIR_STEP, narrow + PAIR_STEP, narrow};  // cols * narrow + PAIR_STEP * wide_tiles == N, wide_tiles < cols
}
