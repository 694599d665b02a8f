// afl_sweep_plan.h -- how the one-sweep streaming CG (afl_cg_sweep.cu) splits a grid, and
// which grids it is the faster streaming form for.
#pragma once

#include <stddef.h>

#include "afl_launch.h"

namespace afl {

constexpr int kSweepRows = 16;  // tile rows, a warp each

struct SweepPlan {
  int tiles_x, tiles_y, chunks, depth;  // z chunks of `depth` planes
  __host__ __device__ int units() const { return tiles_x * tiles_y * chunks; }
};

// Plane steps of the longest CTA's march, `fill` more per unit than its planes.
inline long long sweep_steps(const SweepPlan &pl, int ctas, int fill) {
  const long long units = static_cast<long long>(pl.tiles_x) * pl.tiles_y * pl.chunks;
  return (units + ctas - 1) / ctas * (pl.depth + fill);
}

// Tiles 128 cells wide (4 per thread) unless the last one would be mostly empty (us per
// iteration, tiles of 32 -> of 128: FP64 256 x 256 x 256 177 -> 153, 320 x 256 x 200
// 173 -> 161, 220^3 110 -> 112; 200 x 300 x 300 207 -> 216, 192 x 300 x 300 173 -> 207).
inline bool sweep_wide(const Dims &g) { return (g.nx + 127) / 128 * 128 <= 1.27 * g.nx; }

// z chunks: the fewest that make the longest CTA's march shortest, each with its fill
// (320 x 256 x 200 in tiles of 32: 160 tiles on 296 CTAs leave half the chip idle in one
// chunk).
inline SweepPlan sweep_plan(const Dims &g, int nc, int ctas) {
  SweepPlan pl{}, best{};
  pl.tiles_x = (g.nx + 32 * nc - 1) / (32 * nc);
  pl.tiles_y = (g.ny + kSweepRows - 1) / kSweepRows;
  for (int chunks = 1; chunks <= (g.nz + 15) / 16; ++chunks) {
    pl.depth = (g.nz + chunks - 1) / chunks;
    pl.chunks = (g.nz + pl.depth - 1) / pl.depth;
    if (chunks == 1 || sweep_steps(pl, ctas, 6) < sweep_steps(best, ctas, 6)) best = pl;
  }
  return best;
}

// Rows and planes of the TMA boxes must be 16-byte aligned, and the sweep pays once
// the vectors leave L2 (us per iteration, two passes -> sweep): FP64 160^3 57 -> 51,
// 192 x 160 x 176 73 -> 66, 150 x 300 x 300 193 -> 146, 220^3 136 -> 112, 256^3 208 -> 153;
// mixed 220^3 79 -> 70, 256 x 200 x 256 86 -> 73, 256^3 108 -> 87.  Below that the two
// passes run from L2 and the sweep's chain per plane shows: FP64 64^3 15 -> 28,
// 136 x 140 x 144 41 -> 40; mixed 192^3 50 -> 52, 160^3 33 -> 45.  f32 rows are half as
// long in bytes: only full tiles pay (192 x 300 x 300 112 -> 120).
inline bool sweep_fits(const Dims &g, bool f64, size_t l2_bytes) {
  if (g.n > (1 << 30)) return false;  // cell indices stay clear of 2^31
  // r, q, d twice and the solution; f32 once four of them do
  const size_t bytes = (f64 ? 5 * sizeof(double) : 4 * sizeof(float)) * static_cast<size_t>(g.n);
  return g.nx % (f64 ? 2 : 4) == 0 && bytes > l2_bytes && (f64 || sweep_wide(g));
}

// A plane step takes a CTA about as long whether its tile is full or not, so the sweep
// loses where much of its tiles lies outside the grid or much of the chip is idle.  It pays
// from a share of live cells in all CTAs' plane steps (the two fill planes of a unit
// counted) of 0.60 in FP64, 0.72 in tiles of 32, 0.66 in f32.  us per iteration, share, two
// passes -> sweep; FP64: 512 x 34 x 400 0.63 96 -> 94, 1000 x 1000 x 8 0.66 109 -> 107,
// 250 x 300 x 60 0.67 71 -> 63, but 324 x 566 x 41 0.58 107 -> 121, 512 x 18 x 600 0.51
// 79 -> 92, 7100 x 6 x 531 0.34 265 -> 414; in tiles of 32: 30 x 31792 x 9 0.73 132 -> 127,
// 160 x 160 x 161 0.78 62 -> 59, 96 x 250 x 300 0.92 101 -> 85, but 136 x 136 x 400 0.71
// 104 -> 107, 34 x 500 x 500 0.46 132 -> 168, 6 x 1200 x 1200 0.17 133 -> 450; f32:
// 108 x 69 x 1876 0.68 131 -> 126, 220^3 0.74 96 -> 89, 256 x 200 x 256 as above, but
// 512 x 34 x 800 0.63 111 -> 118, 256 x 17 x 3000 0.50 103 -> 129.
inline bool sweep_pays(const Dims &g, const SweepPlan &pl, int nc, int ctas, bool f64) {
  const double slots =
      double(ctas) * (32 * nc * kSweepRows) * double(sweep_steps(pl, ctas, 2));
  return g.n >= (f64 ? nc == 4 ? 0.60 : 0.72 : 0.66) * slots;
}

}  // namespace afl
