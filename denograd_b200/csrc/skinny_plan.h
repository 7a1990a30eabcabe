// How a projection of a few rows (skinny.cuh) is laid out on the GPU: plain C++, so that it can be walked over all shapes without one.
#pragma once

enum { SK_F16 = 0, SK_BF16 = 1, SK_W8 = 2, SK_NF4 = 3 };

constexpr int SK_WARPS = 16, SK_MAX_STAGES = 12, SK_SMEM = 200 * 1024;
constexpr int SK_TABLE = 256 * 32 * 4;  // NF4: byte -> two codes, a copy per lane
constexpr int sk_align(int n, int to) { return (n + to - 1) / to * to; }
constexpr int sk_runs_x(int type) { return type == SK_NF4 ? 4 : type == SK_W8 ? 2 : 1; }  // 128-byte runs of activations to one of weights
constexpr int sk_units(int type, int nt) { return type == SK_F16 || type == SK_BF16 || (type == SK_W8 && nt > 1) ? 1 : 2; }  // runs of a stage that a warp has offsets for
constexpr int sk_part(int nt, int tp) { return SK_WARPS * tp * nt * 4 * 32 * 4; }         // bytes of the warps' sums
// before the ring: the sums, or the table on a multiple of its size behind them
constexpr int sk_head(int type, int nt, int tp) { return type == SK_NF4 ? 2 * SK_TABLE : sk_part(nt, tp) + 1024; }

// K slices of an int8 projection of up to 16 rows (gemm_small.cu), and the tile of K that they share: slice q has
// [tile * kt + q * kt / slices, .. + kt / slices) of every tile, one after the other, and the slices' sums are added in order.
// No more slices than it takes to have a CTA and a quarter per SM there, so that the launch stays one round of two CTAs per SM and fewer
// CTAs fetch the same activations (8B shapes, 8 rows, us with 2 / 4 / 8 slices: gate and up 25.6 / 29.8 / 31.3, qkv 13.1 / 9.0 / 11.4,
// wo 12.8 / 9.2 / 8.0, down 39 / 27 / 20).
inline int w8_slices(int N, int K, int sm_count) {
  if (K < 8 * 256) return 1;
  const long long tiles = (N + 15) / 16;
  for (int ks = 1, per = 8; ks < 8; ks *= 2, per /= 2)
    if ((tiles + per - 1) / per * 4 >= 5ll * sm_count) return ks;
  return 8;
}
// Activation k tile (halves) of gemm_small.cu.  A lane holds the weights of one k tile at a time, and K slices divide the tile among the
// warps: with int8 weights and 512 halves, eight slices leave a lane 32 bytes in flight, 2 MB on the whole GPU, and the kernel waits
// for memory at 1.4 to 2 TB/s (8B shapes, 8 rows).  So many slices take longer tiles, as far as two CTAs' activations fit an SM.
constexpr int gs_k_tile(int max_rows, int slices, bool w8) { return !w8 || slices < 4 || max_rows > 16 ? 512 : max_rows <= 8 ? 2048 : 1024; }

struct SkPlan {
  bool ok;
  int grid, tr, tiles, tp;  // CTAs; outputs of a pass, 16-row tiles of it, tiles of a warp
  int ks, units, runs, sp;  // warps that share a tile along K, runs of a warp in a stage, runs of a stage; NF4: bytes of a row's scales in a stage
  int slice;                // W8: runs of weights that a warp's slice has one after the other
  int pieces;               // stages to a pass
  int stages, stage_bytes, smem;
};
inline SkPlan sk_plan(int type, bool glu, int M, int N, int K, int block_shift, int sm_count) {
  SkPlan p = {};
  const int nt = M <= 8 ? 1 : 2, to = glu ? 8 : 16, nw = glu ? 2 : 1;  // outputs of a 16-row tile, matrices
  const int row_bytes = type == SK_NF4 ? K / 2 : type == SK_W8 ? K : K * 2;
  p.grid = N < sm_count ? N : sm_count;
  const int per = (N + p.grid - 1) / p.grid;
  auto rows = [&](int passes) {
    p.tr = (per + passes - 1) / passes;
    p.tiles = (p.tr + to - 1) / to;
  };
  auto stage = [&](int runs) {
    const int head = sk_head(type, nt, p.tp) + 4096;  // fragments of a tile may reach up to 31 rows past the ring
    p.runs = runs;
    p.stage_bytes = sk_align(nw * sk_align(runs * p.tr * 128, 1024) + sk_align(runs * sk_runs_x(type) * M * 128, 1024) + nw * sk_align(p.tr * p.sp, 128), 1024);
    p.stages = (SK_SMEM - head) / p.stage_bytes;
    if (p.stages > SK_MAX_STAGES) p.stages = SK_MAX_STAGES;
    p.smem = head + p.stages * p.stage_bytes;
    p.pieces = (row_bytes / 128 + runs - 1) / runs;
  };
  if (row_bytes % 128 != 0) return p;
  if (type == SK_W8) {
    // Every sum is added in gemm_small.cu's order, to the bit: its slices, each of them one warp's.  A pass has as many outputs as the
    // slices leave warps for, and fewer where less than three stages would fit, two beyond 8 rows (8B step, ms with two / three: 8 rows
    // 2.30 / 2.27, 16 rows 2.88 / 2.99).
    const int deep = nt == 1 ? 3 : 2;
    p.ks = w8_slices(N, K, sm_count);
    const int width = p.ks == 1 ? K : gs_k_tile(nt * 8, p.ks, true) / p.ks;
    if (K % width != 0) return p;
    p.slice = width / 128;
    for (int passes = 1;; passes++) {
      rows(passes);
      p.tp = p.tiles * p.ks <= SK_WARPS ? 1 : 2;
      if (p.tiles > 16 || (p.tiles + p.tp - 1) / p.tp * p.ks > SK_WARPS) continue;
      for (p.units = p.slice % 2 == 0 ? sk_units(type, nt) : 1;; p.units--) {
        stage(p.ks * p.units);
        if (p.stages >= deep || p.units == 1) break;
      }
      if (p.stages >= deep || p.tr == 1) break;
    }
    if (p.ks > 1) p.pieces = (K / width + p.ks - 1) / p.ks * (p.slice / p.units);
    p.ok = p.stages >= 2;
    return p;
  }
  rows((per + 16 * to - 1) / (16 * to));
  p.tp = p.tiles <= 8 ? 1 : 2;  // more than 8 tiles: two to a warp, which share its activations' fragments
  const int warps = (p.tiles + p.tp - 1) / p.tp;
  p.ks = 1;
  while (warps * p.ks * 2 <= SK_WARPS && p.ks * 128 < row_bytes) p.ks *= 2;
  for (;; p.ks /= 2) {
    p.units = 1;
    if (type == SK_NF4) {  // at least 16 bytes of scales to a row and stage
      const int run = 512 >> block_shift;
      while (p.ks * p.units * run < 16) p.units *= 2;
      p.sp = p.ks * p.units * run;
    }
    stage(p.ks * p.units);
    if (p.stages >= 3 || p.ks == 1) break;
  }
  p.ok = p.units <= sk_units(type, nt) && p.stages >= 2;  // blocks of 128 and 256 may ask for more runs to a stage, and for more memory
  return p;
}
