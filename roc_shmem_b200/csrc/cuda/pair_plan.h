// pair_plan.h — how wide the tiles of a CTA-pair GEMM (gemm_pair.cuh) are.  Plain C++.
#pragma once

namespace bshmem {
namespace gemm2 {

// Columns of a tile's one accumulator, or of its two (wide form; see gemm_pair.cuh).  What a launch costs is the number of waves
// times the width of a tile, as long as the tensor cores are the bound: 1000 x 7168 x 8192 takes 108 us as two waves of 256 columns
// (112 tiles on 74 pairs), 98 as one of 448 and 95 as one of 416.  Beside that
//  - a tile of one accumulator reads its A rows for half as many columns.  Per k-block it takes as long as (256 + width) / 2
//    columns of a wide one (1000 x 7168 x 8192 by 224 columns: 107 us, also two waves), and under the power cap, where an SM's
//    loads cost clock, 10 % more at the same number of columns (8192 x 8192 x 3584: 367 us, 350 by 512 columns; 8192 x 7168 x 8192:
//    765, and 710 by 448).  With a few k-blocks this turns round, because a wide tile fills and drains the ring more often
//    than it streams (7168 x 8192, 848 deep: 89.7 and 93.7 us; 384 deep: 55.6 and 57.6; 4096 x 4096, 744 deep: 26.5 and 25.4);
//  - of an MN-major B two blocks of 64 columns per CTA and accumulator are loaded whatever the width; what lies beyond it counts half;
//  - the rows of A are a share of a wide tile's loads too, about 26 columns' worth;
//  - a wave has a beginning and an end, worth about 8 columns.
// Without `exact`, row_blocks is an estimate: two accumulators have to be the better choice both where a launch loses half a wave, as
// with unequal groups, and by whole waves, as with equal ones.  Sustained, by 256 and by 512 columns: 16 groups of 1125 rows, 1024
// columns, 2048 deep (better by the first, 2.16 waves paid as three) 83.3 and 88.7 us, 1629 rows 113.5 and 118.0; 8 groups of 1931 rows,
// 2048 columns, 4096 deep 220 and 230; of 750 rows (worse by both) 97 and 109; of 2250 rows (better by both) 248 and 241, 8192 deep 494 and 468.
// `wide_delay`: cycles that a tile's epilogue keeps the tensor cores waiting in the wide form (two per column and k-block).
// `pairs`: that work at the same time; with none (nothing can be launched) as with one.
// `step`: what an accumulator's columns are a multiple of, 32 or, where the epilogue wants more, 64 or 128.
// `narrowest_wide`: the least columns of a tile of two accumulators.
struct Width {
  int cols[2];
  double cost = 0;      // of the launch by whole waves, what an MN-major B adds left out
};
inline Width plan_width(long long row_blocks, int N, int K, int pairs, int step, bool b_mn, bool exact = true, int widest = 512,
                        int wide_delay = 0, int narrowest_wide = 352) {
  constexpr int BN = 256;
  if (pairs < 1) pairs = 1;
  const double blocks = (K + 63) / 64, narrow = 0.91 + blocks / 160 < 1.1 ? 0.91 + blocks / 160 : 1.1;
  struct { double cost, whole; Width w; } best[2] = {{1e30, 1e30, {{BN, 0}}}, {1e30, 1e30, {{BN, 0}}}};      // of one accumulator, of two
  for (int w = widest; w >= 128; w -= step) {
    if (w > BN && w < narrowest_wide) continue;
    const int c0 = w > BN ? (w + 2 * step - 1) / (2 * step) * step : w, c1 = w - c0;
    const int loaded = !b_mn ? w : c1 ? 2 * BN : BN;
    const long long tiles = row_blocks * ((N + w - 1) / w);
    const double per_wave = (c1 ? 26 + 0.95 * 0.5 * (w + loaded) + wide_delay / (2 * blocks) : narrow * 0.5 * (BN + loaded)) + 8;
    const long long waves = (tiles + pairs - 1) / pairs;
    const double whole = (double)waves * per_wave;
    const double cost = exact ? whole : (tiles > pairs / 2 ? 0.5 + (double)tiles / pairs : 1.0) * per_wave;
    auto& b = best[c1 ? 1 : 0];
    if (cost < b.cost) b = {cost, whole, {{c0, c1}, (double)waves * ((c1 ? 26 + 0.95 * w : narrow * 0.5 * (BN + w)) + 8)}};
  }
  return best[1].cost <= best[0].cost && best[1].whole <= best[0].whole ? best[1].w : best[0].w;
}

// Rows of a group whose count is on the device, as far as the host knows: about `about`, as the caller says, else four fifths of its
// capacity, the share that a layer with the usual capacity factor of 1.25 fills.  A layer built for 16384 tokens that gets 1717 (16
// experts of 2048, hidden 1024, two per token: 215 rows for a capacity of 2560) was planned as eight full row blocks per expert
// and took 85.3 us, 78.4 by the widths for one.
inline int group_rows(int capacity, int about) {
  return about > 0 ? (about < capacity ? about : capacity) : (int)((capacity * 4LL + 4) / 5);
}

}  // namespace gemm2
}  // namespace bshmem
