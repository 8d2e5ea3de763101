// Work plan of the dense GEMM (host code without CUDA, so that it can be tested on its own).
#pragma once
#include <cstddef>
#include <cstdint>

namespace ako_gemm {

constexpr int kTileRows = 128;

struct Plan {
  int bn, splits, cg;   // tile width, pieces of K, CTAs per tile
};

// Tile width, CTAs per tile (a pair computes 256 rows) and pieces of K: the candidate with the least estimated
// time. The estimate, in us, is of a call whose workers (CTAs or pairs) each run `per` tiles one after another:
//   first tile   start + blocks x block      (K blocks of 64; a block costs a CTA about the same time
//                                             whatever its tile is: it waits for operands)
//   others       the larger of blocks x steady + overlap and store (the epilogue alone)
//   K in pieces  1.6 + partial sums at 3.2 TB/s, 1 more with 256 columns, for the kernel that adds them up
// Measured, single tiles per worker, estimate in brackets: 128 columns, one CTA: 64 blocks 26.6 (26.6), 32 15.5
// (15.5), 16 10.0 (10.0), 8 7.4 (7.2), 1 4.9 (4.7); a pair: 64 21.2 (21.2), 32 13.4 (13.4), 16 9.5 (9.5), 8 7.5
// (7.6), 1 5.8 (5.8); 256 columns, one CTA: 64 28.8 (28.7), 16 12.0 (11.7), 1 6.3 (6.4); a pair: 64 25.4 (25.4),
// 32 16.3 (16.4), 16 11.6 (11.8), 1 7.2 (7.6). Several: 8192 x 2048 x 4096 on pairs 98 (98), x 512 21.8 (21.4), x 64
// 16.6 (16.9) against 14.5 (14.4) with 128 columns. So pairs win from about 16 blocks per tile on and one CTA
// below; a wave that pairs miss by a little (1100 x 4096 x 4096: 44.3 for 80 pairs, 30.1 for 144 single CTAs),
// and pieces too short for the second kernel, cost what they do.
// Whole call, N = 2048, K = 4096, against one-CTA tiles with lane-number branches everywhere: M = 256: 13.1 (13.3),
// 512: 17.4 (18.0), 640: 20.4 (28.1), 969: 21.3 (25.4), 1536: 26.0 (44.0), 4096: 48.4 (51.0), 8192: 98 (106).
struct Config {
  int bn, cg;
  float start, block, steady, overlap, store;
};
constexpr Config kConfigs[] = {
    {128, 1, 4.4f, 0.347f, 0.290f, 0.7f, 1.6f},
    {128, 2, 5.6f, 0.244f, 0.227f, 0.8f, 1.6f},
    {256, 1, 6.0f, 0.355f, 0.380f, 1.8f, 3.1f},
    {256, 2, 7.3f, 0.283f, 0.360f, 1.0f, 3.1f},
};

inline float estimate(const Config& c, int splits, int64_t m, int64_t n, int64_t k, int sms) {
  const int64_t rows = c.cg * kTileRows;
  const int64_t tiles = (m + rows - 1) / rows * (n / c.bn) * splits, workers = sms / c.cg;
  const int64_t per = (tiles + workers - 1) / workers;
  const float blocks = (float)(k / 64 / splits), more = blocks * c.steady + c.overlap;
  float us = c.start + blocks * c.block + (float)(per - 1) * (more > c.store ? more : c.store);
  if (splits > 1) us += 1.6f + (c.bn == 256 ? 1.f : 0.f) + (float)splits * (float)m * (float)n * 4.f / 3.2e6f;
  return us;
}

// `pairs` false: without CTA pairs. Up to 128 rows a pair would be half empty; without a workspace, 32-column
// tiles give such calls more CTAs.
inline Plan plan(int64_t m, int64_t n, int64_t k, bool have_workspace, int sms, bool pairs) {
  const bool one_row = m <= kTileRows;
  if (one_row && !have_workspace && n / 128 * 4 < 3 * sms) return {32, 1, 1};
  Plan best = {128, 1, 1};
  float least = estimate(kConfigs[0], 1, m, n, k, sms);
  for (const Config& c : kConfigs) {
    if (c.cg == 2 && (!pairs || one_row)) continue;
    for (int s = 1; s <= (have_workspace ? 8 : 1) && k / 64 % s == 0; s *= 2) {
      if (s > 1 && c.bn == 256 && c.cg == 1) break;   // not built
      const float us = estimate(c, s, m, n, k, sms);
      if (us < least) {
        least = us;
        best = {c.bn, s, c.cg};
      }
    }
  }
  return best;
}

inline size_t workspace_bytes(const Plan& pl, int64_t m, int64_t n) {
  return pl.splits > 1 ? (size_t)pl.splits * (size_t)m * (size_t)n * sizeof(float) : 0;
}
// The workspace a caller is told to bring, and refused below: enough for the plan, and not less than what
// callers were told while K was always split until there were 128 items of 128 columns.
inline size_t workspace_bytes(int64_t m, int64_t n, int64_t k, int sms) {
  const size_t need = workspace_bytes(plan(m, n, k, true, sms, true), m, n);
  const int64_t mt = (m + kTileRows - 1) / kTileRows;
  if (mt * (n / 256) * 4 >= 3 * sms) return need;
  int s = 1;
  while (s < 8 && mt * (n / 128) * s < 128 && (k / 64) % (2 * s) == 0) s *= 2;
  const size_t told = workspace_bytes(Plan{128, s, 1}, m, n);
  return need > told ? need : told;
}

// The plan of a call: false if its workspace is too small. `pair_ctas(bn)` tells how many CTAs of the pair
// kernel can be resident; where none can (a partition of the GPU without a free pair of SMs), one-CTA
// tiles, with whatever K split the workspace holds.
template <class PairCtas>
inline bool choose(int64_t m, int64_t n, int64_t k, bool have_workspace, size_t bytes, int sms, PairCtas pair_ctas, Plan& pl) {
  if (have_workspace && bytes < workspace_bytes(m, n, k, sms)) return false;
  pl = plan(m, n, k, have_workspace, sms, true);
  if (pl.cg == 2 && pair_ctas(pl.bn) < 2) {
    pl = plan(m, n, k, have_workspace, sms, false);
    if (workspace_bytes(pl, m, n) > bytes) pl = plan(m, n, k, false, sms, false);
  }
  return true;
}

}  // namespace ako_gemm
