// Work plan of the dense GEMM (host code without CUDA, so that it can be tested on its own).
#pragma once
#include <cstddef>
#include <cstdint>

namespace ako_gemm {

constexpr int kTileRows = 128;

struct Plan {
  int bn, splits, cg;   // tile width, pieces of K, CTAs per tile
};

// Tile width, CTAs per tile and K split by how many work items the GPU gets. A K block of 64 costs a
// CTA about the same time whatever its tile is (it waits for operands, not for the tensor pipe), so
// the plan looks for the widest tiles that still give every SM work: pairs (256 rows) from the second
// row tile on, 256 columns once 128 would need a second wave, K cut into 2, 4 or 8 pieces (summed by
// a second kernel) while less than half of the GPU has work. One-CTA tiles stay for up to 128 rows
// (a pair would be half empty) and where they fit one wave and pairs of the same width do not.
// Measured, whole call, N = 2048, K = 4096, against one-CTA tiles everywhere (us): M = 256: 15.6
// (20.0), 512: 18.5 (20.0), 640: 23.5 (29.2), 969: 22.6 (26.0), 1536: 28.8 (44.5), 4000: 52.3 (57.7),
// 16294: 182 (204); M = 640 as 256 x 128 pairs with K in two, 96 of them for 74 places: 26.7.
// `pairs` false: without CTA pairs.
inline Plan plan(int64_t m, int64_t n, int64_t k, bool have_workspace, int sms, bool pairs) {
  const int64_t mt = (m + kTileRows - 1) / kTileRows, mp = (mt + 1) / 2;
  if (pairs && mt > 1) {
    // more 256 x 128 tiles than one wave of pairs
    if (2 * mp * (n / 128) > sms) {
      if (mt * (n / 128) <= sms) return {128, 1, 1};
      return {256, 1, 2};
    }
    int s = 1;
    while (have_workspace && s < 8 && 4 * mp * (n / 128) * s <= sms && (k / 64) % (2 * s) == 0) s *= 2;
    if (s > 1) return {128, s, 2};
    // between a quarter and a half of the GPU with full-width tiles: those, K in two
    if (have_workspace && 4 * mp * (n / 256) * 3 <= 2 * sms && (k / 64) % 2 == 0) return {256, 2, 2};
    if (4 * mp * (n / 128) >= sms) return {128, 1, 2};
  }
  if (mt * (n / 256) * 4 >= 3 * sms) return {256, 1, 1};
  if (!have_workspace) return {(mt * (n / 128) * 4 >= 3 * sms) ? 128 : 32, 1, 1};
  int s = 1;
  while (s < 8 && mt * (n / 128) * s < 128 && (k / 64) % (2 * s) == 0) s *= 2;
  return {128, s, 1};
}

inline size_t workspace_bytes(const Plan& pl, int64_t m, int64_t n) {
  return pl.splits > 1 ? (size_t)pl.splits * (size_t)m * (size_t)n * sizeof(float) : 0;
}

// The plan of a call: false if its workspace is too small. `pair_ctas(bn)` tells how many CTAs of the pair
// kernel can be resident; where none can (a partition of the GPU without a free pair of SMs), one-CTA
// tiles, with whatever K split the workspace holds.
template <class PairCtas>
inline bool choose(int64_t m, int64_t n, int64_t k, bool have_workspace, size_t bytes, int sms, PairCtas pair_ctas, Plan& pl) {
  pl = plan(m, n, k, have_workspace, sms, true);
  if (workspace_bytes(pl, m, n) > bytes) return false;
  if (pl.cg == 2 && pair_ctas(pl.bn) < 2) {
    pl = plan(m, n, k, have_workspace, sms, false);
    if (workspace_bytes(pl, m, n) > bytes) pl = plan(m, n, k, false, sms, false);
  }
  return true;
}

}  // namespace ako_gemm
