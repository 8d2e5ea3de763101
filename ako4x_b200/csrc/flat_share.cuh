// Work split of the decode attention kernels: the key tiles of all rows (sequences, query tokens) form
// one flat sequence and every CTA takes an equal contiguous share of it (+-1 tile whatever the mix of
// row lengths), which it cuts at row boundaries into segments. A row inside one share is finished by
// its CTA; the segments of a longer row leave one partial each for a merge kernel.
#pragma once
#include "common.cuh"

namespace ako {

struct Share {
  int row;    // row of the first tile
  int skip;   // tiles of that row in front of the share
  int left;   // tiles of the share
  int per;    // tiles of a full share
};

// Finds share `index` of `shares` with 128 threads; `tiles(r)` is the tile count of row r < nrows and
// `empty(r)` is called (by one thread) for the share's part of the rows that have none. s_scan: six ints of
// shared memory.
template <class Tiles, class Empty>
__device__ __forceinline__ Share find_share(int nrows, int index, int shares, int* s_scan, Tiles tiles, Empty empty) {
  constexpr int NT = 128;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  Share sh = {0, 0, 0, 1};
  int first = 0, mine = 0;                          // `first`: the thread's row of the first 128
  for (int r = tid; r < nrows; r += NT) {
    const int n = tiles(r);
    if (r == tid) first = n;
    if (n == 0 && r % shares == index) empty(r);
    mine += n;
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, off);
  if (lane == 0) s_scan[w] = mine;
  if (tid == 0) s_scan[4] = -1;
  __syncthreads();
  const int total = s_scan[0] + s_scan[1] + s_scan[2] + s_scan[3];
  const int per = (total + shares - 1) / shares;
  const int begin = index * per;
  if (begin >= total) return sh;
  int base = 0;
  for (int r0 = 0; r0 < nrows; r0 += NT) {
    const int r = r0 + tid;
    const int n = (r0 == 0) ? first : (r < nrows) ? tiles(r) : 0;
    int x = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += up;
    }
    __syncthreads();
    if (lane == 31) s_scan[w] = x;
    __syncthreads();
    x += base;
    for (int i = 0; i < w; ++i) x += s_scan[i];     // inclusive prefix
    if (x - n <= begin && begin < x) {
      s_scan[4] = r;
      s_scan[5] = begin - (x - n);
    }
    base += s_scan[0] + s_scan[1] + s_scan[2] + s_scan[3];
    __syncthreads();
    if (s_scan[4] >= 0) break;
  }
  sh.row = s_scan[4];
  sh.skip = s_scan[5];
  sh.left = min(per, total - begin);
  sh.per = per;
  return sh;
}

}  // namespace ako
