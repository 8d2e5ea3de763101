// Paged GQA decode: 32 query heads, 8 KV heads, head_dim 128, bf16.
//
// HBM-bound: every KV token costs 4096 bytes (8 heads x 128 x bf16 for K and again for V) and only 4
// query rows reuse it. With page size 1 a token is a random row of the cache, so the kernel is a gather:
// a copy-only probe on B200 reaches 6.4 TB/s with 16-byte register loads (64 contiguous bytes of a row
// per quad of lanes), against 5.4 TB/s with the 1 KB bulk copies that this kernel used before. So
// nothing is staged: a warp's loads ARE its mma operands, there is no barrier and no shared memory in
// the loop, and a dozen independent warps per SM keep the loads of 6 to 8 KB each in flight.
//   * A warp owns one KV head (a CTA: four neighbouring ones of the same tokens, 1 KB of a cache row).
//     Lane (g, t) loads the 16-byte pieces t + 4 j of K of tokens g and g + 8: the A fragments of
//     m16n8k16 with tokens as M, over a permuted order of the reduction in which Q's B fragments are
//     loaded too. S^T = K Q^T is [16 tokens x 8 heads], four of them real.
//   * V is loaded the same way; movmatrix turns an 8 x 8 block of pairs into the A fragment of
//     O^T = V^T P^T ([128 x 8 heads], features as M), and P's own pairs into the B fragment. P goes in as two
//     bf16 pieces (16 bits): in one, its rounding showed in the output (2.2e-3 of an fp64 result at 64 sequences
//     of up to 8 192 tokens, and more the longer a share is; now 1.67e-3, which is the bf16 output's own
//     rounding) for 8 of 24 mma a tile, hidden behind the loads (0 to 0.3 us a call).
//   * K of the next tile is requested when S has been computed, V of it when O has.
//
// Work split: flat_share.cuh, tiles of 16 tokens, one share per pair of CTAs (the two halves of the KV
// heads); a second kernel merges the partials of rows that several shares touch. Measured (whole call,
// bulk copies through shared memory and a planning kernel before -> now): 64 sequences of up to 8 192 tokens
// 245 -> 188 us (6.3 TB/s = 0.96 of the measured copy bandwidth), 256 of them 841 -> 680 (0.99), 16 of up to
// 1 200 25 -> 17, one of 547 12.6 -> 10.2 us. Shares also for batches of short sequences, where one CTA pair
// per sequence needs no merge: equal sequences lose a few us (222 x 64 tokens 13.5 -> 16.4, 888 x 100 67.4 ->
// 71.3, 3 000 x 30 79 -> 94), but one long sequence among them no longer keeps a single pair busy (eight of
// 8 192 tokens among 248 of 256: 580 -> 94; one of 60 000 among 229 of 100: 4 074 -> 78).
#include <algorithm>
#include <cfloat>

#include "flat_share.cuh"

namespace {

constexpr int HQ = 32, HKV = 8, D = 128, GROUP = HQ / HKV;
constexpr int HPC = 4;                    // KV heads per CTA, one per warp
constexpr int HALVES = HKV / HPC;         // CTAs per share
constexpr int TILE = 16;                  // tokens per tile
constexpr int THREADS = HPC * 32;
constexpr int CTAS_PER_SM = 3;
constexpr int ROW_BYTES = HKV * D * 2;    // one token of K (or V)

struct Params {
  const __nv_bfloat16* q;
  const unsigned char* k;
  const unsigned char* v;
  const int32_t* indptr;
  const int32_t* indices;
  __nv_bfloat16* o;
  float* lse;
  float* part_acc;  // [slot][32][128]
  float* part_ml;   // [slot][32][2]
  int2* cut;        // sequences that several shares touch: see below
  float scale_log2;
  int page_size;
  int batch;
  bool whole_rows;  // a share is one sequence
};

// For the merge the split kernel leaves entries {sequence, first share | shares << 16}; one share or none:
// nothing to merge. With no more sequences than shares there is one entry per sequence (written by the CTA
// that starts it), otherwise one per share, for the sequence that starts in it and goes on: the merge has at
// most `shares` of them to look at, however many sequences there are. The partial of share c lies in slot
// sequence + c, or, with one entry per share, in slot 2 c, the first one of a sequence in 2 c + 1.
__device__ __forceinline__ int2 cut_entry(int b, int first, int n) { return make_int2(b, first | n << 16); }

__device__ __forceinline__ void empty_head(const Params& p, int64_t row_head) {   // one thread
  uint4* op = reinterpret_cast<uint4*>(p.o + row_head * D);
  for (int i = 0; i < D / 8; ++i) op[i] = make_uint4(0u, 0u, 0u, 0u);
  p.lse[row_head] = -INFINITY;
}
__device__ __forceinline__ int seq_tokens(const Params& p, int b) {
  return max(0, p.indptr[b + 1] - p.indptr[b]) * p.page_size;
}
__device__ __forceinline__ uint4 ld_row16(const unsigned char* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

__global__ void __launch_bounds__(THREADS, CTAS_PER_SM) gqa_decode_kernel(Params p) {
  __shared__ int s_scan[6];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int half = blockIdx.x % HALVES, share = blockIdx.x / HALVES;
  const int kvh = half * HPC + warp;
  ako::pdl_trigger();  // the merge kernel may be scheduled early; it waits for this grid to finish
  auto seq_tiles = [&](int b) { return (seq_tokens(p, b) + TILE - 1) / TILE; };
  const int shares = gridDim.x / HALVES;
  const bool by_share = p.batch > shares;
  const bool keeper = half == 0 && threadIdx.x == 0;   // writes the entries
  ako::Share sh;
  if (p.whole_rows) {
    sh = {share, 0, seq_tiles(share), 0};
    if (sh.left == 0 && lane < GROUP) empty_head(p, (int64_t)share * HQ + kvh * GROUP + lane);
  } else {
    sh = ako::find_share(p.batch, share, shares, s_scan, seq_tiles, [&](int r) {
      for (int h = 0; h < HQ / HALVES; ++h) empty_head(p, (int64_t)r * HQ + half * (HQ / HALVES) + h);
      if (!by_share && half == 0) p.cut[r] = cut_entry(r, 0, 0);
    });
  }
  int2 cut = cut_entry(0, 0, 0);

  int b = sh.row, ts = sh.skip;
  while (sh.left > 0) {
    const int32_t* idx = p.indices + p.indptr[b];
    const int len = seq_tokens(p, b);
    const int tiles = (len + TILE - 1) / TILE;
    const int te = min(tiles, ts + sh.left);
    if (te <= ts) {                                  // an empty sequence
      ++b;
      ts = 0;
      continue;
    }
    sh.left -= te - ts;

    // this lane's two tokens of a tile: byte offset of its pieces in the caches
    int32_t id[2];
    auto fetch_ids = [&](int tile) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int tok = min(tile * TILE + 8 * i + g, len - 1);   // past the end: a valid row, masked below
        id[i] = __ldg(idx + (p.page_size == 1 ? tok : tok / p.page_size));
      }
    };
    int64_t off[2];
    auto locate = [&](int tile) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        int64_t row = id[i];
        if (p.page_size != 1) row = row * p.page_size + min(tile * TILE + 8 * i + g, len - 1) % p.page_size;
        off[i] = row * ROW_BYTES + kvh * (D * 2) + t * 16;
      }
    };
    uint4 kc[2][4], vc[2][4];
    auto load = [&](uint4 (&x)[2][4], const unsigned char* base) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) x[i][j] = ld_row16(base + off[i] + 64 * j);
    };
    // Q of the four heads as B fragments (n = head g, heads 4-7 are zero), in the order of the K pieces
    uint4 qb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      qb[j] = make_uint4(0u, 0u, 0u, 0u);
      if (g < GROUP)
        qb[j] = __ldg(reinterpret_cast<const uint4*>(p.q + ((int64_t)b * HQ + kvh * GROUP + g) * D + 32 * j + 8 * t));
    }
    // P goes in as two pieces, and once more as one where an output came out NaN or infinite: an infinite value
    // must not meet a piece of zero or of the other sign.
    bool two = true;
    float acc[4][2][4];   // [block j][u]: features 32 j + 8 (g / 2) + (g & 1) + 4 u (regs 0, 1) and + 2 (2, 3), heads 2t, 2t+1
    // heads 2t, 2t+1; l over this lane's tokens. The maxima start at the lowest finite value, so that a score
    // of -inf weighs 0 whatever else a tile or a share holds.
    float m0, m1, l0, l1;
    while (true) {
      fetch_ids(ts);
      locate(ts);
      load(kc, p.k);
      load(vc, p.v);
      fetch_ids(ts + 1);
      m0 = m1 = -FLT_MAX;
      l0 = l1 = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[j][u][i] = 0.f;

      for (int tile = ts; tile < te; ++tile) {
        float s[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t a0[4] = {kc[0][j].x, kc[1][j].x, kc[0][j].y, kc[1][j].y};
          const uint32_t a1[4] = {kc[0][j].z, kc[1][j].z, kc[0][j].w, kc[1][j].w};
          ako::mma_bf16_16816(s, a0, qb[j].x, qb[j].y);
          ako::mma_bf16_16816(s2, a1, qb[j].z, qb[j].w);
        }
        const bool more = tile + 1 < te;
        if (more) {
          locate(tile + 1);
          load(kc, p.k);
        }
        // softmax over the tokens: rows g and g + 8 of this lane, 8 lanes apart by 4
        const bool v0 = tile * TILE + g < len, v1 = tile * TILE + 8 + g < len;
        s[0] = v0 ? (s[0] + s2[0]) * p.scale_log2 : -INFINITY;
        s[1] = v0 ? (s[1] + s2[1]) * p.scale_log2 : -INFINITY;
        s[2] = v1 ? (s[2] + s2[2]) * p.scale_log2 : -INFINITY;
        s[3] = v1 ? (s[3] + s2[3]) * p.scale_log2 : -INFINITY;
        float n0 = fmaxf(s[0], s[2]), n1 = fmaxf(s[1], s[3]);
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) {
          n0 = fmaxf(n0, __shfl_xor_sync(0xffffffffu, n0, o));
          n1 = fmaxf(n1, __shfl_xor_sync(0xffffffffu, n1, o));
        }
        if (__any_sync(0xffffffffu, n0 > m0 || n1 > m1)) {
          n0 = fmaxf(n0, m0);
          n1 = fmaxf(n1, m1);
          const float f0 = ako::fast_exp2(m0 - n0), f1 = ako::fast_exp2(m1 - n1);
          m0 = n0;
          m1 = n1;
          l0 *= f0;
          l1 *= f1;
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              acc[j][u][0] *= f0; acc[j][u][1] *= f1; acc[j][u][2] *= f0; acc[j][u][3] *= f1;
            }
        }
        s[0] = ako::fast_exp2(s[0] - m0);
        s[1] = ako::fast_exp2(s[1] - m1);
        s[2] = ako::fast_exp2(s[2] - m0);
        s[3] = ako::fast_exp2(s[3] - m1);
        l0 += s[0] + s[2];
        l1 += s[1] + s[3];
        if (tile * TILE + TILE > len) {   // past the end: weight 0, but the row read in their place may hold infinities
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (!v0) vc[0][j] = make_uint4(0u, 0u, 0u, 0u);
            if (!v1) vc[1][j] = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        const uint32_t h0 = ako::pack_bf16x2(s[0], s[1]), h1 = ako::pack_bf16x2(s[2], s[3]);
        const uint32_t b0 = ako::movmatrix_trans(h0), b1 = ako::movmatrix_trans(h1);
        // what the rounding of the weights left
        const uint32_t c0 = ako::movmatrix_trans(ako::pack_bf16x2(s[0] - ako::bf16_lo(h0), s[1] - ako::bf16_hi(h0)));
        const uint32_t c1 = ako::movmatrix_trans(ako::pack_bf16x2(s[2] - ako::bf16_lo(h1), s[3] - ako::bf16_hi(h1)));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t a0[4] = {ako::movmatrix_trans(vc[0][j].x), ako::movmatrix_trans(vc[0][j].y), ako::movmatrix_trans(vc[1][j].x), ako::movmatrix_trans(vc[1][j].y)};
          const uint32_t a1[4] = {ako::movmatrix_trans(vc[0][j].z), ako::movmatrix_trans(vc[0][j].w), ako::movmatrix_trans(vc[1][j].z), ako::movmatrix_trans(vc[1][j].w)};
          if (two) {
            ako::mma_bf16_16816(acc[j][0], a0, c0, c1);
            ako::mma_bf16_16816(acc[j][1], a1, c0, c1);
          }
          ako::mma_bf16_16816(acc[j][0], a0, b0, b1);
          ako::mma_bf16_16816(acc[j][1], a1, b0, b1);
        }
        if (more) {
          load(vc, p.v);
          fetch_ids(tile + 2);
        }
      }
      float z = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int i = 0; i < 4; ++i) z = fmaf(acc[j][u][i], 0.f, z);
      if (!two || !__any_sync(0xffffffffu, !(z == 0.f))) break;
      two = false;
    }

#pragma unroll
    for (int o = 4; o <= 16; o <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, o);
      l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    // lanes g = 2 x, 2 x + 1 hold the even and the odd of features 32 j + 8 x .. + 7: swap so that the
    // even lane has the first four and the odd lane the last four
    const bool whole = te - ts == tiles;
    const float i0 = (whole && l0 > 0.f) ? 1.f / l0 : 1.f, i1 = (whole && l1 > 0.f) ? 1.f / l1 : 1.f;
    const bool odd = g & 1;
    const int64_t slot = by_share ? 2 * (int64_t)share + (ts == 0) : (int64_t)b + share;
    if (ts == 0 && !p.whole_rows) {
      cut = cut_entry(b, share, whole ? 1 : 1 + (tiles - te + sh.per - 1) / sh.per);
      if (!by_share && keeper) p.cut[b] = cut;
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int head = kvh * GROUP + 2 * t + hh;
      const float inv = hh ? i1 : i0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = acc[j][0][hh] * inv, c = acc[j][0][2 + hh] * inv, e = acc[j][1][hh] * inv, f = acc[j][1][2 + hh] * inv;
        const float r0 = __shfl_xor_sync(0xffffffffu, odd ? a : e, 4), r1 = __shfl_xor_sync(0xffffffffu, odd ? c : f, 4);
        const float4 x = odd ? make_float4(r0, e, r1, f) : make_float4(a, r0, c, r1);
        if (t < 2) {
          const int col = 32 * j + 8 * (g >> 1) + 4 * (g & 1);
          if (whole)
            *reinterpret_cast<uint2*>(p.o + ((int64_t)b * HQ + head) * D + col) =
                make_uint2(ako::pack_bf16x2(x.x, x.y), ako::pack_bf16x2(x.z, x.w));
          else
            *reinterpret_cast<float4*>(p.part_acc + (slot * HQ + head) * D + col) = x;
        }
      }
      if (t < 2 && g == 0) {
        const float m = hh ? m1 : m0, l = hh ? l1 : l0;
        if (whole)
          p.lse[(int64_t)b * HQ + head] = (l > 0.f) ? m + log2f(l) : -INFINITY;
        else
          *reinterpret_cast<float2*>(p.part_ml + (slot * HQ + head) * 2) = make_float2(m, l);
      }
    }
    ++b;
    ts = 0;
  }
  if (by_share && !p.whole_rows && keeper) p.cut[share] = cut;
}

// Merge: WARPS warps per (sequence, head), every warp 32 threads x 4 columns of every WARPS-th partial;
// a block holds four heads (WARPS = 1) or one (WARPS = 8: few sequences with many partials each, where
// one warp would walk up to 222 partials in a row). Sequences inside one share, and empty ones, are already
// written.
constexpr int MERGE_MAX = 512;                       // shares of a call never exceed this (three CTAs per SM)
template <int WARPS>
__global__ void __launch_bounds__(WARPS == 1 ? 128 : WARPS * 32) gqa_merge_kernel(Params p, int shares) {
  constexpr int HEADS = (WARPS == 1) ? 4 : 1;
  __shared__ float s_w[HEADS][MERGE_MAX];
  __shared__ float4 s_acc[WARPS][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int hl = (WARPS == 1) ? w : 0, part = (WARPS == 1) ? 0 : w;
  const int head = (blockIdx.x % (HQ / HEADS)) * HEADS + hl;
  ako::pdl_wait();
  const int2 cut = p.cut[blockIdx.x / (HQ / HEADS)];
  const int c0 = cut.y & 0xffff, n = cut.y >> 16;
  if (n <= 1) return;
  const bool by_share = p.batch > shares;
  const int64_t oi = (int64_t)cut.x * HQ + head, slot0 = by_share ? 2 * (int64_t)c0 : (int64_t)cut.x + c0;
  auto slot = [&](int i) { return by_share ? 2 * i + (i == 0) : i; };
  uint2* op = reinterpret_cast<uint2*>(p.o + oi * D) + lane;
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + (slot0 * HQ + head);
  const float4* pa = reinterpret_cast<const float4*>(p.part_acc + (slot0 * HQ + head) * D) + lane;
  // every warp of the head finds the maximum over all partials for itself
  float2 mine[MERGE_MAX / 32];
  float M = -INFINITY, L = 0.f;
#pragma unroll
  for (int i = 0; i < MERGE_MAX / 32; ++i) {
    mine[i] = make_float2(-INFINITY, 0.f);
    if (i * 32 < n && i * 32 + lane < n) mine[i] = ml[(int64_t)slot(i * 32 + lane) * HQ];
    M = fmaxf(M, mine[i].x);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
  for (int i = 0; i < MERGE_MAX / 32; ++i)
    if (i * 32 < n) {
      const float wgt = exp2f(mine[i].x - M);
      if (part == 0 && i * 32 + lane < n) s_w[hl][i * 32 + lane] = wgt;
      L = fmaf(mine[i].y, wgt, L);
    }
  if (WARPS == 1) __syncwarp();
  else __syncthreads();
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int i = part; i < n; i += WARPS) {
    const float wgt = s_w[hl][i];
    const float4 x = pa[(int64_t)slot(i) * (HQ * D / 4)];
    acc.x = fmaf(x.x, wgt, acc.x);
    acc.y = fmaf(x.y, wgt, acc.y);
    acc.z = fmaf(x.z, wgt, acc.z);
    acc.w = fmaf(x.w, wgt, acc.w);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
  if (WARPS > 1) {
    s_acc[w][lane] = acc;
    __syncthreads();
    if (w != 0) return;
#pragma unroll
    for (int i = 1; i < WARPS; ++i) {
      const float4 x = s_acc[i][lane];
      acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
    }
  }
  const float inv = (L > 0.f) ? 1.f / L : 0.f;
  *op = make_uint2(ako::pack_bf16x2(acc.x * inv, acc.y * inv), ako::pack_bf16x2(acc.z * inv, acc.w * inv));
  if (lane == 0) p.lse[oi] = (L > 0.f) ? M + log2f(L) : -INFINITY;
}

// Calls that can do without a workspace, with whole sequences as shares: batches that fill the GPU and are
// short on average or many. A long sequence among them is then walked by one pair of CTAs.
bool whole_rows(int64_t batch, int64_t num_kv_indices, int64_t page_size) {
  const int64_t most = (int64_t)CTAS_PER_SM * ako::sm_count() / HALVES;
  return batch >= 4 * most || (batch >= most && num_kv_indices * page_size <= batch * 512);
}
// Shares of a call: all CTAs resident at once, and at least one tile (16 tokens, 64 KB of K and V) each.
int pick_shares(int64_t num_kv_indices, int64_t page_size) {
  const int64_t most = (int64_t)CTAS_PER_SM * ako::sm_count() / HALVES;
  const int64_t tiles = ako::cdiv(num_kv_indices * page_size, (int64_t)TILE);   // at least; rows round up
  int64_t s = tiles < most ? tiles : most;
  if (s > MERGE_MAX) s = MERGE_MAX;
  return (int)(s < 1 ? 1 : s);
}
struct Carve {
  size_t acc, ml, total;   // offsets; the entries are first
};
Carve carve(int64_t batch, int64_t num_kv_indices, int64_t page_size) {
  const int shares = pick_shares(num_kv_indices, page_size);
  const size_t entries = (size_t)(batch < shares ? batch : shares), slots = entries + (size_t)shares;
  Carve c;
  c.acc = (entries * sizeof(int2) + 255) / 256 * 256;
  c.ml = c.acc + slots * HQ * D * sizeof(float);
  // Callers that cannot do without were promised (and are refused below) a size of a slot for every sequence
  // and share, as if each sequence could be cut; at most `shares` can.
  const size_t promised = whole_rows(batch, num_kv_indices, page_size) ? slots : (size_t)batch + (size_t)shares;
  c.total = c.acc + promised * HQ * (D + 2) * sizeof(float);
  return c;
}

}  // namespace

extern "C" size_t ako4x_gqa_paged_decode_workspace_bytes(int64_t batch, int64_t num_kv_indices,
                                                         int64_t page_size) {
  if (batch <= 0) return 0;
  return carve(batch, num_kv_indices, page_size).total;
}

extern "C" int ako4x_gqa_paged_decode(const void* q, const void* k_cache, const void* v_cache,
                                      const int32_t* kv_indptr, const int32_t* kv_indices,
                                      float sm_scale, void* o, float* lse, int64_t batch,
                                      int64_t num_kv_indices, int64_t page_size, void* workspace,
                                      size_t workspace_bytes, void* stream) {
  if (batch < 0 || num_kv_indices < 0 || page_size < 1) return AKO4X_EINVAL;
  if (batch == 0) return AKO4X_OK;
  if (!q || !k_cache || !v_cache || !kv_indptr || !o || !lse) return AKO4X_EINVAL;
  if (num_kv_indices > 0 && !kv_indices) return AKO4X_EINVAL;
  if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)o) & 15) return AKO4X_EINVAL;
  if (batch > 0x7fffffffLL / HQ || page_size > 0x7fffffffLL) return AKO4X_EINVAL;
  int shares = pick_shares(num_kv_indices, page_size);
  const Carve c = carve(batch, num_kv_indices, page_size);
  bool whole = false;
  if (!workspace || workspace_bytes < c.total || ((uintptr_t)workspace & 15)) {
    whole = whole_rows(batch, num_kv_indices, page_size);
    if (!whole) return (!workspace || workspace_bytes < c.total) ? AKO4X_EWORKSPACE : AKO4X_EINVAL;
    shares = (int)batch;
  }
  cudaStream_t st = (cudaStream_t)stream;

  Params p;
  p.q = (const __nv_bfloat16*)q;
  p.k = (const unsigned char*)k_cache;
  p.v = (const unsigned char*)v_cache;
  p.indptr = kv_indptr;
  p.indices = kv_indices;
  p.o = (__nv_bfloat16*)o;
  p.lse = lse;
  p.cut = (int2*)workspace;
  p.part_acc = (float*)((unsigned char*)workspace + c.acc);
  p.part_ml = (float*)((unsigned char*)workspace + c.ml);
  p.scale_log2 = sm_scale * AKO_LOG2E;
  p.page_size = (int)page_size;
  p.batch = (int)batch;
  p.whole_rows = whole;
  gqa_decode_kernel<<<(unsigned)(shares * HALVES), THREADS, 0, st>>>(p);
  AKO_CHECK_LAUNCH();
  if (whole || shares == 1) return AKO4X_OK;          // nothing is cut
  const bool many = shares >= 8 * batch;              // partials per sequence
  const unsigned entries = (unsigned)std::min<int64_t>(batch, shares);
  const cudaError_t e = many ? ako::launch_pdl(true, gqa_merge_kernel<8>, dim3(entries * HQ), dim3(256), 0, st, p, shares)
                             : ako::launch_pdl(true, gqa_merge_kernel<1>, dim3(entries * (HQ / 4)), dim3(128), 0, st, p, shares);
  if (e != cudaSuccess)
    return AKO4X_ELAUNCH;
  return AKO4X_OK;
}

// The kernels of this file have no wait that could give up.
extern "C" int ako4x_gqa_paged_decode_device_status(void) { return AKO4X_OK; }
