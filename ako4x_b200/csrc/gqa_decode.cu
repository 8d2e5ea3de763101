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
//     O^T = V^T P^T ([128 x 8 heads], features as M), and P's own pairs into the B fragment.
//   * K of the next tile is requested when S has been computed, V of it when O has.
//
// Work split: flat_share.cuh, tiles of 16 tokens, one share per pair of CTAs (the two halves of the KV
// heads); a second kernel merges the partials of rows that several shares touch. Measured (whole call,
// bulk copies through shared memory and a planning kernel before -> now): 64 sequences of up to 8 192 tokens
// 245 -> 188 us (6.3 TB/s = 0.96 of the measured copy bandwidth), 256 of them 841 -> 680 (0.99), 16 of up to
// 1 200 25 -> 17, one of 547 12.6 -> 10.2 us.
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

__device__ int g_gqa_status = 0;          // no wait of this kernel can give up: stays 0

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
  int32_t* prefix;  // [batch + 1] tiles in front of a sequence
  float scale_log2;
  int page_size;
  int batch;
  bool whole_rows;  // a share is one sequence
};

__device__ __forceinline__ int seq_tokens(const Params& p, int b) {
  return max(0, p.indptr[b + 1] - p.indptr[b]) * p.page_size;
}
__device__ __forceinline__ uint4 ld_row16(const unsigned char* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
  uint32_t y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
  return y;
}

__global__ void __launch_bounds__(THREADS, CTAS_PER_SM) gqa_decode_kernel(Params p) {
  __shared__ int s_scan[6];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int half = blockIdx.x % HALVES, share = blockIdx.x / HALVES;
  const int kvh = half * HPC + warp;
  ako::pdl_trigger();  // the merge kernel may be scheduled early; it waits for this grid to finish
  auto seq_tiles = [&](int b) { return (seq_tokens(p, b) + TILE - 1) / TILE; };
  ako::Share sh;
  if (p.whole_rows) {
    sh = {share, 0, seq_tiles(share)};
    if (sh.left == 0) {                              // an empty sequence
      const int64_t h0 = (int64_t)share * HQ + kvh * GROUP;
      uint4* op = reinterpret_cast<uint4*>(p.o + h0 * D);
      for (int i = lane; i < GROUP * D / 8; i += 32) op[i] = make_uint4(0u, 0u, 0u, 0u);
      if (lane < GROUP) p.lse[h0 + lane] = -INFINITY;
    }
  } else {
    sh = ako::find_share(p.batch, share, gridDim.x / HALVES, blockIdx.x == 0, p.prefix, s_scan, seq_tiles);
  }

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
    fetch_ids(ts);
    locate(ts);
    load(kc, p.k);
    load(vc, p.v);
    fetch_ids(ts + 1);

    // Q of the four heads as B fragments (n = head g, heads 4-7 are zero), in the order of the K pieces
    uint4 qb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      qb[j] = make_uint4(0u, 0u, 0u, 0u);
      if (g < GROUP)
        qb[j] = __ldg(reinterpret_cast<const uint4*>(p.q + ((int64_t)b * HQ + kvh * GROUP + g) * D + 32 * j + 8 * t));
    }
    float acc[4][2][4];   // [block j][u]: features 32 j + 8 (g / 2) + (g & 1) + 4 u (regs 0, 1) and + 2 (2, 3), heads 2t, 2t+1
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][u][i] = 0.f;
    // heads 2t, 2t+1; l over this lane's tokens. The maxima start at the lowest finite value, so that a score
    // of -inf weighs 0 whatever else a tile or a share holds.
    float m0 = -FLT_MAX, m1 = -FLT_MAX, l0 = 0.f, l1 = 0.f;

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
      const uint32_t b0 = movmatrix_trans(ako::pack_bf16x2(s[0], s[1])), b1 = movmatrix_trans(ako::pack_bf16x2(s[2], s[3]));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t a0[4] = {movmatrix_trans(vc[0][j].x), movmatrix_trans(vc[0][j].y), movmatrix_trans(vc[1][j].x), movmatrix_trans(vc[1][j].y)};
        const uint32_t a1[4] = {movmatrix_trans(vc[0][j].z), movmatrix_trans(vc[0][j].w), movmatrix_trans(vc[1][j].z), movmatrix_trans(vc[1][j].w)};
        ako::mma_bf16_16816(acc[j][0], a0, b0, b1);
        ako::mma_bf16_16816(acc[j][1], a1, b0, b1);
      }
      if (more) {
        load(vc, p.v);
        fetch_ids(tile + 2);
      }
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
    const int64_t slot = (int64_t)b + share;
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
}

// Merge: WARPS warps per (sequence, head), every warp 32 threads x 4 columns of every WARPS-th partial;
// a block holds four heads (WARPS = 1) or one (WARPS = 8: few sequences with many partials each, where
// one warp would walk up to 222 partials in a row). The partials of sequence b are the slots b + c of
// the shares c that touch it; a sequence inside one share is already written, an empty one gets its
// zeros here.
constexpr int MERGE_MAX = 512;                       // shares of a call never exceed this (three CTAs per SM)
template <int WARPS>
__global__ void __launch_bounds__(WARPS == 1 ? 128 : WARPS * 32) gqa_merge_kernel(Params p, int shares) {
  constexpr int HEADS = (WARPS == 1) ? 4 : 1;
  __shared__ float s_w[HEADS][MERGE_MAX];
  __shared__ float4 s_acc[WARPS][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = blockIdx.x / (HQ / HEADS), hl = (WARPS == 1) ? w : 0, part = (WARPS == 1) ? 0 : w;
  const int head = (blockIdx.x % (HQ / HEADS)) * HEADS + hl;
  ako::pdl_wait();
  const int t0 = p.prefix[b], t1 = p.prefix[b + 1], total = p.prefix[p.batch];
  const int64_t oi = (int64_t)b * HQ + head;
  uint2* op = reinterpret_cast<uint2*>(p.o + oi * D) + lane;
  if (t1 <= t0) {
    if (part == 0) {
      *op = make_uint2(0u, 0u);
      if (lane == 0) p.lse[oi] = -INFINITY;
    }
    return;
  }
  const int per = (total + shares - 1) / shares;
  const int c0 = t0 / per, n = (t1 - 1) / per - c0 + 1;
  if (n == 1) return;
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + ((int64_t)(b + c0) * HQ + head);
  const float4* pa = reinterpret_cast<const float4*>(p.part_acc + ((int64_t)(b + c0) * HQ + head) * D) + lane;
  // every warp of the head finds the maximum over all partials for itself
  float2 mine[MERGE_MAX / 32];
  float M = -INFINITY, L = 0.f;
#pragma unroll
  for (int i = 0; i < MERGE_MAX / 32; ++i) {
    mine[i] = make_float2(-INFINITY, 0.f);
    if (i * 32 < n && i * 32 + lane < n) mine[i] = ml[(int64_t)(i * 32 + lane) * HQ];
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
    const float4 x = pa[(int64_t)i * (HQ * D / 4)];
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

// Whole sequences as shares, without partials and without the merge: batches that fill the GPU and are
// short (at most 32 tiles) or many (four times as many sequences as shares fit at once).
bool whole_rows(int64_t batch, int64_t num_kv_indices, int64_t page_size) {
  const int64_t most = (int64_t)CTAS_PER_SM * ako::sm_count() / HALVES;
  return batch >= 4 * most || (batch >= most && num_kv_indices * page_size <= batch * 512);
}
// Shares of a call: all CTAs resident at once, and at least one tile (16 tokens, 64 KB of K and V) each.
int pick_shares(int64_t batch, int64_t num_kv_indices, int64_t page_size) {
  if (whole_rows(batch, num_kv_indices, page_size)) return (int)batch;
  const int64_t most = (int64_t)CTAS_PER_SM * ako::sm_count() / HALVES;
  const int64_t tiles = ako::cdiv(num_kv_indices * page_size, (int64_t)TILE);   // at least; rows round up
  int64_t s = tiles < most ? tiles : most;
  if (s > MERGE_MAX) s = MERGE_MAX;
  return (int)(s < 1 ? 1 : s);
}
struct Carve {
  size_t acc, ml, total;   // offsets; the prefix table is first
};
Carve carve(int64_t batch, int shares) {
  const size_t slots = (size_t)batch + (size_t)shares;
  Carve c;
  c.acc = (((size_t)batch + 1) * sizeof(int32_t) + 255) / 256 * 256;
  c.ml = c.acc + slots * HQ * D * sizeof(float);
  c.total = c.ml + slots * HQ * 2 * sizeof(float);
  return c;
}

}  // namespace

extern "C" size_t ako4x_gqa_paged_decode_workspace_bytes(int64_t batch, int64_t num_kv_indices,
                                                         int64_t page_size) {
  if (batch <= 0 || whole_rows(batch, num_kv_indices, page_size)) return 0;
  return carve(batch, pick_shares(batch, num_kv_indices, page_size)).total;
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
  const bool whole = whole_rows(batch, num_kv_indices, page_size);
  const int shares = pick_shares(batch, num_kv_indices, page_size);
  const Carve c = carve(batch, shares);
  if (!whole) {
    if (!workspace || workspace_bytes < c.total) return AKO4X_EWORKSPACE;
    if ((uintptr_t)workspace & 15) return AKO4X_EINVAL;
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
  p.prefix = (int32_t*)workspace;
  p.part_acc = (float*)((unsigned char*)workspace + c.acc);
  p.part_ml = (float*)((unsigned char*)workspace + c.ml);
  p.scale_log2 = sm_scale * AKO_LOG2E;
  p.page_size = (int)page_size;
  p.batch = (int)batch;
  p.whole_rows = whole;
  gqa_decode_kernel<<<(unsigned)(shares * HALVES), THREADS, 0, st>>>(p);
  AKO_CHECK_LAUNCH();
  if (whole) return AKO4X_OK;
  const bool many = shares >= 8 * batch;              // partials per sequence
  const cudaError_t e = many ? ako::launch_pdl(true, gqa_merge_kernel<8>, dim3((unsigned)(batch * HQ)), dim3(256), 0, st, p, shares)
                             : ako::launch_pdl(true, gqa_merge_kernel<1>, dim3((unsigned)(batch * (HQ / 4))), dim3(128), 0, st, p, shares);
  if (e != cudaSuccess)
    return AKO4X_ELAUNCH;
  return AKO4X_OK;
}

// Status word of the decode kernel of this file. Synchronises the device; meant for tests and
// post-mortems.
extern "C" int ako4x_gqa_paged_decode_device_status(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_gqa_status, sizeof(int)) != cudaSuccess) return AKO4X_ELAUNCH;
  return v;
}
