// Causal paged MLA prefill on the 5th-generation tensor cores (tcgen05 + TMEM) fed by TMA.
//
// Two launches. (1) gather: the keys of all sequences are copied from the paged caches into a
// contiguous [tokens, 576] matrix Kc (ckv | kpe). (2) attention: a PAIR of CTAs (a cluster of two,
// tcgen05 cta_group::2, M = 256) owns 16 consecutive query tokens of one sequence, eight per CTA
// (128 rows: token x head), and ONE half of the 512 output columns; O and the S buffers together
// would not fit TMEM otherwise, so the two halves are separate pairs that both compute S. The Q tile
// (144 KB per CTA) stays in shared memory. Per tile of 128 keys:
//   S  = Q Kc^T        256 x 128, reduction 576 in nine 64-column chunks of Kc, 64 keys per CTA,
//                      through a 6-stage TMA ring; 36 MMAs (bf16, K = 16) into one of two 128-column
//                      TMEM buffers of each CTA;
//   P  = softmax step  eight warps, two threads per row (64 keys each, held in registers from the
//                      one TMEM read on), which exchange the row maximum through shared memory;
//                      P goes back with tcgen05.st as packed bf16 pairs over the first 64 columns of
//                      the S buffer;
//   O  = O alpha + P V 256 x 256, 8 MMAs (N = 256): A operand (P) from TMEM, B = the rows of Kc read
//                      as an MN-major operand (128 columns per CTA), accumulated in TMEM.
// Where a row's maximum grew, its warps rescale their lanes of O in TMEM once the previous PV is done;
// a warp none of whose 32 rows grew skips it. (Letting the maximum lag by up to 2^8 instead makes
// this rare and measured 4 % faster, but then the largest weight of a row is not exactly 1 and its
// bf16 rounding shows: 1.96e-3 instead of 1.81e-3 from fp64 at 8192 keys. Not done.)
//
// Why a pair: one CTA per tile was bound by the bytes that cross shared memory (128 B/clk per SM):
// 644 KB per 128-key tile, of which 294 KB were TMA writes of Q and K chunks and 288 KB S operands.
// A pair reads half of every K chunk and half of V per CTA and leaves room for a resident Q tile:
// 352 KB. Eight ragged prompts (9 101 queries, 39 794 keys): 2 239 -> 1 730 us with the gather, 769
// TFLOP/s of algorithmic flops, 1 180 counting S of both halves.
// Warps: 0-7 softmax, rescale and output, 8 Q/K producer, 9 S issuer (even CTA), 10 V producer,
// 11 PV issuer (even CTA). Rows of a partial last tile and keys past the causal limit are masked;
// every mbarrier wait is bounded and a timeout sets the status word.
#include "mla_prefill_tc.h"

#include <cuda_bf16.h>

#include "ako4x_b200.h"
#include "common.cuh"
#include "tcgen05.cuh"
#include "tma_host.cuh"

namespace {

constexpr int H = 16, DC = 512, DP = 64, DQK = DC + DP;
constexpr int QT = 8;                     // query tokens per CTA
constexpr int PT = 2 * QT;                // query tokens per pair
constexpr int BM = QT * H;                // 128 rows per CTA
constexpr int BK = 128;                   // keys per tile
constexpr int NCH = DQK / 64;             // nine reduction chunks of 64 columns
constexpr int Q_CH_BYTES = BM * 128;      // one 128-row x 64-column bf16 chunk: 16 KB
constexpr int K_CH_BYTES = BK / 2 * 128;  // this CTA's 64 keys of a chunk: 8 KB
constexpr int Q_BYTES = NCH * Q_CH_BYTES;
constexpr int NST = 6;
constexpr int V_BOX_BYTES = BK * 128;     // 128 keys x 64 columns
constexpr int V_BYTES = 2 * V_BOX_BYTES;  // this CTA's 128 columns
constexpr int AUX_BYTES = 3072;           // row exchange [2][2][128], mbarriers, TMEM address, work item
// exactly the 227 KB a CTA may have: no static shared memory in this kernel, so that the dynamic
// region starts on a 1024-byte boundary (checked at entry) and needs no alignment slack
constexpr int SMEM = Q_BYTES + NST * K_CH_BYTES + V_BYTES + AUX_BYTES;
static_assert(SMEM <= 232448, "shared memory per CTA");
constexpr int THREADS = 384;
constexpr int SOFTMAX_WARPS = 8;
constexpr float NEG = -1.0e30f;           // finite stand-in for -inf

// Wait status of the CURRENT call (cleared by the gather kernel that starts every call, so a code
// left by an earlier call cannot make this call's waits give up early; both CTAs of a pair see it)
// and the sticky word that ako_mla_prefill_tc_status() reports.
__device__ int g_pf_status = 0;
__device__ int g_pf_sticky = 0;

struct PfParams {
  const int32_t* qo_indptr;
  const int32_t* kv_indptr;
  __nv_bfloat16* o;
  float* lse;
  float scale_log2;
  int batch, page_size;
};

// ---------------------------------------------------------------------------------------------
// gather: 32 key tokens per CTA
// ---------------------------------------------------------------------------------------------
constexpr int G_TOK = 32, G_VEC = DQK * 2 / 16;  // 72 16-byte vectors per token
static_assert(G_TOK * G_VEC % 256 == 0, "whole passes of the block");

__global__ void __launch_bounds__(256) mla_prefill_gather_kernel(
    const uint4* __restrict__ ckv, const uint4* __restrict__ kpe, const int32_t* __restrict__ kv_indices,
    int page_size, int64_t ntok, uint4* __restrict__ kc) {
  __shared__ int64_t s_row[G_TOK];
  const int tid = threadIdx.x;
  const int64_t g0 = (int64_t)blockIdx.x * G_TOK;
  if (blockIdx.x == 0 && tid == 0) g_pf_status = 0;  // this call's wait status starts clean
  if (tid < G_TOK) {
    const int64_t g = g0 + tid;
    s_row[tid] = (g < ntok) ? (int64_t)kv_indices[g / page_size] * page_size + g % page_size : 0;
  }
  __syncthreads();
  uint4 v[G_TOK * G_VEC / 256];
#pragma unroll
  for (int k = 0; k < G_TOK * G_VEC / 256; ++k) {
    const int i = k * 256 + tid, t = i / G_VEC, c = i % G_VEC;
    if (g0 + t < ntok) v[k] = (c < 64) ? __ldg(ckv + s_row[t] * 64 + c) : __ldg(kpe + s_row[t] * 8 + (c - 64));
  }
#pragma unroll
  for (int k = 0; k < G_TOK * G_VEC / 256; ++k) {
    const int i = k * 256 + tid;
    if (g0 + i / G_VEC < ntok) kc[g0 * G_VEC + i] = v[k];
  }
}

// ---------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS, 1)
mla_prefill_tc_kernel(PfParams p, const __grid_constant__ CUtensorMap tm_qn, const __grid_constant__ CUtensorMap tm_qp,
                      const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int crank = (int)ako::tc::t2_cluster_ctarank();
  const int half = blockIdx.y;  // which 256 output columns
  if (ako::smem_u32(smem_raw) & 1023u) {  // the swizzled operand tiles need this; nothing is started yet
    if (tid == 0) atomicCAS(&g_pf_sticky, 0, 13);
    return;  // the dynamic region starts at the same address in both CTAs: both return
  }
  const uint32_t q_base = ako::smem_u32(smem_raw);
  const uint32_t k_base = q_base + Q_BYTES;
  const uint32_t v_base = k_base + NST * K_CH_BYTES;
  float* xch = reinterpret_cast<float*>(smem_raw + Q_BYTES + NST * K_CH_BYTES + V_BYTES);  // [2][2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(xch + 4 * BM);
  uint64_t* st_full = bars;                // even CTA: bytes of both CTAs
  uint64_t* st_empty = st_full + NST;      // each CTA
  uint64_t* s_full = st_empty + NST;       // each CTA
  uint64_t* pv_done = s_full + 2;          // each CTA: O is up to date, P and V have been read
  uint64_t* p_full = pv_done + 2;          // even CTA: the softmax warps of both CTAs
  uint64_t* xch_full = p_full + 2;         // each CTA: the two warps of a lane quarter
  uint64_t& v_full = xch_full[4];          // even CTA: bytes of both CTAs
  uint32_t& s_tmem = *reinterpret_cast<uint32_t*>(xch_full + 5);
  int* s_work = reinterpret_cast<int*>(xch_full + 6);  // sequence, pair tile inside the sequence (or -1)
  static_assert(4 * BM * 4 + (2 * NST + 6 + 6) * 8 + 8 <= AUX_BYTES, "aux region");

  if (warp == 0) {
    // reversed: within a sequence the later query tiles see more keys, so the long pairs start
    // first and the short ones fill the end of the grid. 32 sequences per step: one thread alone
    // walked 256 of them in 5 us, with every pair.
    int t = (int)((gridDim.x - 1 - blockIdx.x) >> 1), seq = p.batch;
    for (int b0 = 0; b0 < p.batch; b0 += 32) {
      const int b = b0 + lane;
      const int nt = (b < p.batch) ? (p.qo_indptr[b + 1] - p.qo_indptr[b] + PT - 1) / PT : 0;
      int x = nt;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += up;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, t < x);
      if (hit) {
        const int f = __ffs(hit) - 1;
        t -= __shfl_sync(0xffffffffu, x - nt, f);
        seq = b0 + f;
        break;
      }
      t -= __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) {
      s_work[0] = seq;
      s_work[1] = (seq < p.batch) ? t : -1;
    }
  }
  if (tid == 0) {
    for (int s = 0; s < NST; ++s) {
      ako::tc::mbar_init(ako::smem_u32(&st_full[s]), 1);
      ako::tc::mbar_init(ako::smem_u32(&st_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      ako::tc::mbar_init(ako::smem_u32(&s_full[s]), 1);
      ako::tc::mbar_init(ako::smem_u32(&pv_done[s]), 1);
      ako::tc::mbar_init(ako::smem_u32(&p_full[s]), 2 * SOFTMAX_WARPS);
    }
    for (int q = 0; q < 4; ++q) ako::tc::mbar_init(ako::smem_u32(&xch_full[q]), 2);
    ako::tc::mbar_init(ako::smem_u32(&v_full), 1);
    ako::tc::mbar_init_fence();
  }
  if (warp == 9) ako::tc::t2_tmem_alloc(ako::smem_u32(&s_tmem), 512);
  ako::tc::fence_before_thread_sync();
  __syncthreads();
  ako::tc::t2_cluster_sync();  // both CTAs' barriers are initialised before anybody signals across
  ako::tc::fence_after_thread_sync();
  const uint32_t tmem = s_tmem;

  const int b = s_work[0], tile = s_work[1];
  // geometry of this tile (every thread computes the same values; ntk is the pair's)
  int q0 = 0, nq = 0, kv_len = 0, q_len = 0, ntk = 0;
  int64_t kbase = 0;
  if (tile >= 0) {
    const int qb = p.qo_indptr[b];
    q_len = p.qo_indptr[b + 1] - qb;
    q0 = qb + tile * PT + crank * QT;
    nq = min(QT, q_len - tile * PT - crank * QT);  // <= 0 for the empty half of an odd last pair
    kbase = (int64_t)p.kv_indptr[b] * p.page_size;
    kv_len = (p.kv_indptr[b + 1] - p.kv_indptr[b]) * p.page_size;
    // keys visible to the pair's last token: [0, kv_len - q_len + last + 1)
    const int kv_end = max(0, min(kv_len, kv_len - q_len + min(q_len, (tile + 1) * PT)));
    ntk = (kv_end + BK - 1) / BK;
  }

  if (warp < SOFTMAX_WARPS) {
    // ================================ softmax, rescale, output ===================================
    const int quarter = warp & 3, ch = warp >> 2;  // ch: keys [64 ch, 64 ch + 64) of a tile; 128 output columns
    const int r = 32 * quarter + lane;
    const int qtok = r >> 4;
    const bool row_ok = qtok < nq;
    const int kv_lim = row_ok ? max(0, min(kv_len, kv_len - q_len + tile * PT + crank * QT + qtok + 1)) : 0;
    const uint32_t tq = tmem + ((uint32_t)(32 * quarter) << 16);
    const uint32_t to = tq + 256 + 128 * ch;
    const uint32_t xbar = ako::smem_u32(&xch_full[quarter]);
    const uint32_t p_full0 = ako::tc::t2_mapa(ako::smem_u32(&p_full[0]), 0);
    const uint32_t p_full1 = ako::tc::t2_mapa(ako::smem_u32(&p_full[1]), 0);
    const float scale = p.scale_log2;
    float m = NEG, l = 0.f;  // running maximum of the row, sum over this thread's keys
    bool ok = true;
#pragma unroll 1
    for (int j = 0; j < ntk; ++j) {
      const int buf = j & 1;
      if (!ako::tc::mbar_wait_warp(ako::smem_u32(&s_full[buf]), (uint32_t)((j >> 1) & 1), &g_pf_status, 3)) { ok = false; break; }
      ako::tc::fence_after_thread_sync();
      const uint32_t ts = tq + buf * BK;
      float v[2][32];
      ako::tc::tmem_ld32(ts + 64 * ch, v[0]);
      ako::tc::tmem_ld32(ts + 64 * ch + 32, v[1]);
      ako::tc::tmem_ld_wait_regs(v[0]);
      ako::tc::tmem_ld_wait_regs(v[1]);
      const int nvis = kv_lim - j * BK - 64 * ch;  // visible keys of this thread's 64 (may be <= 0 or > 64)
      // no masked key for any row of this warp; warp-uniform, because the aligned TMEM stores below
      // must be reached by the whole warp together
      const bool fast = __all_sync(0xffffffffu, nvis >= 64) && scale > 0.f;
      float tmax = NEG;
      if (fast) {  // four independent chains, the (positive) scale applied once
        float t[4] = {v[0][0], v[0][1], v[0][2], v[0][3]};
#pragma unroll
        for (int i = 4; i < 64; ++i) t[i & 3] = fmaxf(t[i & 3], v[i >> 5][i & 31]);
        tmax = fmaxf(tmax, fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3])) * scale);
      } else {
#pragma unroll
        for (int i = 0; i < 64; ++i) tmax = fmaxf(tmax, (i < nvis) ? v[i >> 5][i & 31] * scale : NEG);
      }
      // the row's other 64 keys belong to the same lane of the other warp of the quarter. Its wait
      // also says that S has been read by both warps, so P may overwrite it.
      xch[(buf * 2 + ch) * BM + r] = tmax;
      ako::tc::fence_before_thread_sync();
      __syncwarp();
      if (lane == 0) ako::tc::mbar_arrive(xbar);
      if (!ako::tc::mbar_wait_warp(xbar, (uint32_t)(j & 1), &g_pf_status, 4)) { ok = false; break; }
      ako::tc::fence_after_thread_sync();
      tmax = fmaxf(tmax, xch[(buf * 2 + (ch ^ 1)) * BM + r]);
      const bool moved = tmax > m;
      const bool rescale = __any_sync(0xffffffffu, moved);  // the same vote in both warps of the quarter
      const float alpha = moved ? ako::fast_exp2(m - tmax) : 1.0f;
      m = fmaxf(m, tmax);
      l *= alpha;
      if (fast) {
        const float2 sc2 = make_float2(scale, scale), nm2 = make_float2(-m, -m);
        float2 sum[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = __ffma2_rn(make_float2(v[h][i], v[h][i + 1]), sc2, nm2);
            const float2 e = make_float2(ako::fast_exp2(x.x), ako::fast_exp2(x.y));
            sum[(i >> 1) & 1] = __fadd2_rn(sum[(i >> 1) & 1], e);
            w[i >> 1] = ako::pack_bf16x2(e.x, e.y);
          }
          ako::tc::tmem_st16(ts + 32 * ch + 16 * h, w);
        }
        l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
      } else {
        float sum = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float e0 = (32 * h + i < nvis) ? ako::fast_exp2(v[h][i] * scale - m) : 0.f;
            const float e1 = (32 * h + i + 1 < nvis) ? ako::fast_exp2(v[h][i + 1] * scale - m) : 0.f;
            sum += e0 + e1;
            w[i >> 1] = ako::pack_bf16x2(e0, e1);
          }
          ako::tc::tmem_st16(ts + 32 * ch + 16 * h, w);
        }
        l += sum;
      }
      if (rescale && j > 0) {
        // S of this tile came after PV of tile j-2, so the phase before this one (tile j-3) is over
        if (!ako::tc::mbar_wait_warp(ako::smem_u32(&pv_done[buf ^ 1]), (uint32_t)(((j - 1) >> 1) & 1), &g_pf_status, 2)) { ok = false; break; }
        ako::tc::fence_after_thread_sync();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float o[32];
          uint32_t w[2][16];
          ako::tc::tmem_ld32(to + 32 * c, o);
          ako::tc::tmem_ld_wait_regs(o);
#pragma unroll
          for (int i = 0; i < 32; ++i) w[i >> 4][i & 15] = __float_as_uint(o[i] * alpha);
          ako::tc::tmem_st16(to + 32 * c, w[0]);
          ako::tc::tmem_st16(to + 32 * c + 16, w[1]);
        }
      }
      ako::tc::tmem_st_wait();
      ako::tc::fence_before_thread_sync();
      __syncwarp();
      // One barrier per buffer: a warp can be one tile ahead of another, never two (S of tile j+2
      // needs PV of tile j), so an arrival cannot complete a phase in a slower warp's place.
      if (lane == 0) ako::tc::t2_arrive_cluster(buf ? p_full1 : p_full0);
    }
    if (ok && tile >= 0) {
      // the slots of the tile before last: every reader has passed the barrier since
      xch[((ntk & 1) * 2 + ch) * BM + r] = l;
      __syncwarp();
      if (lane == 0) ako::tc::mbar_arrive(xbar);
      if (ako::tc::mbar_wait_warp(xbar, (uint32_t)(ntk & 1), &g_pf_status, 1) &&
          (ntk == 0 || ako::tc::mbar_wait_warp(ako::smem_u32(&pv_done[(ntk - 1) & 1]), (uint32_t)(((ntk - 1) >> 1) & 1), &g_pf_status, 12))) {
        ako::tc::fence_after_thread_sync();
        // summed in the order of the keys by both threads of the row
        l = xch[(ntk & 1) * 2 * BM + r] + xch[((ntk & 1) * 2 + 1) * BM + r];
        if (kv_lim <= 0) l = 0.f;
        const float inv = (l > 0.f) ? 1.0f / l : 0.f;
        if (half == 0 && ch == 0 && row_ok)
          p.lse[(int64_t)(q0 + qtok) * H + (r & 15)] = (l > 0.f) ? m + log2f(l) : -INFINITY;
        __nv_bfloat16* dst = p.o + ((int64_t)(q0 + qtok) * H + (r & 15)) * DC + half * 256 + ch * 128;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          float o[32];
          if (ntk > 0) {
            ako::tc::tmem_ld32(to + 32 * c, o);
            ako::tc::tmem_ld_wait_regs(o);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0.f;
          }
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 w;
              w.x = ako::pack_bf16x2(o[i] * inv, o[i + 1] * inv);
              w.y = ako::pack_bf16x2(o[i + 2] * inv, o[i + 3] * inv);
              w.z = ako::pack_bf16x2(o[i + 4] * inv, o[i + 5] * inv);
              w.w = ako::pack_bf16x2(o[i + 6] * inv, o[i + 7] * inv);
              *reinterpret_cast<uint4*>(dst + 32 * c + i) = w;
            }
          }
        }
      }
    }
  } else if (warp == 8 && ntk > 0) {
    // ================================ Q / K producer (each CTA its rows and keys) ================
    // this role and the next three: the whole warp waits, one lane issues
    if (ako::tc::elect_one()) {
      ako::tc::tma_prefetch_desc(&tm_qn);
      ako::tc::tma_prefetch_desc(&tm_qp);
      ako::tc::tma_prefetch_desc(&tm_k);
    }
    int g = 0;
    bool ok = true;
    for (int j = 0; ok && j < ntk; ++j) {
      for (int c = 0; c < NCH; ++c, ++g) {
        const int stage = g % NST;
        if (!ako::tc::mbar_wait_warp(ako::smem_u32(&st_empty[stage]), (uint32_t)(((g / NST) & 1) ^ 1), &g_pf_status, 5)) { ok = false; break; }
        const uint32_t bar = ako::tc::t2_mapa(ako::smem_u32(&st_full[stage]), 0);
        if (ako::tc::elect_one()) {
          // the even CTA announces the bytes of both; the first tile's stages bring the Q chunk along
          if (crank == 0)
            ako::tc::mbar_arrive_expect_tx(ako::smem_u32(&st_full[stage]), 2 * (K_CH_BYTES + (j == 0 ? Q_CH_BYTES : 0)));
          if (j == 0) {
            if (c < DC / 64) ako::tc::t2_tma_load_2d(q_base + c * Q_CH_BYTES, &tm_qn, c * 64, q0 * H, bar);
            else ako::tc::t2_tma_load_2d(q_base + c * Q_CH_BYTES, &tm_qp, 0, q0 * H, bar);
          }
          ako::tc::t2_tma_load_2d(k_base + stage * K_CH_BYTES, &tm_k, c * 64, (int)(kbase + (int64_t)j * BK + crank * (BK / 2)), bar);
        }
        __syncwarp();
      }
    }
  } else if (warp == 10 && ntk > 0) {
    // ================================ V producer (each CTA its 128 columns) ======================
    if (ako::tc::elect_one()) ako::tc::tma_prefetch_desc(&tm_v);
    const uint32_t bar = ako::tc::t2_mapa(ako::smem_u32(&v_full), 0);
    const int x = half * 256 + crank * 128;
    for (int j = 0; j < ntk; ++j) {
      if (j > 0 && !ako::tc::mbar_wait_warp(ako::smem_u32(&pv_done[(j - 1) & 1]), (uint32_t)(((j - 1) >> 1) & 1), &g_pf_status, 6)) break;
      if (ako::tc::elect_one()) {
        if (crank == 0) ako::tc::mbar_arrive_expect_tx(ako::smem_u32(&v_full), 2 * V_BYTES);
        const int y = (int)(kbase + (int64_t)j * BK);
        ako::tc::t2_tma_load_2d(v_base, &tm_v, x, y, bar);
        ako::tc::t2_tma_load_2d(v_base + V_BOX_BYTES, &tm_v, x + 64, y, bar);
      }
      __syncwarp();
    }
  } else if (warp == 9 && crank == 0 && ntk > 0) {
    // ================================ S issuer (for the pair) ====================================
    constexpr uint32_t IDESC_S = ako::tc::idesc_bf16_f32(2 * BM, BK);
    const uint32_t q_lo = ako::tc::smem_desc_lo(q_base), k_lo = ako::tc::smem_desc_lo(k_base);
    int stage = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int j = 0; ok && j < ntk; ++j) {
      const int buf = j & 1;
      // the PV MMAs of tile j-2 have read P out of this buffer
      if (!ako::tc::mbar_wait_warp(ako::smem_u32(&pv_done[buf]), (uint32_t)(((j >> 1) & 1) ^ 1), &g_pf_status, 7)) break;
      const uint32_t d = tmem + buf * BK;
      for (int c = 0; c < NCH; ++c) {
        if (!ako::tc::mbar_wait_warp(ako::smem_u32(&st_full[stage]), ph, &g_pf_status, 8)) { ok = false; break; }
        ako::tc::fence_after_thread_sync();
        const uint32_t a_lo = q_lo + c * (Q_CH_BYTES >> 4);
        const uint32_t b_lo = k_lo + stage * (K_CH_BYTES >> 4);
        if (ako::tc::elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            ako::tc::t2_mma_bf16(d, a_lo + 2 * ks, b_lo + 2 * ks, IDESC_S, (c > 0 || ks > 0) ? 1u : 0u);
          ako::tc::t2_commit_both(ako::smem_u32(&st_empty[stage]));
          if (c == NCH - 1) ako::tc::t2_commit_both(ako::smem_u32(&s_full[buf]));
        }
        __syncwarp();
        if (++stage == NST) { stage = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 11 && crank == 0 && ntk > 0) {
    // ================================ PV issuer (for the pair) ===================================
    // a thread of its own: PV of tile j goes to the tensor pipe the moment P is written, while
    // the S issuer is still waiting on the operand stream of a later tile
    constexpr uint32_t IDESC_PV = ako::tc::idesc_bf16_f32(2 * BM, 256) | ako::tc::kIdescBMnMajor;
    const uint32_t v_lo = ako::tc::smem_desc_lo_mn(v_base, V_BOX_BYTES);
    const uint32_t d = tmem + 256;
    for (int j = 0; j < ntk; ++j) {
      const int buf = j & 1;
      if (!ako::tc::mbar_wait_warp(ako::smem_u32(&p_full[buf]), (uint32_t)((j >> 1) & 1), &g_pf_status, 9)) break;
      if (!ako::tc::mbar_wait_warp(ako::smem_u32(&v_full), (uint32_t)(j & 1), &g_pf_status, 10)) break;
      ako::tc::fence_after_thread_sync();
      if (ako::tc::elect_one()) {
#pragma unroll
        for (int ks = 0; ks < BK / 16; ++ks)  // 16 keys = two 8-row groups of 1024 bytes
          ako::tc::t2_mma_bf16_tmem_a(d, tmem + buf * BK + 8 * ks, v_lo + ks * (2048 >> 4), IDESC_PV, (j > 0 || ks > 0) ? 1u : 0u);
        // P (inside the S buffer) and V have been read, O is up to date. Both CTAs wait for the last of
        // these, so no signal is on its way to a CTA that leaves.
        ako::tc::t2_commit_both(ako::smem_u32(&pv_done[buf]));
      }
      __syncwarp();
    }
  }

  ako::tc::fence_before_thread_sync();
  __syncthreads();
  ako::tc::t2_cluster_sync();  // the peer may still be reading this CTA's shared memory or writing its TMEM
  if (tid == 0) {
    const int code = *reinterpret_cast<volatile int*>(&g_pf_status);
    if (code != 0) atomicCAS(&g_pf_sticky, 0, code);
  }
  if (warp == 9) {
    ako::tc::fence_after_thread_sync();
    ako::tc::t2_tmem_dealloc(tmem, 512);
  }
}

}  // namespace

size_t ako_mla_prefill_tc_workspace_bytes(int64_t batch, int64_t num_kv_indices, int64_t page_size) {
  const int64_t ntok = num_kv_indices * page_size;
  if (ntok <= 0 || batch <= 0) return 0;
  const size_t kc = ((size_t)ntok * DQK * 2 + 255) / 256 * 256;
  // The C ABI promises callers a size of 2 176 bytes per key and refuses less (the values were once
  // copied a second time, transposed). The promise stands; only the first part is used.
  return kc + (size_t)DC * 2 * (((size_t)ntok + 8 * (size_t)batch + 8 + 7) / 8 * 8);
}

int ako_mla_prefill_tc_launch(const void* q_nope, const void* q_pe, const void* ckv_cache, const void* kpe_cache,
                              const int32_t* qo_indptr, const int32_t* kv_indptr, const int32_t* kv_indices,
                              float sm_scale, void* o, float* lse, int64_t total_q, int64_t batch,
                              int64_t num_kv_indices, int64_t page_size, void* workspace, size_t workspace_bytes,
                              cudaStream_t st) {
  const int64_t ntok = num_kv_indices * page_size;
  if (ntok <= 0 || ntok > 0x7fffffffLL || total_q * H > 0x7fffffffLL) return AKO4X_EUNSUPPORTED_SHAPE;
  const size_t need = ako_mla_prefill_tc_workspace_bytes(batch, num_kv_indices, page_size);
  if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255)) return AKO4X_EWORKSPACE;
  unsigned char* kc = (unsigned char*)workspace;
  mla_prefill_gather_kernel<<<(unsigned)ako::cdiv(ntok, G_TOK), 256, 0, st>>>(
      (const uint4*)ckv_cache, (const uint4*)kpe_cache, kv_indices, (int)page_size, ntok, (uint4*)kc);
  AKO_CHECK_LAUNCH();

  CUtensorMap tm_qn, tm_qp, tm_k, tm_v;
  if (!ako::tma::bf16_matrix_map(&tm_qn, q_nope, (uint64_t)total_q * H, DC, DC * 2, BM) ||
      !ako::tma::bf16_matrix_map(&tm_qp, q_pe, (uint64_t)total_q * H, DP, DP * 2, BM) ||
      !ako::tma::bf16_matrix_map(&tm_k, kc, (uint64_t)ntok, DQK, DQK * 2, BK / 2) ||
      !ako::tma::bf16_matrix_map(&tm_v, kc, (uint64_t)ntok, DQK, DQK * 2, BK))
    return AKO4X_ELAUNCH;
  if (!ako::ensure_dynamic_smem<mla_prefill_tc_kernel>(SMEM)) return AKO4X_ELAUNCH;
  PfParams p;
  p.qo_indptr = qo_indptr;
  p.kv_indptr = kv_indptr;
  p.o = (__nv_bfloat16*)o;
  p.lse = lse;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  p.batch = (int)batch;
  p.page_size = (int)page_size;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (ako::cdiv(total_q, PT) + batch)), 2);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, mla_prefill_tc_kernel, p, tm_qn, tm_qp, tm_k, tm_v) != cudaSuccess) return AKO4X_ELAUNCH;
  return AKO4X_OK;
}

int ako_mla_prefill_tc_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_pf_sticky, sizeof(int)) != cudaSuccess) return AKO4X_ELAUNCH;
  return v;
}
