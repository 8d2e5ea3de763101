// Chunked form of the Gated Delta Net prefill recurrence on the tensor cores (mma.sync, bf16 pieces
// of fp32 values); included by gdn_prefill.cu inside its anonymous namespace.
//
// For a chunk of C = 32 tokens with state S0 at its start, gam_i = prod_{l<=i} g_l and
// R_ij = prod_{j<l<=i} g_l (the decay between tokens j and i), unrolling
//   delta_i = beta_i (v_i - g_i S_{i-1} k_i),   S_i = g_i S_{i-1} + delta_i k_i^T
// gives, for every state row on its own,
//   delta = T (v - gam (S0 k)),  T = (I + A)^-1 diag(beta) (its diagonal is beta),
//   A_ij = beta_i R_ij (k_i.k_j) for j < i
//   out_i = gam_i scale (S0 q_i) + sum_{j<=i} P_ij delta_j,  P_ij = scale R_ij (q_i.k_j)
//   S_C   = gam_C S0 + sum_j (R_Cj delta_j) k_j^T
// T and P depend on the tokens only: gdn_chunk_prep_kernel makes them for all chunks at once.
// gdn_chunk_kernel then walks a sequence's chunks with five small matrix products per chunk.
//
// Precision: q, k and v are bf16 already; S, T, P and delta are fp32 and go to the tensor core as
// three bf16 pieces each (8 + 8 + 8 mantissa bits: by truncation the three pieces of an fp32 value
// ADD UP TO IT EXACTLY; T and P are rounded piece by piece, which leaves 2^-26). A product with one
// bf16 factor takes three mma, a product of two fp32 factors takes the six pairs of pieces down to
// 2^-24: the sums are those of an fp32 recurrence in another order. The tensor core truncates where it
// accumulates, which costs an fp32 result twice the error of a rounding and a bias: so what carries most of a
// value is kept out of it or goes in last. The diagonal of T, which is beta, multiplies its right-hand side in
// fp32 outside (the tiles of T hold what is below it); a product's small pieces are summed before the leading
// ones; and a chunk's update is summed from zero and added to the state in fp32. R is the product of its own
// gates, as in the recurrence: never a ratio of two prefix products, so that strong decay elsewhere in a chunk
// costs it nothing, and not an exponential of summed logarithms. Error of the state from an fp64 recurrence,
// rms (8 x 300, 1 x 2 000, 24 x 100 tokens): 6.7e-8, 6.9e-8, 8.3e-8; token by token in fp32 6.4e-8, 6.6e-8,
// 6.7e-8; 1.8e-7, 1.7e-7, 2.0e-7 before that care was taken, for 4 to 7 % less time.
//
// Values that are not finite: a product takes in every token of its 8- or 16-token step, later ones with
// coefficient zero, and 0 x NaN is NaN. A token whose right-hand side or delta is not finite is therefore
// kept out of the tiles of earlier tokens, so that it spoils its row of the state from that token on and
// nothing before it, as in the recurrence. Tiles with finite values only pay the check (1 to 3 %).
//
// Split: the state rows never interact, so a CTA owns 16 rows (v) of one (sequence, head). Two groups
// of four warps share it. The chain group holds S: its warps split k (32 columns each), which makes
// S0 k a sum over the warps but keeps every part of S in registers for the whole sequence, as mma
// accumulators that are at once the A fragments of the next chunk's products. The output group runs
// one step behind on the pieces of S0 and delta that the chain group hands over, off the serial chain.
// Per chunk and pair of warps: 96 mma (24 S0 k, 24 S0 q, <= 12 T, <= 12 P, 24 S update) of 8.2 cycles of
// an SM sub-partition (mma.sync m16n8k16 measured at 2.0 cycles per SM).
//
// What bounds it: one CTA per SM, the chain (2 150 cycles per chunk, of which three exchanges through
// shared memory); two CTAs per SM, the LSU data pipe (ncu: 67 %, 1 130 wavefronts per chunk; tensor pipe
// 39 %). Measured, whole call against the fp32 CUDA-core form this replaces: 8 ragged sequences of
// 7 244 tokens 605 -> 121 us, 1 x 8 192 1 000 -> 288. One group of four warps that also makes the outputs:
// 128 us for the 8 (three CTAs per SM) and 1.2 instead of 1.08 us per chunk for one sequence. Loads by TMA
// instead of cp.async: no difference for 8, 1.22 us per chunk for one.
#pragma once

constexpr int C_TOK = 32;                                // tokens per chunk
constexpr int C_ROWS = 16;                               // state rows per CTA (one m16 tile)
constexpr int C_WARPS = 4;                               // k split
constexpr int C_FRAG_BYTES = 6 * 3 * 32 * 8;             // six 8 x 16 tiles (i, j) on or below the diagonal, three pieces
constexpr int C_COEF_FLOATS = 3 * C_TOK;                 // gam_i, R_Cj, beta_i
constexpr int C_SLOT_BYTES = 2 * C_FRAG_BYTES + C_COEF_FLOATS * 4;   // T, P, coefficients of one (chunk, head)
static_assert(C_SLOT_BYTES % 16 == 0, "slots are copied in 16-byte pieces");

// Workspace slot of chunk c of sequence `seq` that starts at token t0: unique over all sequences
// without a scan of cu_seqlens (every sequence start costs at most one extra partial chunk).
__device__ __forceinline__ int64_t gdn_chunk_slot(int64_t t0, int seq, int c) { return t0 / C_TOK + seq + c; }

// Tile (w, s) of the fragment arrays: rows i = 8w .. 8w+7, columns j = 16s .. 16s+15, s <= w / 2.
__host__ __device__ constexpr int gdn_frag_tile(int w, int s) { return (w < 2) ? w : 2 * w - 2 + s; }

// x = the sum of its three bf16 pieces, exactly; the pieces of two values packed as an mma operand pair.
__device__ __forceinline__ void split3_exact(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
  h = __byte_perm(u0, u1, 0x7632);
  const float2 r = __fadd2_rn(make_float2(x0, x1), make_float2(-__uint_as_float(u0 & 0xffff0000u), -__uint_as_float(u1 & 0xffff0000u)));
  const uint32_t v0 = __float_as_uint(r.x), v1 = __float_as_uint(r.y);
  m = __byte_perm(v0, v1, 0x7632);
  const float2 e = __fadd2_rn(r, make_float2(-__uint_as_float(v0 & 0xffff0000u), -__uint_as_float(v1 & 0xffff0000u)));
  l = __byte_perm(__float_as_uint(e.x), __float_as_uint(e.y), 0x7632);
}
__device__ __forceinline__ void split3_rn(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = ako::pack_bf16x2(x0, x1);
  x0 -= ako::bf16_lo(h);
  x1 -= ako::bf16_hi(h);
  m = ako::pack_bf16x2(x0, x1);
  l = ako::pack_bf16x2(x0 - ako::bf16_lo(m), x1 - ako::bf16_hi(m));
}

// ---- T, P and the decay coefficients of one chunk, for the two v heads of one q/k head ------------
// Grid (slots, q/k heads), 4 warps. k.k and q.k by mma (bf16 operands, exact products); T by forward
// substitution, one warp per head and one column per lane: 496 FMA and 136 broadcast loads per lane.
__global__ void __launch_bounds__(128, 7) gdn_chunk_prep_kernel(
    const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const float* __restrict__ A_log,
    const __nv_bfloat16* __restrict__ a, const float* __restrict__ dt_bias, const __nv_bfloat16* __restrict__ b,
    const int64_t* __restrict__ cu_seqlens, int num_seqs, float scale, unsigned char* __restrict__ ws) {
  // k and q rows; after the products, per warp: A and then T of a head (warps 0, 1), P of a head (2, 3)
  constexpr int A_PITCH = C_TOK + 4, WARP_FLOATS = C_TOK * A_PITCH;
  __shared__ __align__(128) unsigned char s_x[4 * WARP_FLOATS * 4];
  __shared__ float s_g[2][C_TOK][C_TOK + 1];                         // k.k, q.k
  __shared__ float s_gate[2][C_TOK], s_beta[2][C_TOK];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t slot = blockIdx.x;
  const int hq = blockIdx.y;
  ako::pdl_trigger();   // the chunk kernel's prologue may start; it waits before it reads the workspace

  // the sequence of this slot: the last s with cu[s] / 32 + s <= slot, 32 candidates per step
  int lo = 0, hi = num_seqs;
  while (true) {
    const int step = (hi - lo + 31) / 32;
    const int s = lo + lane * step;
    const unsigned below = __ballot_sync(0xffffffffu, s < hi && cu_seqlens[s] / C_TOK + s <= slot);
    const int cnt = __popc(below);
    if (cnt == 0) return;                   // in front of the first sequence
    lo += (cnt - 1) * step;
    hi = min(hi, lo + step);
    if (step == 1) break;
  }
  const int64_t t0 = cu_seqlens[lo], t1 = cu_seqlens[lo + 1];
  const int64_t tb = t0 + (slot - (t0 / C_TOK + lo)) * C_TOK;
  if (tb >= t1) return;                     // a slot that no chunk uses

  const uint32_t sx = ako::smem_u32(s_x);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int idx = tid + 128 * i;          // 2 x 32 rows x 16 pieces of 16 bytes
    const int which = idx >> 9, row = (idx >> 4) & 31, piece = idx & 15;
    const bool valid = tb + row < t1;
    const __nv_bfloat16* src = (which ? q : k) + ((valid ? tb + row : tb) * P_HQ + hq) * P_D + piece * 8;
    ako::cp_async16(sx + which * (C_TOK * 256) + row * 256 + ((piece ^ (row & 7)) << 4), src, valid);
  }
  ako::cp_async_commit();
  if (tid < 64) {
    const int e = tid >> 5, h = 2 * hq + e;
    const int64_t t = tb + lane;
    float gate = 1.f, beta = 0.f;           // tokens past the end: no decay, no update
    if (t < t1) {
      const float y = __bfloat162float(a[t * P_HV + h]) + dt_bias[h];
      const float sp = (y > 20.f) ? y : log1pf(expf(y));
      gate = expf(-expf(A_log[h]) * sp);
      beta = 1.f / (1.f + expf(-__bfloat162float(b[t * P_HV + h])));
    }
    s_gate[e][lane] = gate;
    s_beta[e][lane] = beta;
  }
  ako::cp_async_wait<0>();
  __syncthreads();
  {
    // warps 0, 1: k.k, rows 16 (warp & 1) ..; warps 2, 3: q.k
    const int mt = warp & 1;
    const uint32_t abase = sx + (warp >> 1) * (C_TOK * 256);
    float acc[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[n][c] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t af[4], bf[8];
      const int ar = mt * 16 + (lane & 15);
      ako::ldmatrix_x4(af[0], af[1], af[2], af[3], abase + ar * 256 + (((2 * ks + (lane >> 4)) ^ (ar & 7)) << 4));
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int br = p * 16 + (lane & 7) + ((lane >> 4) << 3);
        ako::ldmatrix_x4(bf[4 * p], bf[4 * p + 1], bf[4 * p + 2], bf[4 * p + 3],
                         sx + br * 256 + (((2 * ks + ((lane >> 3) & 1)) ^ (br & 7)) << 4));
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) ako::mma_bf16_16816(acc[n], af, bf[2 * n], bf[2 * n + 1]);
    }
    float(*g)[C_TOK + 1] = s_g[warp >> 1];
    const int r = mt * 16 + (lane >> 2), c = 2 * (lane & 3);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      g[r][8 * n + c] = acc[n][0];
      g[r][8 * n + c + 1] = acc[n][1];
      g[r + 8][8 * n + c] = acc[n][2];
      g[r + 8][8 * n + c + 1] = acc[n][3];
    }
  }
  __syncthreads();
  // warps 0, 1: T and the coefficients of head e; warps 2, 3: P of head e. Lane = column j.
  const int e = warp & 1, j = lane;
  unsigned char* dst = ws + (slot * P_HV + 2 * hq + e) * C_SLOT_BYTES + (warp >> 1) * C_FRAG_BYTES;
  float* out = reinterpret_cast<float*>(s_x) + warp * WARP_FLOATS;       // [i][j], columns rotated by i
  if (warp < 2) {
    float run = 1.f;
#pragma unroll
    for (int i = 0; i < C_TOK; ++i) {
      if (i > j) run *= s_gate[e][i];
      out[i * A_PITCH + j] = (i > j) ? s_beta[e][i] * run * s_g[0][i][j] : 0.f;
    }
    float* coef = reinterpret_cast<float*>(ws + (slot * P_HV + 2 * hq + e) * C_SLOT_BYTES + 2 * C_FRAG_BYTES);
    float gam = s_gate[e][lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float up = __shfl_up_sync(0xffffffffu, gam, off);
      if (lane >= off) gam *= up;
    }
    coef[lane] = gam;
    coef[C_TOK + lane] = run;
    coef[2 * C_TOK + lane] = s_beta[e][lane];
    __syncwarp();
    const float bj = s_beta[e][j];          // may be NaN: enters at the diagonal, so that zeros above it stay zeros
    float t[C_TOK];
#pragma unroll
    for (int i = 0; i < C_TOK; ++i) {
      float x[4] = {(i == j) ? bj : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int l = 0; l < i; l += 4) {
        const float4 w = *reinterpret_cast<const float4*>(out + i * A_PITCH + l);
        x[0] = fmaf(-w.x, t[l], x[0]);
        if (l + 1 < i) x[1] = fmaf(-w.y, t[l + 1], x[1]);
        if (l + 2 < i) x[2] = fmaf(-w.z, t[l + 2], x[2]);
        if (l + 3 < i) x[3] = fmaf(-w.w, t[l + 3], x[3]);
      }
      t[i] = (x[0] + x[1]) + (x[2] + x[3]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < C_TOK; ++i) out[i * C_TOK + ((j + i) & 31)] = (i == j) ? 0.f : t[i];
  } else {
    float run = 1.f;
#pragma unroll
    for (int i = 0; i < C_TOK; ++i) {
      if (i > j) run *= s_gate[e][i];
      out[i * C_TOK + ((j + i) & 31)] = (i >= j) ? scale * run * s_g[1][i][j] : 0.f;
    }
  }
  __syncwarp();
  // B fragments of mma.m16n8k16 (n = i, k = j): lane (g, t) holds (i = g; j = 2t, 2t+1 | 2t+8, 2t+9)
#pragma unroll
  for (int w = 0; w < 4; ++w) {
#pragma unroll
    for (int s = 0; s <= w / 2; ++s) {
      const int i = 8 * w + (lane >> 2), c = 16 * s + 2 * (lane & 3);
      const float* row = out + i * C_TOK;
      uint32_t f[3][2];
      split3_rn(row[(c + i) & 31], row[(c + 1 + i) & 31], f[0][0], f[1][0], f[2][0]);
      split3_rn(row[(c + 8 + i) & 31], row[(c + 9 + i) & 31], f[0][1], f[1][1], f[2][1]);
#pragma unroll
      for (int p = 0; p < 3; ++p)
        reinterpret_cast<uint2*>(dst)[(gdn_frag_tile(w, s) * 3 + p) * 32 + lane] = make_uint2(f[p][0], f[p][1]);
    }
  }
}

// ---- the recurrence over the chunks of one (sequence, head, 16 state rows) ------------------------
// Shared memory. Everything a chunk reads from global memory is copied here one chunk ahead (two
// stages per group): fetching T, P and v into registers instead tied them to the few scoreboards that
// shared-memory loads wait on as well, 2 700 against 2 240 cycles per chunk in the first version.
constexpr int C_KQ_WARP = C_TOK * 64;                                 // 32 tokens x the warp's 32 columns of k (or q)
constexpr int C_CH_SLOT = C_WARPS * C_KQ_WARP;                        // chain stage: k | T | gam, R_C | v
constexpr int C_CH_COEF = C_CH_SLOT + C_FRAG_BYTES;
constexpr int C_CH_V = C_CH_COEF + C_COEF_FLOATS * 4;
constexpr int C_CH_STAGE = C_CH_V + C_TOK * C_ROWS * 2;
constexpr int C_OUT_SLOT = C_WARPS * C_KQ_WARP;                       // output stage: q | P | gam, R_C
constexpr int C_OUT_COEF = C_OUT_SLOT + C_FRAG_BYTES;
constexpr int C_OUT_STAGE = C_OUT_COEF + C_COEF_FLOATS * 4;
constexpr int C_OFF_OUT = 2 * C_CH_STAGE;
constexpr int C_OFF_S = C_OFF_OUT + 2 * C_OUT_STAGE;                  // pieces of S0, two chunks: [warp][6][lane] uint4
constexpr int C_S_BYTES = C_WARPS * 6 * 512;
constexpr int C_OFF_D = C_OFF_S + 2 * C_S_BYTES;                      // delta pieces, two chunks: [piece][tile][lane] uint2
constexpr int C_D_BYTES = 3 * 4 * 256;
constexpr int C_OFF_E = C_OFF_D + 2 * C_D_BYTES;                      // R_Cj delta_j pieces
constexpr int C_OFF_R = C_OFF_E + C_D_BYTES;                          // right-hand side pieces
constexpr int C_OFF_X = C_OFF_R + C_D_BYTES;                          // partial S0 k: [tile][3 other warps][lane] float4
constexpr int C_OFF_Y = C_OFF_X + 4 * 3 * 512;                        // partial S0 q
constexpr int C_SMEM = C_OFF_Y + 4 * 3 * 512;
constexpr int C_SMEM_ALONE = 120 * 1024;
static_assert(2 * (C_SMEM + 1024) <= 228 * 1024, "two CTAs per SM");

// Named barriers: one per group of four warps, and full / empty pairs for the hand-over of a chunk's
// S0 and delta pieces from the chain group to the output group.
constexpr int C_BAR_CHAIN = 1, C_BAR_OUT = 2, C_BAR_FULL = 3, C_BAR_EMPTY = 5;
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }

// D = A * B.
__device__ __forceinline__ void mma_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// d0 + d1 (+)= A * B with A and B given as three pieces each: the six pairs of pieces above 2^-24.
template <bool FIRST>
__device__ __forceinline__ void mma_6(float (&d0)[4], float (&d1)[4], const uint32_t (&A)[3][4], const uint2 (&B)[3]) {
  if (FIRST) {
    mma_zero(d0, A[0], B[0].x, B[0].y);
    mma_zero(d1, A[1], B[0].x, B[0].y);
  } else {
    ako::mma_bf16_16816(d0, A[0], B[0].x, B[0].y);
    ako::mma_bf16_16816(d1, A[1], B[0].x, B[0].y);
  }
  ako::mma_bf16_16816(d0, A[0], B[1].x, B[1].y);
  ako::mma_bf16_16816(d1, A[2], B[0].x, B[0].y);
  ako::mma_bf16_16816(d0, A[1], B[1].x, B[1].y);
  ako::mma_bf16_16816(d1, A[0], B[2].x, B[2].y);
}
// The same over the first 8 of the 16 tokens: the last step of an even tile, where the other 8 come after
// every token of the tile.
__device__ __forceinline__ void mma_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b));
}
__device__ __forceinline__ void mma_6_half(float (&d0)[4], float (&d1)[4], const uint32_t (&A)[3][4], const uint2 (&B)[3]) {
  mma_k8(d0, A[0][0], A[0][1], B[0].x);
  mma_k8(d1, A[1][0], A[1][1], B[0].x);
  mma_k8(d0, A[0][0], A[0][1], B[1].x);
  mma_k8(d1, A[2][0], A[2][1], B[0].x);
  mma_k8(d0, A[1][0], A[1][1], B[1].x);
  mma_k8(d1, A[0][0], A[0][1], B[2].x);
}
// The A fragments (16 rows x 16 tokens, three pieces) of two neighbouring token tiles.
__device__ __forceinline__ void frag_pieces(uint32_t (&A)[3][4], const uint2* src) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const uint2 x = src[p * 128], y = src[p * 128 + 32];
    A[p][0] = x.x; A[p][1] = x.y; A[p][2] = y.x; A[p][3] = y.y;
  }
}
// ---- values that are not finite ----
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }
__device__ __forceinline__ float not_finite_sum(const float (&x)[4]) {   // 0, or NaN where one of them is not finite
  return fmaf(x[0], 0.f, fmaf(x[1], 0.f, fmaf(x[2], 0.f, x[3] * 0.f)));
}
// Sign bits of the halves of a bf16 pair that are not finite.
__device__ __forceinline__ uint32_t not_finite_pair(uint32_t u) { return ((u & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }
// Of a 16 x 8 tile (lane (g, t): tokens 2t, 2t + 1 of row g and of row g + 8), given as leading pieces: the
// tokens in front of a row's first one that is not finite, as masks of the lane's two pairs.
__device__ __forceinline__ void keep_before(uint32_t lead0, uint32_t lead1, int t, uint32_t& keep0, uint32_t& keep1) {
  const uint32_t b0 = not_finite_pair(lead0), b1 = not_finite_pair(lead1);
  int f0 = (b0 & 0x8000u) ? 2 * t : b0 ? 2 * t + 1 : 8, f1 = (b1 & 0x8000u) ? 2 * t : b1 ? 2 * t + 1 : 8;
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    f0 = min(f0, __shfl_xor_sync(0xffffffffu, f0, o));
    f1 = min(f1, __shfl_xor_sync(0xffffffffu, f1, o));
  }
  keep0 = (2 * t < f0 ? 0xffffu : 0u) | (2 * t + 1 < f0 ? 0xffff0000u : 0u);
  keep1 = (2 * t < f1 ? 0xffffu : 0u) | (2 * t + 1 < f1 ? 0xffff0000u : 0u);
}
// The other tokens become NaN.
__device__ __forceinline__ void spoil(float (&x)[4], uint32_t keep0, uint32_t keep1) {
  const float nan = __uint_as_float(0x7fffffffu);
  if (!(keep0 & 0xffffu)) x[0] = nan;
  if (!(keep0 >> 16)) x[1] = nan;
  if (!(keep1 & 0xffffu)) x[2] = nan;
  if (!(keep1 >> 16)) x[3] = nan;
}

// A group's 128 threads copy `bytes` (a multiple of 16, at most 3 x 2 KB) to shared memory.
template <int BYTES>
__device__ __forceinline__ void copy_group(uint32_t dst, const unsigned char* src, int tid) {
#pragma unroll
  for (int i = 0; i < BYTES / 2048; ++i) ako::cp_async16(dst + (i * 128 + tid) * 16, src + (i * 128 + tid) * 16);
  if (BYTES % 2048 != 0 && tid < (BYTES % 2048) / 16)
    ako::cp_async16(dst + BYTES / 2048 * 2048 + tid * 16, src + BYTES / 2048 * 2048 + tid * 16);
}
// A warp's 32 columns of a chunk's k (or q) rows: 64-byte rows, 16-byte pieces XOR (row / 2). `src` is the
// lane's piece of row lane / 4, `left` the sequence's tokens from that row on; rows past the end are zero.
__device__ __forceinline__ void copy_rows(uint32_t dst, const __nv_bfloat16* src, int left, const __nv_bfloat16* safe) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool valid = 8 * i < left;
    ako::cp_async16(dst + i * 512, valid ? src + i * (8 * P_HQ * P_D) : safe, valid);
  }
}
// B fragments (k = 32 columns, n = 8 tokens) of token tile `tile`: two 16-column steps.
__device__ __forceinline__ void load_token_tile(uint32_t (&bf)[4], uint32_t base, int tile, int lane) {
  const int row = 8 * tile + (lane & 7);
  ako::ldmatrix_x4(bf[0], bf[1], bf[2], bf[3], base + row * 64 + (((lane >> 3) ^ ((row >> 1) & 3)) << 4));
}
// acc[n] = (S0 pieces of this warp's 32 columns) x (token tile (w + n) mod 4), small pieces first; the three tiles that other
// warps finish go to shared memory, tile w itself is accumulator 0.
__device__ __forceinline__ void partial_products(float (&own)[4], const uint32_t (&As)[2][3][4], uint32_t base, float4* part,
                                                 int w, int lane) {
  float acc[4][4];
  uint32_t bf[4][4];
#pragma unroll
  for (int n = 0; n < 4; ++n) load_token_tile(bf[n], base, (w + n) & 3, lane);
#pragma unroll
  for (int n = 0; n < 4; ++n) mma_zero(acc[n], As[0][2], bf[n][0], bf[n][1]);
#pragma unroll
  for (int n = 0; n < 4; ++n) ako::mma_bf16_16816(acc[n], As[1][2], bf[n][2], bf[n][3]);
#pragma unroll
  for (int p = 1; p >= 0; --p)
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int n = 0; n < 4; ++n) ako::mma_bf16_16816(acc[n], As[s][p], bf[n][2 * s], bf[n][2 * s + 1]);
#pragma unroll
  for (int n = 1; n < 4; ++n)
    part[(((w + n) & 3) * 3 + n - 1) * 32 + lane] = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) own[i] = acc[0][i];
}
__device__ __forceinline__ void add_partials(float (&own)[4], const float4* part, int w, int lane) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const float4 x = part[(w * 3 + p) * 32 + lane];
    own[0] += x.x; own[1] += x.y; own[2] += x.z; own[3] += x.w;
  }
}
// A tile of 16 rows x 8 tokens (an mma accumulator) as three exact pieces: half an A fragment.
__device__ __forceinline__ void store_pieces(uint2* dst, const float (&x)[4]) {
  uint32_t f[3][2];
  split3_exact(x[0], x[1], f[0][0], f[1][0], f[2][0]);
  split3_exact(x[2], x[3], f[0][1], f[1][1], f[2][1]);
#pragma unroll
  for (int p = 0; p < 3; ++p) dst[p * 128] = make_uint2(f[p][0], f[p][1]);
}
// d0 + d1 (+)= (pieces of token tiles 0 .. w) x (tile w of T or P): one or two 16-token steps. Of tile w itself
// only the tokens that keep0 and keep1 hold are taken in (`spoilt`, warp-uniform: not all of them). The
// caller makes the masks ahead, off its serial chain: a vote between these loads and products cost 5 %.
template <bool FIRST>
__device__ __forceinline__ void triangular_tile(float (&d0)[4], float (&d1)[4], const uint2* pieces, const uint2* frag, int w,
                                                bool spoilt, uint32_t keep0, uint32_t keep1) {
  uint32_t A[3][4];
  uint2 B[3];
  if (w >= 2) {
    frag_pieces(A, pieces);
    B[0] = frag[0]; B[1] = frag[32]; B[2] = frag[64];
    mma_6<FIRST>(d0, d1, A, B);
    pieces += 64;
    frag += 96;
  } else if (FIRST) {
#pragma unroll
    for (int i = 0; i < 4; ++i) d0[i] = d1[i] = 0.f;
  }
  frag_pieces(A, pieces);
  B[0] = frag[0]; B[1] = frag[32]; B[2] = frag[64];
  if (w & 1) {
    if (spoilt) {
#pragma unroll
      for (int p = 0; p < 3; ++p) { A[p][2] &= keep0; A[p][3] &= keep1; }
    }
    mma_6<false>(d0, d1, A, B);
  } else {
    if (spoilt) {
#pragma unroll
      for (int p = 0; p < 3; ++p) { A[p][0] &= keep0; A[p][1] &= keep1; }
    }
    mma_6_half(d0, d1, A, B);
  }
}

__global__ void __launch_bounds__(2 * C_WARPS * 32, 2) gdn_chunk_kernel(
    const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
    const float* __restrict__ state, const int64_t* __restrict__ cu_seqlens, int64_t total_tokens, float scale,
    __nv_bfloat16* __restrict__ out, float* __restrict__ new_state, const unsigned char* __restrict__ ws) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int GROUP = C_WARPS * 32;
  const int tid = threadIdx.x & (GROUP - 1), lane = tid & 31, w = tid >> 5;
  const bool chain = threadIdx.x < GROUP;
  const int slice = blockIdx.x, h = blockIdx.y, seq = blockIdx.z;
  const int hq = h / (P_HV / P_HQ);
  const int g = lane >> 2, t = lane & 3;
  const int64_t t0 = cu_seqlens[seq], t1 = cu_seqlens[seq + 1];
  const int len = (int)(t1 - t0);
  const int chunks = (len > 0) ? (len + C_TOK - 1) / C_TOK : 0;
  const uint32_t sm = ako::smem_u32(smem);
  const int ft = gdn_frag_tile(w, 0) * 96 + lane;   // its first fragment
  const unsigned char* slot = ws + (gdn_chunk_slot(t0, seq, 0) * P_HV + h) * C_SLOT_BYTES;
  const int64_t kq_off = ((t0 + g) * P_HQ + hq) * P_D + 32 * w + 8 * t;
  const uint32_t kq_dst = w * C_KQ_WARP + g * 64 + ((t ^ ((g >> 1) & 3)) << 4);

  if (chain) {
    // the warp's part of the state: rows g, g + 8, columns 32 w + 8 n + 2 t, + 1
    const int64_t srow = (((int64_t)seq * P_HV + h) * P_D + slice * C_ROWS + g) * P_D + 32 * w + 2 * t;
    float S[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      float2 x = make_float2(0.f, 0.f), y = x;
      if (state != nullptr && len > 0) {   // the definition leaves the new state of an empty sequence at zero
        x = __ldcs(reinterpret_cast<const float2*>(state + srow + 8 * n));
        y = __ldcs(reinterpret_cast<const float2*>(state + srow + 8 * P_D + 8 * n));
      }
      S[n][0] = x.x; S[n][1] = x.y; S[n][2] = y.x; S[n][3] = y.y;
    }
    const __nv_bfloat16* kp = k + kq_off;
    const __nv_bfloat16* vp = v + ((t0 + (tid >> 1)) * P_HV + h) * P_D + slice * C_ROWS + (tid & 1) * 8;
    auto load_k = [&](int c) {
      copy_rows(sm + (c & 1) * C_CH_STAGE + kq_dst, kp, len - c * C_TOK - g, k);
      kp += C_TOK * P_HQ * P_D;
    };
    auto load_rest = [&](int c) {   // T, coefficients, v
      const uint32_t st = sm + (c & 1) * C_CH_STAGE;
      copy_group<C_FRAG_BYTES>(st + C_CH_SLOT, slot, tid);
      if (tid < C_COEF_FLOATS / 4) ako::cp_async16(st + C_CH_COEF + tid * 16, slot + 2 * C_FRAG_BYTES + tid * 16);
      slot += P_HV * C_SLOT_BYTES;
      if (tid < 2 * C_TOK) {
        const bool valid = c * C_TOK + (tid >> 1) < len;
        ako::cp_async16(st + C_CH_V + tid * 16, valid ? vp : v, valid);
        vp += C_TOK * P_HV * P_D;
      }
    };
    if (chunks > 0) load_k(0);
    ako::pdl_wait();   // T, P and the coefficients come from the kernel in front
    if (chunks > 0) load_rest(0);
    ako::cp_async_commit();

    float4* sX = reinterpret_cast<float4*>(smem + C_OFF_X);
    uint2* sR = reinterpret_cast<uint2*>(smem + C_OFF_R) + lane;
    uint2* sE = reinterpret_cast<uint2*>(smem + C_OFF_E) + lane;
    for (int c = 0; c < chunks; ++c) {
      const int b = c & 1;
      if (c + 1 < chunks) load_k(c + 1);
      ako::cp_async_commit();
      // A fragments of S (its accumulators as they lie), three exact pieces
      uint32_t As[2][3][4];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          split3_exact(S[2 * s + (i >> 1)][2 * (i & 1)], S[2 * s + (i >> 1)][2 * (i & 1) + 1], As[s][0][i], As[s][1][i], As[s][2][i]);
      ako::cp_async_wait<1>();
      __syncwarp();
      const uint32_t kbase = sm + b * C_CH_STAGE + w * C_KQ_WARP;
      const unsigned char* stage = smem + b * C_CH_STAGE;
      const float* coef = reinterpret_cast<const float*>(stage + C_CH_COEF);

      // 1. this warp's part of S0 k; the output group gets the pieces of S0
      float x[4];
      partial_products(x, As, kbase, sX, w, lane);
      if (c >= 2) bar_sync(C_BAR_EMPTY + b, 2 * GROUP);
      {
        uint4* dst = reinterpret_cast<uint4*>(smem + C_OFF_S + b * C_S_BYTES) + w * 192 + lane;
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int p = 0; p < 3; ++p) dst[(s * 3 + p) * 32] = make_uint4(As[s][p][0], As[s][p][1], As[s][p][2], As[s][p][3]);
      }
      bar_sync(C_BAR_CHAIN, GROUP);   // the partial sums, and everybody's part of T, coefficients and v
      if (c + 1 < chunks) load_rest(c + 1);   // no warp reads the other stage any more
      ako::cp_async_commit();

      // 2. right-hand side of tile w: v - gam (S0 k), as pieces for the group
      add_partials(x, sX, w, lane);
      bool spoilt;
      uint32_t keep0 = ~0u, keep1 = ~0u;
      float r[4];
      {
        const float2 gam = *reinterpret_cast<const float2*>(coef + 8 * w + 2 * t);
        const __nv_bfloat16* vv = reinterpret_cast<const __nv_bfloat16*>(stage + C_CH_V) + (8 * w + 2 * t) * C_ROWS + g;
        r[0] = __bfloat162float(vv[0]) - gam.x * x[0];
        r[1] = __bfloat162float(vv[C_ROWS]) - gam.y * x[1];
        r[2] = __bfloat162float(vv[8]) - gam.x * x[2];
        r[3] = __bfloat162float(vv[C_ROWS + 8]) - gam.y * x[3];
        store_pieces(sR + w * 32, r);
        spoilt = __any_sync(0xffffffffu, !(not_finite_sum(r) == 0.f));
        if (spoilt)
          keep_before(__byte_perm(__float_as_uint(r[0]), __float_as_uint(r[1]), 0x7632),
                      __byte_perm(__float_as_uint(r[2]), __float_as_uint(r[3]), 0x7632), t, keep0, keep1);
      }
      const float gC = coef[C_TOK - 1];
      const float2 dec = *reinterpret_cast<const float2*>(coef + C_TOK + 8 * w + 2 * t);
      const float2 beta = *reinterpret_cast<const float2*>(coef + 2 * C_TOK + 8 * w + 2 * t);
      bar_sync(C_BAR_CHAIN, GROUP);

      // 3. delta of tile w = T (right-hand side)
      float d0[4], d1[4];
      triangular_tile<true>(d0, d1, sR, reinterpret_cast<const uint2*>(stage + C_CH_SLOT) + ft, w, spoilt, keep0, keep1);
#pragma unroll
      for (int i = 0; i < 4; ++i) d0[i] = fmaf((i & 1) ? beta.y : beta.x, r[i], d0[i] + d1[i]);
      if (spoilt) spoil(d0, keep0, keep1);
      {
        const float e[4] = {d0[0] * dec.x, d0[1] * dec.y, d0[2] * dec.x, d0[3] * dec.y};
        store_pieces(sE + w * 32, e);
      }
      bar_sync(C_BAR_CHAIN, GROUP);
      store_pieces(reinterpret_cast<uint2*>(smem + C_OFF_D + b * C_D_BYTES) + lane + w * 32, d0);
      bar_arrive(C_BAR_FULL + b, 2 * GROUP);

      // 4. the state at the end of the chunk, 16 columns at a time; the leading pieces last
      uint32_t A[2][3][4];
      frag_pieces(A[0], sE);
      frag_pieces(A[1], sE + 64);
#pragma unroll
      for (int n0 = 0; n0 < 4; n0 += 2) {
        uint32_t bf[2][4];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int row = 16 * s + (lane & 15);
          ako::ldmatrix_x4_trans(bf[s][0], bf[s][1], bf[s][2], bf[s][3],
                                 kbase + row * 64 + (((n0 + (lane >> 4)) ^ ((row >> 1) & 3)) << 4));
        }
        float U[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_zero(U[n], A[0][2], bf[0][2 * n], bf[0][2 * n + 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) ako::mma_bf16_16816(U[n], A[1][2], bf[1][2 * n], bf[1][2 * n + 1]);
#pragma unroll
        for (int p = 1; p >= 0; --p)
#pragma unroll
          for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int n = 0; n < 2; ++n) ako::mma_bf16_16816(U[n], A[s][p], bf[s][2 * n], bf[s][2 * n + 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) S[n0 + n][i] = fmaf(gC, S[n0 + n][i], U[n][i]);
      }
      __syncwarp();   // the warp's k of this chunk is read: the next load may overwrite it
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      __stcs(reinterpret_cast<float2*>(new_state + srow + 8 * n), make_float2(S[n][0], S[n][1]));
      __stcs(reinterpret_cast<float2*>(new_state + srow + 8 * P_D + 8 * n), make_float2(S[n][2], S[n][3]));
    }
  } else {
    __nv_bfloat16* out_h = out + h * P_D + slice * C_ROWS;
    const __nv_bfloat16* qp = q + kq_off;
    auto load = [&](int c) {   // q, P, coefficients
      const uint32_t st = sm + C_OFF_OUT + (c & 1) * C_OUT_STAGE;
      copy_rows(st + kq_dst, qp, len - c * C_TOK - g, q);
      qp += C_TOK * P_HQ * P_D;
      copy_group<C_FRAG_BYTES + C_COEF_FLOATS * 4>(st + C_OUT_SLOT, slot + C_FRAG_BYTES, tid);
      slot += P_HV * C_SLOT_BYTES;
      ako::cp_async_commit();
    };
    ako::pdl_wait();
    if (chunks > 0) load(0);
    // tokens outside every sequence: zero, by the CTAs of the first and of the last sequence
    for (int side = 0; side < 2; ++side) {
      if (seq != (side ? (int)gridDim.z - 1 : 0)) continue;
      const int64_t z0 = side ? max(t1, (int64_t)0) : 0, z1 = side ? total_tokens : min(t0, total_tokens);
      for (int64_t i = z0 * 2 + tid; i < z1 * 2; i += GROUP)
        *reinterpret_cast<uint4*>(out_h + (i >> 1) * (P_HV * P_D) + (i & 1) * 8) = make_uint4(0u, 0u, 0u, 0u);
    }
    float4* sY = reinterpret_cast<float4*>(smem + C_OFF_Y);
    out_h += t0 * (P_HV * P_D);
    for (int c = 0; c < chunks; ++c) {
      const int b = c & 1;
      bar_sync(C_BAR_FULL + b, 2 * GROUP);     // S0 and delta of chunk c; the group is done with chunk c - 1
      if (c + 1 < chunks) load(c + 1);
      else ako::cp_async_commit();
      uint32_t As[2][3][4];
      {
        const uint4* src = reinterpret_cast<const uint4*>(smem + C_OFF_S + b * C_S_BYTES) + w * 192 + lane;
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            const uint4 f = src[(s * 3 + p) * 32];
            As[s][p][0] = f.x; As[s][p][1] = f.y; As[s][p][2] = f.z; As[s][p][3] = f.w;
          }
      }
      ako::cp_async_wait<1>();
      __syncwarp();
      const unsigned char* stage = smem + C_OFF_OUT + b * C_OUT_STAGE;
      float y[4];
      partial_products(y, As, sm + C_OFF_OUT + b * C_OUT_STAGE + w * C_KQ_WARP, sY, w, lane);
      bar_sync(C_BAR_OUT, GROUP);
      add_partials(y, sY, w, lane);
      const float2 gam = *reinterpret_cast<const float2*>(reinterpret_cast<const float*>(stage + C_OUT_COEF) + 8 * w + 2 * t);
      float o0[4] = {scale * gam.x * y[0], scale * gam.y * y[1], scale * gam.x * y[2], scale * gam.y * y[3]};
      float o1[4] = {0.f, 0.f, 0.f, 0.f};
      const uint2 own = (reinterpret_cast<const uint2*>(smem + C_OFF_D + b * C_D_BYTES) + lane)[w * 32];   // leading pieces of tile w
      const bool spoilt = __any_sync(0xffffffffu, (not_finite_pair(own.x) | not_finite_pair(own.y)) != 0u);
      uint32_t keep0 = ~0u, keep1 = ~0u;
      if (spoilt) keep_before(own.x, own.y, t, keep0, keep1);
      triangular_tile<false>(o0, o1, reinterpret_cast<const uint2*>(smem + C_OFF_D + b * C_D_BYTES) + lane,
                             reinterpret_cast<const uint2*>(stage + C_OUT_SLOT) + ft, w, spoilt, keep0, keep1);
      if (spoilt) spoil(o0, keep0, keep1);
      if (c + 2 < chunks) bar_arrive(C_BAR_EMPTY + b, 2 * GROUP);
      // transposed across the warp: lane (g, t) gets token g, rows 2t, 2t+1 (and + 8)
      const uint32_t y0 = ako::movmatrix_trans(ako::pack_bf16x2(o0[0] + o1[0], o0[1] + o1[1]));
      const uint32_t y1 = ako::movmatrix_trans(ako::pack_bf16x2(o0[2] + o1[2], o0[3] + o1[3]));
      if (c * C_TOK + 8 * w + g < len) {
        uint32_t* op = reinterpret_cast<uint32_t*>(out_h + (int64_t)(c * C_TOK + 8 * w + g) * (P_HV * P_D)) + t;
        op[0] = y0;
        op[4] = y1;
      }
    }
  }
}

// ---- the same recurrence, one warp per 16 state rows ----------------------------------------------
// With enough sequences to fill the GPU the exchanges between warps are what costs: here a warp holds
// all 128 columns of its 16 rows, so that a chunk needs no exchange at all (everything from S0 k to the
// new S stays in its registers) and the CTA's four warps (64 rows) only share the loads: 264 LSU
// wavefronts per 16 rows and chunk instead of 1 130, 360 mma in a row instead of 96. Bound by the tensor
// pipe (2 950 cycles of a sub-partition per chunk and warp; ncu: 58 %) where at least two warps share one.
// 64 x 128 tokens: 86 us against 128 with the kernel above and 499 token by token.
constexpr int CW_ROWS = 64;
constexpr int CW_V_PITCH = CW_ROWS * 2 + 16;                          // ldmatrix of eight rows: no bank conflict
constexpr int CW_OFF_Q = C_TOK * 256;                                 // stage: k | q | T, P, coefficients | v
constexpr int CW_OFF_SLOT = 2 * C_TOK * 256;
constexpr int CW_OFF_V = CW_OFF_SLOT + C_SLOT_BYTES;
constexpr int CW_STAGE = CW_OFF_V + C_TOK * CW_V_PITCH;
constexpr int CW_SMEM = 2 * CW_STAGE;
static_assert(CW_STAGE % 128 == 0 && 3 * (CW_SMEM + 1024) <= 228 * 1024, "three CTAs per SM");

// Pieces of a 16 x 8 accumulator tile: half of the A fragment of a 16-token step.
__device__ __forceinline__ void tile_pieces(uint32_t (&A)[3][4], int half, const float (&x)[4]) {
  split3_exact(x[0], x[1], A[0][2 * half], A[1][2 * half], A[2][2 * half]);
  split3_exact(x[2], x[3], A[0][2 * half + 1], A[1][2 * half + 1], A[2][2 * half + 1]);
}

__device__ __forceinline__ bool wide_not_finite(const float (&x)[4][4]) {
  const float z = (not_finite_sum(x[0]) + not_finite_sum(x[1])) + (not_finite_sum(x[2]) + not_finite_sum(x[3]));
  return __any_sync(0xffffffffu, !(z == 0.f));
}
// Moves f0 and f1 (rows g, g + 8) up to the row's first token that is not finite.
__device__ __forceinline__ void wide_first_not_finite(const float (&x)[4][4], int& f0, int& f1, int t) {
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (not_finite(x[n][i])) f0 = min(f0, 8 * n + 2 * t + i);
      if (not_finite(x[n][2 + i])) f1 = min(f1, 8 * n + 2 * t + i);
    }
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    f0 = min(f0, __shfl_xor_sync(0xffffffffu, f0, o));
    f1 = min(f1, __shfl_xor_sync(0xffffffffu, f1, o));
  }
}
// Sets the tokens from f0 (f1) on to `value`.
__device__ __forceinline__ void wide_set(float (&x)[4][4], float value, int f0, int f1, int t) {
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (8 * n + 2 * t + i >= f0) x[n][i] = value;
      if (8 * n + 2 * t + i >= f1) x[n][2 + i] = value;
    }
}

__global__ void __launch_bounds__(128, 3) gdn_chunk_wide_kernel(
    const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
    const float* __restrict__ state, const int64_t* __restrict__ cu_seqlens, int64_t total_tokens, float scale,
    __nv_bfloat16* __restrict__ out, float* __restrict__ new_state, const unsigned char* __restrict__ ws) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int half = blockIdx.x, h = blockIdx.y, seq = blockIdx.z;
  const int hq = h / (P_HV / P_HQ);
  const int g = lane >> 2, t = lane & 3;
  const int64_t t0 = cu_seqlens[seq], t1 = cu_seqlens[seq + 1];
  const int len = (int)(t1 - t0);
  const int chunks = (len > 0) ? (len + C_TOK - 1) / C_TOK : 0;
  const uint32_t sm = ako::smem_u32(smem);
  const unsigned char* slot = ws + (gdn_chunk_slot(t0, seq, 0) * P_HV + h) * C_SLOT_BYTES;

  // thread: 16-byte piece tid % 16 of rows tid / 16 + 8 i of k and q; of v piece tid % 8, rows tid / 8 + 16 i
  const __nv_bfloat16* kp = k + ((t0 + (tid >> 4)) * P_HQ + hq) * P_D + (tid & 15) * 8;
  const __nv_bfloat16* qp = q + ((t0 + (tid >> 4)) * P_HQ + hq) * P_D + (tid & 15) * 8;
  const __nv_bfloat16* vp = v + ((t0 + (tid >> 3)) * P_HV + h) * P_D + half * CW_ROWS + (tid & 7) * 8;
  auto load_inputs = [&](int c) {
    const uint32_t st = sm + (c & 1) * CW_STAGE;
    const int left = len - c * C_TOK;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = (tid >> 4) + 8 * i;
      const bool valid = row < left;
      const uint32_t dst = st + row * 256 + (((tid & 15) ^ (row & 7)) << 4);
      ako::cp_async16(dst, valid ? kp + i * (8 * P_HQ * P_D) : k, valid);
      ako::cp_async16(dst + CW_OFF_Q, valid ? qp + i * (8 * P_HQ * P_D) : q, valid);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = (tid >> 3) + 16 * i;
      const bool valid = row < left;
      ako::cp_async16(st + CW_OFF_V + row * CW_V_PITCH + (tid & 7) * 16, valid ? vp + i * (16 * P_HV * P_D) : v, valid);
    }
    kp += C_TOK * P_HQ * P_D;
    qp += C_TOK * P_HQ * P_D;
    vp += C_TOK * P_HV * P_D;
  };
  auto load_slot = [&](int c) {
    copy_group<C_SLOT_BYTES>(sm + (c & 1) * CW_STAGE + CW_OFF_SLOT, slot, tid);
    slot += P_HV * C_SLOT_BYTES;
  };
  if (chunks > 0) load_inputs(0);

  // the warp's rows of the state: g, g + 8 of its 16, columns 8 n + 2 t, + 1
  const int64_t srow = (((int64_t)seq * P_HV + h) * P_D + half * CW_ROWS + w * 16 + g) * P_D + 2 * t;
  float S[16][4];
#pragma unroll
  for (int n = 0; n < 16; ++n) {
    float2 x = make_float2(0.f, 0.f), y = x;
    if (state != nullptr && len > 0) {   // the definition leaves the new state of an empty sequence at zero
      x = __ldcs(reinterpret_cast<const float2*>(state + srow + 8 * n));
      y = __ldcs(reinterpret_cast<const float2*>(state + srow + 8 * P_D + 8 * n));
    }
    S[n][0] = x.x; S[n][1] = x.y; S[n][2] = y.x; S[n][3] = y.y;
  }
  __nv_bfloat16* out_h = out + h * P_D + half * CW_ROWS;
  // tokens outside every sequence: zero, by the CTAs of the first and of the last sequence
  for (int side = 0; side < 2; ++side) {
    if (seq != (side ? (int)gridDim.z - 1 : 0)) continue;
    const int64_t z0 = side ? max(t1, (int64_t)0) : 0, z1 = side ? total_tokens : min(t0, total_tokens);
    for (int64_t i = z0 * 8 + tid; i < z1 * 8; i += 128)
      *reinterpret_cast<uint4*>(out_h + (i >> 3) * (P_HV * P_D) + (i & 7) * 8) = make_uint4(0u, 0u, 0u, 0u);
  }
  out_h += t0 * (P_HV * P_D) + w * 16;
  ako::pdl_wait();   // T, P and the coefficients come from the kernel in front
  if (chunks > 0) load_slot(0);
  ako::cp_async_commit();

  for (int c = 0; c < chunks; ++c) {
    ako::cp_async_wait<0>();
    __syncthreads();               // chunk c is here; nobody reads the other stage any more
    if (c + 1 < chunks) {
      load_inputs(c + 1);
      load_slot(c + 1);
    }
    ako::cp_async_commit();
    const uint32_t st = sm + (c & 1) * CW_STAGE;
    const unsigned char* stage = smem + (c & 1) * CW_STAGE;
    const uint2* sT = reinterpret_cast<const uint2*>(stage + CW_OFF_SLOT) + lane;
    const uint2* sP = sT + C_FRAG_BYTES / 8;
    const float* coef = reinterpret_cast<const float*>(stage + CW_OFF_SLOT + 2 * C_FRAG_BYTES);

    // 1. S0 k and S0 q, four token tiles each
    float x[4][4], y[4][4];
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t As[3][4], bk[8], bq[8];
      tile_pieces(As, 0, S[2 * ks]);
      tile_pieces(As, 1, S[2 * ks + 1]);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int row = p * 16 + (lane & 7) + ((lane >> 4) << 3);
        const uint32_t a = st + row * 256 + (((2 * ks + ((lane >> 3) & 1)) ^ (row & 7)) << 4);
        ako::ldmatrix_x4(bk[4 * p], bk[4 * p + 1], bk[4 * p + 2], bk[4 * p + 3], a);
        ako::ldmatrix_x4(bq[4 * p], bq[4 * p + 1], bq[4 * p + 2], bq[4 * p + 3], a + CW_OFF_Q);
      }
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          if (ks == 0 && p == 0) {
            mma_zero(x[n], As[0], bk[2 * n], bk[2 * n + 1]);
            mma_zero(y[n], As[0], bq[2 * n], bq[2 * n + 1]);
          } else {
            ako::mma_bf16_16816(x[n], As[p], bk[2 * n], bk[2 * n + 1]);
            ako::mma_bf16_16816(y[n], As[p], bq[2 * n], bq[2 * n + 1]);
          }
        }
    }
    // 2. right-hand side v - gam (S0 k), and what S0 adds to the outputs
#pragma unroll
    for (int m = 0; m < 4; m += 2) {
      uint32_t vt[4];                  // tokens 8 m .., rows 0-7 and 8-15; then tokens 8 m + 8 ..
      ako::ldmatrix_x4_trans(vt[0], vt[1], vt[2], vt[3],
                             st + CW_OFF_V + (8 * m + (lane & 7) + ((lane >> 4) << 3)) * CW_V_PITCH + w * 32 + ((lane >> 3) & 1) * 16);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 gam = *reinterpret_cast<const float2*>(coef + 8 * (m + u) + 2 * t);
        float(&xr)[4] = x[m + u];
        float(&yr)[4] = y[m + u];
        xr[0] = ako::bf16_lo(vt[2 * u]) - gam.x * xr[0];
        xr[1] = ako::bf16_hi(vt[2 * u]) - gam.y * xr[1];
        xr[2] = ako::bf16_lo(vt[2 * u + 1]) - gam.x * xr[2];
        xr[3] = ako::bf16_hi(vt[2 * u + 1]) - gam.y * xr[3];
        yr[0] *= scale * gam.x; yr[1] *= scale * gam.y; yr[2] *= scale * gam.x; yr[3] *= scale * gam.y;
      }
    }
    // the first token of rows g and g + 8 that is not finite; it and later ones are left out of the products
    int f0 = C_TOK, f1 = C_TOK;
    bool spoilt = wide_not_finite(x);
    if (spoilt) {
      wide_first_not_finite(x, f0, f1, t);
      wide_set(x, 0.f, f0, f1, t);
    }
    // 3. delta = T (right-hand side), tile by tile
    float d[4][4];
    {
      uint32_t A[2][3][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) tile_pieces(A[n >> 1], n & 1, x[n]);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        float d1[4];
        if (n == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) d[n][i] = d1[i] = 0.f;
        }
#pragma unroll
        for (int s = 0; s <= n / 2; ++s) {
          const uint2* f = sT + gdn_frag_tile(n, s) * 96;
          const uint2 B[3] = {f[0], f[32], f[64]};
          if (s == n / 2 && n % 2 == 0) mma_6_half(d[n], d1, A[s], B);
          else if (s == 0) mma_6<true>(d[n], d1, A[s], B);
          else mma_6<false>(d[n], d1, A[s], B);
        }
        const float2 beta = *reinterpret_cast<const float2*>(coef + 2 * C_TOK + 8 * n + 2 * t);
#pragma unroll
        for (int i = 0; i < 4; ++i) d[n][i] = fmaf((i & 1) ? beta.y : beta.x, x[n][i], d[n][i] + d1[i]);
      }
    }
    if (wide_not_finite(d)) spoilt = true;   // also an overflow
    // 4. outputs
    const float nan = __uint_as_float(0x7fffffffu);
    if (spoilt) {
      wide_first_not_finite(d, f0, f1, t);
      wide_set(d, 0.f, f0, f1, t);
      wide_set(y, nan, f0, f1, t);
    }
    {
      uint32_t A[2][3][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) tile_pieces(A[n >> 1], n & 1, d[n]);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        float o1[4];
        if (n == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) o1[i] = 0.f;
        }
#pragma unroll
        for (int s = 0; s <= n / 2; ++s) {
          const uint2* f = sP + gdn_frag_tile(n, s) * 96;
          const uint2 B[3] = {f[0], f[32], f[64]};
          if (s == n / 2 && n % 2 == 0) {
            mma_6_half(y[n], o1, A[s], B);
          } else if (s == 0) {
            ako::mma_bf16_16816(y[n], A[0][0], B[0].x, B[0].y);
            mma_zero(o1, A[0][1], B[0].x, B[0].y);
            ako::mma_bf16_16816(y[n], A[0][0], B[1].x, B[1].y);
            ako::mma_bf16_16816(o1, A[0][2], B[0].x, B[0].y);
            ako::mma_bf16_16816(y[n], A[0][1], B[1].x, B[1].y);
            ako::mma_bf16_16816(o1, A[0][0], B[2].x, B[2].y);
          } else {
            mma_6<false>(y[n], o1, A[s], B);
          }
        }
        // transposed across the warp: lane (g, t) gets token g, rows 2t, 2t+1 (and + 8)
        const uint32_t y0 = ako::movmatrix_trans(ako::pack_bf16x2(y[n][0] + o1[0], y[n][1] + o1[1]));
        const uint32_t y1 = ako::movmatrix_trans(ako::pack_bf16x2(y[n][2] + o1[2], y[n][3] + o1[3]));
        if (c * C_TOK + 8 * n + g < len) {
          uint32_t* op = reinterpret_cast<uint32_t*>(out_h + (int64_t)(c * C_TOK + 8 * n + g) * (P_HV * P_D)) + t;
          op[0] = y0;
          op[4] = y1;
        }
      }
    }
    // 5. the state at the end of the chunk
    {
      uint32_t A[2][3][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float2 dec = *reinterpret_cast<const float2*>(coef + C_TOK + 8 * n + 2 * t);
        const float e[4] = {d[n][0] * dec.x, d[n][1] * dec.y, d[n][2] * dec.x, d[n][3] * dec.y};
        tile_pieces(A[n >> 1], n & 1, e);
      }
      const float gC = coef[C_TOK - 1], g0 = (spoilt && f0 < C_TOK) ? nan : gC, g1 = (spoilt && f1 < C_TOK) ? nan : gC;
#pragma unroll
      for (int n = 0; n < 16; n += 2) {
        uint32_t bf[2][4];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int row = 16 * s + (lane & 15);
          ako::ldmatrix_x4_trans(bf[s][0], bf[s][1], bf[s][2], bf[s][3], st + row * 256 + (((n + (lane >> 4)) ^ (row & 7)) << 4));
        }
        float U[2][4];
        mma_zero(U[0], A[0][2], bf[0][0], bf[0][1]);
        mma_zero(U[1], A[0][2], bf[0][2], bf[0][3]);
        ako::mma_bf16_16816(U[0], A[1][2], bf[1][0], bf[1][1]);
        ako::mma_bf16_16816(U[1], A[1][2], bf[1][2], bf[1][3]);
#pragma unroll
        for (int p = 1; p >= 0; --p)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            ako::mma_bf16_16816(U[0], A[s][p], bf[s][0], bf[s][1]);
            ako::mma_bf16_16816(U[1], A[s][p], bf[s][2], bf[s][3]);
          }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          S[n][i] = fmaf((i < 2) ? g0 : g1, S[n][i], U[0][i]);
          S[n + 1][i] = fmaf((i < 2) ? g0 : g1, S[n + 1][i], U[1][i]);
        }
      }
    }
  }
#pragma unroll
  for (int n = 0; n < 16; ++n) {
    __stcs(reinterpret_cast<float2*>(new_state + srow + 8 * n), make_float2(S[n][0], S[n][1]));
    __stcs(reinterpret_cast<float2*>(new_state + srow + 8 * P_D + 8 * n), make_float2(S[n][2], S[n][3]));
  }
}
