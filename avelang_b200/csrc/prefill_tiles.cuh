// Pass 1 of the chunked prefill (d_k = d_v = 128): per (chunk, value head) the record that the scan reads.
//     A = strict_lower(beta_i e^{b_i-b_j} k_i.k_j)    Tu = (I + A)^-1 diag(beta)    P = scale lower(e^{b_i-b_j} q_i.k_j)
// Tu and P leave as bf16 hi + lo, lower triangles of 16x16 blocks only, in the layout the scan's MMAs read (see REC_* in prefill_tc.cu):
// 8x8 core matrices of 128 contiguous bytes, which is an accumulator fragment of a warp, register by register, so that the
// tiles go from the accumulators straight to global memory in full 128-byte lines, without staging, barriers or copies.
//
// Persistent CTAs of ten warps, two per SM; a unit is (chunk, key head, up to two of its value heads).  Two warps work a unit ahead, so
// that the other eight never wait for memory: one looks the chunk up (32 units at a time, one a lane), brings K and Q into shared
// memory and has the Gram products [K; Q] K^T formed by eight tcgen05 MMAs into one of two accumulators; the other forms
// the gate sums, the row norms and the per-token factors.
//
// Four warps a value head and one meeting of the four a unit.  Rows of K and Q alternate in groups of eight in the A tile, K's 16-row
// blocks in rising order and Q's in falling order, so that quarter q of the tensor-memory lanes holds block row q of K K^T and
// 3 - q of Q K^T (five blocks of the two triangles for every warp) and the loads return them as accumulator fragments of
// warp-level MMAs.  They are gated in place.  Off the diagonal blocks the gate factors into e^{b_i - b_s} e^{b_s - b_j} with b_s
// the first gate of i's block (both exponents are <= 0); the diagonal blocks take e^{b_i - b_j} element by element and drop
// the half above the diagonal, where the exponent is positive.  Each warp inverts its diagonal block I + A_qq; then T = (I + A)^-1 is
// formed by forward substitution over blocks, eight columns a warp (the columns are independent, so nobody waits for
// another's part; by block rows the last row took 6.3 k cycles while three warps waited), fp32 operands as three bf16 terms.
//
// 132 k (chunk, head) units of a packed batch 1.31 ms, 2.87 when a CTA took one unit with all loads, lookups and Gram products in
// line (6.3 and 2.8 of 21 k cycles) and formed W = T diag(beta e^b) K as well (5 k).  A unit takes 10 k cycles now; 5.0 k warp
// instructions a chunk-head at 0.47 per scheduler-cycle, bound by the latency of dependent steps at five warps a scheduler.
#pragma once
#include "wyblocks.cuh"

namespace ave {
namespace {

// A fragments of a 16x16 block: three bf16 terms, each the four registers of a lane
constexpr int FR_BLOCK = 3 * 512, FR_DIAG = 6 * FR_BLOCK, FR_BYTES = FR_DIAG + 4 * FR_BLOCK;  // -A_rs at r (r - 1) / 2 + s, then D_r
static_assert(16 * AD_LD * 4 <= FR_BLOCK, "a diagonal block is inverted in the place of its fragments");
constexpr int TILES_THREADS = 320;
constexpr int TL_TILE = 0;                                   // [K; Q], two halves of 64 features, 16 groups of 8 rows: K, Q, K, Q, ...; Q's 16-row blocks in falling order
constexpr int TL_HALF = 16384;
constexpr int TL_F = 2 * TL_HALF;                            // [2 heads] fragments of A and of the inverses of its diagonal blocks
constexpr int TL_VEC = TL_F + 2 * FR_BYTES;                  // [2 units][2 heads] vectors of 64 floats
enum { TV_B, TV_BETA, TV_RA, TV_RP, TV_DA, TV_DP, TV_KN, TV_W1, TV_W2, TV_W3, TV_COUNT };
constexpr int TV_FLOATS = TV_COUNT * C;
constexpr int TL_DESC = TL_VEC + 4 * TV_FLOATS * 4;          // [2 units] chunk record (-1: no more units), first head, heads, tokens, ...
constexpr int TL_BARS = TL_DESC + 2 * 32;
constexpr size_t TILES_SMEM = TL_BARS + 128 + 1024;

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float LOG2E = 1.4426950408889634f;
// Two adjacent 8-column groups of 16 rows as accumulator fragments
__device__ __forceinline__ void tmem_ld_frag2(uint32_t taddr, float (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {  // 8x8 of 16 bits, in the register layout of a fragment
  uint32_t y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
// d += A B, A and B in three bf16 terms with those below 2^-24 left out; two accumulators halve the chain of dependent MMAs
__device__ __forceinline__ void mma_frag(float (&d0)[4], float (&d1)[4], const uint8_t* frag, int lane, const uint32_t (&b)[3][2]) {
  const uint4* f = reinterpret_cast<const uint4*>(frag) + lane;
  const uint4 h4 = f[0], m4 = f[32], l4 = f[64];
  const uint32_t h[4] = {h4.x, h4.y, h4.z, h4.w}, m[4] = {m4.x, m4.y, m4.z, m4.w}, l[4] = {l4.x, l4.y, l4.z, l4.w};
  mma_bf16(d0, h, b[0][0], b[0][1]);
  mma_bf16(d1, h, b[1][0], b[1][1]);
  mma_bf16(d0, m, b[0][0], b[0][1]);
  mma_bf16(d1, l, b[0][0], b[0][1]);
  mma_bf16(d0, h, b[2][0], b[2][1]);
  mma_bf16(d1, m, b[1][0], b[1][1]);
}
// 16 rows x 8 columns in accumulator layout -> right operand of a product over those rows, three terms
__device__ __forceinline__ void right_operand(const float (&c)[4], uint32_t (&b)[3][2]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint32_t h, m, l;
    split3(make_float2(c[2 * i], c[2 * i + 1]), h, m, l);
    b[0][i] = transpose8(h); b[1][i] = transpose8(m); b[2][i] = transpose8(l);
  }
}
// hi and lo of a 16x8 block (16-row block r, 8-column group 2 c + nt, c <= r) into their packed triangles
__device__ __forceinline__ void store_half(uint8_t* tri, int r, int c, int nt, int lane, uint32_t h0, uint32_t h1, uint32_t l0, uint32_t l1) {
  uint32_t* p = reinterpret_cast<uint32_t*>(tri + tri_step(c) + (r - c) * 512 + nt * 128) + lane;
  p[0] = h0; p[64] = h1;  // rows 0 .. 7 and 8 .. 15
  p[REC_TRI / 4] = l0; p[REC_TRI / 4 + 64] = l1;
}
// Columns 16 c + 8 nt .. + 7 of T from row block c down, by forward substitution: T_rc = D_r sum_{c <= s < r} (-A_rs) T_sc.
// The columns of a block are independent of one another, so a warp's chain is three MMAs a product long and needs no other warp.
template <int CB>
__device__ __forceinline__ void solve_columns(const uint8_t* frag, const float* vec, int nt, int lane, uint8_t* tu) {
  const float2 be = *reinterpret_cast<const float2*>(vec + TV_BETA * C + 16 * CB + 8 * nt + 2 * (lane & 3));
  auto store = [&](int r, const float (&x)[4]) {
    uint32_t h[2], l[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) split_pair(__fmul2_rn(make_float2(x[2 * i], x[2 * i + 1]), be), h[i], l[i]);
    store_half(tu, r, CB, nt, lane, h[0], h[1], l[0], l[1]);
  };
  uint32_t X[4 - CB][3][2];
  {  // T_cc = D_c
    float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 2; k >= 0; --k) {
      const uint2 w = *reinterpret_cast<const uint2*>(frag + FR_DIAG + CB * FR_BLOCK + k * 512 + lane * 16 + nt * 8);
      const float2 lo = bf16x2_to_float2(w.x), hi = bf16x2_to_float2(w.y);
      x[0] += lo.x; x[1] += lo.y; x[2] += hi.x; x[3] += hi.y;
      X[0][k][0] = transpose8(w.x); X[0][k][1] = transpose8(w.y);
    }
    store(CB, x);
  }
#pragma unroll
  for (int r = CB + 1; r < 4; ++r) {
    float y0[4], y1[4];
    zero(y0); zero(y1);
#pragma unroll
    for (int s = CB; s < r; ++s) mma_frag(y0, y1, frag + (r * (r - 1) / 2 + s) * FR_BLOCK, lane, X[s - CB]);
#pragma unroll
    for (int e = 0; e < 4; ++e) y0[e] += y1[e];
    uint32_t Y[3][2];
    right_operand(y0, Y);
    float x0[4], x1[4];
    zero(x0); zero(x1);
    mma_frag(x0, x1, frag + FR_DIAG + r * FR_BLOCK, lane, Y);
#pragma unroll
    for (int e = 0; e < 4; ++e) x0[e] += x1[e];
    if (r < 3) right_operand(x0, X[r - CB]);
    store(r, x0);
  }
}

__global__ void __launch_bounds__(TILES_THREADS, 2)
chunk_tiles_kernel(const AveGdnArgs a, const int32_t* chunk_start, uint8_t* recs, const __grid_constant__ ScanPlan plan,
                   int n_chunks, int compact_grid) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = tc::align1024(smem_raw);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // (uniform to the compiler)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TL_BARS);
  uint64_t* desc_full = bars;      // [2] the unit's description is in shared memory
  uint64_t* vec_full = bars + 2;   // [2] its token factors are
  uint64_t* gram_full = bars + 4;  // [2] its Gram products are complete
  uint64_t* unit_done = bars + 6;  // [2] all warps are through with it
  uint64_t* head_bar = bars + 8;   // [2] the four warps of a head meet
  uint64_t* frag_free = bars + 10; // [2] they have read the head's fragments
  uint64_t* tile_full = bars + 12; // the unit's tiles are in shared memory
  uint64_t* norm_done = bars + 13; // the row norms have been taken from them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&desc_full[i], 1); tc::mbar_init(&vec_full[i], 32); tc::mbar_init(&gram_full[i], 1); tc::mbar_init(&unit_done[i], 8);
      tc::mbar_init(&head_bar[i], 4); tc::mbar_init(&frag_free[i], 4);
    }
    tc::mbar_init(tile_full, 32); tc::mbar_init(norm_done, 32);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  pdl_wait();
  if (batch_rejected(a, chunk_start, blockIdx.x == 0)) return;
  if (warp == 8) tc::tmem_alloc(tmem_slot, 128);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tm = *tmem_slot;
  const bool l2norm = (a.flags & AVE_GDN_FLAG_QK_L2NORM) != 0;
  const int r = a.Hv / a.Hk, pairs = (r + 1) / 2, rows = a.Hk * pairs;
  int* desc = reinterpret_cast<int*>(smem + TL_DESC);

  if (warp == 8) {
    // ------------------------------------------------------------------ tiles and Gram products, a unit ahead
    int k = 0;
    bool alive = true;
    const int64_t total = (int64_t)n_chunks * rows;
    for (int64_t base = blockIdx.x; base < total && alive; base += 32 * (int64_t)gridDim.x) {
      const int64_t u = base + (int64_t)lane * gridDim.x;
      ChunkRef mine; mine.ok = false; mine.t0 = mine.len = mine.b = mine.cis = 0;
      int my_c = 0;
      if (u < total) {
        my_c = (int)(u / rows);
        bool in = true;
        if (compact_grid) {  // n_seqs x parts x rn: only chunks of this launch's range
          const int per_seq = plan.parts * plan.rn;
          const int n = my_c / per_seq, rest = my_c % per_seq;
          const int cis = plan.part_begin[rest / plan.rn] + plan.r0 + rest % plan.rn;
          const int per = ((a.cu_seqlens ? a.cu_seqlens[n + 1] - a.cu_seqlens[n] : a.T) + C - 1) / C;
          in = cis < per && cis < plan.part_begin[rest / plan.rn + 1];
          my_c = first_record(a, chunk_start, n) + cis;
        }
        if (in) mine = find_chunk(a, chunk_start, my_c);
      }
      const int my_y = (int)(u % rows);
      uint32_t todo = __ballot_sync(0xffffffffu, mine.ok);
      for (; todo != 0u && alive; todo &= todo - 1u, ++k) {
        const int src = __ffs(todo) - 1, buf = k & 1;
        const int c = __shfl_sync(0xffffffffu, my_c, src), b = __shfl_sync(0xffffffffu, mine.b, src), t0 = __shfl_sync(0xffffffffu, mine.t0, src);
        const int len = __shfl_sync(0xffffffffu, mine.len, src), y = __shfl_sync(0xffffffffu, my_y, src);
        const int hk = y / pairs, h0 = hk * r + 2 * (y % pairs), nh = min(2, hk * r + r - h0);
        if (k >= 2 && !tc::mbar_wait_warp(&unit_done[buf], (uint32_t)((k >> 1) & 1) ^ 1u, abort_flag)) { alive = false; break; }
        if (lane == 0) {
          int4* d = reinterpret_cast<int4*>(desc + 8 * buf);
          d[0] = make_int4(c, h0, nh, len); d[1] = make_int4(b, t0, 0, 0);
          tc::mbar_arrive(&desc_full[buf]);
        }
        if (k >= 1) {  // the tiles may be overwritten once the Gram products of the unit before are complete (and the norms taken)
          if (!tc::mbar_wait_warp(&gram_full[buf ^ 1], (uint32_t)((k - 1) >> 1) & 1u, abort_flag)) { alive = false; break; }
          if (l2norm && !tc::mbar_wait_warp(norm_done, (uint32_t)(k - 1) & 1u, abort_flag)) { alive = false; break; }
        }
        const int piece8 = lane & 15, row0 = lane >> 4;
        const __nv_bfloat16* kp = bf(a.k) + b * a.k_stride_b + (int64_t)t0 * a.k_stride_t + (int64_t)hk * a.k_stride_h + 8 * piece8;
        const __nv_bfloat16* qp = bf(a.q) + b * a.q_stride_b + (int64_t)t0 * a.q_stride_t + (int64_t)hk * a.q_stride_h + 8 * piece8;
        const uint32_t tile = tc::smem_u32(smem + TL_TILE) + (piece8 >> 3) * TL_HALF;
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
          const int row = row0 + 2 * i, from = row < len ? row : 0;
          const uint32_t in_group = (row & 7) * 128 + (((piece8 & 7) ^ (row & 7)) << 4);
          cp16(tile + (row >> 3) * 2048 + in_group, kp + from * a.k_stride_t, row < len);
          cp16(tile + ((row >> 3) ^ 6) * 2048 + 1024 + in_group, qp + from * a.q_stride_t, row < len);
        }
        cp_commit();
        cp_wait<0>();
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (l2norm) tc::mbar_arrive(tile_full);
        tc::tc_fence_after_sync();
        if (tc::elect_one()) {
          constexpr uint32_t idesc = tc::idesc_f16(128, 64, 1, 1, false, false);
          const uint32_t at0 = tc::smem_u32(smem + TL_TILE);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            const uint32_t at = at0 + (ks >> 2) * TL_HALF + (ks & 3) * 32;
            tc::mma_ss(tm + 64 * buf, tc::smem_desc_sw128(at, 16, 1024), tc::smem_desc_sw128(at, 16, 2048), idesc, ks != 0 ? 1u : 0u);
          }
          tc::mma_commit(&gram_full[buf]);
        }
        __syncwarp();
      }
    }
    if (alive && k >= 2) alive = tc::mbar_wait_warp(&unit_done[k & 1], (uint32_t)((k >> 1) & 1) ^ 1u, abort_flag);
    if (alive && k >= 1) tc::mbar_wait_warp(&gram_full[(k - 1) & 1], (uint32_t)((k - 1) >> 1) & 1u, abort_flag);  // nothing in flight at the end
    if (lane == 0) {
      desc[8 * (k & 1)] = -1;
      tc::mbar_arrive(&desc_full[k & 1]);
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ gates, norms and the factors of every token, a unit ahead
    for (int k = 0;; ++k) {
      const int buf = k & 1;
      if (!tc::mbar_wait_warp(&desc_full[buf], (uint32_t)(k >> 1) & 1u, abort_flag)) break;
      const int c = desc[8 * buf], h0 = desc[8 * buf + 1], nh = desc[8 * buf + 2], len = desc[8 * buf + 3], b = desc[8 * buf + 4], t0 = desc[8 * buf + 5];
      if (c < 0) { tc::mbar_arrive(&vec_full[buf]); break; }
      float g[2][2], be[2][2];  // gates and betas of tokens lane and lane + 32
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const bool in = hh < nh && lane + 32 * e < len;
          const int64_t off = b * a.g_stride_b + (int64_t)(t0 + lane + 32 * e) * a.g_stride_t + h0 + hh;
          g[hh][e] = in ? a.g[off] : 0.f;
          be[hh][e] = in ? a.beta[off] : 0.f;
        }
      // in-chunk cumulative gates, an inclusive scan of 64 values, of both heads side by side
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float x = __shfl_up_sync(0xffffffffu, g[hh][e], o);
            if (lane >= o) g[hh][e] += x;
          }
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) g[hh][1] += __shfl_sync(0xffffffffu, g[hh][0], 31);
      float kn[2] = {1.f, 1.f}, qn[2] = {1.f, 1.f};
      if (l2norm) {
        if (!tc::mbar_wait_warp(tile_full, (uint32_t)k & 1u, abort_flag)) break;
#pragma unroll 1
        for (int e = 0; e < 2; ++e) {
          const int i = lane + 32 * e;
          const uint8_t* k_row = smem + TL_TILE + (i >> 3) * 2048 + (i & 7) * 128;
          const uint8_t* q_row = smem + TL_TILE + ((i >> 3) ^ 6) * 2048 + 1024 + (i & 7) * 128;
          float2 sk = make_float2(0.f, 0.f), sq = sk;
#pragma unroll 2
          for (int p = 0; p < 16; ++p) {  // the swizzle permutes pieces inside a row, a sum needs no decode
            const int at = (p >> 3) * TL_HALF + (((p + lane) & 7) << 4);
            const uint4 kr = *reinterpret_cast<const uint4*>(k_row + at), qr = *reinterpret_cast<const uint4*>(q_row + at);
            const uint32_t kw[4] = {kr.x, kr.y, kr.z, kr.w}, qw[4] = {qr.x, qr.y, qr.z, qr.w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const float2 kf = bf16x2_to_float2(kw[w]), qf = bf16x2_to_float2(qw[w]);
              sk = __ffma2_rn(kf, kf, sk); sq = __ffma2_rn(qf, qf, sq);
            }
          }
          const float rk = rsqrtf(sk.x + sk.y + 1e-6f), rq = rsqrtf(sq.x + sq.y + 1e-6f);
          if (e == 0) { kn[0] = rk; qn[0] = rq; } else { kn[1] = rk; qn[1] = rq; }
        }
        tc::mbar_arrive(norm_done);
      }
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        const float v0 = hh ? g[1][0] : g[0][0], v1 = hh ? g[1][1] : g[0][1], be0 = hh ? be[1][0] : be[0][0], be1 = hh ? be[1][1] : be[0][1];
        const float bs1 = __shfl_sync(0xffffffffu, v0, 16), bs2 = __shfl_sync(0xffffffffu, v1, 0), bs3 = __shfl_sync(0xffffffffu, v1, 16);
        const float bC = __shfl_sync(0xffffffffu, v1, 31);
        float* vec = reinterpret_cast<float*>(smem + TL_VEC) + (2 * buf + hh) * TV_FLOATS;
        float* sc = reinterpret_cast<float*>(recs + ((int64_t)c * a.Hv + h0 + hh) * REC_BYTES + REC_SCAL);
        const float decay = __expf(bC);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = lane + 32 * e;
          const float x = e ? v1 : v0, beta = e ? be1 : be0, q = i < len ? qn[e] * a.scale : 0.f, bk = beta * kn[e];
          const float u0 = ex2_approx((x - __shfl_sync(0xffffffffu, x, lane & 16)) * LOG2E);
          vec[TV_B * C + i] = x; vec[TV_BETA * C + i] = beta;
          vec[TV_RA * C + i] = -bk * u0; vec[TV_RP * C + i] = q * u0;
          vec[TV_DA * C + i] = bk; vec[TV_DP * C + i] = q;
          vec[TV_KN * C + i] = kn[e];
          if (e == 0) vec[TV_W1 * C + i] = i < 16 ? ex2_approx((bs1 - x) * LOG2E) * kn[e] : 0.f;
          if (e == 0) vec[TV_W2 * C + i] = ex2_approx((bs2 - x) * LOG2E) * kn[e];
          vec[TV_W3 * C + i] = i < 48 ? ex2_approx((bs3 - x) * LOG2E) * kn[e] : 0.f;
          if (hh < nh) {
            const float eb = __expf(x);
            sc[i] = eb * qn[e] * a.scale;              // o_i = qs_i (H q_i) + (scale P Vn)_i: the output scale is folded in here and in P
            sc[C + i] = __expf(bC - x) * kn[e];        // Vd_j = ks_j Vn_j
            sc[2 * C + i] = i < len ? eb * kn[e] : 0.f;  // X_j = kx_j (H k_j)
            sc[3 * C + i] = decay;
          }
        }
      }
      tc::mbar_arrive(&vec_full[buf]);
    }
  } else {
    // ------------------------------------------------------------------ four warps a head, one row of blocks each
    // (They meet at an mbarrier, not a named one, so that a wait that expires ends every warp's loop.)
    const int hh = warp >> 2, q = warp & 3, gr = lane >> 2, t = lane & 3;
    uint32_t met = 0, units = 0;
    auto head_meet = [&]() {
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&head_bar[hh]);
      return tc::mbar_wait_warp(&head_bar[hh], met++ & 1u, abort_flag);
    };
    for (int k = 0;; ++k) {
      const int buf = k & 1;
      const uint32_t ph = (uint32_t)(k >> 1) & 1u;
      if (!tc::mbar_wait_warp(&vec_full[buf], ph, abort_flag)) break;
      const int c = desc[8 * buf], h0 = desc[8 * buf + 1], nh = desc[8 * buf + 2];
      if (c < 0) break;
      const float* vec = reinterpret_cast<const float*>(smem + TL_VEC) + (2 * buf + hh) * TV_FLOATS;
      uint8_t* rec = recs + ((int64_t)c * a.Hv + h0 + hh) * REC_BYTES;
      if (hh < nh) {
        uint8_t* frag = smem + TL_F + hh * FR_BYTES;
        const float* bs = vec + TV_B * C;
        const uint32_t acc = tm + 64 * buf + ((uint32_t)(32 * q) << 16);
        if (!tc::mbar_wait_warp(&gram_full[buf], ph, abort_flag)) break;
        tc::tc_fence_after_sync();
        // element (row 16 q + gr + 8 hf, column 16 x + 8 nt + 2 t + e) of K K^T is f[hf][4 nt + e], of Q K^T f[hf][4 nt + 2 + e]
        auto load = [&](float (&f)[2][8], int x) {
          tmem_ld_frag2(acc + 16 * x, f[0]);
          tmem_ld_frag2(acc + (16u << 16) + 16 * x, f[1]);
          tc::tmem_ld_wait();
        };
        {  // diagonal block: A in fp32, inverted by this warp, its inverse as a left operand
          float f[2][8];
          load(f, q);
          if (units > 0 && !tc::mbar_wait_warp(&frag_free[hh], (uint32_t)(units - 1) & 1u, abort_flag)) break;
          ++units;
          uint8_t* dst = frag + FR_DIAG + q * FR_BLOCK;
          float* ad = reinterpret_cast<float*>(dst);
#pragma unroll
          for (int hf = 0; hf < 2; ++hf)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              const int i = gr + 8 * hf, j = 8 * nt + 2 * t;
              const float fa = vec[TV_DA * C + 16 * q + i], bi = bs[16 * q + i];
              const float2 kn = *reinterpret_cast<const float2*>(vec + TV_KN * C + 16 * q + j), bj = *reinterpret_cast<const float2*>(bs + 16 * q + j);
              const float x = f[hf][4 * nt] * fa * kn.x * ex2_approx((bi - bj.x) * LOG2E), y = f[hf][4 * nt + 1] * fa * kn.y * ex2_approx((bi - bj.y) * LOG2E);
              *reinterpret_cast<float2*>(ad + i * AD_LD + j) = make_float2(i > j ? x : 0.f, i > j + 1 ? y : 0.f);
            }
          __syncwarp();
          wy_invert_block(ad, lane & 15, lane < 16);
          __syncwarp();
          uint32_t h[4], m[4], l[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {  // rows gr + 8 (e & 1), columns 8 (e >> 1) + 2 t, + 1 (the block is transposed)
            const float* at = ad + (8 * (e >> 1) + 2 * t) * AD_LD + gr + 8 * (e & 1);
            split3(make_float2(at[0], at[AD_LD]), h[e], m[e], l[e]);
          }
          __syncwarp();
          uint4* out = reinterpret_cast<uint4*>(dst) + lane;
          out[0] = make_uint4(h[0], h[1], h[2], h[3]);
          out[32] = make_uint4(m[0], m[1], m[2], m[3]);
          out[64] = make_uint4(l[0], l[1], l[2], l[3]);
        }
        {  // -A left of it
          const float2 ra = make_float2(vec[TV_RA * C + 16 * q + gr], vec[TV_RA * C + 16 * q + gr + 8]);
          const float* w = vec + (TV_W1 + q - 1) * C;  // (q = 0 has no such block)
#pragma unroll 1
          for (int x = 0; x < q; ++x) {
            float f[2][8];
            load(f, x);
            uint32_t h[4], m[4], l[4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              const float2 wj = *reinterpret_cast<const float2*>(w + 16 * x + 8 * nt + 2 * t);
              split3(__fmul2_rn(__fmul2_rn(make_float2(f[0][4 * nt], f[0][4 * nt + 1]), wj), make_float2(ra.x, ra.x)), h[2 * nt], m[2 * nt], l[2 * nt]);
              split3(__fmul2_rn(__fmul2_rn(make_float2(f[1][4 * nt], f[1][4 * nt + 1]), wj), make_float2(ra.y, ra.y)), h[2 * nt + 1], m[2 * nt + 1], l[2 * nt + 1]);
            }
            uint4* out = reinterpret_cast<uint4*>(frag + (q * (q - 1) / 2 + x) * FR_BLOCK) + lane;
            out[0] = make_uint4(h[0], h[1], h[2], h[3]);
            out[32] = make_uint4(m[0], m[1], m[2], m[3]);
            out[64] = make_uint4(l[0], l[1], l[2], l[3]);
          }
        }
        // P, rows of block 3 - q (so that A and P are five blocks for every warp): before the four warps meet by those with the
        // fewest blocks of A, behind the substitution by the others
        bool ok = true;
#pragma unroll 1
        for (int step = 0; step < 2; ++step) {
          if ((q < 2) == (step == 0)) {
            const int pr = 3 - q;
            const float* w = vec + (TV_W1 + pr - 1) * C;  // (pr = 0 has no off-diagonal block)
            const float2 rp = make_float2(vec[TV_RP * C + 16 * pr + gr], vec[TV_RP * C + 16 * pr + gr + 8]);
#pragma unroll 1
            for (int x = 0; x <= pr; ++x) {
              float f[2][8];
              load(f, x);
#pragma unroll
              for (int nt = 0; nt < 2; ++nt) {
                float2 p0 = make_float2(f[0][4 * nt + 2], f[0][4 * nt + 3]), p1 = make_float2(f[1][4 * nt + 2], f[1][4 * nt + 3]);
                const int j = 16 * x + 8 * nt + 2 * t;
                if (x < pr) {
                  const float2 wj = *reinterpret_cast<const float2*>(w + j);
                  p0 = __fmul2_rn(__fmul2_rn(p0, wj), make_float2(rp.x, rp.x));
                  p1 = __fmul2_rn(__fmul2_rn(p1, wj), make_float2(rp.y, rp.y));
                } else {
                  const float2 kn = *reinterpret_cast<const float2*>(vec + TV_KN * C + j), bj = *reinterpret_cast<const float2*>(bs + j);
                  const int i0 = 16 * x + gr, i1 = i0 + 8;
                  const float f0 = vec[TV_DP * C + i0], f1 = vec[TV_DP * C + i1], b0 = bs[i0], b1 = bs[i1];
                  p0.x *= f0 * kn.x * ex2_approx((b0 - bj.x) * LOG2E); p0.y *= f0 * kn.y * ex2_approx((b0 - bj.y) * LOG2E);
                  p1.x *= f1 * kn.x * ex2_approx((b1 - bj.x) * LOG2E); p1.y *= f1 * kn.y * ex2_approx((b1 - bj.y) * LOG2E);
                  p0 = make_float2(i0 >= j ? p0.x : 0.f, i0 > j ? p0.y : 0.f);
                  p1 = make_float2(i1 >= j ? p1.x : 0.f, i1 > j ? p1.y : 0.f);
                }
                uint32_t h0, l0, h1, l1;
                split_pair(p0, h0, l0); split_pair(p1, h1, l1);
                store_half(rec + REC_PT, pr, x, nt, lane, h0, h1, l0, l1);
              }
            }
          }
          if (step == 0) {
            ok = head_meet();
            if (!ok) break;
            uint8_t* tu = rec + REC_TU;
            if (q < 2) {
              solve_columns<0>(frag, vec, q, lane, tu);
            } else {
              solve_columns<1>(frag, vec, q - 2, lane, tu);
              solve_columns<2>(frag, vec, q - 2, lane, tu);
              solve_columns<3>(frag, vec, q - 2, lane, tu);
            }
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&frag_free[hh]);
          }
        }
        if (!ok) break;
        tc::tc_fence_before_sync();
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&unit_done[buf]);
    }
  }
  __syncwarp();
  tc::tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && a.status != nullptr) atomicOr(a.status, AVE_GDN_DEV_WAIT_EXPIRED);
  if (warp == 8) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tm, 128);
  }
}

}  // namespace
}  // namespace ave
