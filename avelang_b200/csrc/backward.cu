// Backward pass of the gated delta rule (d_k = d_v = 128), chunked (64 tokens), with fp32-level accuracy.
//
// Per chunk (M0 the state that enters it, b the in-chunk cumulative gate, G_ij = e^{b_i - b_j}, S the output scale):
//     A = strict_lower(beta_i G_ij k_i.k_j)    T = (I + A)^-1      P = lower(G_ij q_i.k_j)      D_i = e^{b_C - b_i}
//     Vn = T diag(beta) (V - diag(e^b) K M0)   O = S (diag(e^b) Q M0 + P Vn)    M1 = e^{b_C} M0 + K^T diag(D) Vn
// and in reverse, with E the gradient of M1:
//     dVn = S P^T dO + diag(D) K E             Ut = T^T dVn
//     dM0 = e^{b_C} E + S Q^T diag(e^b) dO - K^T diag(beta e^b) Ut
//     dV  = diag(beta) Ut
//     dQ  = S diag(e^b) dO M0^T + X K          X = S lower(dO Vn^T) o G
//     dK  = row + col,  row = Y K - diag(beta e^b) Ut M0^T,   col = Y^T K + X^T Q + diag(D) Vn E^T,
//           Y = -diag(beta) strict_lower(Ut Vn^T) o G     (the gradient of A collapses to -strict_lower(Ut Vn^T))
//     dbeta_i = Ut_i.v_i + (k_i.row_i) / beta_i
//     db_i    = q_i.dq_i + k_i.row_i - k_i.col_i,  and  dg_t = sum_{i >= t} db_i + sum_j k_j.(D_j (Vn E^T)_j) + e^{b_C} <E, M0>
//           (b_i rides on q_i and on the row side of k_i with a plus sign, on the column side of k_i with a minus sign).
//
// Three launches.  bwd_prep: T, P and b of every (chunk, value head), in parallel.  bwd_scans: the states and Vn, chunk after
// chunk, and beside them the state gradients and Ut, chunk after chunk from the end (neither needs anything of the other).
// bwd_grads: everything else, in parallel over (chunk, key head), summing over the value heads that share the key head.
//
// The contractions run on bf16 MMAs (bwd_prep: warp-level, the others: tcgen05) with fp32 accumulation.  q, k, v and dO are bf16
// and enter as they are; every fp32 operand enters as three bf16 terms x = h + m + l (24 significant bits), so a product with
// one fp32 operand is three MMAs and one with two is six (h h, h m, m h, h l, l h, m m): the accuracy of fp32 arithmetic, which
// the gradient of the gate needs, because it is a difference of large sums.
// Two sequences of 4096 tokens, 32 value heads: 0.82 ms (prep 0.08, scans 0.30, gradients 0.44) against 22.1 ms for the
// token-by-token reverse sweep this replaced (a 64 KiB tile written and read per token).
#include <type_traits>

#include "common.cuh"
#include "recslots.cuh"
#include "tc.cuh"
#include "wyblocks.cuh"

namespace ave {
namespace {

constexpr int BD = 128, BCH = 64;
constexpr int IMG = BCH * BCH * 2;              // one bf16 [64][64] tile
constexpr int PREP_P = 3 * IMG, PREP_SC = 6 * IMG, SC_BYTES = 3 * BCH * 4, PREP_BYTES = PREP_SC + SC_BYTES;  // T h m l | P h m l | b | beta | b's low part
constexpr int STATE_FLOATS = BD * BD, VEC_FLOATS = BD * BCH;

// 246528 bytes a (slot, value head).  The key heads are independent of one another, so a call with less scratch than all of
// them need takes them in several passes over the same scratch, one after the other.  A pass is a call on its own heads: Hk
// and Hv of its argument block are theirs, and its pointers start at their first; hk_all and hv_all are the heads of the
// whole call, the pitch of the states and of the results.
struct BwdScratch {
  uint8_t* prep;   // [slots][Hv][PREP_BYTES]; the tiles are stored as the swizzled shared-memory images the scans read
  float *m0, *e;   // [slots][Hv][d_k / 8][d_v][8]: H = M0^T and E^T of every chunk
  float *vn, *u;   // [slots][Hv][64 tokens / 8][d_v][8]: Vn^T and Ut^T
  int hk_all, hv_all;
};

// ---------------------------------------------------------------------------------------------- T, P and b of every chunk
// One CTA of eight warps per (chunk, key head, up to two of its value heads); the Gram products are shared by the two.  Bound by the
// latency of its dependent steps, like the forward pass's preparation, whose block algebra it uses: warps 0..3 form the
// fragments of A, 4..7 those of P, then a warp per row of blocks forms T.  P and T leave through the same shared memory, by
// bulk copies.  4096 (chunk, value head) units: 78 us against 116 for one head per CTA with the block products spread
// over CTA barriers.
constexpr int PREP_T = 256;
constexpr int PR_K = 0, PR_Q = 16384, PR_OUT = 0, PR_OUT_HEAD = 3 * IMG, PR_F = 2 * PR_OUT_HEAD, PR_F_HEAD = 16384, PR_SC = PR_F + 2 * PR_F_HEAD,
              PR_SMEM = PR_SC + 2 * SC_BYTES;
static_assert(PR_Q + 16384 <= PR_F && WY_BYTES <= PR_F_HEAD, "shared memory");

template <int R>
__device__ __forceinline__ void bwd_prep_row(uint8_t* smem, int hh, int lane, bool lead, uint8_t* rec) {
  float T[R + 1][2][4];
  wy_row<R>(T, smem + PR_F + hh * PR_F_HEAD, lane);
  if (lead) tc::bulk_wait_read<0>();  // P has been read out of the head's region
  head_sync(hh);
  const uint32_t region = tc::smem_u32(smem + PR_OUT + hh * PR_OUT_HEAD);
#pragma unroll
  for (int c = 0; c <= R; ++c) {
    uint32_t h[4], m[4], l[4];
    split_acc(T[c][0], T[c][1], h, m, l);
    const uint32_t at = region + at_a<128>(16 * R, 2 * c, lane);
    stsm4(at, h[0], h[1], h[2], h[3]);
    stsm4(at + IMG, m[0], m[1], m[2], m[3]);
    stsm4(at + 2 * IMG, l[0], l[1], l[2], l[3]);
  }
  tc::fence_proxy_async_smem();
  head_sync(hh);
  if (lead) {
    tc::bulk_store(rec, smem + PR_OUT + hh * PR_OUT_HEAD, PR_OUT_HEAD);
    tc::bulk_commit();
    tc::bulk_wait_read<0>();  // shared memory must stay intact until the copy has read it
  }
}

__global__ void __launch_bounds__(PREP_T, 2) bwd_prep_kernel(const AveGdnBwdArgs a, BwdScratch ws) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (!offsets_ok(a, blockIdx.x == 0 && blockIdx.y == 0)) return;
  const SlotChunk c = chunk_of_slot(a, blockIdx.x);
  if (!c.ok) return;
  const int r = a.Hv / a.Hk, pairs = (r + 1) / 2;
  const int hk = blockIdx.y / pairs, h0 = hk * r + 2 * (blockIdx.y % pairs), nh = min(2, hk * r + r - h0);
  uint8_t* rec0 = ws.prep + ((int64_t)blockIdx.x * a.Hv + h0) * PREP_BYTES;
  const uint32_t sb = tc::smem_u32(smem);
  load_tile<BCH, 16, PREP_T>(sb + PR_K, bf(a.k) + c.b * a.k_stride_b + (int64_t)c.t0 * a.k_stride_t + hk * a.k_stride_h, a.k_stride_t, c.len, tid);
  load_tile<BCH, 16, PREP_T>(sb + PR_Q, bf(a.q) + c.b * a.q_stride_b + (int64_t)c.t0 * a.q_stride_t + hk * a.q_stride_h, a.q_stride_t, c.len, tid);
  cp_commit();
  if (warp < nh) {  // inclusive scan of the gates; beyond the end of the sequence b stays and beta is 0
    // b reaches hundreds while e^{b_i - b_j} of near tokens matters: it is summed in double and kept as two floats, so that
    // the differences are as exact as the gates themselves
    const int64_t off = c.b * a.g_stride_b + (int64_t)c.t0 * a.g_stride_t + h0 + warp;
    double v0 = lane < c.len ? a.g[off + lane * a.g_stride_t] : 0.f, v1 = lane + 32 < c.len ? a.g[off + (lane + 32) * a.g_stride_t] : 0.f;
    const float be0 = lane < c.len ? a.beta[off + lane * a.g_stride_t] : 0.f, be1 = lane + 32 < c.len ? a.beta[off + (lane + 32) * a.g_stride_t] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t0 = __shfl_up_sync(0xffffffffu, v0, o), t1 = __shfl_up_sync(0xffffffffu, v1, o);
      if (lane >= o) { v0 += t0; v1 += t1; }
    }
    v1 += __shfl_sync(0xffffffffu, v0, 31);
    float* sc = reinterpret_cast<float*>(rec0 + warp * PREP_BYTES + PREP_SC);
    float* bs = reinterpret_cast<float*>(smem + PR_SC + warp * SC_BYTES);
    const float x0 = (float)v0, x1 = (float)v1, l0 = (float)(v0 - x0), l1 = (float)(v1 - x1);
    bs[lane] = sc[lane] = x0; bs[lane + 32] = sc[lane + 32] = x1;
    bs[BCH + lane] = sc[BCH + lane] = be0; bs[BCH + lane + 32] = sc[BCH + lane + 32] = be1;
    bs[2 * BCH + lane] = sc[2 * BCH + lane] = l0; bs[2 * BCH + lane + 32] = sc[2 * BCH + lane + 32] = l1;
  }
  cp_wait<0>();
  __syncthreads();
  // Warps 0..3: rows of K block m against the blocks from it on (A transposed); warps 4..7: rows of Q block m against the K blocks
  // up to it.  acc[2 x] and acc[2 x + 1]: the x-th of those blocks.
  const int m = warp & 3;
  const bool is_p = warp >= 4;
  const int first = is_p ? 0 : m, count = is_p ? m + 1 : 4 - m;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) zero(acc[i]);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    uint32_t af[4];
    ldsm4(af, sb + (is_p ? PR_Q : PR_K) + at_a<256>(16 * m, 2 * ks, lane));
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      if (x >= count) break;
      uint32_t b[4];
      ldsm4(b, sb + PR_K + at_b<256>(16 * (first + x), 2 * ks, lane));
      mma_bf16(acc[2 * x], af, b[0], b[1]);
      mma_bf16(acc[2 * x + 1], af, b[2], b[3]);
    }
  }
  __syncthreads();  // K and Q make room for P, later T; their blocks above the diagonal are zero
  for (int e = tid; e < nh * 3 * 6 * 32; e += PREP_T) {
    const int blk = (e >> 5) % 6, brow = (blk < 3 ? 0 : blk < 5 ? 1 : 2), bcol = (blk < 3 ? blk + 1 : blk < 5 ? blk - 1 : 3);
    *reinterpret_cast<uint4*>(smem + PR_OUT + ((e >> 5) / 6) * IMG + piece<128>(16 * brow + ((e & 31) >> 1), 2 * bcol + (e & 1))) = make_uint4(0u, 0u, 0u, 0u);
  }
#pragma unroll 1
  for (int hh = 0; hh < nh; ++hh) {
    const float* bs = reinterpret_cast<const float*>(smem + PR_SC + hh * SC_BYTES);
    uint8_t* frag = smem + PR_F + hh * PR_F_HEAD;
    if (!is_p) {  // element (row j = 16 m + g + 8 hf, column i = 16 s + 8 nt + 2 t + e) of the transposed A
      float* ad = reinterpret_cast<float*>(frag + WY_DIAG) + m * 16 * AD_LD;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = g + 8 * (e >> 1), i = 8 * nt + 2 * t + (e & 1);
          const float x = bs[BCH + 16 * m + i] * gate_between(bs, 16 * m + i, 16 * m + j) * acc[nt][e];
          ad[i * AD_LD + j] = i > j ? x : 0.f;
        }
#pragma unroll
      for (int x = 1; x < 4; ++x) {
        if (x >= count) break;
        const int s = m + x;
        uint32_t ah[4], am[4], al[4];
#pragma unroll
        for (int idx = 0; idx < 4; ++idx) {  // (column tile idx & 1, row half idx >> 1)
          const int i = 16 * s + 8 * (idx & 1) + 2 * t, j = 16 * m + g + 8 * (idx >> 1);
          const float* p = acc[2 * x + (idx & 1)] + 2 * (idx >> 1);
          split3(make_float2(bs[BCH + i] * gate_between(bs, i, j) * p[0], bs[BCH + i + 1] * gate_between(bs, i + 1, j) * p[1]), ah[idx], am[idx], al[idx]);
        }
        uint4* f = reinterpret_cast<uint4*>(frag + (s * (s - 1) / 2 + m) * WY_BLOCK) + lane;
        f[0] = make_uint4(ah[0], ah[1], ah[2], ah[3]);
        f[32] = make_uint4(am[0], am[1], am[2], am[3]);
        f[64] = make_uint4(al[0], al[1], al[2], al[3]);
      }
    } else {  // element (row i = 16 m + g + 8 hf, column j = 16 x + 8 nt + 2 t + e) of P
      const uint32_t region = sb + PR_OUT + hh * PR_OUT_HEAD;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        if (x >= count) break;
        uint32_t ph[4], pm[4], pl[4];
#pragma unroll
        for (int idx = 0; idx < 4; ++idx) {  // (column tile idx >> 1, row half idx & 1)
          const int i = 16 * m + g + 8 * (idx & 1), j = 16 * x + 8 * (idx >> 1) + 2 * t;
          const float* p = acc[2 * x + (idx >> 1)] + 2 * (idx & 1);
          const float y0 = gate_between(bs, i, j) * p[0], y1 = gate_between(bs, i, j + 1) * p[1];
          split3(make_float2(i >= j ? y0 : 0.f, i > j ? y1 : 0.f), ph[idx], pm[idx], pl[idx]);
        }
        const uint32_t at = region + at_a<128>(16 * m, 2 * x, lane);
        stsm4(at, ph[0], ph[1], ph[2], ph[3]);
        stsm4(at + IMG, pm[0], pm[1], pm[2], pm[3]);
        stsm4(at + 2 * IMG, pl[0], pl[1], pl[2], pl[3]);
      }
    }
  }
  tc::fence_proxy_async_smem();
  __syncthreads();
  const int hh = warp >> 2;
  if (hh >= nh) return;
  uint8_t* rec = rec0 + hh * PREP_BYTES;
  // rows cost R + 1 units of work and warps 0 and 4, 1 and 5, ... share a scheduler: opposite orders
  const int row = hh == 0 ? 3 - warp : warp - 4;
  const bool lead = row == 0 && lane == 0;  // in the warp with the least work
  if (lead) {
    tc::bulk_store(rec + PREP_P, smem + PR_OUT + hh * PR_OUT_HEAD, PR_OUT_HEAD);
    tc::bulk_commit();
  }
  if (row >= 2) wy_invert(smem + PR_F + hh * PR_F_HEAD, row & 1, lane);
  head_sync(hh);
  switch (row) {
    case 3: bwd_prep_row<3>(smem, hh, lane, lead, rec); break;
    case 2: bwd_prep_row<2>(smem, hh, lane, lead, rec); break;
    case 1: bwd_prep_row<1>(smem, hh, lane, lead, rec); break;
    default: bwd_prep_row<0>(smem, hh, lane, lead, rec); break;
  }
}

// ---------------------------------------------------------------------------------------------- the two scans
// One CTA of 16 warps per (sequence, value head) and direction, in one launch.  The state stays transposed, S = H or E, d_v on the
// 128 tensor-memory lanes: a thread keeps 32 of a row's 128 elements in fp32 registers, and S, the left operand of the first
// product, X and (reverse) dO^T live in tensor memory as three bf16 terms each.  A chunk is three dependent products,
//     x = S K^T,   y = (f(x, V or dO P)) T or T^T,   S += (f(y)) K   (reverse: and the scaled dO)^T Q,
// with a pass of all threads over the result behind each; the product of the pass's tile is issued by two threads, into
// accumulators (or column halves) of their own.  The chain is bound by these hand-offs, about 1 k cycles each beside 0.8 k of
// MMAs.  Tiles of the next chunk land meanwhile.  Two sequences of 4096 tokens, 32 value heads: 0.30 ms; on warp-level MMAs, whose
// pipe was full (504 and 756 of them a warp and chunk, 16 cycles each), the two scans took 0.27 + 0.38 ms one after the other.
constexpr int SC_T = 512, SC_LT = 256;  // the first SC_LT threads copy tiles; warps 10 and 13 issue the first products
constexpr int SC_K = 0, FW_V = 16384, FW_TI = 32768, FW_SC = FW_TI + 3 * IMG, FW_STAGE = FW_SC + 1024;
constexpr int RV_Q = 16384, RV_DO = 32768, RV_TI = 49152, RV_PI = RV_TI + 3 * IMG, RV_SC = RV_PI + 3 * IMG, RV_STAGE = RV_SC + 1024;
constexpr int SC_FAC = 2 * RV_STAGE, SC_BAR = SC_FAC + 2 * BCH * 16, SC_SMEM = SC_BAR + 64;
static_assert(FW_STAGE % 1024 == 0 && RV_STAGE % 1024 == 0 && SC_SMEM <= 227 * 1024, "shared memory");
// tensor-memory columns.  State terms: [half of d_k][term][32]; the increment's accumulator takes the first 64 of each half.
constexpr uint32_t TS_S = 0, TS_HALF = 96, TS_X = 192, TS_DO = 288, TS_ACC = 384, TS_ACC2 = 448;

// The fp32 records of a chunk, [d_v][N]: eight elements of a row are one 32-byte unit, units in the order [N / 8][d_v], so that
// the scans (a lane is a row) and bwd_grads (a lane is half a unit) both move whole lines.
__device__ __forceinline__ void store_unit(float* rec, int unit, int row, const float* v) {
  float* p = rec + (unit * BD + row) * 8;
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]),
               "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}
// N fp32 values -> three terms, N / 2 tensor-memory columns each, `step` columns apart
template <int N>
__device__ __forceinline__ void store_terms(uint32_t at, uint32_t step, const float (&x)[N]) {
  uint32_t h[N / 2], m[N / 2], l[N / 2];
#pragma unroll
  for (int i = 0; i < N / 2; ++i) split3(make_float2(x[2 * i], x[2 * i + 1]), h[i], m[i], l[i]);
  tc::tmem_st_n(at, h);
  tc::tmem_st_n(at + step, m);
  tc::tmem_st_n(at + 2 * step, l);
}

template <bool kRev>
__device__ __forceinline__ void bwd_scan(const AveGdnBwdArgs& a, const BwdScratch& ws, int unit, uint8_t* smem) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = unit / a.Hv, h = unit % a.Hv, hk = h / (a.Hv / a.Hk);
  const SeqSpan sp = seq_span(a.cu_seqlens, n, a.T, nullptr);
  const int64_t tile = ((int64_t)n * ws.hv_all + h) * STATE_FLOATS;
  if (sp.len == 0) {  // empty sequence: the state gradient passes through
    if (kRev && a.d_initial_state != nullptr)
      for (int e = tid; e < STATE_FLOATS; e += SC_T) a.d_initial_state[tile + e] = a.d_final_state ? a.d_final_state[tile + e] : 0.f;
    return;
  }
  constexpr int STAGE = kRev ? RV_STAGE : FW_STAGE, TI = kRev ? RV_TI : FW_TI, SC = kRev ? RV_SC : FW_SC, ROWS = kRev ? RV_DO : FW_V;
  const int64_t slot0 = first_slot(a, n);
  const int n_chunks = (sp.len + BCH - 1) / BCH;
  const __nv_bfloat16* kp = bf(a.k) + sp.b * a.k_stride_b + (int64_t)sp.t0 * a.k_stride_t + hk * a.k_stride_h;
  const __nv_bfloat16* qp = bf(a.q) + sp.b * a.q_stride_b + (int64_t)sp.t0 * a.q_stride_t + hk * a.q_stride_h;
  const __nv_bfloat16* vp = bf(a.v) + sp.b * a.v_stride_b + (int64_t)sp.t0 * a.v_stride_t + h * a.v_stride_h;
  const __nv_bfloat16* dop = bf(a.d_o) + sp.b * a.do_stride_b + (int64_t)sp.t0 * a.do_stride_t + h * a.do_stride_h;
  const uint32_t sb = tc::smem_u32(smem);
  float4* fac_of = reinterpret_cast<float4*>(smem + SC_FAC);    // per stage and token: forward beta, e^b, D; reverse D, S e^b, -beta e^b
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SC_BAR);  // one per product, then one per stage
  volatile uint32_t* abort_flag = reinterpret_cast<uint32_t*>(smem + SC_BAR + 48);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SC_BAR + 56);
  auto load = [&](int c) {
    const uint32_t st = sb + (c & 1) * STAGE;
    const int len = min(BCH, sp.len - c * BCH);
    if (tid < SC_LT) {
      auto tiles = [&](int at, const __nv_bfloat16* src, int64_t stride) {  // [64 tokens][128] as two tiles of 128-byte rows
        load_tile<BCH, 8, SC_LT>(st + at, src + (int64_t)c * BCH * stride, stride, len, tid);
        load_tile<BCH, 8, SC_LT>(st + at + 8192, src + (int64_t)c * BCH * stride + 64, stride, len, tid);
      };
      tiles(SC_K, kp, a.k_stride_t);
      if constexpr (kRev) {
        tiles(RV_Q, qp, a.q_stride_t);
        tiles(RV_DO, dop, a.do_stride_t);
      } else {
        tiles(FW_V, vp, a.v_stride_t);
      }
      cp_commit();
    }
    if (tid == 0) {
      const uint8_t* rec = ws.prep + ((slot0 + c) * a.Hv + h) * PREP_BYTES;
      uint8_t* dst = smem + (c & 1) * STAGE;
      tc::mbar_expect_tx(&bars[3 + (c & 1)], kRev ? PREP_BYTES : 3 * IMG + SC_BYTES);
      if constexpr (kRev) {
        tc::bulk_load(dst + RV_TI, rec, PREP_BYTES, &bars[3 + (c & 1)]);
      } else {
        tc::bulk_load(dst + FW_TI, rec, 3 * IMG, &bars[3 + (c & 1)]);
        tc::bulk_load(dst + FW_SC, rec + PREP_SC, SC_BYTES, &bars[3 + (c & 1)]);
      }
    }
  };
  if (tid == 0) {
    for (int i = 0; i < 5; ++i) tc::mbar_init(&bars[i], i < 3 ? 2 : 1);  // commits of the two issuers; the records of the two stages
    *abort_flag = 0u;
    tc::fence_barrier_init();
  }
  load(kRev ? n_chunks - 1 : 0);
  if (warp == 2) tc::tmem_alloc(tmem_slot, 512);
  // this thread: row `row` of d_v; 16 tokens from 16 grp; 32 columns of d_k from 32 grp
  const int grp = warp >> 2, quarter = warp & 3, row = 32 * quarter + lane;
  float S[32];
  {
    const float* src = kRev ? a.d_final_state : a.initial_state;
#pragma unroll
    for (int i = 0; i < 32; ++i) S[i] = src != nullptr ? src[tile + (int64_t)(32 * grp + i) * BD + row] : 0.f;
  }
  // all of a chunk's tiles are there for the MMAs (behind the next barrier).  The fence waits for this thread's outstanding
  // accesses to global memory, so it stands where few are.
  auto landed = [&](int c, uint32_t n_th) {
    cp_wait<0>();
    tc::fence_proxy_async_smem();
    tc::mbar_wait_warp(&bars[3 + (c & 1)], n_th >> 1 & 1, abort_flag);  // the stage's (n_th / 2)-th use
    if (tid >= SC_T - BCH) {
      const int i = tid - (SC_T - BCH);
      const float* bs = reinterpret_cast<const float*>(smem + (c & 1) * STAGE + SC);
      const float eb = __expf(bs[i]), be = bs[BCH + i], D = gate_between(bs, BCH - 1, i);
      fac_of[(c & 1) * BCH + i] = kRev ? make_float4(D, i < sp.len - c * BCH ? a.scale * eb : 0.f, -be * eb, 0.f) : make_float4(be, eb, D, 0.f);
    }
  };
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  landed(kRev ? n_chunks - 1 : 0, 0);
  const uint32_t tm = *tmem_slot, lanes = tm + ((uint32_t)(32 * quarter) << 16);
  const uint32_t s_cols = lanes + TS_S + (grp >> 1) * TS_HALF;
  auto issue_do_p = [&](int c) {  // dO^T P of a chunk, ahead of it
    tc::tc_fence_after_sync();
    const uint32_t st = sb + (c & 1) * STAGE;
    const uint64_t od = tc::smem_desc_sw128(st + RV_DO, 8192, 1024), pd = tc::smem_desc_sw128(st + RV_PI, 8192, 1024);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        tc::mma_ss(tm + TS_ACC2, od + ks * (2048 >> 4), pd + ((i * IMG + ks * 2048) >> 4), tc::idesc_f16(128, 64, 1, 1, true, true), (i | ks) != 0 ? 1u : 0u);
    tc::mma_commit(&bars[0]);  // counts for the chunk's first product
  };
  store_terms<32>(s_cols + 16 * (grp & 1), 32, S);
  if constexpr (kRev) {
    __syncthreads();
    if (warp == 10 && tc::elect_one()) issue_do_p(n_chunks - 1);
    __syncwarp();
  }
#pragma unroll 1
  for (int it = 0; it < n_chunks; ++it) {
    const int c = kRev ? n_chunks - 1 - it : it, c_next = kRev ? c - 1 : c + 1;
    const uint32_t st = sb + (c & 1) * STAGE, phase = it & 1;
    uint8_t* stage = smem + (c & 1) * STAGE;
    const float* bs = reinterpret_cast<const float*>(stage + SC);
    const int64_t rec = (slot0 + c) * a.Hv + h;
    const float4* fac = fac_of + (c & 1) * BCH;
    const bool last = it + 1 == n_chunks, update = kRev ? !last || a.d_initial_state != nullptr : !last;
    tc::tmem_st_wait();
    tc::tc_fence_before_sync();
    __syncthreads();
    if ((warp == 13 || (!kRev && warp == 10)) && tc::elect_one()) {  // S K^T; forward: its terms over two accumulators
      tc::tc_fence_after_sync();
      constexpr uint32_t id = tc::idesc_f16(128, 64, 1, 1, false, false);
      const uint64_t kd = tc::smem_desc_sw128(st + SC_K, 16, 1024);
      auto step = [&](int i, int ks, uint32_t acc, bool more) {
        tc::mma_ts(tm + acc, tm + TS_S + (ks >> 2) * TS_HALF + 32 * i + 8 * (ks & 3), kd + (uint64_t)(((ks >> 2) * 8192 + (ks & 3) * 32) >> 4), id, more ? 1u : 0u);
      };
      if constexpr (kRev) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) step(i, ks, TS_ACC, (i | ks) != 0);
      } else {
        const bool first = warp == 13;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) step(first ? 0 : 2, ks, first ? TS_ACC : TS_ACC2, ks != 0);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) step(1, first ? ks : 4 + ks, first ? TS_ACC : TS_ACC2, true);
      }
      tc::mma_commit(&bars[0]);
    }
    __syncwarp();
    const float decay = __expf(bs[BCH - 1]);
    float rows[16];  // V^T or dO^T
#pragma unroll
    for (int i = 0; i < 16; ++i)
      rows[i] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(stage + ROWS + (row >> 6) * 8192 + piece<128>(16 * grp + i, (row & 63) >> 3) + 2 * (row & 7)));
    if constexpr (kRev) {
      if (update) {
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = fac[16 * grp + i].y * rows[i];
        store_terms<16>(lanes + TS_DO + 8 * grp, 32, x);
      }
    }
    float* s_rec = (kRev ? ws.e : ws.m0) + rec * STATE_FLOATS;
    if (!last) load(c_next);
    tc::mbar_wait_warp(&bars[0], phase, abort_flag);
    tc::tc_fence_after_sync();
    {
      uint32_t u[16], w[16];
      tc::tmem_ld16(lanes + TS_ACC + 16 * grp, u);
      tc::tmem_ld16(lanes + TS_ACC2 + 16 * grp, w);
      tc::tmem_ld_wait();
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float4 f = fac[16 * grp + i];
        if (kRev) x[i] = fmaf(a.scale, __uint_as_float(w[i]), f.x * __uint_as_float(u[i]));       // D (E^T K^T) + S (dO^T P)
        else x[i] = f.x * (rows[i] - f.y * (__uint_as_float(u[i]) + __uint_as_float(w[i])));       // beta (V^T - e^b (K M0)^T)
      }
      store_terms<16>(lanes + TS_X + 8 * grp, 32, x);
    }
    tc::tmem_st_wait();
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp < 2 && tc::elect_one()) {  // X T^T or X T, the six term products over two accumulators
      tc::tc_fence_after_sync();
      constexpr int L[2][3] = {{0, 0, 1}, {0, 2, 1}}, R[2][3] = {{0, 1, 0}, {2, 0, 1}};  // hh hm mh | hl lh mm
      const uint32_t acc = tm + (warp == 0 ? TS_ACC : TS_ACC2);
      const uint64_t td = tc::smem_desc_sw128(st + TI, kRev ? 8192 : 16, 1024);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const uint32_t l = tm + TS_X + 32 * (warp == 0 ? L[0][j] : L[1][j]);
        const uint64_t r = td + (uint64_t)((warp == 0 ? R[0][j] : R[1][j]) * (IMG >> 4));
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          // T is lower triangular: tokens up to 16 kr + 15 (the first step, kr = 3, covers all), or from 16 ks on
          const int kr = 3 - ks;
          if constexpr (kRev) tc::mma_ts(acc, l + 8 * kr, r + kr * (2048 >> 4), tc::idesc_f16(128, 16 * (kr + 1), 1, 1, false, true), (j | ks) != 0 ? 1u : 0u);
          else
            tc::mma_ts(acc + 16 * ks, l + 8 * ks, r + ks * ((2048 + 32) >> 4), tc::idesc_f16(128, 64 - 16 * ks, 1, 1, false, false), (j | ks) != 0 ? 1u : 0u);
        }
      }
      tc::mma_commit(&bars[1]);
      if (kRev && update) {  // (S e^b dO)^T Q, this issuer's half of d_k, opens the increment
        const uint64_t qd = tc::smem_desc_sw128(st + RV_Q + warp * 8192, 8192, 1024);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            tc::mma_ts(tm + TS_S + warp * TS_HALF, tm + TS_DO + 32 * i + 8 * ks, qd + ks * (2048 >> 4), tc::idesc_f16(128, 64, 1, 1, false, true), (i | ks) != 0 ? 1u : 0u);
      }
    }
    __syncwarp();
    store_unit(s_rec, 4 * grp, row, S);
    store_unit(s_rec, 4 * grp + 1, row, S + 8);
    tc::mbar_wait_warp(&bars[1], phase, abort_flag);
    tc::tc_fence_after_sync();
    {
      uint32_t u[16], w[16];
      tc::tmem_ld16(lanes + TS_ACC + 16 * grp, u);
      tc::tmem_ld16(lanes + TS_ACC2 + 16 * grp, w);
      tc::tmem_ld_wait();
      float y[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) y[i] = __uint_as_float(u[i]) + __uint_as_float(w[i]);
      float* dst = (kRev ? ws.u : ws.vn) + rec * VEC_FLOATS;
      if (update) {
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = y[i] * fac[16 * grp + i].z;
        store_terms<16>(lanes + TS_X + 8 * grp, 32, f);
        tc::tmem_st_wait();
        if (!last) landed(c_next, it + 1);
        tc::tc_fence_before_sync();
        __syncthreads();
        if (warp < 2 && tc::elect_one()) {  // the increment: X K, this issuer's half of d_k
          tc::tc_fence_after_sync();
          const uint64_t kd = tc::smem_desc_sw128(st + SC_K + warp * 8192, 8192, 1024);
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              tc::mma_ts(tm + TS_S + warp * TS_HALF, tm + TS_X + 32 * i + 8 * ks, kd + ks * (2048 >> 4), tc::idesc_f16(128, 64, 1, 1, false, true), kRev || (i | ks) != 0 ? 1u : 0u);
          tc::mma_commit(&bars[2]);
        }
        __syncwarp();
      }
      store_unit(dst, 2 * grp, row, y);
      store_unit(dst, 2 * grp + 1, row, y + 8);
      store_unit(s_rec, 4 * grp + 2, row, S + 16);
      store_unit(s_rec, 4 * grp + 3, row, S + 24);
    }
    if (!update) break;
    tc::mbar_wait_warp(&bars[2], phase, abort_flag);
    tc::tc_fence_after_sync();
    if (kRev && !last && warp == 10 && tc::elect_one()) issue_do_p(c_next);  // the tensor core idles during the pass below
    __syncwarp();
    {
      uint32_t d[32];
      tc::tmem_ld32(s_cols + 32 * (grp & 1), d);
      tc::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) S[i] = fmaf(decay, S[i], __uint_as_float(d[i]));
      // the two warps of this half and quarter have both read the accumulator: the new terms take its columns
      tc::tc_fence_before_sync();
      asm volatile("bar.sync %0, 64;" ::"r"(1 + 4 * (grp >> 1) + quarter) : "memory");
      tc::tc_fence_after_sync();
      if (!last) store_terms<32>(s_cols + 16 * (grp & 1), 32, S);
    }
  }
  if (kRev && a.d_initial_state != nullptr) {
#pragma unroll
    for (int i = 0; i < 32; ++i) a.d_initial_state[tile + (int64_t)(32 * grp + i) * BD + row] = S[i];
  }
  tc::tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0u && a.status != nullptr) atomicOr(a.status, AVE_GDN_DEV_WAIT_EXPIRED);
  if (warp == 2) tc::tmem_dealloc(tm, 512);
}
__global__ void __launch_bounds__(SC_T, 1) bwd_scans_kernel(const AveGdnBwdArgs a, BwdScratch ws) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (!offsets_ok(a, false)) return;
  const int units = a.n_seqs * a.Hv;
  if ((int)blockIdx.x < units) bwd_scan<true>(a, ws, blockIdx.x, smem);
  else bwd_scan<false>(a, ws, blockIdx.x - units, smem);
}

// ---------------------------------------------------------------------------------------------- the gradients of one chunk
// A persistent CTA of 16 warps walks (chunk, key head) pairs.  All products run on tcgen05: X and Y (64 x 64) and, transposed
// (128 d_k lanes x 64 tokens, so that the tile that differs per product is the narrow operand), dO M0^T, Ut M0^T and Vn E^T over
// d_v, and X K, Y K, X^T Q + Y^T K over the tokens.  fp32 operands are three bf16 tiles each.  M0 and E pass through shared
// memory 16 d_v rows at a time, split on the way in, two steps deep.  One thread needs about 100 cycles per MMA of this size,
// so four warps issue, each into accumulators of its own; the records of the next head are asked for (into L2) a head ahead.
// Two sequences of 4096 tokens, 32 value heads: 0.44 ms (0.57 with X and Y on warp-level MMAs, one issuer, one pair per CTA;
// 0.73 with every product on warp-level MMAs, whose pipe takes 16 cycles for each).
constexpr int GR_CTAS = 148;  // one CTA per SM
constexpr int GR_T = 512, GR_DV = 16, GR_TERM = GR_DV * BD * 2, GR_STAGE = 6 * GR_TERM;
constexpr int GR_K = 0, GR_Q = 16384, GR_DO = 32768, GR_VN = 49152, GR_U = GR_VN + 3 * 16384, GR_ST = GR_U + 3 * 16384,
              GR_X = GR_ST, GR_Y = GR_X + 3 * IMG,  // X and Y take the place of the two stages once those are consumed
              GR_RED = GR_ST + 2 * GR_STAGE, GR_UV = GR_RED + 4 * BCH * 8, GR_SC = GR_UV + 8 * BCH * 4, GR_F = GR_SC + SC_BYTES + 144,
              GR_BAR = GR_F + BCH * 16, GR_SMEM = GR_BAR + 64;
static_assert(GR_Y + 3 * IMG <= GR_RED && GR_SMEM <= 227 * 1024, "shared memory");
enum { TG_Q = 0, TG_R = 64, TG_S = 128, TG_XK = 192, TG_YK = 256, TG_COL = 320, TG_DQ = 384, TG_DK = 448 };  // tensor-memory columns

// fp32 [128][64] -> three bf16 tiles of 128-byte rows
__device__ __forceinline__ void fetch_tile(float4 (&x)[4], const float* src, int tid) {
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = __ldcs(reinterpret_cast<const float4*>(src) + tid + i * GR_T);
}
__device__ __forceinline__ void split_tile(uint8_t* dst, const float4 (&x)[4], int tid) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = tid + i * GR_T, unit = e >> 8, row = (e >> 1) & (BD - 1);
    uint32_t h[2], m[2], l[2];
    split3(make_float2(x[i].x, x[i].y), h[0], m[0], l[0]);
    split3(make_float2(x[i].z, x[i].w), h[1], m[1], l[1]);
    uint8_t* p = dst + piece<128>(row, unit) + 8 * (e & 1);
    *reinterpret_cast<uint2*>(p) = make_uint2(h[0], h[1]);
    *reinterpret_cast<uint2*>(p + 16384) = make_uint2(m[0], m[1]);
    *reinterpret_cast<uint2*>(p + 32768) = make_uint2(l[0], l[1]);
  }
}
// half a unit of a 16-row step (d_v), unit = warp, row = lane / 2 -> the three tiles of the step, [128 d_k / 64][16 rows][128 bytes]
__device__ __forceinline__ void split_step(uint8_t* dst, const float4& x, int warp, int lane) {
  uint32_t h[2], m[2], l[2];
  split3(make_float2(x.x, x.y), h[0], m[0], l[0]);
  split3(make_float2(x.z, x.w), h[1], m[1], l[1]);
  uint8_t* p = dst + (warp >> 3) * (GR_TERM / 2) + piece<128>(lane >> 1, warp & 7) + 8 * (lane & 1);
  *reinterpret_cast<uint2*>(p) = make_uint2(h[0], h[1]);
  *reinterpret_cast<uint2*>(p + GR_TERM) = make_uint2(m[0], m[1]);
  *reinterpret_cast<uint2*>(p + 2 * GR_TERM) = make_uint2(l[0], l[1]);
}
__device__ __forceinline__ float quad_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  return x + __shfl_xor_sync(0xffffffffu, x, 2);
}
// v[lane & 15] of the 16 values summed over the lanes
__device__ __forceinline__ float lane_sums(float (&v)[16], int lane) {
#pragma unroll
  for (int o = 8; o >= 1; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float give = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}
// Per-head gradients kept in fp32 (the C entry point), or summed over the heads of a key head and rounded to bf16: eight tokens
// of one d_k column per lane.
template <bool kSum>
__device__ __forceinline__ void store_dqk(const AveGdnBwdArgs& a, const BwdScratch& ws, float* dst, const SlotChunk& c, int head, int tok0, int dk, const float (&x)[8]) {
  const int64_t row = (int64_t)c.b * a.T + c.t0 + tok0;
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    if (kSum) {  // even lanes store token i, odd lanes token i + 1, two columns each
      const bool odd = dk & 1;
      const float y = __shfl_xor_sync(0xffffffffu, odd ? x[i] : x[i + 1], 1);
      const int j = i + (odd ? 1 : 0);
      if (tok0 + j < c.len)
        *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(dst) + ((row + j) * ws.hk_all + head) * BD + (dk & ~1)) =
            odd ? pack_bf16x2(y, x[i + 1]) : pack_bf16x2(x[i], y);
    } else {
      if (tok0 + i < c.len) dst[((row + i) * ws.hv_all + head) * BD + dk] = x[i];
      if (tok0 + i + 1 < c.len) dst[((row + i + 1) * ws.hv_all + head) * BD + dk] = x[i + 1];
    }
  }
}

template <bool kSum>
__global__ void __launch_bounds__(GR_T, 1) bwd_grads_kernel(const AveGdnBwdArgs a, BwdScratch ws, int64_t slots) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (!offsets_ok(a, false)) return;
  const int r = a.Hv / a.Hk;
  const uint32_t sb = tc::smem_u32(smem);
  float2* red = reinterpret_cast<float2*>(smem + GR_RED);  // [4 d_k quarters][64 tokens]: q.dq + k.row - k.col, k.row
  float* uv = reinterpret_cast<float*>(smem + GR_UV);      // [8 d_v blocks][64 tokens]: u.v
  float* bs = reinterpret_cast<float*>(smem + GR_SC);
  float* betas = bs + BCH;
  float* dots = bs + 3 * BCH;  // [16] partial <E, M0> | [16] partial k.state | the carry of the suffix sum
  float4* fac = reinterpret_cast<float4*>(smem + GR_F);    // per token: factors of dO M0^T, Ut M0^T, Vn E^T
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + GR_BAR);  // the two stages, and everything
  volatile uint32_t* abort_flag = reinterpret_cast<uint32_t*>(smem + GR_BAR + 32);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + GR_BAR + 40);
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) tc::mbar_init(&bars[i], i < 2 ? 4 : 3);  // commits: one per issuing warp
    *abort_flag = 0u;
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, 512);
  const int wm = warp & 1, wn = warp >> 1;  // dV: token half, 16 d_v columns
  uint32_t tm = 0;
  uint32_t phase = 0;  // bit i: parity of the next completion of bars[i]

  // Persistent: the CTA walks its (chunk, key head) pairs and asks for the next head's tiles while it works on one.
  const int64_t pairs = slots * a.Hk;
#pragma unroll 1
  for (int64_t p = blockIdx.x; p < pairs; p += gridDim.x) {
    const int64_t slot = p / a.Hk;
    const int hk = (int)(p % a.Hk);
    const SlotChunk c = chunk_of_slot(a, slot);
    if (!c.ok) continue;
    const int64_t row0 = (int64_t)c.b * a.T + c.t0;
    auto load_half_tiles = [&](int at, const __nv_bfloat16* src, int64_t stride) {  // [64 tokens][128] as two tiles of 128-byte rows
      load_tile<BCH, 8, GR_T>(sb + at, src, stride, c.len, tid);
      load_tile<BCH, 8, GR_T>(sb + at + 8192, src + 64, stride, c.len, tid);
    };
    __syncthreads();  // the tiles and sums of the pair before are no longer read
    load_half_tiles(GR_K, bf(a.k) + c.b * a.k_stride_b + (int64_t)c.t0 * a.k_stride_t + hk * a.k_stride_h, a.k_stride_t);
    load_half_tiles(GR_Q, bf(a.q) + c.b * a.q_stride_b + (int64_t)c.t0 * a.q_stride_t + hk * a.q_stride_h, a.q_stride_t);

#pragma unroll 1
    for (int hh = 0; hh < r; ++hh) {
      const int h = hk * r + hh;
      const int64_t rec = slot * a.Hv + h;
      if (hh > 0) __syncthreads();  // the tiles and sums of the previous head are no longer read
      load_half_tiles(GR_DO, bf(a.d_o) + c.b * a.do_stride_b + (int64_t)c.t0 * a.do_stride_t + h * a.do_stride_h, a.do_stride_t);
      cp_commit();
      if (tid == 0) {  // the next head's records towards L2
        const int64_t np = hh + 1 < r ? p : p + gridDim.x;
        if (np < pairs) {
          const int64_t nrec = (np / a.Hk) * a.Hv + (np % a.Hk) * r + (hh + 1 < r ? hh + 1 : 0);
          tc::bulk_prefetch_l2(ws.vn + nrec * VEC_FLOATS, VEC_FLOATS * 4);
          tc::bulk_prefetch_l2(ws.u + nrec * VEC_FLOATS, VEC_FLOATS * 4);
          tc::bulk_prefetch_l2(ws.m0 + nrec * STATE_FLOATS, STATE_FLOATS * 4);
          tc::bulk_prefetch_l2(ws.e + nrec * STATE_FLOATS, STATE_FLOATS * 4);
        }
      }
      constexpr int STEP = 2 * GR_DV;  // float4s from one step of d_v rows to the next
      const int first = (warp * BD + (lane >> 1)) * 2 + (lane & 1);
      const float4* hp = reinterpret_cast<const float4*>(ws.m0 + rec * STATE_FLOATS) + first;
      const float4* ep = reinterpret_cast<const float4*>(ws.e + rec * STATE_FLOATS) + first;
      float4 hx[2], ex[2];
      {
        float4 vn[4], ut[4];
        fetch_tile(vn, ws.vn + rec * VEC_FLOATS, tid);
        fetch_tile(ut, ws.u + rec * VEC_FLOATS, tid);
#pragma unroll
        for (int s = 0; s < 2; ++s) { hx[s] = __ldcs(hp + s * STEP); ex[s] = __ldcs(ep + s * STEP); }
        split_tile(smem + GR_VN, vn, tid);
        split_tile(smem + GR_U, ut, tid);
      }
      if (tid < 3 * BCH) bs[tid] = reinterpret_cast<const float*>(ws.prep + rec * PREP_BYTES + PREP_SC)[tid];
      cp_wait<0>();
      tc::tc_fence_before_sync();
      __syncthreads();
      tc::tc_fence_after_sync();
      tm = *tmem_slot;
      if (tid < BCH) {
        const float eb = __expf(bs[tid]), be = fabsf(betas[tid]) < 1e-20f ? 1e-20f : betas[tid];
        fac[tid] = make_float4(a.scale * eb, -be * eb, gate_between(bs, BCH - 1, tid), 0.f);
      }
      float dot = 0.f;
#pragma unroll 1
      for (int s0 = 0; s0 < 8; s0 += 2)
#pragma unroll
      for (int st = 0; st < 2; ++st) {
        const int s = s0 + st;
        uint8_t* stage = smem + GR_ST + st * GR_STAGE;
        if (s >= 2) { tc::mbar_wait_warp(&bars[st], phase >> st & 1, abort_flag); phase ^= 1u << st; }
        split_step(stage, hx[st], warp, lane);
        split_step(stage + 3 * GR_TERM, ex[st], warp, lane);
        dot = fmaf(hx[st].x, ex[st].x, fmaf(hx[st].y, ex[st].y, fmaf(hx[st].z, ex[st].z, fmaf(hx[st].w, ex[st].w, dot))));
        tc::fence_proxy_async_smem();  // waits for loads in flight: the next ones go out behind it
        if (s < 6) { hx[st] = __ldcs(hp + (s + 2) * STEP); ex[st] = __ldcs(ep + (s + 2) * STEP); }
        __syncthreads();
        if (warp < 4 && tc::elect_one()) {  // four issuers; X and Y take the columns of X K and Y K, which come after them
          constexpr uint32_t id_k = tc::idesc_f16(128, 64, 1, 1, true, false), id_mn = tc::idesc_f16(128, 64, 1, 1, true, true),
                             id_x = tc::idesc_f16(64, 64, 1, 1, false, true), id_y = tc::idesc_f16(64, 64, 1, 1, true, true);
          const uint32_t so = sb + GR_ST + st * GR_STAGE, acc = s > 0 ? 1u : 0u;
          const uint64_t mo = tc::smem_desc_sw128(so, GR_TERM / 2, 1024), eo = tc::smem_desc_sw128(so + 3 * GR_TERM, GR_TERM / 2, 1024),
                         u = tc::smem_desc_sw128(sb + GR_U + s * 2048, 8192, 1024), v = tc::smem_desc_sw128(sb + GR_VN + s * 2048, 8192, 1024),
                         o = tc::smem_desc_sw128(sb + GR_DO + (s >> 2) * 8192 + (s & 3) * 32, 16, 1024);
          if (warp == 3) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              tc::mma_ss(tm + TG_Q, mo + i * (GR_TERM >> 4), o, id_k, i > 0 ? 1u : acc);
              tc::mma_ss(tm + TG_XK, o, v + i * (16384 >> 4), id_x, i > 0 ? 1u : acc);
            }
          } else {
            const uint64_t left = warp == 0 ? mo : warp == 1 ? eo : u, right = warp == 0 ? u : v;
            const uint32_t step = (warp == 2 ? 16384 : GR_TERM) >> 4, id = warp == 2 ? id_y : id_mn, dst = tm + (warp == 0 ? TG_R : warp == 1 ? TG_S : TG_YK);
#pragma unroll
            for (int i = 0; i < 6; ++i) {  // hh hm mh hl lh mm
              constexpr int L[6] = {0, 0, 1, 0, 2, 1}, R[6] = {0, 1, 0, 2, 0, 1};
              tc::mma_ss(dst, left + L[i] * step, right + R[i] * (16384 >> 4), id, i > 0 ? 1u : acc);
            }
          }
          tc::mma_commit(&bars[st]);
        }
        __syncwarp();
      }
      dot = warp_sum(dot);
      if (lane == 0) dots[warp] = dot;
#pragma unroll
      for (int st = 0; st < 2; ++st) { tc::mbar_wait_warp(&bars[st], phase >> st & 1, abort_flag); phase ^= 1u << st; }
      // X = S lower(dO Vn^T) o G and Y = -beta strict_lower(Ut Vn^T) o G, 16 rows per quarter of the tensor-memory lanes, take the
      // place of the stages; blocks above the diagonal are zero
      tc::tc_fence_after_sync();
      const int m = warp & 3, nq = warp >> 2, last = 2 * m + 1;
      float ax[2][4], ay[2][4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t at = tm + ((uint32_t)(32 * m) << 16) + 8 * (nq + 4 * e);
        tc::tmem_ld_frag(at + TG_XK, ax[e]);
        tc::tmem_ld_frag(at + TG_YK, ay[e]);
      }
      tc::tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int nt = nq + 4 * e;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int i = 16 * m + g + 8 * half, j = 8 * nt + 2 * t;
          float2 x = make_float2(0.f, 0.f), y = x;
          if (nt <= last) {
            const float e0 = gate_between(bs, i, j), e1 = gate_between(bs, i, j + 1);
            const float be = -(fabsf(betas[i]) < 1e-20f ? 1e-20f : betas[i]);
            x = make_float2(i >= j ? a.scale * e0 * ax[e][2 * half] : 0.f, i > j ? a.scale * e1 * ax[e][2 * half + 1] : 0.f);
            y = make_float2(i > j ? be * e0 * ay[e][2 * half] : 0.f, i > j + 1 ? be * e1 * ay[e][2 * half + 1] : 0.f);
          }
          uint32_t xh, xm, xl;
          uint8_t* dst = smem + GR_X + piece<128>(i, nt) + 4 * t;
          split3(x, xh, xm, xl);
          *reinterpret_cast<uint32_t*>(dst) = xh; *reinterpret_cast<uint32_t*>(dst + IMG) = xm; *reinterpret_cast<uint32_t*>(dst + 2 * IMG) = xl;
          dst += GR_Y - GR_X;
          split3(y, xh, xm, xl);
          *reinterpret_cast<uint32_t*>(dst) = xh; *reinterpret_cast<uint32_t*>(dst + IMG) = xm; *reinterpret_cast<uint32_t*>(dst + 2 * IMG) = xl;
        }
      }
      tc::fence_proxy_async_smem();
      uint32_t vv[2][2][2];  // this warp's part of V (see dV below)
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const int tok = 32 * wm + 16 * mt + g + 8 * half;
            vv[mt][half][kk] = tok < c.len ? __ldg(reinterpret_cast<const uint32_t*>(bf(a.v) + c.b * a.v_stride_b + (int64_t)(c.t0 + tok) * a.v_stride_t + h * a.v_stride_h + 16 * wn + 8 * kk + 2 * t)) : 0u;
          }
      tc::tc_fence_before_sync();
      __syncthreads();
      if (warp < 3 && tc::elect_one()) {  // X K, Y K, X^T Q + Y^T K
        tc::tc_fence_after_sync();
        constexpr uint32_t id_k = tc::idesc_f16(128, 64, 1, 1, true, false), id_mn = tc::idesc_f16(128, 64, 1, 1, true, true);
        const uint64_t ka = tc::smem_desc_sw128(sb + GR_K, 8192, 1024), qa = tc::smem_desc_sw128(sb + GR_Q, 8192, 1024);
        const uint64_t x = tc::smem_desc_sw128(sb + GR_X, 8192, 1024), y = tc::smem_desc_sw128(sb + GR_Y, 8192, 1024);
#pragma unroll 1
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t acc = ks > 0 ? 1u : 0u;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const uint32_t more = i > 0 ? 1u : acc, term = i * (IMG >> 4), rows = ks * (2048 >> 4);
            if (warp == 0) tc::mma_ss(tm + TG_XK, ka + rows, x + term + ks * 2, id_k, more);
            if (warp == 1) tc::mma_ss(tm + TG_YK, ka + rows, y + term + ks * 2, id_k, more);
            if (warp == 2) {
              tc::mma_ss(tm + TG_COL, qa + rows, x + term + rows, id_mn, more);
              tc::mma_ss(tm + TG_COL, ka + rows, y + term + rows, id_mn, 1u);
            }
          }
        }
        tc::mma_commit(&bars[2]);
      }
      __syncwarp();
      {  // dV = beta Ut and the row sums of Ut o V: this warp's 16 d_v columns and 32 tokens
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          uint32_t uh[4], um[4], ul[4];
          const uint32_t ua = sb + GR_U + at_at<128>(16 * wn, 4 * wm + 2 * mt, lane);
          ldsm4t(uh, ua); ldsm4t(um, ua + 16384); ldsm4t(ul, ua + 32768);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int tok = 32 * wm + 16 * mt + g + 8 * half;
            float s = 0.f;
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              const int idx = half + 2 * kk, col = 16 * wn + 8 * kk + 2 * t;
              const float2 x = bf16x2_to_float2(uh[idx]), y = bf16x2_to_float2(um[idx]), z = bf16x2_to_float2(ul[idx]);
              const float2 ut = make_float2(x.x + (y.x + z.x), x.y + (y.y + z.y));
              if (tok < c.len) {
                const float2 v = bf16x2_to_float2(vv[mt][half][kk]);
                s = fmaf(ut.x, v.x, fmaf(ut.y, v.y, s));
                const float be = betas[tok];
                if (kSum) *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(a.d_v) + ((row0 + tok) * ws.hv_all + h) * BD + col) = pack_bf16x2(be * ut.x, be * ut.y);
                else *reinterpret_cast<float2*>(a.d_v + ((row0 + tok) * ws.hv_all + h) * BD + col) = make_float2(be * ut.x, be * ut.y);
              }
            }
            s = quad_sum(s);
            if (t == 0) uv[wn * BCH + tok] = s;
          }
        }
      }
      tc::mbar_wait_warp(&bars[2], phase >> 2 & 1, abort_flag);
      phase ^= 4u;
      tc::tc_fence_after_sync();
      const int quarter = warp & 3, dk = 32 * quarter + lane;  // a warp reads the tensor-memory lanes of its quarter
      float states = 0.f;
#pragma unroll 1
      for (int pc = 0; pc < 2; ++pc) {
        const int tok0 = 16 * (warp >> 2) + 8 * pc;
        const uint32_t at = tm + ((uint32_t)(32 * quarter) << 16) + tok0;
        uint32_t xq[8], xr[8], xs[8], xk[8], yk[8], xc[8];
        tc::tmem_ld8(at + TG_Q, xq); tc::tmem_ld8(at + TG_R, xr); tc::tmem_ld8(at + TG_S, xs);
        tc::tmem_ld8(at + TG_XK, xk); tc::tmem_ld8(at + TG_YK, yk); tc::tmem_ld8(at + TG_COL, xc);
        tc::tmem_ld_wait();
        float v[16], dq[8], dkv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t off = (dk >> 6) * 8192 + piece<128>(tok0 + i, (dk & 63) >> 3) + 2 * (dk & 7);
          const float k = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(smem + GR_K + off));
          const float q = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(smem + GR_Q + off));
          const float4 f = fac[tok0 + i];
          const float gq = fmaf(f.x, __uint_as_float(xq[i]), __uint_as_float(xk[i]));
          const float row = fmaf(f.y, __uint_as_float(xr[i]), __uint_as_float(yk[i]));
          const float state = f.z * __uint_as_float(xs[i]), col = state + __uint_as_float(xc[i]);
          v[2 * i] = fmaf(q, gq, k * (row - col)); v[2 * i + 1] = k * row;
          states = fmaf(k, state, states);
          dq[i] = gq; dkv[i] = row + col;
        }
        const float sums = lane_sums(v, lane);
        if (lane < 16) reinterpret_cast<float*>(red + quarter * BCH + tok0)[lane] = sums;
        if (kSum && r > 1) {  // the sums over the heads so far wait in tensor memory
          if (hh > 0) {
            tc::tmem_ld8(at + TG_DQ, xq); tc::tmem_ld8(at + TG_DK, xr);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) { dq[i] += __uint_as_float(xq[i]); dkv[i] += __uint_as_float(xr[i]); }
          }
          if (hh < r - 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) { xq[i] = __float_as_uint(dq[i]); xr[i] = __float_as_uint(dkv[i]); }
            tc::tmem_st8(at + TG_DQ, xq); tc::tmem_st8(at + TG_DK, xr);
            tc::tmem_st_wait();
          }
        }
        if (!kSum || hh == r - 1) {
          store_dqk<kSum>(a, ws, a.d_q, c, kSum ? hk : h, tok0, dk, dq);
          store_dqk<kSum>(a, ws, a.d_k, c, kSum ? hk : h, tok0, dk, dkv);
        }
      }
      states = warp_sum(states);
      if (lane == 0) dots[16 + warp] = states;
      tc::tc_fence_before_sync();
      __syncthreads();
      if (tid < BCH) {  // dbeta, and dg as a suffix sum of db
        float2 s = red[tid];
        float su = 0.f, em = 0.f, st = 0.f;
#pragma unroll
        for (int w = 1; w < 4; ++w) { s.x += red[w * BCH + tid].x; s.y += red[w * BCH + tid].y; }
#pragma unroll
        for (int w = 0; w < 8; ++w) su += uv[w * BCH + tid];
#pragma unroll
        for (int w = 0; w < 16; ++w) { em += dots[w]; st += dots[16 + w]; }
        const float be = fabsf(betas[tid]) < 1e-20f ? 1e-20f : betas[tid];
        const int64_t off = (row0 + tid) * ws.hv_all + h;
        if (tid < c.len) a.d_beta[off] = su + s.y / be;
        float db = s.x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float x = __shfl_down_sync(0xffffffffu, db, o);
          if (lane + o < 32) db += x;
        }
        if (tid == 32) dots[32] = db;
        asm volatile("bar.sync 1, 64;" ::: "memory");
        if (warp == 0) db += dots[32];
        if (tid < c.len) a.d_g[off] = db + st + __expf(bs[BCH - 1]) * em;
      }
    }
  }
  __syncthreads();
  if (tid == 0 && *abort_flag != 0u && a.status != nullptr) atomicOr(a.status, AVE_GDN_DEV_WAIT_EXPIRED);
  if (warp == 1) tc::tmem_dealloc(*tmem_slot, 512);
}

// Scratch of a pass over nk key heads.
BwdScratch scratch_layout(const AveGdnBwdArgs& a, int nk, size_t* total) {
  BwdScratch ws;
  ws.hk_all = a.Hk; ws.hv_all = a.Hv;
  const size_t recs = (size_t)record_slots(a) * nk * (a.Hv / a.Hk);
  uint8_t* p = reinterpret_cast<uint8_t*>(a.workspace);
  size_t off = 0;
  auto take = [&](size_t bytes) { uint8_t* q = p + off; off += (recs * bytes + 255) & ~(size_t)255; return q; };
  ws.prep = take(PREP_BYTES);
  ws.m0 = reinterpret_cast<float*>(take(STATE_FLOATS * 4));
  ws.e = reinterpret_cast<float*>(take(STATE_FLOATS * 4));
  ws.vn = reinterpret_cast<float*>(take(VEC_FLOATS * 4));
  ws.u = reinterpret_cast<float*>(take(VEC_FLOATS * 4));
  if (total != nullptr) *total = off;
  return ws;
}

// The argument block of a pass over the nk key heads from hk0 on.
AveGdnBwdArgs pass_args(const AveGdnBwdArgs& a, int hk0, int nk) {
  const int r = a.Hv / a.Hk, h0 = hk0 * r;
  const bool sum = (a.flags & AVE_GDN_FLAG_BWD_SUMMED) != 0;
  AveGdnBwdArgs p = a;
  auto skip = [](auto& ptr, int64_t bytes) { if (ptr != nullptr) ptr = reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(reinterpret_cast<uintptr_t>(ptr) + bytes); };
  p.Hk = nk; p.Hv = nk * r;
  skip(p.q, hk0 * a.q_stride_h * 2); skip(p.k, hk0 * a.k_stride_h * 2);
  skip(p.v, h0 * a.v_stride_h * 2); skip(p.d_o, h0 * a.do_stride_h * 2);
  skip(p.g, (int64_t)h0 * 4); skip(p.beta, (int64_t)h0 * 4);
  for (auto* s : {&p.initial_state, &p.d_final_state}) skip(*s, (int64_t)h0 * STATE_FLOATS * 4);
  skip(p.d_initial_state, (int64_t)h0 * STATE_FLOATS * 4);
  for (auto* d : {&p.d_q, &p.d_k}) skip(*d, (int64_t)(sum ? hk0 * 2 : h0 * 4) * BD);
  skip(p.d_v, (int64_t)h0 * BD * (sum ? 2 : 4));
  skip(p.d_g, (int64_t)h0 * 4); skip(p.d_beta, (int64_t)h0 * 4);
  return p;
}

}  // namespace

// Bytes for a pass over nk of the a.Hk key heads.
size_t backward_workspace_bytes(const AveGdnBwdArgs& a, int nk) {
  size_t total = 0;
  scratch_layout(a, nk, &total);
  return total;
}

int launch_backward(const AveGdnBwdArgs& a, cudaStream_t stream) {
  if (a.n_seqs * a.Hv == 0 || a.T == 0) return AVE_GDN_OK;
  static bool attr_set_dev[64] = {};
  int dev = 0;
  AVE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return AVE_GDN_UNSUPPORTED;
  if (!attr_set_dev[dev]) {
    AVE_CUDA_TRY(cudaFuncSetAttribute(bwd_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(bwd_scans_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SC_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(bwd_grads_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(bwd_grads_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM));
    attr_set_dev[dev] = true;  // repeating the calls from another thread is harmless
  }
  int passes = 1, nk = a.Hk;  // as few passes as the scratch allows, of equal size
  while (nk > 1 && backward_workspace_bytes(a, nk) > a.workspace_bytes) nk = (a.Hk + passes) / (passes + 1), ++passes;
  const unsigned slots = (unsigned)record_slots(a);
  const bool sum = (a.flags & AVE_GDN_FLAG_BWD_SUMMED) != 0;
  for (int hk0 = 0; hk0 < a.Hk; hk0 += nk) {
    const AveGdnBwdArgs p = pass_args(a, hk0, min(nk, a.Hk - hk0));
    const BwdScratch ws = scratch_layout(a, p.Hk, nullptr);
    bwd_prep_kernel<<<dim3(slots, (unsigned)(p.Hk * ((p.Hv / p.Hk + 1) / 2))), PREP_T, PR_SMEM, stream>>>(p, ws);
    AVE_CUDA_TRY(cudaGetLastError());
    bwd_scans_kernel<<<2 * p.n_seqs * p.Hv, SC_T, SC_SMEM, stream>>>(p, ws);
    AVE_CUDA_TRY(cudaGetLastError());
    (sum ? bwd_grads_kernel<true> : bwd_grads_kernel<false>)<<<(unsigned)min((int64_t)GR_CTAS, (int64_t)slots * p.Hk), GR_T, GR_SMEM, stream>>>(p, ws, slots);
    AVE_CUDA_TRY(cudaGetLastError());
  }
  return AVE_GDN_OK;
}

}  // namespace ave
