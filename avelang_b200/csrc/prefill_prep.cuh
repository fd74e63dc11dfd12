// Pass 1 of the chunked prefill (d_k = d_v = 128): per (chunk, value head) the tiles the scan reads.
//     A = strict_lower(beta_i e^{b_i-b_j} k_i.k_j)    T = (I + A)^-1    P = scale lower(e^{b_i-b_j} q_i.k_j)
//     Tu = T diag(beta)    W^T = K^T (T diag(beta e^b))^T
// P, Tu and W^T leave as bf16 hi + lo tiles, each as the swizzled shared-memory image the scan's MMAs read.
//
// One CTA of eight warps per (chunk, key head, up to two of its value heads); K, Q and the Gram products K K^T and Q K^T
// are shared by the two.  The pass is bound by the instructions it issues and by their latency, so the products run on
// warp-level MMAs whose fragments are handed on in registers: the Gram fragments are gated in place; A is formed transposed
// (k_j.k_i, rows j), because that fragment is, element for element, the right operand of the block substitution; a row of
// 16x16 blocks of T,
//     T_rc = -(sum_{c < s <= r} T_rs A_sc) D_c,   D_c = (I + A_cc)^-1,
// is computed by one warp with every block staying in its accumulators (left operands again, in place); and the same
// accumulators scaled by beta e^b are the right operands of W^T.  fp32 operands enter as three bf16 terms (24 bits), the
// last product as two, like the tiles themselves.  Off the diagonal blocks the gate factors into
// e^{b_i - b_s} e^{b_s - b_j} with b_s the first gate of i's block (both exponents are <= 0), so 64 + 96 exponentials
// serve all but the diagonal blocks.  (Those take e^{b_i - b_j} element by element and drop the half above the diagonal, where
// the exponent is positive.)
// 132 k (chunk, head) units of a packed batch: 2.85 ms, 8.0 k warp instructions a unit; the form that took one head per CTA
// through tcgen05 products and CTA barriers needed 12.4 k instructions and 3.84 ms.
#pragma once
#include "wyblocks.cuh"

namespace ave {
namespace {

constexpr int PREP_THREADS = 256;
constexpr int PP_K = 0, PP_R = 16384;                         // K tile; per head a 16 KB region (head 0's holds the Q tile first)
constexpr int PP_F = PP_R + 2 * 16384, PP_F_HEAD = 16384;     // per head: off-diagonal A fragments | diagonal blocks; later W^T
static_assert(WY_BYTES <= PP_F_HEAD, "fragments and diagonal blocks must fit");
constexpr int PP_V = PP_F + 2 * PP_F_HEAD;                    // per head: vectors of 64 floats
enum { V_B, V_BETA, V_RA, V_RP, V_DA, V_DP, V_FW, V_W1, V_W2, V_W3, V_COUNT };
constexpr int PP_N = PP_V + 2 * V_COUNT * C * 4;              // row norms of k | q
constexpr size_t PREP_SMEM = PP_N + 2 * C * 4;

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float LOG2E = 1.4426950408889634f;
// Row R of 16x16 blocks of T, and with it rows / columns 16 R .. 16 R + 15 of Tu and W^T.  Called by one warp per R; the
// four warps of the head meet at named barriers.  `lead` (one lane of the head's warps) moves finished tiles out.
template <int R>
__device__ __forceinline__ void prep_row(uint8_t* smem, int hh, int lane, bool lead, const PrepOut& out, int64_t rec) {
  const int t = lane & 3;
  uint8_t* frag = smem + PP_F + hh * PP_F_HEAD;
  const float* vec = reinterpret_cast<const float*>(smem + PP_V) + hh * V_COUNT * C;
  float T[R + 1][2][4];
  wy_row<R>(T, frag, lane);
  if (lead) tc::bulk_wait_read<0>();  // the P tiles have been read out of the head's region
  head_sync(hh);                      // and nobody needs the fragments any more
  const uint32_t region = tc::smem_u32(smem + PP_R + hh * 16384);
#pragma unroll
  for (int c = 0; c <= R; ++c) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const float2 be = *reinterpret_cast<const float2*>(vec + V_BETA * C + 16 * c + 8 * nt + 2 * t);
      split_pair(__fmul2_rn(make_float2(T[c][nt][0], T[c][nt][1]), be), hi[2 * nt], lo[2 * nt]);
      split_pair(__fmul2_rn(make_float2(T[c][nt][2], T[c][nt][3]), be), hi[2 * nt + 1], lo[2 * nt + 1]);
    }
    const uint32_t at = region + at_a<128>(16 * R, 2 * c, lane);
    stsm4(at, hi[0], hi[1], hi[2], hi[3]);
    stsm4(at + REC_P, lo[0], lo[1], lo[2], lo[3]);
  }
  tc::fence_proxy_async_smem();
  head_sync(hh);
  if (lead) {
    tc::bulk_store(out.tu_hi + rec * (C * C), smem + PP_R + hh * 16384, REC_P);
    tc::bulk_store(out.tu_lo + rec * (C * C), smem + PP_R + hh * 16384 + REC_P, REC_P);
    tc::bulk_commit();
  }
  // W^T[d_k][16 R ..] = sum_c K_c^T Tw_Rc^T, 64 rows of d_k at a time: the first half through the fragments' space, the
  // second through the region once Tu has left it
  uint32_t wh[R + 1][4], wl[R + 1][4];
#pragma unroll
  for (int c = 0; c <= R; ++c)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const float2 fw = *reinterpret_cast<const float2*>(vec + V_FW * C + 16 * c + 8 * nt + 2 * t);
      split_pair(__fmul2_rn(make_float2(T[c][nt][0], T[c][nt][1]), fw), wh[c][nt], wl[c][nt]);
      split_pair(__fmul2_rn(make_float2(T[c][nt][2], T[c][nt][3]), fw), wh[c][2 + nt], wl[c][2 + nt]);
    }
  const uint32_t k_tile = tc::smem_u32(smem + PP_K);
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const uint32_t dst = half == 0 ? tc::smem_u32(frag) : region;
    if (half == 1) {
      if (lead) tc::bulk_wait_read<1>();  // all but the newest group: the Tu tiles
      head_sync(hh);
    }
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      float acc[2][4];
      zero(acc[0]); zero(acc[1]);
#pragma unroll
      for (int c = 0; c <= R; ++c) {
        uint32_t k[4];
        ldsm4t(k, k_tile + at_at<256>(16 * c, 8 * half + 2 * mt, lane));
        mma_bf16(acc[0], k, wh[c][0], wh[c][1]);
        mma_bf16(acc[1], k, wh[c][2], wh[c][3]);
        mma_bf16(acc[0], k, wl[c][0], wl[c][1]);
        mma_bf16(acc[1], k, wl[c][2], wl[c][3]);
      }
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        split_pair(make_float2(acc[nt][0], acc[nt][1]), hi[2 * nt], lo[2 * nt]);
        split_pair(make_float2(acc[nt][2], acc[nt][3]), hi[2 * nt + 1], lo[2 * nt + 1]);
      }
      const uint32_t at = dst + at_a<128>(16 * mt, 2 * R, lane);
      stsm4(at, hi[0], hi[1], hi[2], hi[3]);
      stsm4(at + REC_W / 2, lo[0], lo[1], lo[2], lo[3]);
    }
    tc::fence_proxy_async_smem();
    head_sync(hh);
    if (lead) {
      const uint8_t* src = half == 0 ? frag : smem + PP_R + hh * 16384;
      tc::bulk_store(out.w_hi + rec * (C * D) + half * (C * D / 2), src, REC_W / 2);
      tc::bulk_store(out.w_lo + rec * (C * D) + half * (C * D / 2), src + REC_W / 2, REC_W / 2);
      tc::bulk_commit();
    }
  }
  if (lead) tc::bulk_wait_read<0>();  // shared memory must stay intact until the copies have read it
}

__global__ void __launch_bounds__(PREP_THREADS, 2)
chunk_prep_kernel(const AveGdnArgs a, const int32_t* chunk_start, PrepOut out, const __grid_constant__ ScanPlan plan,
                  int compact_grid) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  pdl_trigger();
  pdl_wait();
  if (batch_rejected(a, chunk_start, blockIdx.x == 0 && blockIdx.y == 0)) return;
  // Whole-batch launches index every chunk of the batch; range launches use the compact grid
  // n_seqs x parts x rn so that no CTA is spent on chunks outside the range.
  int c = blockIdx.x;
  if (compact_grid) {
    const int per_seq = plan.parts * plan.rn;
    const int n = blockIdx.x / per_seq, rest = blockIdx.x % per_seq;
    const int cis = plan.part_begin[rest / plan.rn] + plan.r0 + rest % plan.rn;
    const int per = ((a.cu_seqlens ? a.cu_seqlens[n + 1] - a.cu_seqlens[n] : a.T) + C - 1) / C;
    if (cis >= per || cis >= plan.part_begin[rest / plan.rn + 1]) return;
    c = first_record(a, chunk_start, n) + cis;
  }
  const ChunkRef cr = find_chunk(a, chunk_start, c);  // (a compact grid only ever names chunks of this launch's range)
  if (!cr.ok) return;
  const int r = a.Hv / a.Hk, pairs = (r + 1) / 2;
  const int hk = blockIdx.y / pairs, h0 = hk * r + 2 * (blockIdx.y % pairs), nh = min(2, hk * r + r - h0);
  const uint32_t sb = tc::smem_u32(smem);
  float* kn = reinterpret_cast<float*>(smem + PP_N);
  float* qn = kn + C;
  float* vecs = reinterpret_cast<float*>(smem + PP_V);

  load_tile<C, 16, PREP_THREADS>(sb + PP_K, reinterpret_cast<const __nv_bfloat16*>(a.k) + cr.b * a.k_stride_b + (int64_t)cr.t0 * a.k_stride_t + (int64_t)hk * a.k_stride_h,
                                 a.k_stride_t, cr.len, tid);
  load_tile<C, 16, PREP_THREADS>(sb + PP_R, reinterpret_cast<const __nv_bfloat16*>(a.q) + cr.b * a.q_stride_b + (int64_t)cr.t0 * a.q_stride_t + (int64_t)hk * a.q_stride_h,
                                 a.q_stride_t, cr.len, tid);
  cp_commit();
  if (warp < nh) {  // in-chunk cumulative gate: inclusive scan of 64 values by one warp per head
    const int64_t off = cr.b * a.g_stride_b + (int64_t)cr.t0 * a.g_stride_t + h0 + warp;
    float* vec = vecs + warp * V_COUNT * C;
    const bool in0 = lane < cr.len, in1 = lane + 32 < cr.len;
    float v0 = in0 ? a.g[off + lane * a.g_stride_t] : 0.f, v1 = in1 ? a.g[off + (lane + 32) * a.g_stride_t] : 0.f;
    vec[V_BETA * C + lane] = in0 ? a.beta[off + lane * a.g_stride_t] : 0.f;
    vec[V_BETA * C + lane + 32] = in1 ? a.beta[off + (lane + 32) * a.g_stride_t] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t0 = __shfl_up_sync(0xffffffffu, v0, o), t1 = __shfl_up_sync(0xffffffffu, v1, o);
      if (lane >= o) { v0 += t0; v1 += t1; }
    }
    v1 += __shfl_sync(0xffffffffu, v0, 31);
    vec[V_B * C + lane] = v0; vec[V_B * C + lane + 32] = v1;
  }
  cp_wait<0>();
  __syncthreads();

  // Gram products.  Warps 0..3: rows of K block `warp` against the blocks from it on (A transposed); warps 4..7: rows of Q
  // block `warp - 4` against the K blocks up to it.  acc[2 x] and acc[2 x + 1]: the x-th of those blocks.
  const int m = warp & 3;
  const bool is_p = warp >= 4;
  const int first = is_p ? 0 : m, count = is_p ? m + 1 : 4 - m;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) zero(acc[i]);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    uint32_t af[4];
    ldsm4(af, sb + (is_p ? PP_R : PP_K) + at_a<256>(16 * m, 2 * ks, lane));
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      if (x >= count) break;
      uint32_t b[4];
      ldsm4(b, sb + PP_K + at_b<256>(16 * (first + x), 2 * ks, lane));
      mma_bf16(acc[2 * x], af, b[0], b[1]);
      mma_bf16(acc[2 * x + 1], af, b[2], b[3]);
    }
  }
  if (a.flags & AVE_GDN_FLAG_QK_L2NORM) {  // four threads per row; the swizzle permutes pieces inside a row, a sum needs no decode
    const int i = tid >> 2, part = tid & 3;
    float sk = 0.f, sq = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint4 kr = *reinterpret_cast<const uint4*>(smem + PP_K + i * 256 + ((part + 4 * e) << 4));
      const uint4 qr = *reinterpret_cast<const uint4*>(smem + PP_R + i * 256 + ((part + 4 * e) << 4));
      const uint32_t kw[4] = {kr.x, kr.y, kr.z, kr.w}, qw[4] = {qr.x, qr.y, qr.z, qr.w};
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float2 kf = bf16x2_to_float2(kw[w]), qf = bf16x2_to_float2(qw[w]);
        sk += kf.x * kf.x + kf.y * kf.y; sq += qf.x * qf.x + qf.y * qf.y;
      }
    }
    sk += __shfl_xor_sync(0xffffffffu, sk, 1); sk += __shfl_xor_sync(0xffffffffu, sk, 2);
    sq += __shfl_xor_sync(0xffffffffu, sq, 1); sq += __shfl_xor_sync(0xffffffffu, sq, 2);
    if (part == 0) { kn[i] = rsqrtf(sk + 1e-6f); qn[i] = rsqrtf(sq + 1e-6f); }
  } else if (tid < C) { kn[tid] = 1.f; qn[tid] = 1.f; }
  __syncthreads();
  if (tid < 128) {  // per-token factors, and the scale vectors of the scan
    const int hh = tid >> 6, i = tid & 63;
    if (hh < nh) {
      float* vec = vecs + hh * V_COUNT * C;
      const float* bs = vec + V_B * C;
      const float b = bs[i], bC = bs[C - 1], be = vec[V_BETA * C + i], k = kn[i], q = i < cr.len ? qn[i] * a.scale : 0.f;
      const float u = ex2_approx((b - bs[i & 48]) * LOG2E);
      vec[V_RA * C + i] = be * k * u; vec[V_RP * C + i] = q * u;
      vec[V_DA * C + i] = be * k; vec[V_DP * C + i] = q;
      vec[V_FW * C + i] = be * __expf(b) * k;
#pragma unroll
      for (int s = 1; s < 4; ++s) vec[(V_W1 + s - 1) * C + i] = i < 16 * s ? ex2_approx((bs[16 * s] - b) * LOG2E) * k : 0.f;
      float* sc = out.scal + ((int64_t)c * a.Hv + h0 + hh) * SCAL_FLOATS;
      sc[i] = __expf(b) * qn[i] * a.scale;     // o_i = qs_i (H q_i) + (scale P Vn)_i: the output scale is folded in here and in P
      sc[C + i] = __expf(bC - b) * k;          // Vd_j = ks_j Vn_j
      sc[2 * C + i] = __expf(bC);
    }
  } else {  // blocks above the diagonal are zero in P and in Tu: once per region
    for (int e = tid - 128; e < nh * 2 * 6 * 32; e += 128) {
      const int blk = (e >> 5) % 6, row = (blk < 3 ? 0 : blk < 5 ? 1 : 2), col = (blk < 3 ? blk + 1 : blk < 5 ? blk - 1 : 3);
      *reinterpret_cast<uint4*>(smem + PP_R + ((e >> 5) / 6) * REC_P + piece<128>(16 * row + ((e & 31) >> 1), 2 * col + (e & 1))) =
          make_uint4(0u, 0u, 0u, 0u);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int hh = 0; hh < nh; ++hh) {
    const float* vec = vecs + hh * V_COUNT * C;
    const float* bs = vec + V_B * C;
    if (!is_p) {  // element (row j = 16 m + g + 8 hf, column i = 16 s + 8 nt + 2 t + e) of the transposed A
      float* ad = reinterpret_cast<float*>(smem + PP_F + hh * PP_F_HEAD + WY_DIAG) + m * 16 * AD_LD;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = g + 8 * (e >> 1), i = 8 * nt + 2 * t + (e & 1);
          const float x = acc[nt][e] * vec[V_DA * C + 16 * m + i] * kn[16 * m + j] * ex2_approx((bs[16 * m + i] - bs[16 * m + j]) * LOG2E);
          ad[i * AD_LD + j] = i > j ? x : 0.f;
        }
#pragma unroll
      for (int x = 1; x < 4; ++x) {
        if (x >= count) break;
        const int s = m + x;
        const float w0 = vec[(V_W1 + s - 1) * C + 16 * m + g], w1 = vec[(V_W1 + s - 1) * C + 16 * m + g + 8];
        const float2 r0 = *reinterpret_cast<const float2*>(vec + V_RA * C + 16 * s + 2 * t), r1 = *reinterpret_cast<const float2*>(vec + V_RA * C + 16 * s + 8 + 2 * t);
        uint32_t ah[4], am[4], al[4];
        auto gate = [&](int idx, const float* p, float2 rr, float w) {
          split3(__fmul2_rn(__fmul2_rn(make_float2(p[0], p[1]), rr), make_float2(w, w)), ah[idx], am[idx], al[idx]);
        };
        gate(0, acc[2 * x], r0, w0); gate(1, acc[2 * x + 1], r1, w0);
        gate(2, acc[2 * x] + 2, r0, w1); gate(3, acc[2 * x + 1] + 2, r1, w1);
        uint4* f = reinterpret_cast<uint4*>(smem + PP_F + hh * PP_F_HEAD + (s * (s - 1) / 2 + m) * WY_BLOCK) + lane;
        f[0] = make_uint4(ah[0], ah[1], ah[2], ah[3]);
        f[32] = make_uint4(am[0], am[1], am[2], am[3]);
        f[64] = make_uint4(al[0], al[1], al[2], al[3]);
      }
    } else {  // element (row i = 16 m + g + 8 hf, column j = 16 x + 8 nt + 2 t + e) of P
      const uint32_t region = sb + PP_R + hh * 16384;
      const float* w = vec + (V_W1 + m - 1) * C;  // (m = 0 has no off-diagonal block)
      const float p0 = vec[V_RP * C + 16 * m + g], p1 = vec[V_RP * C + 16 * m + g + 8];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        if (x >= count) break;
        uint32_t hi[4], lo[4];
        if (x < m) {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const float2 wj = *reinterpret_cast<const float2*>(w + 16 * x + 8 * nt + 2 * t);
            const float* p = acc[2 * x + nt];
            split_pair(__fmul2_rn(__fmul2_rn(make_float2(p[0], p[1]), wj), make_float2(p0, p0)), hi[2 * nt], lo[2 * nt]);
            split_pair(__fmul2_rn(__fmul2_rn(make_float2(p[2], p[3]), wj), make_float2(p1, p1)), hi[2 * nt + 1], lo[2 * nt + 1]);
          }
        } else {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              const int i = g + 8 * hf, j = 8 * nt + 2 * t;
              const float f = vec[V_DP * C + 16 * m + i], bi = bs[16 * m + i];
              const float* p = acc[2 * x + nt] + 2 * hf;
              const float y0 = p[0] * f * kn[16 * m + j] * ex2_approx((bi - bs[16 * m + j]) * LOG2E);
              const float y1 = p[1] * f * kn[16 * m + j + 1] * ex2_approx((bi - bs[16 * m + j + 1]) * LOG2E);
              split_pair(make_float2(i >= j ? y0 : 0.f, i > j ? y1 : 0.f), hi[2 * nt + hf], lo[2 * nt + hf]);
            }
        }
        const uint32_t at = region + at_a<128>(16 * m, 2 * x, lane);
        stsm4(at, hi[0], hi[1], hi[2], hi[3]);
        stsm4(at + REC_P, lo[0], lo[1], lo[2], lo[3]);
      }
    }
  }
  tc::fence_proxy_async_smem();
  __syncthreads();

  const int hh = warp >> 2;
  if (hh >= nh) return;
  const int64_t rec = (int64_t)c * a.Hv + h0 + hh;
  // Block row R of T costs R + 1 units of work and the warps 0 and 4, 1 and 5, ... share a scheduler, so the second head
  // hands its rows out in the opposite order
  const int row = hh == 0 ? 3 - warp : warp - 4;
  const bool lead = row == 0 && lane == 0;  // in the warp with the least work
  if (lead) {
    tc::bulk_store(out.p_hi + rec * (C * C), smem + PP_R + hh * 16384, REC_P);
    tc::bulk_store(out.p_lo + rec * (C * C), smem + PP_R + hh * 16384 + REC_P, REC_P);
    tc::bulk_commit();
  }
  if (row >= 2) wy_invert(smem + PP_F + hh * PP_F_HEAD, row & 1, lane);
  head_sync(hh);
  switch (row) {
    case 3: prep_row<3>(smem, hh, lane, lead, out, rec); break;
    case 2: prep_row<2>(smem, hh, lane, lead, out, rec); break;
    case 1: prep_row<1>(smem, hh, lane, lead, out, rec); break;
    default: prep_row<0>(smem, hh, lane, lead, out, rec); break;
  }
}

}  // namespace
}  // namespace ave
