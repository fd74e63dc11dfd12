// Chunked gated-delta-rule prefill for d_k = d_v = 64 (chunk 64), fp32 accuracy.
//
// The recurrence over the chunks is linear in the state (H = M^T, [d_v][d_k]; b the in-chunk cumulative gate, T, P as in
// the WY form, D_i = e^{b_C - b_i}):
//     H' = H Phi + Gam,   Z = T^T diag(D) K,   Phi = e^{b_C} I - K^T diag(beta e^b) Z,   Gam = V^T diag(beta) Z
//     Vn = T diag(beta) (V - diag(e^b) K H^T),   O = scale (diag(e^b) Q H^T + P Vn)
// so only one 64x64x64 product per chunk is sequential.  Three launches: d64_prep forms T, P, Phi and Gam of every (chunk,
// head) in parallel; d64_chain carries the state along a sequence, in fp32 on the CUDA cores, 16 of the 64 independent
// rows of H per CTA; d64_out forms the outputs of every chunk in parallel from the states, with the gated norm fused.
// The parallel launches use warp-level bf16 MMAs; bf16 inputs enter as they are and every fp32 operand as three bf16 terms
// (24 bits).
// A chain of SIMT chunk steps (18 us each, all four products and the copies in one CTA) took 104.8 us for 256 tokens and
// four heads.
#include "blockalg.cuh"
#include "common.cuh"
#include "recslots.cuh"
#include "tc.cuh"
#include "warpmma.cuh"

namespace ave {
namespace {

constexpr int CH = 64, DH = 64, IMG = CH * CH * 2, THREADS = 256;
// one record per (chunk slot, head)
constexpr int R_T = 0, R_P = 3 * IMG, R_PHI = 6 * IMG, R_GAM = R_PHI + DH * DH * 4, R_H = R_GAM + DH * DH * 4, R_SC = R_H + DH * DH * 4,
              SC_FLOATS = 5 * CH, REC_BYTES = R_SC + SC_FLOATS * 4;  // T h m l | P h m l | Phi | Gam | H | b, beta, low b, |q|^-1, |k|^-1

// three bf16 terms of a pair -> images at `at`, `at` + IMG, `at` + 2 IMG
__device__ __forceinline__ void put3(uint8_t* at, float x, float y) {
  uint32_t h, m, l;
  split3(make_float2(x, y), h, m, l);
  *reinterpret_cast<uint32_t*>(at) = h;
  *reinterpret_cast<uint32_t*>(at + IMG) = m;
  *reinterpret_cast<uint32_t*>(at + 2 * IMG) = l;
}
// acc[0..3] (16 rows x 32 columns) += A B over one 16-wide step, A exact, B three terms stored with rows = contraction
// index (kTrans) or rows = columns
template <bool kTrans>
__device__ __forceinline__ void step3(float (&acc)[4][4], const uint32_t (&af)[4], uint32_t b_tile, int k0, int n0, int lane) {
#pragma unroll
  for (int np = 0; np < 2; ++np)
#pragma unroll
    for (int term = 0; term < 3; ++term) {
      uint32_t b[4];
      if (kTrans) ldsm4t(b, b_tile + term * IMG + at_bt<128>(k0, (n0 >> 3) + 2 * np, lane));
      else ldsm4(b, b_tile + term * IMG + at_b<128>(n0 + 16 * np, k0 >> 3, lane));
      mma_bf16(acc[2 * np], af, b[0], b[1]);
      mma_bf16(acc[2 * np + 1], af, b[2], b[3]);
    }
}

// ---------------------------------------------------------------------------------------------- T, P, Phi, Gam
constexpr int PQ_K = 0, PQ_Q = 8192, PQ_V = 16384, PQ_TD = 24576, PQ_Z2 = PQ_TD + 3 * IMG, PQ_BLK = PQ_Z2 + 3 * IMG;
constexpr int PQ_A = PQ_BLK, PQ_D = PQ_A + 10 * BLK_FLOATS * 4, PQ_E = PQ_D + 4 * BLK_FLOATS * 4, PQ_BLK_END = PQ_E + 10 * BLK_FLOATS * 4;
constexpr int PQ_Z1 = PQ_BLK;  // the blocks are dead when Z exists
static_assert(PQ_Z1 + 3 * IMG <= PQ_BLK_END, "Z must fit where the blocks were");
constexpr int PQ_SC = PQ_BLK_END, PQ_SMEM = PQ_SC + SC_FLOATS * 4;

__global__ void __launch_bounds__(THREADS) d64_prep_kernel(const AveGdnArgs a, uint8_t* recs) {
  extern __shared__ __align__(1024) uint8_t smem[];
  float* Ab = reinterpret_cast<float*>(smem + PQ_A);
  float* Di = reinterpret_cast<float*>(smem + PQ_D);
  float* Eb = reinterpret_cast<float*>(smem + PQ_E);
  float* E2b = Eb + 6 * BLK_FLOATS;
  float* E3b = E2b + 3 * BLK_FLOATS;
  float* bs = reinterpret_cast<float*>(smem + PQ_SC);
  float *betas = bs + CH, *qn = bs + 3 * CH, *kn = bs + 4 * CH;
  const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  pdl_trigger();
  pdl_wait();
  if (!offsets_ok(a, blockIdx.x == 0 && h == 0)) return;
  const SlotChunk c = chunk_of_slot(a, blockIdx.x);
  if (!c.ok) return;
  const int hk = h / (a.Hv / a.Hk);
  uint8_t* rec = recs + ((int64_t)blockIdx.x * a.Hv + h) * REC_BYTES;
  const uint32_t sb = tc::smem_u32(smem);
  load_tile<CH, 8, THREADS>(sb + PQ_K, bf(a.k) + c.b * a.k_stride_b + (int64_t)c.t0 * a.k_stride_t + (int64_t)hk * a.k_stride_h, a.k_stride_t, c.len, tid);
  load_tile<CH, 8, THREADS>(sb + PQ_Q, bf(a.q) + c.b * a.q_stride_b + (int64_t)c.t0 * a.q_stride_t + (int64_t)hk * a.q_stride_h, a.q_stride_t, c.len, tid);
  load_tile<CH, 8, THREADS>(sb + PQ_V, bf(a.v) + c.b * a.v_stride_b + (int64_t)c.t0 * a.v_stride_t + (int64_t)h * a.v_stride_h, a.v_stride_t, c.len, tid);
  cp_commit();
  if (warp == 0) {  // inclusive scan of the gates in double, kept as two floats
    const int64_t off = c.b * a.g_stride_b + (int64_t)c.t0 * a.g_stride_t + h;
    const bool in0 = lane < c.len, in1 = lane + 32 < c.len;
    double v0 = in0 ? a.g[off + lane * a.g_stride_t] : 0.f, v1 = in1 ? a.g[off + (lane + 32) * a.g_stride_t] : 0.f;
    betas[lane] = in0 ? a.beta[off + lane * a.g_stride_t] : 0.f;
    betas[lane + 32] = in1 ? a.beta[off + (lane + 32) * a.g_stride_t] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t0 = __shfl_up_sync(0xffffffffu, v0, o), t1 = __shfl_up_sync(0xffffffffu, v1, o);
      if (lane >= o) { v0 += t0; v1 += t1; }
    }
    v1 += __shfl_sync(0xffffffffu, v0, 31);
    bs[lane] = (float)v0; bs[lane + 32] = (float)v1;
    bs[2 * CH + lane] = (float)(v0 - (float)v0); bs[2 * CH + lane + 32] = (float)(v1 - (float)v1);
  }
  cp_wait<0>();
  __syncthreads();
  if (a.flags & AVE_GDN_FLAG_QK_L2NORM) {  // four threads per row
    const int i = tid >> 2, part = tid & 3;
    float sk = 0.f, sq = 0.f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint4 kr = *reinterpret_cast<const uint4*>(smem + PQ_K + i * 128 + ((part + 4 * e) << 4));
      const uint4 qr = *reinterpret_cast<const uint4*>(smem + PQ_Q + i * 128 + ((part + 4 * e) << 4));
      const uint32_t kw[4] = {kr.x, kr.y, kr.z, kr.w}, qw[4] = {qr.x, qr.y, qr.z, qr.w};
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float2 kf = bf16x2_to_float2(kw[w]), qf = bf16x2_to_float2(qw[w]);
        sk += kf.x * kf.x + kf.y * kf.y; sq += qf.x * qf.x + qf.y * qf.y;
      }
    }
    sk = sk + __shfl_xor_sync(0xffffffffu, sk, 1); sk += __shfl_xor_sync(0xffffffffu, sk, 2);
    sq = sq + __shfl_xor_sync(0xffffffffu, sq, 1); sq += __shfl_xor_sync(0xffffffffu, sq, 2);
    if (part == 0) { kn[i] = rsqrtf(sk + 1e-6f); qn[i] = rsqrtf(sq + 1e-6f); }
  } else if (tid < CH) { kn[tid] = 1.f; qn[tid] = 1.f; }
  __syncthreads();
  for (int e = tid; e < SC_FLOATS; e += THREADS) reinterpret_cast<float*>(rec + R_SC)[e] = bs[e];
  {  // warps 0..3: rows 16m.. of K K^T -> A;  warps 4..7: rows 16m.. of Q K^T -> P.  Blocks above the diagonal are skipped.
    const int m = warp & 3;
    const bool is_p = warp >= 4;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) zero(acc[i]);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t af[4];
      ldsm4(af, sb + (is_p ? PQ_Q : PQ_K) + at_a<128>(16 * m, 2 * ks, lane));
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        if (np > m) break;
        uint32_t b[4];
        ldsm4(b, sb + PQ_K + at_b<128>(16 * np, 2 * ks, lane));
        mma_bf16(acc[2 * np], af, b[0], b[1]);
        mma_bf16(acc[2 * np + 1], af, b[2], b[3]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int i = 16 * m + g + 8 * half, j = 8 * nt + 2 * t;
        const float x0 = gate_between(bs, i, j) * kn[j] * acc[nt][2 * half], x1 = gate_between(bs, i, j + 1) * kn[j + 1] * acc[nt][2 * half + 1];
        if (is_p) {
          const float f = qn[i];
          put3(rec + R_P + piece<128>(i, nt) + 4 * t, i >= j ? f * x0 : 0.f, i > j ? f * x1 : 0.f);
        } else if (nt <= 2 * m + 1) {
          const float f = betas[i] * kn[i];
          *reinterpret_cast<float2*>(Ab + tri(m, nt >> 1) * BLK_FLOATS + (i & 15) * BLK_LD + (j & 15)) =
              make_float2(i > j ? f * x0 : 0.f, i > j + 1 ? f * x1 : 0.f);
        }
      }
  }
  __syncthreads();
  // T = (I + A)^-1 by 16x16 blocks: D = blockdiag(I + A_rr), E = D^-1 (A - A_D), T = (I - E + E^2 - E^3) D^-1
  if (tid < 64) {
    const int r = tid >> 4, k = tid & 15;
    const float* Arr = Ab + tri(r, r) * BLK_FLOATS;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s0 = (i == k) ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) {
        const float av = Arr[i * BLK_LD + j];
        if (j & 1) s1 = fmaf(-av, x[j], s1); else s0 = fmaf(-av, x[j], s0);
      }
      x[i] = s0 + s1;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) Di[r * BLK_FLOATS + i * BLK_LD + k] = x[i];
  }
  __syncthreads();
  constexpr int RR[6] = {1, 2, 2, 3, 3, 3}, CC[6] = {0, 0, 1, 0, 1, 2};
  auto Eblk = [&](int r, int cc) { return Eb + (tri(r, cc) - r) * BLK_FLOATS; };
  auto plain = [](const float* L) { return [L](int row, int col) { return L[row * BLK_LD + col]; }; };
  if (warp < 6) {
    const int r = RR[warp], cc = CC[warp];
    float acc[2][4] = {};
    block_mma(acc, plain(Di + r * BLK_FLOATS), Ab + tri(r, cc) * BLK_FLOATS, lane);
    block_store(Eblk(r, cc), acc, lane);
  }
  __syncthreads();
  if (warp < 3) {  // E^2: (2,0), (3,1), (3,0)
    float acc[2][4] = {};
    if (warp == 0) block_mma(acc, plain(Eblk(2, 1)), Eblk(1, 0), lane);
    else if (warp == 1) block_mma(acc, plain(Eblk(3, 2)), Eblk(2, 1), lane);
    else { block_mma(acc, plain(Eblk(3, 1)), Eblk(1, 0), lane); block_mma(acc, plain(Eblk(3, 2)), Eblk(2, 0), lane); }
    block_store(E2b + warp * BLK_FLOATS, acc, lane);
  }
  __syncthreads();
  if (warp == 0) {
    float acc[2][4] = {};
    block_mma(acc, plain(Eblk(3, 2)), E2b, lane);
    block_store(E3b, acc, lane);
  }
  __syncthreads();
  if (warp < 6) {
    const int r = RR[warp], cc = CC[warp];
    const float* e1 = Eblk(r, cc);
    const float* e2 = (r - cc >= 2) ? E2b + ((r == 2) ? 0 : (cc == 1 ? 1 : 2)) * BLK_FLOATS : nullptr;
    const float* e3 = (r - cc == 3) ? E3b : nullptr;
    float acc[2][4] = {};
    block_mma(acc, [&](int row, int col) {
      float v = -e1[row * BLK_LD + col];
      if (e2 != nullptr) v += e2[row * BLK_LD + col];
      if (e3 != nullptr) v -= e3[row * BLK_LD + col];
      return v;
    }, Di + cc * BLK_FLOATS, lane);
    block_store(Ab + tri(r, cc) * BLK_FLOATS, acc, lane);
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < 2; ++it) {  // T to the record, diag(D |k|^-1) T as an operand tile
    const int i = (tid >> 3) + 32 * it, rb = i >> 4, pc = tid & 7, cb = pc >> 1;
    const float d = gate_between(bs, CH - 1, i) * kn[i];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      float2 x = make_float2(0.f, 0.f);
      if (cb <= rb) {
        const float* src = ((rb == cb) ? Di + rb * BLK_FLOATS : Ab + tri(rb, cb) * BLK_FLOATS) + (i & 15) * BLK_LD + (pc & 1) * 8 + 2 * w;
        const int j = 8 * pc + 2 * w;
        x = make_float2(j <= i ? src[0] : 0.f, j + 1 <= i ? src[1] : 0.f);
      }
      put3(rec + R_T + piece<128>(i, pc) + 4 * w, x.x, x.y);
      put3(smem + PQ_TD + piece<128>(i, pc) + 4 * w, d * x.x, d * x.y);
    }
  }
  __syncthreads();
  const int m = warp & 3, n0 = 32 * (warp >> 2);  // this warp's 16 rows and 32 columns of Z, Phi and Gam
  {
    float z[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) zero(z[i]);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {  // Z_j takes the tokens from j on
      if (ks < m) continue;
#pragma unroll
      for (int term = 2; term >= 0; --term) {
        uint32_t af[4];
        ldsm4t(af, sb + PQ_TD + term * IMG + at_at<128>(16 * ks, 2 * m, lane));
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t b[4];
          ldsm4t(b, sb + PQ_K + at_bt<128>(16 * ks, (n0 >> 3) + 2 * np, lane));
          mma_bf16(z[2 * np], af, b[0], b[1]);
          mma_bf16(z[2 * np + 1], af, b[2], b[3]);
        }
      }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int j = 16 * m + g + 8 * half;
      const float f2 = betas[j], f1 = f2 * __expf(bs[j]) * kn[j];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const uint32_t at = piece<128>(j, (n0 >> 3) + nt) + 4 * t;
        put3(smem + PQ_Z1 + at, f1 * z[nt][2 * half], f1 * z[nt][2 * half + 1]);
        put3(smem + PQ_Z2 + at, f2 * z[nt][2 * half], f2 * z[nt][2 * half + 1]);
      }
    }
  }
  __syncthreads();
  float phi[4][4], gam[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) { zero(phi[i]); zero(gam[i]); }
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    uint32_t kf[4], vf[4];
    ldsm4t(kf, sb + PQ_K + at_at<128>(16 * ks, 2 * m, lane));
    ldsm4t(vf, sb + PQ_V + at_at<128>(16 * ks, 2 * m, lane));
    step3<true>(phi, kf, sb + PQ_Z1, 16 * ks, n0, lane);
    step3<true>(gam, vf, sb + PQ_Z2, 16 * ks, n0, lane);
  }
  const float decay = __expf(bs[CH - 1]);
#pragma unroll
  for (int half = 0; half < 2; ++half)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int row = 16 * m + g + 8 * half, col = n0 + 8 * nt + 2 * t;
      *reinterpret_cast<float2*>(rec + R_PHI + (row * DH + col) * 4) =
          make_float2((row == col ? decay : 0.f) - phi[nt][2 * half], (row == col + 1 ? decay : 0.f) - phi[nt][2 * half + 1]);
      *reinterpret_cast<float2*>(rec + R_GAM + (row * DH + col) * 4) = make_float2(gam[nt][2 * half], gam[nt][2 * half + 1]);
    }
}

// ---------------------------------------------------------------------------------------------- the chain of states
// One CTA of 128 threads per (sequence, head, 16 rows of H); a thread owns two rows and four columns.
constexpr int CN_T = 128, CN_ROWS = 16, CN_LD = DH + 4;
constexpr int CN_PHI = 0, CN_GAM = DH * DH * 4, CN_STAGE = CN_GAM + CN_ROWS * DH * 4, CN_SMEM = 3 * CN_STAGE;

__global__ void __launch_bounds__(CN_T) d64_chain_kernel(const AveGdnArgs a, uint8_t* recs) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(16) float Hs[2][CN_ROWS][CN_LD];
  const int tid = threadIdx.x, n = blockIdx.x, h = blockIdx.y, row0 = blockIdx.z * CN_ROWS;
  pdl_trigger();
  pdl_wait();
  if (!offsets_ok(a, false)) return;
  const SeqSpan sp = seq_span(a.cu_seqlens, n, a.T, nullptr);
  if (!sp.ok) return;
  int slot = n;
  if (a.state_indices != nullptr) {
    slot = a.state_indices[n];
    if (slot >= a.num_slots && a.status != nullptr && tid == 0) atomicOr(a.status, AVE_GDN_DEV_BAD_SLOT);
    if (slot < 0 || slot >= a.num_slots) return;  // no state access; d64_out writes zeros
  }
  const int64_t tile = ((int64_t)slot * a.Hv + h) * (DH * DH);
  const int rr = (tid >> 4) * 2, col = (tid & 15) * 4;
  const int n_chunks = (sp.len + CH - 1) / CH;
  uint8_t* rec = recs + (first_slot(a, n) * a.Hv + h) * REC_BYTES;
  const int64_t step = (int64_t)a.Hv * REC_BYTES;
  const uint32_t sb = tc::smem_u32(smem);
  auto load = [&](int c) {  // Phi whole, 16 rows of Gam
    const uint8_t* src = rec + c * step;
    const uint32_t st = sb + (c % 3) * CN_STAGE;
#pragma unroll
    for (int i = 0; i < DH * DH * 4 / 16 / CN_T; ++i) cp16(st + CN_PHI + (tid + i * CN_T) * 16, src + R_PHI + (tid + i * CN_T) * 16, true);
#pragma unroll
    for (int i = 0; i < CN_ROWS * DH * 4 / 16 / CN_T; ++i) cp16(st + CN_GAM + (tid + i * CN_T) * 16, src + R_GAM + row0 * DH * 4 + (tid + i * CN_T) * 16, true);
  };
  if (n_chunks > 0) load(0);
  cp_commit();
  if (n_chunks > 1) load(1);
  cp_commit();
  float4 H[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = a.initial_state ? a.initial_state[tile + (int64_t)(col + e) * DH + row0 + rr + r] : 0.f;
    H[r] = make_float4(x[0], x[1], x[2], x[3]);
  }
  for (int c = 0; c < n_chunks; ++c) {
    float* keep = reinterpret_cast<float*>(rec + c * step + R_H) + (row0 + rr) * DH + col;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      *reinterpret_cast<float4*>(keep + r * DH) = H[r];
      *reinterpret_cast<float4*>(&Hs[c & 1][rr + r][col]) = H[r];
    }
    cp_wait<1>();
    __syncthreads();  // H is complete, chunk c has landed, and chunk c - 1's buffers are free
    if (c + 2 < n_chunks) load(c + 2);
    cp_commit();
    const uint8_t* st = smem + (c % 3) * CN_STAGE;
    const float* phi = reinterpret_cast<const float*>(st + CN_PHI) + col;
    const float4 g0 = *reinterpret_cast<const float4*>(st + CN_GAM + (rr * DH + col) * 4), g1 = *reinterpret_cast<const float4*>(st + CN_GAM + ((rr + 1) * DH + col) * 4);
    float2 x[2][2] = {{make_float2(g0.x, g0.y), make_float2(g0.z, g0.w)}, {make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)}};
    float2 y[2][2] = {};
#pragma unroll 4
    for (int k = 0; k < DH; k += 4) {
      const float4 h0 = *reinterpret_cast<const float4*>(&Hs[c & 1][rr][k]), h1 = *reinterpret_cast<const float4*>(&Hs[c & 1][rr + 1][k]);
      const float ha[4] = {h0.x, h0.y, h0.z, h0.w}, hb[4] = {h1.x, h1.y, h1.z, h1.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 p = *reinterpret_cast<const float4*>(phi + (k + e) * DH);
        float2 (&d)[2][2] = (e & 1) ? y : x;
        d[0][0] = __ffma2_rn(make_float2(ha[e], ha[e]), make_float2(p.x, p.y), d[0][0]);
        d[0][1] = __ffma2_rn(make_float2(ha[e], ha[e]), make_float2(p.z, p.w), d[0][1]);
        d[1][0] = __ffma2_rn(make_float2(hb[e], hb[e]), make_float2(p.x, p.y), d[1][0]);
        d[1][1] = __ffma2_rn(make_float2(hb[e], hb[e]), make_float2(p.z, p.w), d[1][1]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
      H[r] = make_float4(x[r][0].x + y[r][0].x, x[r][0].y + y[r][0].y, x[r][1].x + y[r][1].x, x[r][1].y + y[r][1].y);
  }
  if (a.final_state != nullptr) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float x[4] = {H[r].x, H[r].y, H[r].z, H[r].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) a.final_state[tile + (int64_t)(col + e) * DH + row0 + rr + r] = x[e];
    }
  }
}

// ---------------------------------------------------------------------------------------------- the outputs of one chunk
constexpr int OT_K = 0, OT_Q = 8192, OT_V = 16384, OT_T = 24576, OT_P = OT_T + 3 * IMG, OT_H = OT_P + 3 * IMG, OT_X = OT_H + 3 * IMG,
              OT_SC = OT_X + 3 * IMG, OT_RED = OT_SC + SC_FLOATS * 4, OT_SMEM = OT_RED + 2 * CH * 4;

__global__ void __launch_bounds__(THREADS) d64_out_kernel(const AveGdnArgs a, const uint8_t* recs) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  pdl_trigger();
  pdl_wait();
  if (!offsets_ok(a, false)) return;
  const SlotChunk c = chunk_of_slot(a, blockIdx.x);
  if (!c.ok) return;
  const int hk = h / (a.Hv / a.Hk);
  const uint8_t* rec = recs + ((int64_t)blockIdx.x * a.Hv + h) * REC_BYTES;
  __nv_bfloat16* og = reinterpret_cast<__nv_bfloat16*>(a.o) + c.b * a.o_stride_b + (int64_t)c.t0 * a.o_stride_t + (int64_t)h * a.o_stride_h;
  if (a.state_indices != nullptr) {
    const int slot = a.state_indices[c.n];
    if (slot < 0 || slot >= a.num_slots) {  // skipped sequence: zero output
      for (int e = tid; e < c.len * DH; e += THREADS) og[(int64_t)(e / DH) * a.o_stride_t + e % DH] = __float2bfloat16(0.f);
      return;
    }
  }
  const uint32_t sb = tc::smem_u32(smem);
  float* bs = reinterpret_cast<float*>(smem + OT_SC);
  float *betas = bs + CH, *qn = bs + 3 * CH, *kn = bs + 4 * CH;
  float* red = reinterpret_cast<float*>(smem + OT_RED);  // [column half][64 tokens]
  load_tile<CH, 8, THREADS>(sb + OT_K, bf(a.k) + c.b * a.k_stride_b + (int64_t)c.t0 * a.k_stride_t + (int64_t)hk * a.k_stride_h, a.k_stride_t, c.len, tid);
  load_tile<CH, 8, THREADS>(sb + OT_Q, bf(a.q) + c.b * a.q_stride_b + (int64_t)c.t0 * a.q_stride_t + (int64_t)hk * a.q_stride_h, a.q_stride_t, c.len, tid);
  load_tile<CH, 8, THREADS>(sb + OT_V, bf(a.v) + c.b * a.v_stride_b + (int64_t)c.t0 * a.v_stride_t + (int64_t)h * a.v_stride_h, a.v_stride_t, c.len, tid);
  load_flat<6 * IMG, THREADS>(sb + OT_T, rec + R_T, tid);
  load_flat<SC_FLOATS * 4, THREADS>(sb + OT_SC, rec + R_SC, tid);
  cp_commit();
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // H -> three tiles, rows d_v
    const int e = tid + i * THREADS, row = e >> 4, q4 = e & 15;
    const float4 x = *reinterpret_cast<const float4*>(rec + R_H + (row * DH + 4 * q4) * 4);
    uint8_t* at = smem + OT_H + piece<128>(row, q4 >> 1) + 8 * (q4 & 1);
    put3(at, x.x, x.y);
    put3(at + 4, x.z, x.w);
  }
  cp_wait<0>();
  __syncthreads();
  const int m = warp & 3, n0 = 32 * (warp >> 2);  // 16 tokens, 32 d_v columns
  float x[4][4], o[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) { zero(x[i]); zero(o[i]); }
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    uint32_t kf[4], qf[4];
    ldsm4(kf, sb + OT_K + at_a<128>(16 * m, 2 * ks, lane));
    ldsm4(qf, sb + OT_Q + at_a<128>(16 * m, 2 * ks, lane));
    step3<false>(x, kf, sb + OT_H, 16 * ks, n0, lane);
    step3<false>(o, qf, sb + OT_H, 16 * ks, n0, lane);
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {  // X = beta (V - e^b K H^T)
    const int i = 16 * m + g + 8 * half;
    const float eb = __expf(bs[i]), fk = eb * kn[i], fq = eb * qn[i], be = betas[i];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const uint32_t at = piece<128>(i, (n0 >> 3) + nt) + 4 * t;
      const float2 v = bf16x2_to_float2(*reinterpret_cast<const uint32_t*>(smem + OT_V + at));
      put3(smem + OT_X + at, be * (v.x - fk * x[nt][2 * half]), be * (v.y - fk * x[nt][2 * half + 1]));
      o[nt][2 * half] *= fq; o[nt][2 * half + 1] *= fq;
    }
  }
  __syncthreads();
  // d += L R over the tokens up to block m, both with three terms (rows of R = contraction index)
  auto lower6 = [&](float (&d)[4][4], uint32_t left, uint32_t right) {
    for (int ks = 0; ks <= m; ++ks) {
      uint32_t ah[4], am[4], al[4];
      const uint32_t la = left + at_a<128>(16 * m, 2 * ks, lane);
      ldsm4(ah, la); ldsm4(am, la + IMG); ldsm4(al, la + 2 * IMG);
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        uint32_t bh[4], bm[4], bl[4];
        const uint32_t ra = right + at_bt<128>(16 * ks, (n0 >> 3) + 2 * np, lane);
        ldsm4t(bh, ra); ldsm4t(bm, ra + IMG); ldsm4t(bl, ra + 2 * IMG);
        mma6(d[2 * np], ah, am, al, bh[0], bh[1], bm[0], bm[1], bl[0], bl[1]);
        mma6(d[2 * np + 1], ah, am, al, bh[2], bh[3], bm[2], bm[3], bl[2], bl[3]);
      }
    }
  };
#pragma unroll
  for (int i = 0; i < 4; ++i) zero(x[i]);
  lower6(x, sb + OT_T, sb + OT_X);  // Vn, over the tiles of H (read by everyone above, before the barrier)
#pragma unroll
  for (int half = 0; half < 2; ++half)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
      put3(smem + OT_H + piece<128>(16 * m + g + 8 * half, (n0 >> 3) + nt) + 4 * t, x[nt][2 * half], x[nt][2 * half + 1]);
  __syncthreads();
  lower6(o, sb + OT_P, sb + OT_H);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] *= a.scale;
  if (a.z != nullptr) {  // gated RMSNorm over the 64 features of a token: two warps hold a row
    const bool gate_first = (a.flags & AVE_GDN_FLAG_GATE_FIRST) != 0;
    float2 gate[2][4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = 16 * m + g + 8 * half;
      float ss = 0.f;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        uint32_t zr = 0u;
        if (i < c.len)
          zr = *reinterpret_cast<const uint32_t*>(bf(a.z) + c.b * a.z_stride_b + (int64_t)(c.t0 + i) * a.z_stride_t + (int64_t)h * a.z_stride_h + n0 + 8 * nt + 2 * t);
        gate[half][nt] = silu2(bf16x2_to_float2(zr));
        if (gate_first) { o[nt][2 * half] *= gate[half][nt].x; o[nt][2 * half + 1] *= gate[half][nt].y; }
        ss += o[nt][2 * half] * o[nt][2 * half] + o[nt][2 * half + 1] * o[nt][2 * half + 1];
      }
      ss += __shfl_xor_sync(0xffffffffu, ss, 1);
      ss += __shfl_xor_sync(0xffffffffu, ss, 2);
      if (t == 0) red[(warp >> 2) * CH + i] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = 16 * m + g + 8 * half;
      const float rinv = rsqrtf((red[i] + red[CH + i]) * (1.0f / DH) + a.norm_eps);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int col = n0 + 8 * nt + 2 * t;
        const float w0 = a.norm_weight ? a.norm_weight[col] : 1.f, w1 = a.norm_weight ? a.norm_weight[col + 1] : 1.f;
        o[nt][2 * half] *= rinv * w0 * (gate_first ? 1.f : gate[half][nt].x);
        o[nt][2 * half + 1] *= rinv * w1 * (gate_first ? 1.f : gate[half][nt].y);
      }
    }
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int i = 16 * m + g + 8 * half;
    if (i < c.len) {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
        *reinterpret_cast<uint32_t*>(og + (int64_t)i * a.o_stride_t + n0 + 8 * nt + 2 * t) = pack_bf16x2(o[nt][2 * half], o[nt][2 * half + 1]);
    }
  }
}

}  // namespace

size_t prefill_d64_workspace_bytes(const AveGdnArgs& a) { return (size_t)record_slots(a) * a.Hv * REC_BYTES; }

int launch_prefill_d64(const AveGdnArgs& a, cudaStream_t stream) {
  if (a.n_seqs == 0) return AVE_GDN_OK;
  static bool attr_set_dev[64] = {};  // the opt-in is per function and per device
  int dev = 0;
  AVE_CUDA_TRY(cudaGetDevice(&dev));
  if (!attr_set_dev[dev & 63]) {
    AVE_CUDA_TRY(cudaFuncSetAttribute(d64_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PQ_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(d64_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CN_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(d64_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OT_SMEM));
    attr_set_dev[dev & 63] = true;  // repeating the calls from another thread is harmless
  }
  uint8_t* recs = reinterpret_cast<uint8_t*>(a.workspace);
  const dim3 chunks((unsigned)record_slots(a), (unsigned)a.Hv);
  AVE_CUDA_TRY(launch_after(d64_prep_kernel, chunks, THREADS, PQ_SMEM, stream, a, recs));
  AVE_CUDA_TRY(launch_after(d64_chain_kernel, dim3((unsigned)a.n_seqs, (unsigned)a.Hv, DH / CN_ROWS), CN_T, CN_SMEM, stream, a, recs));
  AVE_CUDA_TRY(launch_after(d64_out_kernel, chunks, THREADS, OT_SMEM, stream, a, recs));
  return AVE_GDN_OK;
}

}  // namespace ave
