// T = (I + A)^-1 of a 64x64 strictly lower triangular A on warp-level MMAs, by 16x16 blocks, shared by the forward and the backward
// chunk preparations.  The caller leaves, per head, the off-diagonal blocks of A as ready-made right operands (three bf16
// terms; block (s, m) at (s (s - 1) / 2 + m) WY_BLOCK, its fragments in the order of the accumulators of the transposed
// product) and the diagonal blocks as fp32, and gets each row of blocks of T in the accumulators of one warp.
#pragma once
#include "warpmma.cuh"

namespace ave {
namespace {

constexpr int AD_LD = 20;                                     // row pitch (floats) of a 16x16 fp32 block
constexpr int WY_BLOCK = 3 * 512, WY_DIAG = 6 * WY_BLOCK, WY_BYTES = WY_DIAG + 4 * 16 * AD_LD * 4;

// the four warps of one head
__device__ __forceinline__ void head_sync(int hh) {
  __syncwarp();
  asm volatile("bar.sync %0, 128;" ::"r"(1 + hh) : "memory");
}

// A diagonal block in place: (I + A_bb)^-1, transposed.  A lane per column k; lanes that are not `owner` repeat another's work.
__device__ __forceinline__ void wy_invert_block(float* ad, int k, bool owner) {
  float x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float s0 = (i == k) ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
    for (int j4 = 0; j4 < (i + 3) / 4; ++j4) {
      const float4 av = *reinterpret_cast<const float4*>(ad + i * AD_LD + 4 * j4);
      s0 = fmaf(-av.x, x[4 * j4], s0);
      if (4 * j4 + 1 < i) s1 = fmaf(-av.y, x[4 * j4 + 1], s1);
      if (4 * j4 + 2 < i) s0 = fmaf(-av.z, x[4 * j4 + 2], s0);
      if (4 * j4 + 3 < i) s1 = fmaf(-av.w, x[4 * j4 + 3], s1);
    }
    x[i] = s0 + s1;
  }
  __syncwarp();  // every lane has read the block: its inverse, transposed, takes its place
  if (owner)
#pragma unroll
    for (int i4 = 0; i4 < 4; ++i4)
      *reinterpret_cast<float4*>(ad + k * AD_LD + 4 * i4) = make_float4(x[4 * i4], x[4 * i4 + 1], x[4 * i4 + 2], x[4 * i4 + 3]);
}
// The diagonal blocks 2 part and 2 part + 1, by one warp.
__device__ __forceinline__ void wy_invert(uint8_t* frag, int part, int lane) {
  wy_invert_block(reinterpret_cast<float*>(frag + WY_DIAG) + (2 * part + (lane >> 4)) * 16 * AD_LD, lane & 15, true);
}
// Row R of 16x16 blocks of T: T_rc = -(sum_{c < s <= r} T_rs A_sc) D_c, D_c = (I + A_cc)^-1; every block stays in accumulators.
template <int R>
__device__ __forceinline__ void wy_row(float (&T)[R + 1][2][4], const uint8_t* frag, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const float* Dt = reinterpret_cast<const float*>(frag + WY_DIAG);  // D_c transposed: [c][column][row]
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) T[R][nt][e] = Dt[R * 16 * AD_LD + (8 * nt + 2 * t + (e & 1)) * AD_LD + g + 8 * (e >> 1)];
  if constexpr (R > 0) {
    uint32_t th[R][4], tm[R][4], tl[R][4];  // T_rs as left operand, [R - s]
    split_acc(T[R][0], T[R][1], th[0], tm[0], tl[0]);
#pragma unroll
    for (int c = R - 1; c >= 0; --c) {
      float y[2][4];
      zero(y[0]); zero(y[1]);
#pragma unroll
      for (int s = c + 1; s <= R; ++s) {
        const uint4* f = reinterpret_cast<const uint4*>(frag + (s * (s - 1) / 2 + c) * WY_BLOCK) + lane;
        const uint4 ah = f[0], am = f[32], al = f[64];
        mma6(y[0], th[R - s], tm[R - s], tl[R - s], ah.x, ah.y, am.x, am.y, al.x, al.y);
        mma6(y[1], th[R - s], tm[R - s], tl[R - s], ah.z, ah.w, am.z, am.w, al.z, al.w);
      }
      uint32_t yh[4], ym[4], yl[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) { y[0][e] = -y[0][e]; y[1][e] = -y[1][e]; }
      split_acc(y[0], y[1], yh, ym, yl);
      zero(T[c][0]); zero(T[c][1]);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float* d = Dt + c * 16 * AD_LD + (8 * nt + g) * AD_LD + 2 * t;
        uint32_t dh[2], dm[2], dl[2];
        split3(*reinterpret_cast<const float2*>(d), dh[0], dm[0], dl[0]);
        split3(*reinterpret_cast<const float2*>(d + 8), dh[1], dm[1], dl[1]);
        mma6(T[c][nt], yh, ym, yl, dh[0], dh[1], dm[0], dm[1], dl[0], dl[1]);
      }
      if (c > 0) split_acc(T[c][0], T[c][1], th[R - c], tm[R - c], tl[R - c]);
    }
  }
}

}  // namespace
}  // namespace ave
