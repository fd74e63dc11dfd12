#pragma once
#include <stdint.h>

namespace ave {
namespace {

// 16x16 fp32 block algebra on warp MMAs (m16n8k8 tf32), used for the inverse of a unit lower triangular 64x64 matrix.
// Blocks live in shared memory as [16][BLK_LD] fp32.  Each product is issued as three tf32 MMAs per fragment
// (hi*hi + lo*hi + hi*lo) so the result carries fp32-level accuracy.
constexpr int BLK_LD = 20;                 // row stride (floats): conflict-free left-operand fragment loads
constexpr int BLK_FLOATS = 16 * BLK_LD;    // 320
__host__ __device__ constexpr int tri(int r, int c) { return r * (r + 1) / 2 + c; }  // lower-triangular block index

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// acc[nt] (+)= L * R for one 16x16 block pair; `lget(row, col)` returns element (row, col) of the left operand.
template <class LGet>
__device__ __forceinline__ void block_mma(float (&acc)[2][4], LGet lget, const float* __restrict__ R, int lane) {
  const int g = lane >> 2, t = lane & 3;
  float lh[2][4] = {}, hl[2][4] = {};  // separate chains for the lo*hi and hi*lo terms: shorter dependent MMA chains
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    const float af[4] = {lget(g, 8 * ks + t), lget(g + 8, 8 * ks + t), lget(g, 8 * ks + t + 4), lget(g + 8, 8 * ks + t + 4)};
    uint32_t ah[4], al[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) { ah[e] = to_tf32(af[e]); al[e] = to_tf32(af[e] - __uint_as_float(ah[e])); }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const float bf[2] = {R[(8 * ks + t) * BLK_LD + 8 * nt + g], R[(8 * ks + t + 4) * BLK_LD + 8 * nt + g]};
      uint32_t bh[2], bl[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) { bh[e] = to_tf32(bf[e]); bl[e] = to_tf32(bf[e] - __uint_as_float(bh[e])); }
      mma_tf32(acc[nt], ah, bh);
      mma_tf32(lh[nt], al, bh);
      mma_tf32(hl[nt], ah, bl);
    }
  }
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[nt][e] += lh[nt][e] + hl[nt][e];
}
// accumulator fragment -> block in shared memory (optionally negated)
__device__ __forceinline__ void block_store(float* __restrict__ dst, const float (&acc)[2][4], int lane, float sign = 1.f) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    *reinterpret_cast<float2*>(dst + g * BLK_LD + 8 * nt + 2 * t) = make_float2(sign * acc[nt][0], sign * acc[nt][1]);
    *reinterpret_cast<float2*>(dst + (g + 8) * BLK_LD + 8 * nt + 2 * t) = make_float2(sign * acc[nt][2], sign * acc[nt][3]);
  }
}

}  // namespace
}  // namespace ave
