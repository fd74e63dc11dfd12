// Warp-level bf16 MMAs (m16n8k16, fp32 accumulate) with fp32 operands carried as two or three bf16 terms, the shared-memory
// tile layout their operands are read from, and asynchronous copies into such tiles.
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace ave {
namespace {

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void stsm4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void stsm4t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Tiles are stored in rows of ROWB bytes; the 16-byte piece c of row r sits at piece c ^ (r & 7).
template <int ROWB>
__device__ __forceinline__ uint32_t piece(int row, int c) { return (uint32_t)(row * ROWB + ((c ^ (row & 7)) << 4)); }
// Lane addresses of the four ldmatrix patterns (r0, c0: first row and first 16-byte piece of the 16x16 block in the tile)
template <int ROWB>  // left operand, tile rows = its rows
__device__ __forceinline__ uint32_t at_a(int r0, int c0, int lane) { return piece<ROWB>(r0 + (lane & 15), c0 + (lane >> 4)); }
template <int ROWB>  // left operand, tile rows = contraction index (with .trans)
__device__ __forceinline__ uint32_t at_at(int r0, int c0, int lane) { return piece<ROWB>(r0 + (lane & 7) + ((lane >> 4) << 3), c0 + ((lane >> 3) & 1)); }
template <int ROWB>  // right operand of two adjacent column tiles, tile rows = its columns
__device__ __forceinline__ uint32_t at_b(int r0, int c0, int lane) { return piece<ROWB>(r0 + (lane & 7) + ((lane >> 4) << 3), c0 + ((lane >> 3) & 1)); }
template <int ROWB>  // right operand of two adjacent column tiles, tile rows = contraction index (with .trans)
__device__ __forceinline__ uint32_t at_bt(int r0, int c0, int lane) { return piece<ROWB>(r0 + (lane & 15), c0 + (lane >> 4)); }

// x - h for a pair of bf16 values h (exact where h is x rounded): a mixed-precision multiply-add takes the halves of the register as they
// are, where widening them first costs a shift, a mask and a packed multiply-add (a pair split into two terms 8.6 -> 6.8 cycles a warp)
__device__ __forceinline__ float2 residual(float2 x, uint32_t h) {
  float2 r;
  asm("{\n .reg .b16 lo, hi;\n mov.b32 {lo, hi}, %2;\n fma.rn.f32.bf16 %0, lo, %5, %3;\n fma.rn.f32.bf16 %1, hi, %5, %4;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "r"(h), "f"(x.x), "f"(x.y), "h"((unsigned short)0xbf80));  // -1
  return r;
}
// x = h + m + l in bf16, exact to 24 bits
__device__ __forceinline__ void split3(float2 x, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16x2(x.x, x.y);
  const float2 r = residual(x, h);
  m = pack_bf16x2(r.x, r.y);
  const float2 s = residual(r, m);
  l = pack_bf16x2(s.x, s.y);
}
// two adjacent accumulator tiles (columns 0..15) -> left operand of a product over those columns, three terms
__device__ __forceinline__ void split_acc(const float (&c0)[4], const float (&c1)[4], uint32_t (&h)[4], uint32_t (&m)[4], uint32_t (&l)[4]) {
  split3(make_float2(c0[0], c0[1]), h[0], m[0], l[0]);
  split3(make_float2(c0[2], c0[3]), h[1], m[1], l[1]);
  split3(make_float2(c1[0], c1[1]), h[2], m[2], l[2]);
  split3(make_float2(c1[2], c1[3]), h[3], m[3], l[3]);
}
// d += (ah + am + al) (bh + bm + bl), the terms below 2^-24 left out
__device__ __forceinline__ void mma6(float (&d)[4], const uint32_t (&ah)[4], const uint32_t (&am)[4], const uint32_t (&al)[4],
                                     uint32_t bh0, uint32_t bh1, uint32_t bm0, uint32_t bm1, uint32_t bl0, uint32_t bl1) {
  mma_bf16(d, ah, bh0, bh1);
  mma_bf16(d, ah, bm0, bm1);
  mma_bf16(d, am, bh0, bh1);
  mma_bf16(d, ah, bl0, bl1);
  mma_bf16(d, al, bh0, bh1);
  mma_bf16(d, am, bm0, bm1);
}
// x = h + l in bf16, 16 bits
__device__ __forceinline__ void split_pair(float2 x, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16x2(x.x, x.y);
  const float2 l = residual(x, hi);
  lo = pack_bf16x2(l.x, l.y);
}
__device__ __forceinline__ void zero(float (&d)[4]) { d[0] = d[1] = d[2] = d[3] = 0.f; }

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;  // the rest of the 16 bytes is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// `rows` x `PIECES` 16-byte pieces of a strided bf16 matrix into a tile; rows from `len` on are zero
template <int ROWS, int PIECES, int THREADS>
__device__ __forceinline__ void load_tile(uint32_t dst, const __nv_bfloat16* src, int64_t stride, int len, int tid) {
#pragma unroll
  for (int i = 0; i < ROWS * PIECES / THREADS; ++i) {
    const int e = tid + i * THREADS, row = e / PIECES, c = e % PIECES;
    cp16(dst + piece<PIECES * 16>(row, c), src + (int64_t)(row < len ? row : 0) * stride + c * 8, row < len);
  }
}
template <int BYTES, int THREADS>
__device__ __forceinline__ void load_flat(uint32_t dst, const uint8_t* src, int tid) {
#pragma unroll
  for (int i = 0; i < (BYTES / 16 + THREADS - 1) / THREADS; ++i) {
    const int e = tid + i * THREADS;
    if (BYTES / 16 % THREADS == 0 || e < BYTES / 16) cp16(dst + e * 16, src + e * 16, true);
  }
}
__device__ __forceinline__ const __nv_bfloat16* bf(const void* p) { return reinterpret_cast<const __nv_bfloat16*>(p); }

}  // namespace
}  // namespace ave
