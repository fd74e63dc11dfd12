// Chunk records without a table: chunk j of sequence n has record slot floor(first token of n / 64) + n + j.  The slots are unique,
// and the sequence of a slot is found by bisection, because the first slots increase strictly from sequence to sequence.
// Both hold only while the offsets of a packed batch are monotone and stay inside [0, T], so every kernel that reads or
// writes such records asks offsets_ok first.  Shared by the d = 64 prefill and the backward pass (Args: their argument block).
#pragma once
#include "common.cuh"

namespace ave {
namespace {

constexpr int SLOT_CHUNK = 64;

struct SlotChunk { int n, b, t0, len; bool ok; };  // sequence, batch row, first token and length of a chunk
template <class Args>
__device__ __forceinline__ int64_t first_slot(const Args& a, int n) {
  return (a.cu_seqlens ? (int64_t)a.cu_seqlens[n] : (int64_t)n * a.T) / SLOT_CHUNK + n;
}
template <class Args>
__device__ __forceinline__ SlotChunk chunk_of_slot(const Args& a, int64_t slot) {
  int lo = 0, hi = a.n_seqs;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first_slot(a, mid) <= slot) lo = mid; else hi = mid;
  }
  SlotChunk c{lo, 0, 0, 0, false};
  const SeqSpan sp = seq_span(a.cu_seqlens, lo, a.T, nullptr);
  const int64_t j = slot - first_slot(a, lo);
  if (!sp.ok || j < 0 || j * SLOT_CHUNK >= sp.len) return c;
  c.b = sp.b; c.t0 = sp.t0 + (int)j * SLOT_CHUNK; c.len = min(SLOT_CHUNK, sp.len - (int)j * SLOT_CHUNK); c.ok = true;
  return c;
}
// A packed batch whose offsets are not monotone inside [0, T] is skipped as a whole.  Called by the whole CTA.
template <class Args>
__device__ __forceinline__ bool offsets_ok(const Args& a, bool flag) {
  if (a.cu_seqlens == nullptr) return true;
  int bad = 0;
  for (int n = threadIdx.x; n < a.n_seqs; n += blockDim.x) {
    const int x = a.cu_seqlens[n], y = a.cu_seqlens[n + 1];
    bad |= (x < 0 || y < x || y > a.T) ? 1 : 0;
  }
  bad = __syncthreads_or(bad);
  if (bad && flag && threadIdx.x == 0 && a.status != nullptr) atomicOr(a.status, AVE_GDN_DEV_BAD_SEQLEN);
  return bad == 0;
}
template <class Args>
inline int64_t record_slots(const Args& a) { return (int64_t)a.B * a.T / SLOT_CHUNK + a.n_seqs + 1; }

// e^{b_i - b_j} for i >= j (at most 1 elsewhere); sc: b[64] | 64 other floats | low part of b[64] (b as two floats, so that near
// differences are exact)
__device__ __forceinline__ float gate_between(const float* sc, int i, int j) {
  return __expf(fminf((sc[i] - sc[j]) + (sc[2 * SLOT_CHUNK + i] - sc[2 * SLOT_CHUNK + j]), 0.f));
}

}  // namespace
}  // namespace ave
