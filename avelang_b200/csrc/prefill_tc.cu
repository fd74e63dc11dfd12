// Chunked gated-delta-rule prefill on the tensor cores (d_k = d_v = 128, chunk 64).
//
// Pass 1, chunk_tiles (prefill_tiles.cuh; parallel over chunks): in-chunk cumulative gate b, T = (I+A)^-1 with
//   A = strict_lower(beta_i e^{b_i-b_j} k_i.k_j), P = scale * lower_incl(e^{b_i-b_j} q_i.k_j).  P and Tu = T diag(beta) leave as
//   bf16 hi+lo pairs (the tensor cores then see 16 significant bits), lower triangles only, plus per-token scale vectors.
// Pass 2, chunk_scan (prefill_scan.cuh; one CTA per (sequence, value head)): the recurrence over chunks with the state kept on chip.
//   With a gate tensor z the un-normalised output goes to fp32 scratch and a gated-RMSNorm launch finishes it
//   (optionally storing each row into every GPU's buffer: the fused all-gather).
// All waits are bounded; on give-up the CTA drains, frees its tensor memory and sets a status bit.
#include <mutex>

#include "common.cuh"
#include "tc.cuh"

namespace ave {
namespace {

constexpr int C = 64;     // chunk
constexpr int D = 128;    // d_k = d_v
// A record: what pass 1 leaves per (chunk, value head) for the scan.  Tu and P are lower triangles of 16x16 blocks as bf16 hi
// and lo, packed by 16-token steps of the contraction: step c holds rows 16 c .. 63, eight of them after eight, each as two 8x8 core
// matrices of 128 bytes.  qs[64] | ks[64] | kx[64] | decay[64] in fp32 behind them.
constexpr int REC_TRI = 5120, REC_TU = 0, REC_PT = 2 * REC_TRI, REC_SCAL = 4 * REC_TRI, REC_BYTES = REC_SCAL + 4 * C * 4;
__host__ __device__ constexpr int tri_step(int c) { return 2048 * c - 256 * c * (c - 1); }  // byte offset of step c

struct ChunkRef { int n, b, t0, len, cis; bool ok; };  // cis: index of the chunk inside its sequence

// Records are numbered by chunk.  A packed batch comes with chunk tables (see below) or, when all of its chains run at once
// anyway, without (chunk_start == nullptr): then sequence n starts at record floor(first token / 64) + n, which leaves gaps
// but needs no launch in front of pass 1, and the sequence of a record is found by bisection.
__device__ __forceinline__ int first_record(const AveGdnArgs& a, const int32_t* chunk_start, int n) {
  if (a.cu_seqlens == nullptr) return n * ((a.T + C - 1) / C);
  return chunk_start != nullptr ? chunk_start[n] : a.cu_seqlens[n] / C + n;
}
// Whether the offsets of a packed batch are not monotone inside [0, T]: nothing runs then.  Called by whole warps.
__device__ __forceinline__ bool batch_rejected(const AveGdnArgs& a, const int32_t* chunk_start, bool flag = false) {
  if (a.cu_seqlens == nullptr) return false;
  if (chunk_start != nullptr) return chunk_start[a.n_seqs] < 0;
  bool bad = false;
  for (int n = threadIdx.x & 31; n < a.n_seqs; n += 32) {
    const int x = a.cu_seqlens[n], y = a.cu_seqlens[n + 1];
    bad |= x < 0 || y < x || y > a.T;
  }
  bad = __any_sync(0xffffffffu, bad);
  if (bad && flag && threadIdx.x == 0 && a.status != nullptr) atomicOr(a.status, AVE_GDN_DEV_BAD_SEQLEN);
  return bad;
}
__device__ __forceinline__ ChunkRef find_chunk(const AveGdnArgs& a, const int32_t* chunk_start, int c) {
  ChunkRef r; r.ok = false;
  if (a.cu_seqlens == nullptr) {
    const int per = (a.T + C - 1) / C;
    r.n = c / per; r.b = r.n;
    if (r.n >= a.B) return r;
    r.cis = c - r.n * per;
    r.t0 = r.cis * C; r.len = min(C, a.T - r.t0); r.ok = true;
    return r;
  }
  int lo = 0;
  if (chunk_start != nullptr) {
    if (c >= chunk_start[a.n_seqs]) return r;
    lo = chunk_start[a.n_seqs + 1 + c];  // chunk -> sequence map, stored behind the prefix table
  } else {
    int hi = a.n_seqs;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (a.cu_seqlens[mid] / C + mid <= c) lo = mid; else hi = mid;
    }
  }
  const int s0 = a.cu_seqlens[lo], s1 = a.cu_seqlens[lo + 1];
  if (s0 < 0 || s1 < s0 || s1 > a.T) return r;
  r.n = lo; r.b = 0; r.cis = c - first_record(a, chunk_start, lo); r.t0 = s0 + r.cis * C; r.len = min(C, s1 - r.t0); r.ok = r.cis >= 0 && r.len > 0;
  return r;
}

// One CTA builds the chunk tables of a packed batch: chunk_start[n] = chunks of sequences 0..n-1, chunk_start[n_seqs] =
// their total, then the chunk -> sequence map and the scan's launch order.  The scratch behind the tables is sized for
// T/64 + n_seqs chunks, which holds exactly when the offsets are monotone and stay inside [0, T]; a table that breaks this
// would send later sequences' records past their regions, so the whole batch is skipped instead: the total is stored as -1
// (every CTA of the following launches tests it and leaves) and the status word gets AVE_GDN_DEV_BAD_SEQLEN.
// Everything behind this launch waits for it, so it is all latency: a block scan by shuffles and a warp per sequence for
// the map take 3 us where a serial sum and map took 7.5 us (one sequence) to 13 us (64 sequences, 4123 chunks).
__global__ void chunk_table_tc_kernel(const int32_t* cu_seqlens, int n_seqs, int T, int32_t* chunk_start,
                                      int max_chunks, uint32_t* __restrict__ status) {
  __shared__ int part[1024], first[1024], warp_sum_s[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x, warps = threads >> 5;
  pdl_trigger();
  pdl_wait();
  const int per = (n_seqs + threads - 1) / threads;
  const int lo = min(tid * per, n_seqs), hi = min(lo + per, n_seqs);
  int s = 0, bad = 0;
  for (int n = lo; n < hi; ++n) {
    const int a0 = cu_seqlens[n], a1 = cu_seqlens[n + 1];
    bad |= (a0 < 0 || a1 < a0 || a1 > T) ? 1 : 0;
    s += max(0, (a1 - a0 + C - 1) / C);
  }
  int incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) warp_sum_s[warp] = incl;
  bad = __syncthreads_or(bad);
  int before = 0, total = 0;
  for (int w = 0; w < warps; ++w) {
    const int x = warp_sum_s[w];
    before += w < warp ? x : 0;
    total += x;
  }
  bad |= total > max_chunks ? 1 : 0;
  if (tid == 0) {
    chunk_start[n_seqs] = bad ? -1 : total;
    if (bad && status != nullptr) atomicOr(status, AVE_GDN_DEV_BAD_SEQLEN);
  }
  if (bad) return;
  int run = before + incl - s;
  int32_t* chunk_seq = chunk_start + n_seqs + 1;  // chunk_seq[c] = sequence that owns chunk c
  // Launch order of the scan's CTAs: longest sequences first, so that the last CTAs to start are short ones and the
  // SMs finish together (one CTA walks one sequence's chain).  Exact ranking where a thread has one sequence; beyond that
  // the tail is short against the total anyway and the order is the input order.
  int32_t* order = chunk_seq + max_chunks;
  if (per > 1) {
    for (int n = lo; n < hi; ++n) {
      chunk_start[n] = run;
      const int cnt = max(0, (cu_seqlens[n + 1] - cu_seqlens[n] + C - 1) / C);
      for (int i = 0; i < cnt; ++i) chunk_seq[run + i] = n;
      run += cnt;
      order[n] = n;
    }
    return;
  }
  if (tid < n_seqs) { chunk_start[tid] = run; first[tid] = run; part[tid] = s; }
  __syncthreads();
  for (int n = warp; n < n_seqs; n += warps)
    for (int i = lane; i < part[n]; i += 32) chunk_seq[first[n] + i] = n;
  if (tid < n_seqs) {
    int rank = 0;
    for (int m = 0; m < n_seqs; ++m) rank += (part[m] > s || (part[m] == s && m < tid)) ? 1 : 0;
    order[rank] = tid;
  }
}

struct GdnMaps {
  CUtensorMap q, k, v;
  CUtensorMap o, o32;  // 32 features of 64 tokens: the result, and the rows that wait in fp32 scratch
  bool o_ok;           // the result's layout can be described by a map
};

// How one launch cuts the chunks of every sequence.
//   parts : a sequence's chunks are cut into up to `parts` consecutive parts, [part_begin[p], part_begin[p+1]), that are
//           scanned at the same time by different CTAs.  Part 0 starts from the true initial state.  A later part p runs
//           two chains: a local one from a zero state (its outputs miss the contribution of the state M0(p) that enters
//           the part) and a transition chain, the same recurrence with v = 0 started from the identity, whose state is
//           the part's transition matrix F (M_end = F M0 + local end state) and whose "output" is qt_t = scale F_t^T q_t,
//           so that the missing contribution is M0(p)^T qt_t: one GEMM per part once M0(p) is known.
//   ranges: independently, a launch covers only the chunk offsets [r0, r0 + rn) inside every part, so that pass 1 of a
//           later range runs while pass 2 walks an earlier one; a chain's state crosses launches in the carry buffer.
constexpr int MAX_PARTS = 16;
struct ScanPlan {
  int parts;
  int part_begin[MAX_PARTS + 1];  // part_begin[parts] = 1 << 24
  int r0, rn;
};
constexpr int PACK_BYTES = 2 * 128 * 128 * 2;  // bf16 hi image | lo image of one [128][128] operand
constexpr int QT_BYTES = 2 * 128 * 64 * 2;     // bf16 hi image | lo image of one chunk's qt^T [128 d_k][64 tokens]
// byte offset of the 16-byte piece (8 consecutive k) of row `row` in a K-major [128 rows][128 k] bf16 operand stored as
// two 64-wide K halves of 128-byte rows with the 128-byte swizzle (the layout tcgen05.mma reads)
__device__ __forceinline__ uint32_t kmajor_piece_off(int row, int k8) {
  return (uint32_t)((k8 >> 3) * 16384 + row * 128 + (((k8 & 7) ^ (row & 7)) << 4));
}

}  // namespace
}  // namespace ave

#include "prefill_tiles.cuh"  // pass 1
#include "prefill_scan.cuh"   // pass 2

namespace ave {
namespace {

// ------------------------------------------------------------------------------------------------ parts: combine and fix-up
// Once every chain of a multi-part sequence has run, the carry buffer holds, per (sequence, value head): chain 0 = the
// true state after part 0, chain 2p-1 = the end state Psi_p of part p's local chain, chain 2p = part p's transition
// matrix F_p (row-major [k][d]: M_end = F_p M0 + Psi_p).
// Serial combine over the parts of one (sequence, value head, 8-column slice of d_v): M0(1) = state after part 0,
// M0(p+1) = F_p M0(p) + Psi_p in fp32 on the CUDA cores; the last one is the sequence's final state.  M0(p) for p >= 2
// also leaves as the bf16 hi/lo operand image the fix-up kernel's MMAs read (B[d_v][k]); the image of M0(1) was written
// by the scan itself.  The steps are serial and everything behind them waits, so each is kept short: the next F lands in
// shared memory by asynchronous copies while this one is multiplied (row pitch 132: 16-byte reads of eight rows meet eight
// different bank groups), and a thread takes two rows, four columns and half of the contraction, which needs six 16-byte
// reads for 32 multiply-adds.
constexpr int COMBINE_PITCH = 132;
constexpr int COMBINE_F = D * COMBINE_PITCH * 4, COMBINE_CUR = (D + 4) * 8 * 4;  // (a gap of one row between the shares of the contraction)
constexpr size_t combine_smem(int stages) { return stages * (size_t)COMBINE_F + 2 * COMBINE_CUR; }
// COLS columns a CTA: 8, or 4 while that still is one wave (its step is shorter, but F passes through twice as many SMs).
// Bound by shared-memory reads and the issue of the copies, 2 us a step: 15 steps for 4 heads 30 us (42 us when the lanes of a
// quarter warp read one row at four offsets of 128 bytes, 8 wavefronts a load; 55 us with one row a thread, scalar reads and F
// staged through registers).  STAGES of the ring: three, or one where two parts leave a single step, so that three CTAs share an SM
// (32 heads: 24 us with three stages and 3.5 waves).
template <int COLS, int STAGES>
__global__ void __launch_bounds__(256)
part_combine_kernel(const AveGdnArgs a, const int32_t* chunk_start, const float* carry, uint8_t* m0_pack, const __grid_constant__ ScanPlan plan) {
  pdl_wait();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int cb = blockIdx.x, h = blockIdx.y, n = blockIdx.z, tid = threadIdx.x;
  if (batch_rejected(a, chunk_start)) return;
  const SeqSpan sp = seq_span(a.cu_seqlens, n, a.T, nullptr);
  if (!sp.ok || (a.cu_seqlens != nullptr && a.max_seqlen > 0 && sp.len > a.max_seqlen)) return;
  const int seq_chunks = (sp.len + C - 1) / C;
  if (seq_chunks <= plan.part_begin[1]) return;  // a plain chain: the scan wrote the final state itself
  const int slot = a.state_indices ? a.state_indices[n] : n;
  if (slot < 0 || slot >= a.num_slots) return;
  int active = 1;
  for (int p = 1; p < plan.parts; ++p) active += plan.part_begin[p] < seq_chunks ? 1 : 0;
  if (active == 2 && a.final_state == nullptr) return;  // nothing to produce
  const int chains = 2 * plan.parts - 1;
  auto tile_of = [&](int chain) { return carry + (((int64_t)n * chains + chain) * a.Hv + h) * (int64_t)(D * D); };
  constexpr int SPLIT = 16 / COLS, SHARE = D / SPLIT;  // threads that share a contraction, and its length for each
  auto cur_at = [&](int b, int k, int j) -> float& {
    return reinterpret_cast<float*>(smem_raw + STAGES * COMBINE_F + b * COMBINE_CUR)[(k + k / SHARE) * COLS + j];
  };
  const uint32_t sb = tc::smem_u32(smem_raw);
  // this thread: rows k and k + 64, columns j0 .. j0 + 3, contraction indices d0 .. d0 + SHARE - 1
  // (the lanes of a quarter warp, which a 16-byte shared load serves together, read eight rows, so no two meet in a bank)
  const int part = (tid >> 3) & 3, dh = part & 1, j0 = COLS == 8 ? (part >> 1) * 4 : 0, k = (tid >> 5) * 8 + (tid & 7), d0 = (part & (SPLIT - 1)) * SHARE;
  auto fetch = [&](int p) {  // F_p into buffer p % 3
    if (p >= active) { cp_commit(); return; }
    const float* F = tile_of(2 * p);
#pragma unroll
    for (int i = 0; i < D * D / 4 / 256; ++i) {
      const int e = tid + 256 * i, row = e >> 5, c4 = e & 31;
      cp16(sb + (p % STAGES) * COMBINE_F + row * COMBINE_PITCH * 4 + c4 * 16, F + 4 * e, true);
    }
    cp_commit();
  };
  auto psi_of = [&](int p) {
    return p < active ? *reinterpret_cast<const float4*>(tile_of(2 * p - 1) + (int64_t)(k + 64 * dh) * D + cb * COLS + j0) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  fetch(1);
  if (STAGES > 1) fetch(2);
  float4 psi_next = psi_of(1);
  for (int e = tid; e < D * COLS; e += 256) cur_at(0, e / COLS, e % COLS) = tile_of(0)[(e / COLS) * D + cb * COLS + e % COLS];
  int b = 0;
  for (int p = 1; p < active; ++p) {
    cp_wait<(STAGES > 1 ? 1 : 0)>();
    __syncthreads();  // F_p and cur are complete; F_{p-1} has been read
    if (STAGES > 1) fetch(p + 2);
    const float4 psi = psi_next;
    psi_next = psi_of(p + 1);
    const float* F0 = reinterpret_cast<const float*>(smem_raw + (p % STAGES) * COMBINE_F) + k * COMBINE_PITCH + d0;
    float2 x[2][2] = {};
#pragma unroll 4
    for (int d = 0; d < SHARE; d += 4) {
      const float4 f0 = *reinterpret_cast<const float4*>(F0 + d), f1 = *reinterpret_cast<const float4*>(F0 + 64 * COMBINE_PITCH + d);
      const float fa[4] = {f0.x, f0.y, f0.z, f0.w}, fb[4] = {f1.x, f1.y, f1.z, f1.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 c4 = *reinterpret_cast<const float4*>(&cur_at(b, d0 + d + e, j0));
        x[0][0] = __ffma2_rn(make_float2(fa[e], fa[e]), make_float2(c4.x, c4.y), x[0][0]);
        x[0][1] = __ffma2_rn(make_float2(fa[e], fa[e]), make_float2(c4.z, c4.w), x[0][1]);
        x[1][0] = __ffma2_rn(make_float2(fb[e], fb[e]), make_float2(c4.x, c4.y), x[1][0]);
        x[1][1] = __ffma2_rn(make_float2(fb[e], fb[e]), make_float2(c4.z, c4.w), x[1][1]);
      }
    }
    {  // the shares of the contraction meet; two of them finish one of the two rows each
      float v[8] = {x[0][0].x, x[0][0].y, x[0][1].x, x[0][1].y, x[1][0].x, x[1][0].y, x[1][1].x, x[1][1].y};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float mine = dh ? v[4 + i] : v[i], other = dh ? v[i] : v[4 + i];
        v[i] = mine + __shfl_xor_sync(0xffffffffu, other, 8);
        if (SPLIT == 4) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 16);
      }
      if (SPLIT == 2 || part < 2) *reinterpret_cast<float4*>(&cur_at(b ^ 1, k + 64 * dh, j0)) = make_float4(v[0] + psi.x, v[1] + psi.y, v[2] + psi.z, v[3] + psi.w);
    }
    b ^= 1;
    if (p + 1 == active) break;
    __syncthreads();
    if (tid < 16 * COLS) {  // operand image of M0(p+1): B[row = d_v][k] = M0[k][d_v]; a 16-byte piece of hi and of lo
      const int k8 = tid / COLS, v = tid % COLS;
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) split_pair(make_float2(cur_at(b, 8 * k8 + 2 * w, v), cur_at(b, 8 * k8 + 2 * w + 1, v)), hi[w], lo[w]);
      uint8_t* img = m0_pack + (((int64_t)n * (plan.parts - 1) + p) * a.Hv + h) * (int64_t)PACK_BYTES;
      const uint32_t off = kmajor_piece_off(cb * COLS + v, k8);
      *reinterpret_cast<uint4*>(img + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(img + D * D * 2 + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
  __syncthreads();
  if (a.final_state != nullptr) {
    float* dst = a.final_state + ((int64_t)slot * a.Hv + h) * (int64_t)(D * D);
    for (int e = tid; e < D * COLS; e += 256) dst[(e / COLS) * D + cb * COLS + e % COLS] = cur_at(b, e / COLS, e % COLS);
  }
}

// Fix-up of the parts after the first.  For a chunk of 64 tokens of one value head,
//   o = o_local + qt M0(part)        (qt = the transition chain's rows, [64 tokens][128 d_k])
// is one product on tcgen05, transposed like the scan's (128 d_v lanes x 64 tokens), with both operands as bf16 hi+lo pairs (hi hi +
// hi lo + lo hi): A = the image of M0(part), B = the qt^T images the scan wrote (MN-major, brought in by bulk copies).  The
// accumulator is staged in shared memory, so that everything that touches global memory runs in the layout of
// the streaming norm kernel: a half-warp per token row, 8 adjacent features per lane, 16- and 32-byte accesses, the
// RMS over d_v as four shuffles.  (Reading o_local and z straight from the accumulator's layout, a row or a column per
// thread, measured three to four times slower: 2- or 4-byte accesses and tens of instructions per element.)
// A CTA serves one (sequence, part, head) with the M0 image resident.  Its two groups of eight warps walk the chunks independently, the last ones
// first: what the scan wrote last is still in L2.  A group has images, staged rows, accumulator and barriers of its own, and asks for the next chunk's images as
// soon as its product has read these, so that they arrive under the staging and the norm.  Bound by memory traffic (96 KB a chunk with a gate) and
// by the serial steps of a chunk, which the groups overlap.  A whole call, 8192 tokens x 32 heads / 32768 x 4 heads: two CTAs an SM of one group each, whose
// images were in the place of the staged rows, 259.9 / 185.0 us, the last chunks first 258.6 / 183.5, two groups 253.6 / 171.8 (256.8 / 179.0 with
// the next chunk's rows prefetched into L2 as well).
constexpr int FIN_GROUP = 256, FIN_THREADS = 2 * FIN_GROUP;
constexpr int FIN_M0 = 0, FIN_Q = PACK_BYTES, FIN_ST = QT_BYTES, FIN_GROUP_BYTES = QT_BYTES + C * D * 4, FIN_BARS = FIN_Q + 2 * FIN_GROUP_BYTES;
constexpr size_t FIN_SMEM = FIN_BARS + 64 + 1024;
__global__ void __launch_bounds__(FIN_THREADS, 1)
part_finish_kernel(const AveGdnArgs a, const int32_t* chunk_start, const float* o_f32,
                   const uint8_t* qt_img, const uint8_t* m0_pack, const __grid_constant__ ScanPlan plan) {
  extern __shared__ uint8_t smem_raw[];
  pdl_wait();
  uint8_t* smem = tc::align1024(smem_raw);
  const int grp = __shfl_sync(0xffffffffu, (int)(threadIdx.x / FIN_GROUP), 0);
  uint8_t* mine = smem + FIN_Q + grp * FIN_GROUP_BYTES;
  float* stage = reinterpret_cast<float*>(mine + FIN_ST);  // [64 tokens][128] product rows, neighbouring 16-byte pieces swapped by token
  auto piece16 = [&](int t, int p) { return stage + t * D + 4 * (p ^ (((p >> 3) ^ t) & 1)); };
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FIN_BARS);
  uint64_t* m0_full = bars;
  uint64_t* q_full = bars + 1 + grp;
  uint64_t* mma_bar = bars + 3 + grp;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int h = blockIdx.y, tid = threadIdx.x % FIN_GROUP, warp = tid >> 5, lane = tid & 31;  // within the group
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(FIN_GROUP) : "memory"); };
  auto group_all = [&](bool x) {  // the same, with one answer for the whole group
    int all;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.and.pred q, %2, %3, p;\n selp.s32 %0, 1, 0, q;\n}"
                 : "=r"(all) : "r"((int)x), "r"(1 + grp), "n"(FIN_GROUP) : "memory");
    return all != 0;
  };
  const int n = blockIdx.z / (plan.parts - 1), part = 1 + blockIdx.z % (plan.parts - 1);
  if (batch_rejected(a, chunk_start)) return;
  const SeqSpan sp = seq_span(a.cu_seqlens, n, a.T, nullptr);
  if (!sp.ok || (a.cu_seqlens != nullptr && a.max_seqlen > 0 && sp.len > a.max_seqlen)) return;
  const int seq_chunks = (sp.len + C - 1) / C;
  const int c_end = min(plan.part_begin[part + 1], seq_chunks), c_begin = plan.part_begin[part] + 2 * (int)blockIdx.x + grp, stride = 2 * gridDim.x;
  if (c_begin - grp >= c_end) return;
  auto from_end = [&](int i) { return plan.part_begin[part] + c_end - 1 - i; };
  const int slot = a.state_indices ? a.state_indices[n] : n;
  const bool skipped = slot < 0 || slot >= a.num_slots;  // the scan skipped the sequence: its rows are zero
  const int64_t rec0 = first_record(a, chunk_start, n);  // record of the sequence's chunk 0

  auto load_qt = [&](int c) {  // called by one thread
    tc::mbar_expect_tx(q_full, QT_BYTES);
    tc::bulk_load(mine, qt_img + ((rec0 + c) * a.Hv + h) * (int64_t)QT_BYTES, QT_BYTES, q_full);
  };
  if (threadIdx.x == 0) {
    for (int i = 0; i < 5; ++i) tc::mbar_init(bars + i, 1);
    *abort_flag = 0;
    tc::fence_barrier_init();
    if (!skipped) {
      const uint8_t* img = m0_pack + (((int64_t)n * (plan.parts - 1) + (part - 1)) * a.Hv + h) * (int64_t)PACK_BYTES;
      tc::mbar_expect_tx(m0_full, PACK_BYTES);
      tc::bulk_load(smem + FIN_M0, img, PACK_BYTES, m0_full);
    }
  }
  if (grp == 0 && warp == 1) tc::tmem_alloc(tmem_slot, 128);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  int asked = 0;  // images that this group's first thread has asked for
  if (tid == 0 && !skipped && c_begin < c_end) { load_qt(from_end(c_begin)); ++asked; }
  const uint32_t tm = *tmem_slot + 64 * grp;
  const int hw = tid >> 4, sub = tid & 15;  // streaming pass: half-warp index (16 of them) and lane inside it
  const bool gate_first = (a.flags & AVE_GDN_FLAG_GATE_FIRST) != 0;
  float2 wv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    wv[i] = a.norm_weight ? make_float2(a.norm_weight[8 * sub + 2 * i], a.norm_weight[8 * sub + 2 * i + 1]) : make_float2(1.f, 1.f);
  // A wait that has expired ends the group's walk: no rows from a product that is not there, no further images.
  bool ok = true, landed = true;  // ok: the same for the whole group between its meetings

  int it = 0;
  for (int i = c_begin; i < c_end && ok; i += stride, ++it) {
    const int c = from_end(i);
    const int64_t tok0 = sp.t0 + (int64_t)c * C;
    const int rows = min(C, sp.len - c * C);
    // the rows this half-warp will stream (hw, hw + 16, hw + 32, hw + 48) are fetched before the product is waited for
    float4 ol[4][2];
    uint4 zraw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = hw + 16 * u;
      ol[u][0] = ol[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      zraw[u] = make_uint4(0u, 0u, 0u, 0u);
      if (!skipped && r < rows) {
        const float* src = o_f32 + (((int64_t)sp.b * a.T + tok0 + r) * a.Hv + h) * D + 8 * sub;
        ol[u][0] = *reinterpret_cast<const float4*>(src);
        ol[u][1] = *reinterpret_cast<const float4*>(src + 4);
      }
      if (a.z != nullptr && r < rows)
        zraw[u] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(a.z) + sp.b * a.z_stride_b +
                                                  (tok0 + r) * a.z_stride_t + (int64_t)h * a.z_stride_h + 8 * sub);
    }
    if (!skipped) {
      if (warp == 0) {
        landed = __all_sync(0xffffffffu, (it > 0 || tc::mbar_wait_warp(m0_full, 0, abort_flag)) && tc::mbar_wait_warp(q_full, (uint32_t)it & 1u, abort_flag)) != 0;
        tc::tc_fence_after_sync();
        if (landed && tc::elect_one()) {
          constexpr uint32_t idesc = tc::idesc_f16(128, 64, 1, 1, false, true);  // A K-major, B MN-major (token rows)
          const uint32_t sq = tc::smem_u32(mine), sm = tc::smem_u32(smem + FIN_M0);
#pragma unroll 1
          for (int t = 0; t < 3; ++t) {  // hi hi, hi lo, lo hi
            const uint32_t qb = sq + (t == 1 ? QT_BYTES / 2 : 0), mb = sm + (t == 2 ? PACK_BYTES / 2 : 0);
#pragma unroll
            for (int k = 0; k < 8; ++k)  // 16 d_k rows of qt^T per step: 2048 bytes
              tc::mma_ss(tm, tc::smem_desc_sw128(mb + (uint32_t)((k >> 2) * 16384 + (k & 3) * 32), 16, 1024),
                         tc::smem_desc_sw128(qb + k * 2048, 16, 1024), idesc, (t | k) != 0 ? 1u : 0u);
          }
          tc::mma_commit(mma_bar);
        }
        __syncwarp();
      }
      ok = __all_sync(0xffffffffu, tc::mbar_wait(mma_bar, (uint32_t)it & 1u, abort_flag)) != 0;
      tc::tc_fence_after_sync();
      if (ok && tid == 0 && i + stride < c_end) { load_qt(c - stride); ++asked; }  // the product has read the images
      if (ok) {  // accumulator (a d_v row per thread, 32 tokens) -> staged token rows
        const int d = (warp & 3) * 32 + lane, first = 32 * (warp >> 2);
        uint32_t acc[32];
        tc::tmem_ld32(tm + ((uint32_t)((warp & 3) * 32) << 16) + first, acc);
        tc::tmem_ld_wait();
#pragma unroll
        for (int t = 0; t < 32; ++t) piece16(first + t, d >> 2)[d & 3] = __uint_as_float(acc[t]);
      }
    }
    tc::tc_fence_before_sync();
    ok = group_all(ok);  // staged rows complete; the accumulator is free for the next product
    tc::tc_fence_after_sync();
    if (ok) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = hw + 16 * u;
        float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0;
        if (!skipped && r < rows) {
          p0 = *reinterpret_cast<const float4*>(piece16(r, 2 * sub));
          p1 = *reinterpret_cast<const float4*>(piece16(r, 2 * sub + 1));
        }
        float2 x[4] = {make_float2(ol[u][0].x + p0.x, ol[u][0].y + p0.y), make_float2(ol[u][0].z + p0.z, ol[u][0].w + p0.w),
                       make_float2(ol[u][1].x + p1.x, ol[u][1].y + p1.y), make_float2(ol[u][1].z + p1.z, ol[u][1].w + p1.w)};
        uint32_t packed[4];
        if (a.z != nullptr) {
          const float2 gate[4] = {silu2(bf16x2_to_float2(zraw[u].x)), silu2(bf16x2_to_float2(zraw[u].y)),
                                  silu2(bf16x2_to_float2(zraw[u].z)), silu2(bf16x2_to_float2(zraw[u].w))};
          float2 ss2 = make_float2(0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (gate_first) x[i] = __fmul2_rn(x[i], gate[i]);
            ss2 = __ffma2_rn(x[i], x[i], ss2);
          }
          float ss = ss2.x + ss2.y;
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);  // stays inside the half-warp
          const float rinv = rsqrtf(ss * (1.0f / D) + a.norm_eps);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float2 y2 = __fmul2_rn(__fmul2_rn(x[i], make_float2(rinv, rinv)), wv[i]);
            if (!gate_first) y2 = __fmul2_rn(y2, gate[i]);
            packed[i] = pack_bf16x2(y2.x, y2.y);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) packed[i] = pack_bf16x2(x[i].x, x[i].y);
        }
        if (r < rows)
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.o) + sp.b * a.o_stride_b + (tok0 + r) * a.o_stride_t +
                                    (int64_t)h * a.o_stride_h + 8 * sub) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      }
    }
    group_sync();  // the staged rows have been read
  }
  if (!ok) {  // nothing of this group is on its way when the CTA ends
    if (warp == 0 && landed) tc::drain(mma_bar, (uint32_t)(it - 1) & 1u);
    if (tid == 0) tc::drain(q_full, (uint32_t)(asked - 1) & 1u);
    if (threadIdx.x == 0) tc::drain(m0_full, 0u);
  }
  tc::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u && threadIdx.x == 0 && a.status != nullptr) atomicOr(a.status, AVE_GDN_DEV_WAIT_EXPIRED);
  if (grp == 0 && warp == 1) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tm, 128);
  }
}

// ------------------------------------------------------------------------------------------------ schedule and scratch
constexpr int SEG_MAX = 8;
constexpr int PART0_X4 = 4;         // length of part 0 in quarters of a later part's length
constexpr int NUM_SMS = 148;        // B200; the schedule is a pure function of the arguments, so that the workspace
                                    // query and the launch agree without a device being current
struct WsLayout {
  size_t chunk_start, recs, o_f32, qt_img, carry, m0_pack, total;
  int64_t chunks;
  int max_chunks;      // bound of the longest sequence, in chunks
  int parts;           // see ScanPlan
  int part_begin[MAX_PARTS + 1];
  int segments;        // chunk ranges handled by separate launches
  int seg_begin[9];    // range i covers chunk offsets [seg_begin[i], seg_begin[i+1])
};

// The longest chain, in chunks, is known for dense batches and for packed ones that come with the max_seqlen bound; otherwise only its bound T is.
int longest_chunks(const AveGdnArgs& a) { return ((a.cu_seqlens != nullptr && a.max_seqlen > 0 ? min(a.max_seqlen, a.T) : a.T) + C - 1) / C; }

// Length of the parts after the first and of the first, in chunks.  Part 0 runs one chain and needs no fix-up, a later part runs two chains and its rows wait for
// the fix-up, so part 0 is made PART0_X4 / 4 times as long as the others; lengths are even.
int part_length(int chunks, int S) { return max(2, (4 * chunks / (4 * (S - 1) + PART0_X4) + 1) & ~1); }
int first_part_length(int chunks, int S) { return S > 1 ? max(2, (chunks - (S - 1) * part_length(chunks, S) + 1) & ~1) : 0; }

// Most parts whose 2S - 1 chains per head still get an SM each
int most_parts(int64_t heads_total) {
  const int64_t per_head = (NUM_SMS / heads_total + 1) / 2;
  return per_head < MAX_PARTS ? (int)per_head : MAX_PARTS;
}
// Two parts take three chains a head.  They are taken while these leave a third of the SMs and the chains are long enough for the
// fix-up, which with a gate also holds the later part's norms back.
bool two_parts(int64_t heads_total, int chunks, bool gated) { return 3 * heads_total <= 2 * NUM_SMS / 3 && chunks >= (gated ? 112 : 64); }

// The parts that a call may bring the scratch for instead, with which it then runs: the largest count with eight chunks a part or more.  Its scratch grows
// with the length, so that a buffer for the longest of a caller's prompts serves the shorter ones; with the wanted parts four heads need 24.0 MB
// at 20 chunks and 5.4 MB at 21.
int parts_least(const AveGdnArgs& a, bool plain) {
  const int64_t heads_total = (int64_t)a.n_seqs * a.Hv;
  const int max_chunks = longest_chunks(a);
  if (plain || (a.o_peers != nullptr && a.n_peers > 1) || heads_total <= 0 || max_chunks < 32) return 1;
  int S = most_parts(heads_total);
  while (S > 1 && max_chunks / S < 8) --S;
  return S >= 3 || (S == 2 && two_parts(heads_total, max_chunks, a.z != nullptr)) ? S : 1;
}

// Parts: with few chains most SMs idle while every chain walks its chunks one after the other.  Cutting the sequences into S parts that run at
// the same time shortens the walk S-fold at the price of a second (transition) chain per later part, a combine and one GEMM-shaped fix-up.  Not
// with the fused all-gather: there the fix-up would push most rows to the peers after the scan instead of beside it.
int parts_wanted(const AveGdnArgs& a, bool plain) {
  const int64_t heads_total = (int64_t)a.n_seqs * a.Hv;
  const int max_chunks = longest_chunks(a);
  if (plain || (a.o_peers != nullptr && a.n_peers > 1) || heads_total <= 0 || max_chunks < 12) return 1;
  // What a call with S parts takes beside what it takes anyway, in ns: its longest chain's steps, which get longer with the SMs that hold chains, their
  // start, the fix-up, and what goes with any.  Fitted to 1156 measurements (4 to 96 chains of 8 to 256 chunks, whole and in 2 to 16 parts, with a gate and
  // without; 3.4 % off on the mean, as good with either).
  auto scan = [&](int S) {
    const int64_t chains = heads_total * (2 * S - 1), steps = S > 1 ? max(part_length(max_chunks, S), first_part_length(max_chunks, S)) : max_chunks;
    return steps * (1870 + 34 * chains / 10) + 122 * chains;
  };
  auto cost = [&](int S) {
    return scan(S) + (S == 1 ? 0 : S == 2 ? 10500 : 13000 + 460 * (S - 1)) +
           (S > 1 ? 147 * heads_total * max(0, max_chunks - first_part_length(max_chunks, S)) / 10 : 0) + 10100 + 3 * heads_total * max_chunks;
  };
  int most = most_parts(heads_total);
  while (most > 1 && max_chunks / most < 2) --most;
  int S = most;
  for (int i = most - 1; i >= 3; --i) if (cost(i) < cost(S)) S = i;
  if (max_chunks < 32) {
    // Of several packed sequences without a bound only the sum is known.  Each may end inside the first part or soon behind it, and what parts take beside
    // the scan is paid for nothing (whole / parts: 3 x 650 tokens x 4 heads gated 37.8 / 52.6 us, 2 x 975 x 8 51.7 / 59.8; 1853 and 97 x 4 69.8 / 53.7, with its bound 56).
    if (a.cu_seqlens != nullptr && a.n_seqs > 1 && a.max_seqlen <= 0) return 1;
    // Short chains: two parts as well, and whole unless parts are clearly ahead (4 heads x 1024 tokens 45.8 -> 40.0 us, 16 x 1536 65.7 -> 58.0).  Not beyond 16 chains: at
    // 24 two parts win only with a gate, and not always (whole / two, 1536 tokens 74 / 67 us, without a gate 58 / 57; 1024 55 / 56 and 43 / 48).
    if (most >= 2 && cost(2) < cost(S)) S = 2;
    if (S < 2 || heads_total > 16 || 20 * cost(S) >= 19 * cost(1)) S = 1;
  } else if (S >= 3) {  // two only where clearly ahead (24 heads x 2048 tokens 88.6 -> 82.4; 8 heads x 6144 tokens 103 with nine parts, 92.9 with eight)
    if (20 * cost(2) < 19 * cost(S)) S = 2;
  } else if (S == 2 && !two_parts(heads_total, max_chunks, a.z != nullptr)) {
    // Both lines of two parts are those of slower forms of pass 1, the combine and the fix-up: two parts win at them and would win beyond (32 heads gated, whole / two:
    // 2048 tokens 96.1 / 86.5 us, 4096 176 / 141, 6144 258 / 199; without a gate 2048 79.7 / 77.0; 48 heads x 8192 gated 382 / 318).
    S = 1;
  }
  // The single tokens of a mixed step stream their states, 64 KB in and out in about 1.75 us an SM, through the SMs that the chains leave, and the fix-up finds no
  // room before they are through.  Where they take longer than the scan, not more parts than by the rule above (without the gate, parts / not: 16
  // heads, 200 single tokens and a prompt of 1700 123 / 99 us, 8 heads, 200 and 1200 74 / 57; 8 heads, 200 and 2500, six parts / five 88 / 81).
  const int least = parts_least(a, plain);
  if (least < S && (int64_t)a.token_begin * a.Hv * 1750 > scan(S) * (NUM_SMS - heads_total * (2 * S - 1))) S = least;
  return max(S, 1);
}

WsLayout ws_layout_of(const AveGdnArgs& a, bool plain, int parts) {
  WsLayout L;
  L.chunks = a.cu_seqlens ? (int64_t)a.T / C + a.n_seqs : (int64_t)a.B * ((a.T + C - 1) / C);
  const size_t recs = (size_t)L.chunks * a.Hv;
  auto up = [](size_t x) { return (x + 1023) & ~(size_t)1023; };
  const int max_chunks = longest_chunks(a);
  L.max_chunks = max_chunks;
  const int64_t heads_total = (int64_t)a.n_seqs * a.Hv;
  const bool push = a.o_peers != nullptr && a.n_peers > 1;
  L.parts = parts;
  L.part_begin[0] = 0;
  for (int p = 1; p <= MAX_PARTS; ++p) L.part_begin[p] = p < parts ? first_part_length(max_chunks, parts) + (p - 1) * part_length(max_chunks, parts) : (1 << 24);
  // Ranges: with the fused all-gather a launch of its own norms the rows and pushes them to every peer over NVLink, which takes about
  // as long as a chain itself; with few long chains that runs beside the chains of the next range, and only the last range's push is
  // exposed, so the ranges are equal and as many as the event pool allows.  (Without peers ranges do not pay any more: pass 1 of
  // the whole batch takes less than the two launches and the state's way through the carry buffer, about 10 us a range.  One
  // launch against two ranges or more: 2 x 4096 tokens x 32 heads 228 us / 244, 32768 x 4 218 / 239, 8192 x 16 196 / 217.)
  L.seg_begin[0] = 0;
  L.segments = 1;
  L.seg_begin[1] = 1 << 24;  // every chunk (times 64 still fits an int)
  if (!plain && push && heads_total <= 74 && max_chunks >= 32) {
    const int len = (max_chunks + SEG_MAX - 1) / SEG_MAX;
    L.segments = 0;
    while (L.seg_begin[L.segments] < max_chunks) {
      L.seg_begin[L.segments + 1] = L.segments == SEG_MAX - 1 ? max_chunks : min(max_chunks, L.seg_begin[L.segments] + len);
      ++L.segments;
    }
  }
  size_t off = 0;
  L.chunk_start = off; off = up(off + (2 * (size_t)a.n_seqs + 1 + (size_t)L.chunks) * 4);  // prefix table, chunk -> sequence map, scan order
  L.recs = off; off = up(off + recs * (size_t)REC_BYTES);
  L.o_f32 = off;
  if (L.parts > 1 || a.z != nullptr) off = up(off + (size_t)a.B * a.T * a.Hv * D * 4);  // rows waiting for the fix-up / the norm
  L.qt_img = off;
  if (L.parts > 1) off = up(off + recs * (size_t)QT_BYTES);                             // the transition chains' rows (operand images)
  L.carry = off;
  if (L.segments > 1 || L.parts > 1) off = up(off + (size_t)a.n_seqs * (2 * L.parts - 1) * a.Hv * D * D * 4);
  L.m0_pack = off;
  if (L.parts > 1) off = up(off + (size_t)a.n_seqs * (L.parts - 1) * a.Hv * PACK_BYTES);
  L.total = off;
  return L;
}

// `plain`: one part, one range, everything on the caller's stream (the schedule of the fixed-scratch entry point).
WsLayout ws_layout(const AveGdnArgs& a, bool plain) {
  const WsLayout L = ws_layout_of(a, plain, parts_wanted(a, plain));
  return plain || a.workspace == nullptr || a.workspace_bytes >= L.total ? L : ws_layout_of(a, plain, parts_least(a, plain));
}

}  // namespace

int launch_decode(const AveGdnArgs& a, cudaStream_t stream);
int launch_decode_beside(const AveGdnArgs& a, const AveGdnArgs& prefill, cudaStream_t stream);
int launch_shared_slots(const AveGdnArgs& a, const AveGdnArgs& prefill, cudaStream_t stream);
int launch_gated_rmsnorm_f32in_batched(const AveGdnNormArgs& a, cudaStream_t stream, const void* const* peers, int n_peers,
                                       int64_t peer_off, int batches, int64_t xs_b, int64_t zs_b, int64_t ys_b);

// More chains than SMs: the walk of the longest chains decides, so the tables are built, which sort the sequences for the scan.
// 32 heads, one sequence of 203 tokens: 33.9 us with the tables, 31.3 without.
static bool needs_tables(const AveGdnArgs& a) { return a.cu_seqlens != nullptr && (int64_t)a.n_seqs * a.Hv > NUM_SMS; }

// What a caller is told to bring, and what a call is refused below
size_t prefill_tc_workspace_bytes(const AveGdnArgs& a, bool plain) {
  return max(ws_layout_of(a, plain, parts_wanted(a, plain)).total, ws_layout_of(a, plain, parts_least(a, plain)).total);
}
size_t prefill_tc_workspace_least(const AveGdnArgs& a) {
  return min(ws_layout_of(a, false, parts_wanted(a, false)).total, ws_layout_of(a, false, parts_least(a, false)).total);
}

int prefill_tc_parts(const AveGdnArgs& a) { return ws_layout(a, false).parts; }

// Kernels one call enqueues, mirroring launch_prefill_tc below.
int prefill_tc_launch_count(const AveGdnArgs& a, bool plain) {
  const WsLayout L = ws_layout(a, plain);
  if (L.chunks == 0 || a.n_seqs == 0) return 0;
  const bool tables = needs_tables(a);
  const bool push = a.o_peers != nullptr && a.n_peers > 1;
  int n = tables ? 1 : 0;                                  // chunk tables
  n += 2 * L.segments;                                     // pass 1 and pass 2 of every range
  if (a.z != nullptr) n += (a.cu_seqlens == nullptr ? L.segments : 1) * (push || a.B == 1 ? 1 : a.B);  // norm_rows: one launch, or one per batch row
  if (L.parts > 1) n += 2;                                 // combine and fix-up
  return n;
}

// Helper streams and events for the ranges.  Pass 2 runs on a high-priority stream so that, when a
// range's pass 1 completes and both its pass 2 and the next range's pass 1 become runnable, the few whole-SM pass-2
// CTAs are placed first.  Each device owns a small pool of such sets; a call takes the set its stream hashes to, so
// calls on different streams usually overlap instead of queueing behind one another's helper streams.  A device's sets
// and the whole enqueue sequence of a call are guarded by that device's mutex: the record/wait pairs of two host
// threads never interleave, which is what makes a set shareable at all (a wait binds to the event's latest record at
// the time of the call).
struct SideSet {
  cudaStream_t prep = nullptr, scan = nullptr, norm = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr, join_norm = nullptr;
  cudaEvent_t done[SEG_MAX] = {}, scanned[SEG_MAX] = {};
  bool ready = false;
};
constexpr int SIDE_SETS = 4, MAX_DEVICES = 64;
struct DeviceSide {
  std::mutex mu;
  SideSet sets[SIDE_SETS];
  bool attr_set = false;
};
static DeviceSide g_side[MAX_DEVICES];

static void destroy_side_set(SideSet& s) {
  if (s.prep) cudaStreamDestroy(s.prep);
  if (s.scan) cudaStreamDestroy(s.scan);
  if (s.norm) cudaStreamDestroy(s.norm);
  for (cudaEvent_t e : {s.fork, s.join, s.join_norm}) if (e) cudaEventDestroy(e);
  for (int i = 0; i < SEG_MAX; ++i) { if (s.done[i]) cudaEventDestroy(s.done[i]); if (s.scanned[i]) cudaEventDestroy(s.scanned[i]); }
  s = SideSet{};
}
// Called with the device's mutex held.  A set is built in a local and published only when every piece exists.
static SideSet* side_set(DeviceSide& dev, cudaStream_t stream) {
  SideSet& slot = dev.sets[(reinterpret_cast<uintptr_t>(stream) >> 4) % SIDE_SETS];
  if (slot.ready) return &slot;
  SideSet s;
  int lo = 0, hi = 0;
  bool ok = cudaDeviceGetStreamPriorityRange(&lo, &hi) == cudaSuccess;
  ok = ok && cudaStreamCreateWithPriority(&s.prep, cudaStreamNonBlocking, lo) == cudaSuccess;
  ok = ok && cudaStreamCreateWithPriority(&s.scan, cudaStreamNonBlocking, hi) == cudaSuccess;
  ok = ok && cudaStreamCreateWithPriority(&s.norm, cudaStreamNonBlocking, lo) == cudaSuccess;
  ok = ok && cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming) == cudaSuccess;
  ok = ok && cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming) == cudaSuccess;
  ok = ok && cudaEventCreateWithFlags(&s.join_norm, cudaEventDisableTiming) == cudaSuccess;
  for (int i = 0; i < SEG_MAX; ++i) {
    ok = ok && cudaEventCreateWithFlags(&s.done[i], cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaEventCreateWithFlags(&s.scanned[i], cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) { destroy_side_set(s); return nullptr; }
  s.ready = true;
  slot = s;
  return &slot;
}

// Gated RMSNorm over the fp32 output for tokens [t_begin, t_end) of every batch row.
static int norm_rows(const AveGdnArgs& a, float* o_f32, int t_begin, int t_end, cudaStream_t stream) {
  if (t_end <= t_begin) return AVE_GDN_OK;
  AveGdnNormArgs nb{};
  nb.struct_size = sizeof(nb);
  nb.flags = a.flags & AVE_GDN_FLAG_GATE_FIRST;
  nb.rows = (int64_t)(t_end - t_begin) * a.Hv;
  nb.d = D; nb.heads = a.Hv; nb.eps = a.norm_eps; nb.weight = a.norm_weight;
  nb.x = o_f32 + (int64_t)t_begin * a.Hv * D;
  nb.x_stride_t = (int64_t)a.Hv * D; nb.x_stride_h = D;
  nb.z = reinterpret_cast<const __nv_bfloat16*>(a.z) + (int64_t)t_begin * a.z_stride_t;
  nb.z_stride_t = a.z_stride_t; nb.z_stride_h = a.z_stride_h;
  nb.y = reinterpret_cast<__nv_bfloat16*>(a.o) + (int64_t)t_begin * a.o_stride_t;
  nb.y_stride_t = a.o_stride_t; nb.y_stride_h = a.o_stride_h;
  // With peers the launch covers every batch row at once (many short launches keep too few peer stores in flight);
  // without, one launch per batch row measured 1-2 % faster on four rows of a million norm rows each.
  const bool push = a.o_peers != nullptr && a.n_peers > 1;
  const int64_t xs_b = (int64_t)a.T * a.Hv * D;
  if (push || a.B == 1)
    return launch_gated_rmsnorm_f32in_batched(nb, stream, a.o_peers, a.n_peers, (int64_t)t_begin * a.o_stride_t, a.B, xs_b,
                                              a.z_stride_b, a.o_stride_b);
  for (int b = 0; b < a.B; ++b) {
    AveGdnNormArgs one = nb;
    one.x = reinterpret_cast<const float*>(nb.x) + b * xs_b;
    one.z = reinterpret_cast<const __nv_bfloat16*>(nb.z) + b * a.z_stride_b;
    one.y = reinterpret_cast<__nv_bfloat16*>(nb.y) + b * a.o_stride_b;
    const int rc = launch_gated_rmsnorm_f32in_batched(one, stream, a.o_peers, a.n_peers,
                                                      (int64_t)b * a.o_stride_b + (int64_t)t_begin * a.o_stride_t, 1, 0, 0, 0);
    if (rc != AVE_GDN_OK) return rc;
  }
  return AVE_GDN_OK;
}

// Enqueues one prefill, and the single-token part of a mixed step with it (`decode`).  Thread-safe: the enqueue sequence of a call runs under the device's mutex (see SideSet).
int launch_prefill_tc(const AveGdnArgs& a, cudaStream_t stream, bool plain, const AveGdnArgs* decode) {
  const WsLayout L = ws_layout(a, plain);
  if (L.chunks == 0 || a.n_seqs == 0) return decode != nullptr ? launch_decode(*decode, stream) : AVE_GDN_OK;
  char* ws = reinterpret_cast<char*>(a.workspace);
  int32_t* chunk_start = needs_tables(a) ? reinterpret_cast<int32_t*>(ws + L.chunk_start) : nullptr;
  uint8_t* recs = reinterpret_cast<uint8_t*>(ws + L.recs);

  GdnMaps maps;
  {
    int rc;
    const uint32_t box4[4] = {64, 1, 64, 1};
    const uint64_t dq[4] = {D, (uint64_t)a.Hk, (uint64_t)a.T, (uint64_t)a.B};
    const uint64_t sq[4] = {2, (uint64_t)a.q_stride_h * 2, (uint64_t)a.q_stride_t * 2, (uint64_t)(a.B > 1 ? a.q_stride_b : a.q_stride_t * a.T) * 2};
    const uint64_t sk[4] = {2, (uint64_t)a.k_stride_h * 2, (uint64_t)a.k_stride_t * 2, (uint64_t)(a.B > 1 ? a.k_stride_b : a.k_stride_t * a.T) * 2};
    if ((rc = make_tmap(&maps.q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.q), 4, dq, sq, box4, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
    if ((rc = make_tmap(&maps.k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.k), 4, dq, sk, box4, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
    const uint32_t boxv[4] = {64, 1, 64, 1};
    const uint64_t dv4[4] = {D, (uint64_t)a.Hv, (uint64_t)a.T, (uint64_t)a.B};
    const uint64_t sv[4] = {2, (uint64_t)a.v_stride_h * 2, (uint64_t)a.v_stride_t * 2, (uint64_t)(a.B > 1 ? a.v_stride_b : a.v_stride_t * a.T) * 2};
    if ((rc = make_tmap(&maps.v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.v), 4, dv4, sv, boxv, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  }

  int dev_id = 0;
  AVE_CUDA_TRY(cudaGetDevice(&dev_id));
  if (dev_id < 0 || dev_id >= MAX_DEVICES) return AVE_GDN_UNSUPPORTED;
  DeviceSide& dev = g_side[dev_id];
  std::lock_guard<std::mutex> guard(dev.mu);
  if (!dev.attr_set) {
    AVE_CUDA_TRY(cudaFuncSetAttribute(chunk_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILES_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(chunk_scan_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCAN_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(chunk_scan_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCAN_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(part_finish_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FIN_SMEM));
    AVE_CUDA_TRY(cudaFuncSetAttribute(part_combine_kernel<4, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)combine_smem(3)));
    AVE_CUDA_TRY(cudaFuncSetAttribute(part_combine_kernel<8, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)combine_smem(3)));
    AVE_CUDA_TRY(cudaFuncSetAttribute(part_combine_kernel<8, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)combine_smem(1)));
    dev.attr_set = true;
  }
  if (chunk_start != nullptr) {
    AVE_CUDA_TRY(launch_after(chunk_table_tc_kernel, 1, a.n_seqs <= 256 ? 256 : 1024, 0, stream, a.cu_seqlens, a.n_seqs, a.T, chunk_start, (int)L.chunks, a.status));
  }
  float* o_f32 = L.parts > 1 || a.z != nullptr ? reinterpret_cast<float*>(ws + L.o_f32) : nullptr;
  {
    const uint32_t box[4] = {32, 1, 64, 1};
    const uint64_t dims[4] = {D, (uint64_t)a.Hv, (uint64_t)a.T, (uint64_t)a.B};
    maps.o_ok = false;
    if (a.z == nullptr) {
      const uint64_t so[4] = {2, (uint64_t)a.o_stride_h * 2, (uint64_t)a.o_stride_t * 2, (uint64_t)(a.B > 1 ? a.o_stride_b : a.o_stride_t * a.T) * 2};
      const int last_error = g_last_cuda_error;
      maps.o_ok = make_tmap(&maps.o, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.o, 4, dims, so, box, CU_TENSOR_MAP_SWIZZLE_64B) == AVE_GDN_OK;
      if (!maps.o_ok) g_last_cuda_error = last_error;  // (no fault: 16-byte stores then)
    }
    if (o_f32 != nullptr) {
      const uint64_t row = (uint64_t)a.Hv * D * 4, s32[4] = {4, D * 4, row, row * a.T};
      const int rc = make_tmap(&maps.o32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, o_f32, 4, dims, s32, box, CU_TENSOR_MAP_SWIZZLE_128B);
      if (rc != AVE_GDN_OK) return rc;
    }
  }
  uint8_t* qt_img = L.parts > 1 ? reinterpret_cast<uint8_t*>(ws + L.qt_img) : nullptr;
  float* carry = reinterpret_cast<float*>(ws + L.carry);
  uint8_t* m0_pack = reinterpret_cast<uint8_t*>(ws + L.m0_pack);
  const int32_t* seq_order = chunk_start != nullptr ? chunk_start + a.n_seqs + 1 + L.chunks : nullptr;
  ScanPlan plan;
  plan.parts = L.parts;
  for (int p = 0; p <= MAX_PARTS; ++p) plan.part_begin[p] = L.part_begin[p];
  const int64_t tile_rows = (int64_t)a.Hk * ((a.Hv / a.Hk + 1) / 2);  // a unit of pass 1 takes up to two value heads of a key head
  auto tiles_grid = [&](int64_t chunks) { return dim3((unsigned)min(chunks * tile_rows, (int64_t)(2 * NUM_SMS))); };  // persistent, two CTAs an SM
  const unsigned scan_grid = (unsigned)a.n_seqs * (unsigned)(2 * L.parts - 1) * (unsigned)a.Hv;
  const auto scan = L.parts > 1 ? chunk_scan_kernel<true> : chunk_scan_kernel<false>;

  // What follows pass 2 on the caller's stream
  auto finish = [&]() -> int {
    if (L.parts <= 1) return a.z != nullptr ? norm_rows(a, o_f32, a.token_begin, a.T, stream) : AVE_GDN_OK;
    // Parts: the combine and the fix-up of the later ones.  With two parts the fix-up needs nothing from the combine, which then only forms
    // final states: it follows pass 2 directly, and the combine, all latency, runs beside it on a helper stream.  Dense layouts: so does the gated
    // norm of the tokens no fix-up touches, beside either; packed layouts: the norm covers every row, and the fix-up behind it rewrites those of
    // later parts.  32 heads x 8192 tokens 318.1 us with the combine in front of the fix-up, 313.5 beside it (without a gate 281.2, 277.5), 32768
    // tokens 1166, 1149; one packed sequence of 12000 491, 486; 2 x 8192 tokens x 16 heads 311, 311 (314 with the combine at a high priority).
    const bool dense_gate = a.z != nullptr && a.cu_seqlens == nullptr, two = L.parts == 2;
    SideSet* side = dense_gate || two ? side_set(dev, stream) : nullptr;
    int rc = AVE_GDN_OK;
    auto step = [&](cudaError_t e) { if (e != cudaSuccess && rc == AVE_GDN_OK) rc = cuda_fail(e); return rc == AVE_GDN_OK; };
    auto combine = [&](cudaStream_t on) {
      const int cols = (int64_t)a.n_seqs * a.Hv * (D / 4) <= NUM_SMS ? 4 : 8, stages = cols == 8 && two ? 1 : 3;
      const auto kernel = cols == 4 ? part_combine_kernel<4, 3> : stages == 1 ? part_combine_kernel<8, 1> : part_combine_kernel<8, 3>;
      step(launch_after(kernel, dim3((unsigned)(D / cols), (unsigned)a.Hv, (unsigned)a.n_seqs), 256, combine_smem(stages), on, a, chunk_start, carry, m0_pack, plan));
    };
    auto fix_up = [&]() {
      int part_len = 0;  // the longest of the later parts
      for (int p = 1; p < L.parts; ++p) part_len = max(part_len, min(L.part_begin[p + 1], L.max_chunks) - L.part_begin[p]);
      const int64_t groups = (int64_t)a.n_seqs * (L.parts - 1) * a.Hv;
      int split = (int)(NUM_SMS / (groups > 0 ? groups : 1));  // CTAs per (sequence, part, head), two chunks at a time each: about one wave
      split = max(1, min(split, (part_len + 1) / 2));
      step(launch_after(part_finish_kernel, dim3((unsigned)split, (unsigned)a.Hv, (unsigned)(a.n_seqs * (L.parts - 1))), FIN_THREADS, FIN_SMEM, stream,
                        a, chunk_start, o_f32, qt_img, m0_pack, plan));
    };
    const bool norm_beside = side != nullptr && dense_gate, combine_beside = side != nullptr && two;
    bool on_norm = false;
    auto norm_of_part0 = [&]() {
      on_norm = norm_beside && step(cudaStreamWaitEvent(side->norm, side->fork, 0));
      if (on_norm) rc = norm_rows(a, o_f32, 0, min(a.T, L.part_begin[1] * C), side->norm);
    };
    if (side != nullptr) AVE_CUDA_TRY(cudaEventRecord(side->fork, stream));
    if (a.z != nullptr && !norm_beside) rc = norm_rows(a, o_f32, a.token_begin, dense_gate ? min(a.T, L.part_begin[1] * C) : a.T, stream);
    if (!combine_beside) norm_of_part0();  // beside the combine
    if (rc == AVE_GDN_OK && !combine_beside) combine(stream);
    if (rc == AVE_GDN_OK) fix_up();
    cudaStream_t aside = norm_beside ? side->prep : combine_beside ? side->norm : nullptr;  // (in a mixed step, a packed layout, `prep` has the single tokens)
    const bool forked = combine_beside && rc == AVE_GDN_OK && step(cudaStreamWaitEvent(aside, side->fork, 0));
    if (forked) combine(aside);
    if (combine_beside && rc == AVE_GDN_OK) norm_of_part0();
    // (the joins after an error too, so that a surrounding stream capture stays well formed)
    if (forked) { step(cudaEventRecord(side->done[0], aside)); step(cudaStreamWaitEvent(stream, side->done[0], 0)); }
    if (on_norm) { step(cudaEventRecord(side->join_norm, side->norm)); step(cudaStreamWaitEvent(stream, side->join_norm, 0)); }
    return rc;
  };

  SideSet* side = L.segments > 1 ? side_set(dev, stream) : nullptr;
  if (side == nullptr) {
    // One launch per pass on the caller's stream.  The single tokens of a mixed step run beside pass 2, on a helper stream: pass 2 holds one SM a
    // chain and is bound by latency, they are bound by memory and take the SMs that its chains leave or never had.  They fork behind
    // pass 1, so that pass 2, which is launched dependent on it, has its SMs first; the gated norm follows pass 2 and runs beside the rest of them.
    // Those that share a slot with a prompt come in front of pass 2.
    // 61 sequences beside three prompts of 1500 tokens, 32 heads: one part behind the other 128 us, 96.3 so; 200
    // beside one of 100: 176, 165; 128 beside 2048 tokens 218, 150.  (With an event that completes when pass 2's CTAs have started, the
    // runtime held the single tokens back until pass 2 was complete: 128.)
    plan.r0 = 0; plan.rn = 1 << 24;  // every chunk (times 64 still fits an int)
    SideSet* beside = decode != nullptr ? side_set(dev, stream) : nullptr;
    if (decode != nullptr && beside == nullptr) {
      const int drc = launch_decode(*decode, stream);
      if (drc != AVE_GDN_OK) return drc;
    }
    int rc = AVE_GDN_OK;
    auto step = [&](cudaError_t e) { if (e != cudaSuccess && rc == AVE_GDN_OK) rc = cuda_fail(e); return rc == AVE_GDN_OK; };
    if (rc == AVE_GDN_OK) step(launch_after(chunk_tiles_kernel, tiles_grid(L.chunks), TILES_THREADS, TILES_SMEM, stream, a, chunk_start, recs, plan, (int)L.chunks, 0));
    if (rc == AVE_GDN_OK && beside != nullptr) rc = launch_shared_slots(*decode, a, stream);
    const bool forked = rc == AVE_GDN_OK && beside != nullptr && step(cudaEventRecord(beside->fork, stream)) && step(cudaStreamWaitEvent(beside->prep, beside->fork, 0));
    if (rc == AVE_GDN_OK)
      step(launch_after(scan, scan_grid, SCAN_THREADS, SCAN_SMEM, stream, a, maps, chunk_start, recs, o_f32, qt_img, carry, m0_pack, seq_order, plan));
    if (rc == AVE_GDN_OK && forked) rc = launch_decode_beside(*decode, a, beside->prep);
    if (rc == AVE_GDN_OK) rc = finish();
    if (forked) {  // after an error too, so that a surrounding stream capture stays well formed
      step(cudaEventRecord(beside->join, beside->prep));
      step(cudaStreamWaitEvent(stream, beside->join, 0));
    }
    return rc;
  }

  // Pass 1 of all ranges back to back on one helper stream, pass 2 of range i on a second once pass 1 of range i is
  // done, and (dense layouts) the gated norm of range i on a third once pass 2 of range i is done; all
  // fork from the caller's stream and join back into it through events.  After an error the joins are still enqueued,
  // so that a surrounding stream capture stays well formed.
  const bool norm_per_range = a.z != nullptr && a.cu_seqlens == nullptr;
  AVE_CUDA_TRY(cudaEventRecord(side->fork, stream));
  int rc = AVE_GDN_OK;
  auto step = [&](cudaError_t e) { if (e != cudaSuccess && rc == AVE_GDN_OK) rc = cuda_fail(e); return e == cudaSuccess; };
  step(cudaStreamWaitEvent(side->prep, side->fork, 0));
  step(cudaStreamWaitEvent(side->scan, side->fork, 0));
  if (norm_per_range) step(cudaStreamWaitEvent(side->norm, side->fork, 0));
  for (int i = 0; i < L.segments && rc == AVE_GDN_OK; ++i) {
    plan.r0 = L.seg_begin[i]; plan.rn = L.seg_begin[i + 1] - L.seg_begin[i];
    if (plan.rn <= 0) continue;
    chunk_tiles_kernel<<<tiles_grid((int64_t)a.n_seqs * plan.rn), TILES_THREADS, TILES_SMEM, side->prep>>>(a, chunk_start, recs, plan, a.n_seqs * plan.rn, 1);
    if (!step(cudaGetLastError())) break;
    if (!step(cudaEventRecord(side->done[i], side->prep))) break;
    if (!step(cudaStreamWaitEvent(side->scan, side->done[i], 0))) break;
    scan<<<scan_grid, SCAN_THREADS, SCAN_SMEM, side->scan>>>(a, maps, chunk_start, recs, o_f32, qt_img, carry, m0_pack, seq_order, plan);
    if (!step(cudaGetLastError())) break;
    if (norm_per_range) {
      if (!step(cudaEventRecord(side->scanned[i], side->scan))) break;
      if (!step(cudaStreamWaitEvent(side->norm, side->scanned[i], 0))) break;
      const int nrc = norm_rows(a, o_f32, min(a.T, plan.r0 * C), min(a.T, (plan.r0 + plan.rn) * C), side->norm);
      if (nrc != AVE_GDN_OK && rc == AVE_GDN_OK) rc = nrc;
    }
  }
  if (rc == AVE_GDN_OK && a.z != nullptr && !norm_per_range) rc = norm_rows(a, o_f32, a.token_begin, a.T, side->scan);  // packed layout: after the last scan
  step(cudaEventRecord(side->join, side->scan));
  step(cudaStreamWaitEvent(stream, side->join, 0));
  step(cudaEventRecord(side->join_norm, norm_per_range ? side->norm : side->prep));
  step(cudaStreamWaitEvent(stream, side->join_norm, 0));
  return rc;
}

}  // namespace ave

// ------------------------------------------------------------------------------------------------ no-allocation variant
// Some callers may not allocate device memory at all: code that runs between a framework's memory-pool snapshot
// and its release (serving runtimes that hand every byte of HBM to a paged state/KV pool at start-up and forbid
// later driver allocations), plug-in callbacks that only receive pre-registered buffers, and latency-critical
// paths where an allocator call is not allowed.  For them the prefill scratch lives in this fixed array, which
// every GPU that loads the library carries until the process exits.
namespace ave {
int validate_prefill_args(const AveGdnArgs* a);
constexpr size_t kStaticScratchBytes = AVE_GDN_NOALLOC_SCRATCH_BYTES;  // 64 MiB
}
static __device__ __align__(256) unsigned char g_static_prefill_scratch[ave::kStaticScratchBytes];

// The array's name is only a host-side handle; the device address is looked up once per device (with that device
// current) and cached.  That first call on a device should be made outside any stream capture.
extern "C" int ave_gdn_chunk_prefill_noalloc(const AveGdnArgs* args, void* stream) {
  using namespace ave;
  const int rc = validate_prefill_args(args);
  if (rc != AVE_GDN_OK) return rc;
  if ((int64_t)args->B * args->T == 0 || args->n_seqs == 0) return AVE_GDN_OK;
  if (args->dk != 128 || args->dv != 128) return AVE_GDN_UNSUPPORTED;
  // The plain schedule: one launch per pass on the caller's stream, no helper streams or events, the least scratch.  A request is judged by
  // the records' size that the documented limits were given for; what a call uses of the array is less.
  constexpr size_t kJudgedRecord = 66304;
  const size_t records = (size_t)(args->cu_seqlens ? (int64_t)args->T / C + args->n_seqs : (int64_t)args->B * ((args->T + C - 1) / C)) * args->Hv;
  if (prefill_tc_workspace_bytes(*args, true) + records * (kJudgedRecord - REC_BYTES) > kStaticScratchBytes) return AVE_GDN_WORKSPACE_TOO_SMALL;
  static std::mutex mu;
  static void* scratch_of_device[64] = {};
  int dev = 0;
  AVE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return AVE_GDN_UNSUPPORTED;
  void* scratch = nullptr;
  {
    std::lock_guard<std::mutex> guard(mu);
    if (scratch_of_device[dev] == nullptr) {
      void* p = nullptr;
      AVE_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_prefill_scratch));
      scratch_of_device[dev] = p;
    }
    scratch = scratch_of_device[dev];
  }
  AveGdnArgs local = *args;
  local.workspace = scratch;
  local.workspace_bytes = kStaticScratchBytes;
  // every scratch record a launch reads is written earlier in the same launch sequence, so nothing needs clearing
  return launch_prefill_tc(local, reinterpret_cast<cudaStream_t>(stream), true, nullptr);
}
