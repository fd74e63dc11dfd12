// Blackwell (sm_100a) building blocks in inline PTX: mbarrier with bounded waits, TMA (tiled and bulk)
// copies, tensor-memory allocation, tcgen05 MMA / commit / ld / st, and the shared-memory and instruction
// descriptors the MMA reads.  No cluster multicast is used anywhere.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ave {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The first multiple of 1024 bytes in the dynamic shared memory.  An offset is added to the pointer itself: rounding its address
// as an integer loses the address space, and every access behind it becomes a generic one (the scale vectors of a chunk then cost
// the scan's epilogue 300 to 500 cycles a stage; 32 heads x 8192 tokens 398 us, with shared loads 374).
__device__ __forceinline__ uint8_t* align1024(uint8_t* smem) { return smem + ((0u - smem_u32(smem)) & 1023u); }

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after kWaitLimit polls that found the phase incomplete, or as soon as another role has raised *abort_flag.
// Returns false on give-up (the caller raises the flag, records a status bit and leaves its loop).
// The loops stay rolled, here and below: with those that the compiler unrolls a kernel of many roles outgrows the SM's 32 KB of instruction cache (the prefill's
// scan missed 145 lines a chunk; 39 with this, roles that are uniform to the compiler and a rolled loop for the outputs; 8192 tokens x 32 heads 297 -> 260 us).
constexpr uint32_t kWaitLimit = 1u << 24;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag) {
  uint32_t left = kWaitLimit;
#pragma unroll 1
  while (!mbar_try_wait(bar, parity))
    if (*abort_flag != 0u || --left == 0u) { *abort_flag = 1u; return false; }
  return true;
}

// The same in a loop that the compiler unrolls and that looks for the flag at every 64th poll, for the GEMM, whose few roles have the room: 4096^3 108.7 us
// with the other, 106.4 with this, 1000 x 12352 x 2048 42.8 and 42.3.
__device__ __forceinline__ bool mbar_wait_unrolled(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag) {
  for (uint32_t it = 0; it < kWaitLimit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 63u && *abort_flag != 0u) return false;
  }
  *abort_flag = 1u;
  return false;
}

// Bounded waits for two or three phases at once.  The polls are independent, so the latencies of phases that are
// already complete overlap instead of adding up.
__device__ __forceinline__ bool mbar_wait2(uint64_t* b0, uint32_t p0, uint64_t* b1, uint32_t p1, volatile uint32_t* abort_flag) {
  uint32_t left = kWaitLimit;
  bool d0 = false, d1 = false;  // seen complete, once and for all
#pragma unroll 1
  for (;;) {
    d0 |= mbar_try_wait(b0, p0); d1 |= mbar_try_wait(b1, p1);
    if (d0 & d1) return true;
    if (*abort_flag != 0u || --left == 0u) { *abort_flag = 1u; return false; }
  }
}
__device__ __forceinline__ bool mbar_wait3(uint64_t* b0, uint32_t p0, uint64_t* b1, uint32_t p1, uint64_t* b2, uint32_t p2,
                                           volatile uint32_t* abort_flag) {
  uint32_t left = kWaitLimit;
  bool d0 = false, d1 = false, d2 = false;
#pragma unroll 1
  for (;;) {
    d0 |= mbar_try_wait(b0, p0); d1 |= mbar_try_wait(b1, p1); d2 |= mbar_try_wait(b2, p2);
    if (d0 & d1 & d2) return true;
    if (*abort_flag != 0u || --left == 0u) { *abort_flag = 1u; return false; }
  }
}

// Bounded wait called by all 32 lanes of a converged warp.  Every lane polls: letting lane 0 poll alone and
// broadcasting the outcome was measured and doubled the time of the scan (0.90 ms against 0.46 ms on an 8192-token
// sequence), so the hand-off latency is not a matter of the number of pollers.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag) {
  return mbar_wait(bar, parity, abort_flag);
}

// A hardware barrier as a hand-off: `threads` of them arrive or wait, whole warps, and those that wait go on when all are there.  30 cycles from the
// last arrival to the first instruction behind the wait, an mbarrier 85 to 100 (alone on an SM; more beside others' shared-memory traffic).
// A wait on it is not bounded, so it is only for roles that come to it as often as they are waited for whatever happens, bounded waits of theirs
// that expire included.  And nobody may arrive again before the waiting warps have gone on (the barrier counts threads and knows no parity: it
// would complete without them), so a warp may arrive only where its own waits see to that; one whose wait has expired (`alive` false, the same for the
// whole warp) waits with the others.
struct NamedBar { uint32_t id, threads; };
__device__ __forceinline__ void named_sync(NamedBar b) { asm volatile("bar.sync %0, %1;" ::"r"(b.id), "r"(b.threads) : "memory"); }
__device__ __forceinline__ void mbar_arrive(NamedBar b, bool alive) {
  if (alive) asm volatile("bar.arrive %0, %1;" ::"r"(b.id), "r"(b.threads) : "memory");
  else named_sync(b);
}
__device__ __forceinline__ void mbar_wait_warp(NamedBar b, uint32_t, volatile uint32_t*) { named_sync(b); }

// In front of a CTA's end, for a phase that copies or MMAs of its own complete: waited for whatever the flag says, again with a limit.
__device__ __forceinline__ void drain(uint64_t* bar, uint32_t parity) {
  uint32_t left = kWaitLimit;
#pragma unroll 1
  while (!mbar_try_wait(bar, parity) && --left != 0u) {}
}

// One lane of a converged warp; the enclosing control flow stays warp-uniform.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}

// Per-warpgroup register budget (all four warps of an aligned warpgroup execute it together).  The sum over the
// CTA's warpgroups must stay within the kernel's launch-time allocation or the increase never completes.
// A decrease to more, or an increase to fewer, registers than the warp currently owns is an illegal instruction,
// so the direction is derived from the launch-time count.
template <int N, int LAUNCH_REGS>
__device__ __forceinline__ void reg_set() {
  static_assert(N % 8 == 0 && N >= 24 && N <= 256, "register count must be a multiple of 8 in [24, 256]");
  if constexpr (N > LAUNCH_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
  else if constexpr (N < LAUNCH_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// ---------------------------------------------------------------- proxies / fences
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
// untiled bulk copy global -> shared (both 16-byte aligned, size a multiple of 16)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// a run of global memory towards L2 (16-byte aligned, size a multiple of 16)
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<uint64_t>(src)), "r"(bytes) : "memory");
}
// untiled bulk copy shared -> global (both 16-byte aligned, size a multiple of 16), tracked by the thread's bulk group
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(reinterpret_cast<uint64_t>(dst)),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
// tiled copy shared -> global, tracked the same way; what lies outside the tensor is not written
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)),
               "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------- thread-block clusters (distributed shared memory)
__device__ __forceinline__ uint32_t mapa(uint32_t saddr, uint32_t rank) {  // address of the same location in CTA `rank` of the cluster
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// every thread of every CTA of the cluster; shared-memory writes before it are visible after it
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}

// ---------------------------------------------------------------- tensor memory
// One full warp allocates; the base address (lane 0, first column) lands in *slot (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

// ---------------------------------------------------------------- descriptors
// 64-bit shared-memory matrix descriptor, 128-byte swizzle.  K-major operand: rows of 128 bytes, 8-row groups
// `sbo` bytes apart (lbo unused).  MN-major operand: 128 bytes (64 elements) of MN contiguous per k-row, groups of
// 8 k-rows `sbo` bytes apart, successive 64-element MN groups `lbo` bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3fffu);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fffu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  d |= (uint64_t)2 << 61;  // 128-byte swizzle
  return d;
}
// The two words of such a descriptor, or of one without swizzle (K-major: 8x8 core matrices of 128 contiguous bytes, `lbo` bytes from one to the next along
// K and `sbo` along M or N), for a tile that lies `off` bytes behind one whose address / 16 is known: the low word is that plus
// desc_lo, the high word is desc_hi, both constants.  (An address put together, shifted and masked for every MMA costs more than a small MMA.)
__host__ __device__ constexpr uint32_t desc_lo(int off, int lbo_bytes) { return (uint32_t)(off >> 4) | (uint32_t)(lbo_bytes >> 4) << 16; }
__host__ __device__ constexpr uint32_t desc_hi(int sbo_bytes, bool swizzled) { return (uint32_t)(sbo_bytes >> 4) | 1u << 14 | (swizzled ? 2u << 29 : 0u); }
__device__ __forceinline__ uint64_t smem_desc(uint32_t lo, uint32_t hi) { return (uint64_t)hi << 32 | lo; }
// 32-bit instruction descriptor for kind::f16 with fp32 accumulate.  fmt: 0 = f16, 1 = bf16.
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N, int a_fmt, int b_fmt, bool a_mn_major, bool b_mn_major,
                                                 bool a_neg = false, bool b_neg = false) {
  return (1u << 4) | ((uint32_t)a_fmt << 7) | ((uint32_t)b_fmt << 10) | ((uint32_t)a_neg << 13) | ((uint32_t)b_neg << 14) |
         ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ---------------------------------------------------------------- MMA
// D[tmem] (+)= A[smem] * B[smem]; issued by one thread.
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// mbarrier arrives once every tcgen05 operation issued so far by this thread has completed
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// the same for all MMAs of this warp, whose elected lane has issued them; `bar` is used by nothing else
__device__ __forceinline__ void drain_mmas(uint64_t* bar) {
  if (elect_one()) mma_commit(bar);
  __syncwarp();
  drain(bar, 0u);
}

// ---------------------------------------------------------------- TMEM <-> registers (warp-collective; a warp reaches
// only the 32 lanes of its quarter: lanes 32*(warp_id % 4) ...)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// 16 lanes x 8 columns in the accumulator layout of the warp-level m16n8 MMAs
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, float (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(taddr) : "memory");
}
// the same for eight and four adjacent groups of 8 columns, four registers a group
__device__ __forceinline__ void tmem_ld_frags(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_frags(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// N consecutive 32-bit columns of this warp's 32 lanes
template <int N>
__device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t (&r)[N]) {
  static_assert(N == 16 || N == 32, "column count");
  if constexpr (N == 32) tmem_ld32(taddr, r); else tmem_ld16(taddr, r);
}
template <int N>
__device__ __forceinline__ void tmem_st_n(uint32_t taddr, const uint32_t (&r)[N]) {
  static_assert(N == 8 || N == 16, "column count");
  if constexpr (N == 16) tmem_st16(taddr, r); else tmem_st8(taddr, r);
}

}  // namespace tc

// ---------------------------------------------------------------- host side: tensor maps without linking libcuda
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn();
// rank-N bf16 (or other 2-byte) tensor map with 128-byte swizzle; dims/strides innermost first, strides in bytes
// (strides[0] is implied by the element size and not passed to the driver).
int make_tmap(CUtensorMap* out, CUtensorMapDataType dt, int elem_bytes, void* base, int rank, const uint64_t* dims,
              const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swz);

}  // namespace ave
