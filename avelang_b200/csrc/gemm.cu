// C[M,N] = A[M,K] * B[N,K]^T, bf16 operands, fp32 accumulation in tensor memory, bf16 result.
//
// Persistent kernel, one CTA per SM, 128x256 output tiles, K in steps of 64 (one 128-byte swizzle span):
//   warp 0      TMA producer: A and B tiles into a 4-stage shared-memory ring
//   warp 1      issues tcgen05.mma (128x256x16 per instruction) into one of two 256-column TMEM accumulators
//   warps 2..5  epilogue: TMEM -> registers -> bf16 -> global, overlapped with the next tile's main loop
// Tiles are walked in groups of 16 row-tiles so the A rows of a group stay in L2 while B is swept.
#include <mutex>

#include "common.cuh"
#include "tc.cuh"

namespace ave {
namespace {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int GEMM_THREADS = 192;
constexpr int GROUP_M = 16;
constexpr size_t GEMM_SMEM = (size_t)STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
// row-parallel form: each epilogue warp also has a [32 rows][128 columns] bf16 staging tile, so that rows leave as
// 256 contiguous bytes (stores of 16 bytes per row, as the plain epilogue issues them, make poor NVLink packets)
constexpr int EPI_STAGE_BYTES = 32 * 256;
constexpr int SKINNY_STAGES = 10, SKINNY_RING = 200 * 1024;  // ring depth limit and bytes of the few-row-tiles form
constexpr int SKINNY_SMEM = SKINNY_RING + A_BYTES + 1024;    // an MMA reads 128 rows of A wherever the tile ends
constexpr size_t GEMM_SMEM_SCATTER = GEMM_SMEM + 4 * EPI_STAGE_BYTES;

// Row-parallel form: instead of one result matrix, every 128-row piece of this rank's partial product goes to the rank
// that owns those rows (rows_per_owner consecutive rows each), into slot `rank` of the owner's staging buffer
// [n_ranks][rows_per_owner][N] -- plain peer stores over NVLink from the GEMM's own epilogue, tile by tile, while the
// main loop of the next tile runs.  dst == nullptr: the ordinary single-matrix epilogue.
struct GemmScatter { const uint64_t* dst; int n_ranks, rank; int64_t rows_per_owner; };

struct TileCoord { int m, n; };
__device__ __forceinline__ TileCoord tile_coord(int tile, int mt, int nt) {
  const int per_group = GROUP_M * nt;
  const int g = tile / per_group, r = tile % per_group;
  const int rows = min(GROUP_M, mt - g * GROUP_M);
  return {g * GROUP_M + r % rows, r / rows};
}

__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_nt_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    __nv_bfloat16* __restrict__ C, int64_t M, int64_t N, int64_t K, int64_t ldc, uint32_t* status, int bn,
                    const GemmScatter sc) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = tc::align1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full = bars;                 // [STAGES]
  uint64_t* empty = bars + STAGES;       // [STAGES]
  uint64_t* acc_full = bars + 2 * STAGES;      // [2]
  uint64_t* acc_empty = bars + 2 * STAGES + 2; // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // bn: width of a column tile, a multiple of 16 up to BN chosen by the launcher so that the column tiles are of
  // (nearly) equal width; shared memory and tensor memory are laid out for BN
  const int mt = (int)((M + BM - 1) / BM), nt = (int)((N + bn - 1) / bn), kb_count = (int)((K + BK - 1) / BK);
  const int n_tiles = mt * nt;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { tc::mbar_init(&acc_full[b], 1); tc::mbar_init(&acc_empty[b], 4); }
    *abort_flag = 0;
    tc::fence_barrier_init();
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, 512);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const TileCoord tcd = tile_coord(tile, mt, nt);
        for (int kb = 0; kb < kb_count; ++kb) {
          if (!tc::mbar_wait_unrolled(&empty[s], ph ^ 1u, abort_flag)) goto producer_done;
          tc::mbar_expect_tx(&full[s], (uint32_t)(A_BYTES + bn * BK * 2));
          tc::tma_load_2d(smem + s * STAGE_BYTES, &tmA, &full[s], kb * BK, tcd.m * BM);
          tc::tma_load_2d(smem + s * STAGE_BYTES + A_BYTES, &tmB, &full[s], kb * BK, tcd.n * bn);
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
      }
    }
  producer_done:;
  } else if (warp == 1) {
    if (lane == 0) {
      int s = 0; uint32_t ph = 0; int local = 0;
      for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++local) {
        const uint32_t idesc = tc::idesc_f16(BM, bn, 1, 1, false, false);
        const int buf = local & 1;
        const uint32_t acc_ph = (uint32_t)(local >> 1) & 1u;
        if (!tc::mbar_wait_unrolled(&acc_empty[buf], acc_ph ^ 1u, abort_flag)) break;
        tc::tc_fence_after_sync();
        const uint32_t d = tmem_base + (uint32_t)buf * BN;
        bool ok = true;
        for (int kb = 0; kb < kb_count; ++kb) {
          if (!tc::mbar_wait_unrolled(&full[s], ph, abort_flag)) { ok = false; break; }
          tc::tc_fence_after_sync();
          const uint32_t a_addr = tc::smem_u32(smem + s * STAGE_BYTES);
          const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            tc::mma_ss(d, tc::smem_desc_sw128(a_addr + k * 32, 16, 1024), tc::smem_desc_sw128(b_addr + k * 32, 16, 1024), idesc,
                       (kb | k) != 0 ? 1u : 0u);
          }
          tc::mma_commit(&empty[s]);
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        tc::mma_commit(&acc_full[buf]);
      }
    }
  } else {
    const int quarter = warp & 3;  // TMEM lanes this warp may touch
    int local = 0;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++local) {
      const TileCoord tcd = tile_coord(tile, mt, nt);
      const int buf = local & 1;
      const uint32_t acc_ph = (uint32_t)(local >> 1) & 1u;
      if (!tc::mbar_wait_unrolled(&acc_full[buf], acc_ph, abort_flag)) break;
      tc::tc_fence_after_sync();
      const int64_t row = (int64_t)tcd.m * BM + quarter * 32 + lane;
      __nv_bfloat16* crow = C + row * ldc + (int64_t)tcd.n * bn;
      const int64_t n_left = min((int64_t)bn, N - (int64_t)tcd.n * bn);
      const int col_groups = (int)((n_left + 31) / 32);  // 32-column groups that hold results
      if (sc.dst != nullptr) {
        // Row-parallel form: 128 columns at a time through this warp's staging tile (16-byte pieces, piece p of row r
        // at p ^ (r & 15): conflict-free both ways), then out two rows per instruction, 256 contiguous bytes each, to
        // the slot of the rank that owns the row.
        uint8_t* st = smem + STAGES * STAGE_BYTES + 256 + (warp - 2) * EPI_STAGE_BYTES;
        const int64_t row_first = (int64_t)tcd.m * BM + quarter * 32;
        const int owner0 = (int)min(row_first / sc.rows_per_owner, (int64_t)sc.n_ranks - 1);
        const int64_t boundary = (int64_t)(owner0 + 1) * sc.rows_per_owner;  // first row of the next owner
        const int halves = (int)((n_left + 127) / 128);
#pragma unroll 1
        for (int half = 0; half < halves; ++half) {
#pragma unroll 1
          for (int c4 = 0; c4 < 4; ++c4) {
            if (half * 128 + c4 * 32 >= n_left) break;
            uint32_t r[32];
            tc::tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + half * 128 + c4 * 32), r);
            tc::tmem_ld_wait();
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 pk;
              pk.x = pack_bf16x2(__uint_as_float(r[v * 8 + 0]), __uint_as_float(r[v * 8 + 1]));
              pk.y = pack_bf16x2(__uint_as_float(r[v * 8 + 2]), __uint_as_float(r[v * 8 + 3]));
              pk.z = pack_bf16x2(__uint_as_float(r[v * 8 + 4]), __uint_as_float(r[v * 8 + 5]));
              pk.w = pack_bf16x2(__uint_as_float(r[v * 8 + 6]), __uint_as_float(r[v * 8 + 7]));
              *reinterpret_cast<uint4*>(st + lane * 256 + (((c4 * 4 + v) ^ (lane & 15)) << 4)) = pk;
            }
          }
          if (half == halves - 1) {  // the accumulator is out of tensor memory: the next tile's MMAs may overwrite it
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
          }
          __syncwarp();
          const int p = lane & 15;
          const int64_t col = (int64_t)half * 128 + p * 8;
#pragma unroll 4
          for (int it = 0; it < 16; ++it) {
            const int a = 2 * it + (lane >> 4);
            const int64_t grow = row_first + a;
            if (grow < M && col < n_left) {
              const uint4 pk = *reinterpret_cast<const uint4*>(st + a * 256 + ((p ^ (a & 15)) << 4));
              // a 32-row block meets at most two owners unless an owner has fewer than 32 rows
              const int owner = sc.rows_per_owner >= 32 ? (grow >= boundary ? owner0 + 1 : owner0)
                                                        : (int)min(grow / sc.rows_per_owner, (int64_t)sc.n_ranks - 1);
              __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(sc.dst[owner]) +
                                   ((int64_t)sc.rank * sc.rows_per_owner + (grow - (int64_t)owner * sc.rows_per_owner)) * ldc +
                                   (int64_t)tcd.n * bn + col;
              *reinterpret_cast<uint4*>(dst) = pk;
            }
          }
          __syncwarp();
        }
        continue;
      }
#pragma unroll 1
      for (int c = 0; c < col_groups; ++c) {
        uint32_t r[32];
        tc::tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c * 32), r);
        tc::tmem_ld_wait();
        if (row < M) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int col = c * 32 + v * 8;
            if (col + 8 <= n_left) {
              uint4 pk;
              pk.x = pack_bf16x2(__uint_as_float(r[v * 8 + 0]), __uint_as_float(r[v * 8 + 1]));
              pk.y = pack_bf16x2(__uint_as_float(r[v * 8 + 2]), __uint_as_float(r[v * 8 + 3]));
              pk.z = pack_bf16x2(__uint_as_float(r[v * 8 + 4]), __uint_as_float(r[v * 8 + 5]));
              pk.w = pack_bf16x2(__uint_as_float(r[v * 8 + 6]), __uint_as_float(r[v * 8 + 7]));
              *reinterpret_cast<uint4*>(crow + col) = pk;
            } else {
              for (int e = 0; e < 8; ++e)
                if (col + e < n_left) crow[col + e] = __float2bfloat16(__uint_as_float(r[v * 8 + e]));
            }
          }
        }
      }
      tc::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
    }
  }

  tc::tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && status != nullptr) atomicOr(status, AVE_GDN_DEV_WAIT_EXPIRED);
  if (warp == 1) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem_base, 512);
  }
}

// The form for few row tiles (decode batches, short prompts), where 128 x 256 tiles leave most SMs idle and the time is
// that of streaming B: one tile per cluster of `split` CTAs, each of which takes a contiguous share of K; column tiles are
// as narrow as it takes to give every SM a part of B (see skinny_plan).  The partial accumulators meet in shared memory:
// CTA r owns rows [r * slice, (r + 1) * slice) of the tile, every CTA stores its part of them into r's (drained) operand
// ring over distributed shared memory, and r sums the parts in rank order, rounds once and stores whole rows.
// M = 64, operands not in L2: N = 12352, K = 2048 in 16.9 us and N = 2048, K = 4096 in 12.6 us, of which 4.5 us are launch,
// prologue and exchange; 22.5 and 28.3 us with the persistent kernel (49 and 8 tiles).
struct SkinnyPlan { int bn, split, stages, ks, a_rows; };  // tile width, CTAs per tile, ring depth, 64-blocks per stage, A rows
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, __nv_bfloat16* __restrict__ C,
                   int64_t M, int64_t N, int64_t K, int64_t ldc, uint32_t* status, const SkinnyPlan plan, uint32_t tmem_cols) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = tc::align1024(smem_raw);
  __shared__ uint64_t full[SKINNY_STAGES], empty[SKINNY_STAGES], acc_full;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bn = plan.bn, split = plan.split, stages = plan.stages;
  const int a_bytes = plan.a_rows * BK * 2, b_bytes = bn * BK * 2, stage_bytes = plan.ks * (a_bytes + b_bytes);
  const int nt = (int)((N + bn - 1) / bn), kb_count = (int)((K + plan.ks * BK - 1) / (plan.ks * BK));  // in stages of ks x 64
  const int rank = (int)(blockIdx.x % split), tile = (int)(blockIdx.x / split), tm = tile / nt, tn = tile % nt;
  const int per = (kb_count + split - 1) / split, kb0 = rank * per, kb1 = min(kb_count, kb0 + per);

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
    tc::mbar_init(&acc_full, 1);
    abort_flag = 0;
    tc::fence_barrier_init();
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 1) tc::tmem_alloc(&tmem_slot, tmem_cols);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();

  // Both issuing warps run their loops whole and elect a lane for the instructions themselves.  A stage holds `ks` blocks
  // of 64 along K, [A][A].. [B][B].., behind one barrier: a wait, its loads or MMAs and the release cost about 700 cycles
  // whatever their size, which at 64 per stage (8 to 16 KB) was longer than the data took to arrive.
  if (warp == 0) {
    int s = 0; uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!tc::mbar_wait_unrolled(&empty[s], ph ^ 1u, &abort_flag)) break;
      if (tc::elect_one()) {
        uint8_t* st = smem + s * stage_bytes;
        tc::mbar_expect_tx(&full[s], (uint32_t)stage_bytes);
        for (int j = 0; j < plan.ks; ++j) tc::tma_load_2d(st + plan.ks * a_bytes + j * b_bytes, &tmB, &full[s], (kb * plan.ks + j) * BK, tn * bn);
        for (int j = 0; j < plan.ks; ++j) tc::tma_load_2d(st + j * a_bytes, &tmA, &full[s], (kb * plan.ks + j) * BK, tm * BM);
      }
      __syncwarp();
      if (++s == stages) { s = 0; ph ^= 1u; }
    }
  } else if (warp == 1) {
    const uint32_t idesc = tc::idesc_f16(BM, bn, 1, 1, false, false);
    int s = 0; uint32_t ph = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!tc::mbar_wait_unrolled(&full[s], ph, &abort_flag)) { ok = false; break; }
      tc::tc_fence_after_sync();
      if (tc::elect_one()) {
        // with fewer than 128 rows in the A tile the MMA reads whatever lies behind it: those lanes are never read back
        const uint32_t base = tc::smem_u32(smem) + (uint32_t)(s * stage_bytes);
        for (int j = 0; j < plan.ks; ++j) {
          const uint64_t da = tc::smem_desc_sw128(base + (uint32_t)(j * a_bytes), 16, 1024);
          const uint64_t db = tc::smem_desc_sw128(base + (uint32_t)(plan.ks * a_bytes + j * b_bytes), 16, 1024);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            tc::mma_ss(tmem_base, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > kb0 || j > 0 || k != 0) ? 1u : 0u);
        }
        tc::mma_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == stages) { s = 0; ph ^= 1u; }
    }
    if (ok && tc::elect_one()) tc::mma_commit(&acc_full);
  }
  __syncwarp();  // the other lanes of the issuing warps must not poll beside them
  // the accumulator is complete, so every operand tile has landed and been read
  const bool ok = tc::mbar_wait_unrolled(&acc_full, 0, &abort_flag);
  tc::tc_fence_after_sync();
  __syncwarp();
  tc::cluster_sync();  // ... in every CTA of the cluster: the rings may be overwritten
  const int rows = (int)min((int64_t)BM, M - (int64_t)tm * BM), slice = (rows + split - 1) / split, pitch = bn + 4;
  if (ok && warp >= 2) {
    const int row = (warp & 3) * 32 + lane;
    const bool live = row < rows;
    const int owner = live ? row / slice : 0;
    const uint32_t dst = tc::mapa(tc::smem_u32(smem) + (uint32_t)(((rank * slice + (row - owner * slice)) * pitch) * 4), (uint32_t)owner);
#pragma unroll 1
    for (int c = 0; c < bn; c += 16) {
      uint32_t r[16];
      tc::tmem_ld16(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, r);
      tc::tmem_ld_wait();
      if (live) {
#pragma unroll
        for (int v = 0; v < 4; ++v) tc::st_cluster_v4(dst + (uint32_t)(c + 4 * v) * 4, r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
      }
    }
  }
  tc::tc_fence_before_sync();
  __syncwarp();
  tc::cluster_sync();
  {
    const float* part = reinterpret_cast<const float*>(smem);
    const int mine = min(slice, rows - rank * slice), vec = bn / 8;
    for (int i = threadIdx.x; i < mine * vec; i += GEMM_THREADS) {
      const int r = i / vec, c = (i - r * vec) * 8;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
      for (int s = 0; s < split; ++s) {
        const float4 a = *reinterpret_cast<const float4*>(part + (s * slice + r) * pitch + c);
        const float4 b = *reinterpret_cast<const float4*>(part + (s * slice + r) * pitch + c + 4);
        x.x += a.x; x.y += a.y; x.z += a.z; x.w += a.w;
        y.x += b.x; y.y += b.y; y.z += b.z; y.w += b.w;
      }
      const int64_t col = (int64_t)tn * bn + c;
      __nv_bfloat16* dst = C + ((int64_t)tm * BM + rank * slice + r) * ldc + col;
      if (col + 8 <= N) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
      } else {
        const float f[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        for (int e = 0; e < 8; ++e)
          if (col + e < N) dst[e] = __float2bfloat16(f[e]);
      }
    }
  }
  if (threadIdx.x == 0 && !ok && status != nullptr) atomicOr(status, AVE_GDN_DEV_WAIT_EXPIRED);
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem_base, tmem_cols);
  }
}

// Tile width, K split and ring depth for a product with few row tiles: among the cluster sizes that still give every tile
// its SMs, the one with the fewest bytes through the busiest SM (its operand tiles, plus what the exchange costs).
// `clusters[s]`: clusters of s CTAs that run at once.  A cluster lives inside one GPC, so it is not 148 / s (a plan of 49
// clusters of 3 needed a second wave and took twice the time).
SkinnyPlan skinny_plan(int64_t M, int64_t N, int64_t K, const int* clusters) {
  const int64_t mt = (M + BM - 1) / BM, kb = (K + BK - 1) / BK;
  const int64_t a_rows = M < BM ? (M + 7) / 8 * 8 : BM;
  SkinnyPlan best{};
  int64_t best_cost = INT64_MAX;
  for (int split = 1; split <= 8; ++split) {
    const int64_t tiles_n = clusters[split] / mt;
    if (tiles_n == 0) continue;
    const int64_t bn = ((N + tiles_n - 1) / tiles_n + 15) / 16 * 16, block = (a_rows + bn) * BK * 2;
    if (bn > BN) continue;
    // blocks of 64 per stage: up to 48 KB a stage, at least three stages, no padding of K beyond one block per CTA
    int ks = 1;
    while (ks < 8 && 2 * ks * block <= 49152 && 2 * ks * split <= kb) ks *= 2;
    const int64_t steps = (kb + ks - 1) / ks, per = (steps + split - 1) / split;
    if ((split - 1) * per >= steps) continue;  // no CTA without work
    // a stage costs at least the 16 KB that arrive during its waits, and a block of 64 at least the 8 KB that arrive during
    // its four MMAs, which read 128 rows of A however narrow they are; two cluster barriers are worth 64 KB of streaming
    const int64_t stage = ks * block, exchange = split == 1 ? 0 : 65536 + a_rows * bn * 4;
    const int64_t least = ks > 2 ? ks * 8192 : 16384;
    const int64_t cost = per * (stage > least ? stage : least) + exchange;
    if (cost < best_cost) {
      best_cost = cost;
      const int fit = (int)(SKINNY_RING / stage);
      best = {(int)bn, split, fit < SKINNY_STAGES ? fit : SKINNY_STAGES, ks, (int)a_rows};
    }
  }
  return best;
}

// Clusters of 1..8 CTAs of the kernel above that fit the device at once, asked once per device (nullptr: it would not say).
const int* skinny_clusters(int dev, int sms) {
  static std::mutex mu;
  static int table[64][9] = {};
  std::lock_guard<std::mutex> guard(mu);
  int* t = table[dev & 63];
  if (t[0] == 0) {
    if (cudaFuncSetAttribute(gemm_skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SKINNY_SMEM) != cudaSuccess) return nullptr;
    for (int s = 1; s <= 8; ++s) {
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)s; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3((unsigned)(s * sms)); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = SKINNY_SMEM;
      cfg.attrs = at; cfg.numAttrs = 1;
      int n = 0;
      if (s > 1 && cudaOccupancyMaxActiveClusters(&n, gemm_skinny_kernel, &cfg) != cudaSuccess) n = 0;
      t[s] = s == 1 ? sms : n;
    }
    (void)cudaGetLastError();
    t[0] = 1;
  }
  return t;
}

// Second phase of the row-parallel form, after every rank's first phase (a cross-rank barrier lies between): the owner
// sums its rows over the n_ranks slots of its staging buffer in fp32, in slot order (the same bits on every run),
// rounds once to bf16 and stores the row into every rank's result matrix.  One 16-byte piece per thread and step.
__global__ void __launch_bounds__(256) reduce_push_kernel(const __nv_bfloat16* __restrict__ stage, const uint64_t* __restrict__ out_peers,
                                                          int n_ranks, int rank, int64_t rows_per_owner, int64_t M, int64_t N, int64_t ldc) {
  const int64_t row0 = (int64_t)rank * rows_per_owner;
  const int64_t rows = max((int64_t)0, min(rows_per_owner, M - row0));
  const int64_t vec_per_row = N / 8, total = rows * vec_per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / vec_per_row, c = (i - r * vec_per_row) * 8;
    float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    for (int s = 0; s < n_ranks; ++s) {
      const uint4 v = *reinterpret_cast<const uint4*>(stage + ((int64_t)s * rows_per_owner + r) * N + c);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = bf16x2_to_float2(w[e]);
        acc[e].x += f.x; acc[e].y += f.y;
      }
    }
    uint4 pk;
    pk.x = pack_bf16x2(acc[0].x, acc[0].y); pk.y = pack_bf16x2(acc[1].x, acc[1].y);
    pk.z = pack_bf16x2(acc[2].x, acc[2].y); pk.w = pack_bf16x2(acc[3].x, acc[3].y);
    for (int d = 0; d < n_ranks; ++d)
      *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out_peers[d]) + (row0 + r) * ldc + c) = pk;
  }
}

}  // namespace

int launch_gemm_bf16_nt_impl(const AveGemmArgs& a, cudaStream_t stream, const GemmScatter& sc);
int launch_gemm_bf16_nt(const AveGemmArgs& a, cudaStream_t stream) { return launch_gemm_bf16_nt_impl(a, stream, GemmScatter{nullptr, 1, 0, 0}); }

int launch_gemm_bf16_nt_scatter(const AveGemmReduceArgs& r, cudaStream_t stream) {
  AveGemmArgs a{};
  a.struct_size = sizeof(AveGemmArgs);
  a.a = r.a; a.b = r.b; a.c = r.stage;  // the tensor-map-free C pointer is replaced per row by the owner's slot
  a.M = r.M; a.N = r.N; a.K = r.K; a.lda = r.lda; a.ldb = r.ldb; a.ldc = r.N;
  a.status = r.status;
  return launch_gemm_bf16_nt_impl(a, stream, GemmScatter{reinterpret_cast<const uint64_t*>(r.stage_peers), r.n_ranks, r.rank, r.rows_per_owner});
}

int launch_gemm_reduce_push(const AveGemmReduceArgs& r, cudaStream_t stream) {
  int dev = 0, sms = 148;
  AVE_CUDA_TRY(cudaGetDevice(&dev));
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  reduce_push_kernel<<<sms * 8, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(r.stage), reinterpret_cast<const uint64_t*>(r.out_peers),
                                                 r.n_ranks, r.rank, r.rows_per_owner, r.M, r.N, r.ldc);
  AVE_CUDA_TRY(cudaGetLastError());
  return AVE_GDN_OK;
}

int launch_gemm_bf16_nt_impl(const AveGemmArgs& a, cudaStream_t stream, const GemmScatter& sc) {
  int dev = 0, sms = 148;
  AVE_CUDA_TRY(cudaGetDevice(&dev));
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  CUtensorMap tmA, tmB;
  const uint64_t dimsA[2] = {(uint64_t)a.K, (uint64_t)a.M}, strA[2] = {2, (uint64_t)a.lda * 2};
  const uint64_t dimsB[2] = {(uint64_t)a.K, (uint64_t)a.N}, strB[2] = {2, (uint64_t)a.ldb * 2};
  // Column tiles of equal width: as few tiles as BN = 256 allows, each as narrow as that count permits (a multiple of
  // 16, the granularity of the MMA's N).  N = 1544 becomes 7 tiles of 224 columns instead of 6 of 256 and one of 8,
  // whose MMAs and A-tile loads would be spent on 8 columns of output.
  const int64_t n_tiles_n = (a.N + BN - 1) / BN;
  int bn = (int)(((a.N + n_tiles_n - 1) / n_tiles_n + 15) / 16 * 16);
  // fewer tiles than SMs: the form that spreads a tile over narrower columns and a split of K
  SkinnyPlan sp{};
  if (sc.dst == nullptr && (a.M + BM - 1) / BM * n_tiles_n < sms) {
    const int* clusters = skinny_clusters(dev, sms);
    if (clusters != nullptr) sp = skinny_plan(a.M, a.N, a.K, clusters);
  }
  if (sp.bn != 0) bn = sp.bn;
  const uint32_t boxA[2] = {BK, sp.bn != 0 ? (uint32_t)sp.a_rows : (uint32_t)BM}, boxB[2] = {BK, (uint32_t)bn};
  int rc = make_tmap(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.a), 2, dimsA, strA, boxA, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != AVE_GDN_OK) return rc;
  rc = make_tmap(&tmB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.b), 2, dimsB, strB, boxB, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != AVE_GDN_OK) return rc;
  static bool attr_set_dev[64] = {};
  if (!attr_set_dev[dev & 63]) {
    AVE_CUDA_TRY(cudaFuncSetAttribute(gemm_bf16_nt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_SCATTER));
    attr_set_dev[dev & 63] = true;
  }
  if (sp.bn != 0) {
    uint32_t cols = 32;
    while ((int)cols < bn) cols *= 2;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)sp.split; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(((a.M + BM - 1) / BM) * ((a.N + bn - 1) / bn) * sp.split));
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = SKINNY_SMEM;
    cfg.stream = stream;
    cfg.attrs = at; cfg.numAttrs = 2;
    AVE_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_skinny_kernel, tmA, tmB, reinterpret_cast<__nv_bfloat16*>(a.c), a.M, a.N, a.K, a.ldc, a.status,
                                    sp, cols));
    return AVE_GDN_OK;
  }
  const int64_t tiles = ((a.M + BM - 1) / BM) * ((a.N + bn - 1) / bn);
  const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
  AVE_CUDA_TRY(launch_after(gemm_bf16_nt_kernel, grid, GEMM_THREADS, sc.dst != nullptr ? GEMM_SMEM_SCATTER : GEMM_SMEM, stream, tmA, tmB,
                            reinterpret_cast<__nv_bfloat16*>(a.c), a.M, a.N, a.K, a.ldc, a.status, bn, sc));
  AVE_CUDA_TRY(cudaGetLastError());
  return AVE_GDN_OK;
}

}  // namespace ave
