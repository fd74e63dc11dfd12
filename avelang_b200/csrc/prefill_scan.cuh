// Pass 2 of the chunked prefill: one CTA per chain walks its chunks with the state on chip, transposed (H = M^T, rows = d_v = TMEM
// lanes) so that every MMA has M = 128:
//     X^T  = kx H K^T                     (A = H hi/lo from TMEM, B = K tile, K-major)
//     Vn^T = V^T Tu^T - X^T Tu^T          (A = V tile MN-major / X hi/lo from TMEM, B = Tu hi/lo, packed triangles)
//     O^T  = qs H Q^T + Vn^T P^T          (A = H or Vn hi/lo from TMEM, B = Q or P hi/lo)
//     H   <- decay H + Vd^T K             (A = Vd hi/lo from TMEM, B = K, MN-major), Vd_j = ks_j Vn_j
// with kx_j = e^{b_j}, qs_i = scale e^{b_i}, ks_j = e^{b_C - b_j}, decay = e^{b_C}.  The fp32 state lives in the chain-epilogue threads'
// registers; its bf16 hi/lo image is rewritten to TMEM every chunk.  Pass 1 could also hand over W = Tu diag(kx) K, which
// makes Vn = U - H W one product: a hand-off less in a step, but W is twice as many bytes as everything else in a record and a third
// of pass 1.  K itself is exact in bf16, so H K^T takes 16 MMAs where H W^T takes 24.  (262144 packed tokens x 32 heads: 5.75 ms with W,
// 3.73 without, both after a rest, back to back the power cap makes it 4.1 to 4.3; 8192 tokens 370 us / 344; 4 heads x 32768 254 / 215; 1024 63.4 / 60.6.)
// A step takes 3.9 to 4.2 k cycles, of which the tensor pipe is busy 2.4 k: H K^T 0.85 k, X 0.55 k, its product 0.45 k, Vd 0.35 k, the increment
// 0.7 k, the new state 0.7 k, each of them about a third hand-over (arrival or commit, wake-up, first load).  What it took to get there from 4.55 k
// (8192 tokens x 32 heads 313 -> 260 us, 4 heads x 32768 212 -> 186, 262144 packed tokens 4.17 -> 3.75 ms, all with everything around the scan):
//   - the code that a step runs fits the 32 KB of the SM's instruction cache (rolled waits, outputs in a rolled loop, descriptors from constants and roles that the
//     compiler knows to be uniform took the kernel from 83 to 67 KB): every step fetched 116 lines of 128 bytes, 40 now, from the cache that the SMs of a GPC share, and
//     chains ran up to a third slower where more of a GPC's SMs held one;
//   - the two groups of epilogue warps hand over by halves: a group's tokens of X and Vd, and features of the state, have barriers of their own, so
//     that the products begin with one half while the other is converted, and an increment's first features are taken while the rest is formed;
//   - arrivals that the chain waits for are hardware barriers (30 cycles, an mbarrier 85 to 250);
//   - outputs leave by asynchronous copies: the transition chains' steps were a fifth longer when 32 lines were written an instruction.
// Later: O1 taken whole before the rows are formed (drained 1.0 to 1.25 k cycles into a step it held X's product back): 253.5 -> 249.3 us.
// The conversions are bound by the instructions of a scheduler (a pair of values into two bf16 terms takes 7 cycles of it).
// O2 waits for the increment: side by side they shared the pipe and the increment came 200 cycles later; H K^T in the increment's columns and not
// in O2's lets O2 end beside the next step.  Measured and dropped: the state a chunk behind the chain by
// S(c+1) = decay H(c) K(c+1)^T + Vd(c) (K(c+1) K(c)^T)^T, with three splits of 16 epilogue warps (3.08, 3.52 and 4.48 ms where this
// form then took 2.73: 11 to 15 k instructions a chunk, and the code of 20 warps misses the instruction cache); the gated norm in
// the output warps (layer of 8192 tokens 344 -> 374 us with eight of them, 422 with four).
#pragma once

namespace ave {
namespace {

// Warpgroup 0: warp 0 loader, warps 1 and 2 MMA issuers; warpgroups 1..NG: chain epilogue, each covering all 128 TMEM
// lanes and 1/NG of the columns; the last warpgroup: output.  (Four epilogue groups at 80 registers were measured: no
// faster, the epilogue is bound by the instructions issued per scheduler, not by the work per thread.)
constexpr int NG = 2;
constexpr int SCAN_THREADS = 32 * (4 + 4 * NG + 4);
constexpr int REGS_LAUNCH = 128;
constexpr int REGS_CTRL = 72, REGS_CHAIN = 168, REGS_OUT = 104;
static_assert(NG == 2, "the register split below is for two epilogue groups");
static_assert(REGS_CTRL + NG * REGS_CHAIN + REGS_OUT <= (NG + 2) * REGS_LAUNCH, "register redistribution exceeds the launch allocation");
static_assert(SCAN_THREADS * REGS_LAUNCH <= 65536, "launch allocation exceeds the register file");
constexpr int HC = D / NG;   // columns of H (d_k) per chain-epilogue group
constexpr int VC = C / NG;   // columns of Vn (tokens) per group
constexpr size_t SCAN_SMEM_MAX = 232448;
// A stage of the ring: the Q, K and V tiles of a chunk and its record
constexpr int CS_Q = 0, CS_K = 16384, CS_V = 32768, CS_REC = 49152, CS_STAGE = CS_REC + REC_BYTES, CS_STAGES = 3;
constexpr int CS_BARS = CS_STAGES * CS_STAGE;
constexpr size_t SCAN_SMEM = CS_BARS + 256 + 1024;
static_assert(CS_STAGE % 1024 == 0, "swizzled tiles need 1024-byte alignment");
static_assert(SCAN_SMEM <= SCAN_SMEM_MAX, "shared memory of an SM");
// TMEM columns: hi and lo image of H, accumulator of Vn (then the images of Vd), images of Vn, outputs, state increment.  H K^T
// and the images of X take columns of the increment, which they are never alive beside.
constexpr uint32_t TC_HHI = 0, TC_HLO = 64, TC_VN = 128, TC_VI = 192, TC_O1 = 256, TC_O2 = 320, TC_DH = 384, TC_X = TC_DH;
// The bf16 hi and lo images of an accumulator of 64 tokens reuse its columns, 16 tokens by 16 tokens (hi in the first eight columns, lo in the others), so
// a warp overwrites only columns it has itself read and needs no barrier between reading the accumulator and writing the images.
__host__ __device__ constexpr uint32_t img_col(uint32_t base, int k, bool lo) { return base + (uint32_t)(16 * k + (lo ? 8 : 0)); }  // 16-token step k

// The products.  `at` is the shared address / 16 of the stage, everything else a constant: with descriptors formed address by address in rolled loops a
// warp issued an MMA every 30 to 70 cycles, and the triangles' products, 8 to 32 cycles each, waited for it.
// D[:, 16 k ..] (+)= +-A[:, 16 k .. 16 k + 15] Tri[16 k .., 16 k .. 16 k + 15]^T over the 16-token steps k0 <= k < k1 of the packed lower triangle at `tri` in
// the stage, for (A hi, Tri hi), (A lo, Tri hi), (A hi, Tri lo); `first` overwrites D: step 0 covers all of its columns.  A: bf16 image in TMEM.
template <bool kNeg, int k0, int k1, int tri>
__device__ __forceinline__ void issue_tri(uint32_t d_tmem, uint32_t a_base, uint32_t at, bool first) {
#pragma unroll
  for (int t = 0; t < 3; ++t)
#pragma unroll
    for (int k = k0; k < k1; ++k)
      tc::mma_ts(d_tmem + 16 * k, img_col(a_base, k, t == 1),
                 tc::smem_desc(at + tc::desc_lo(tri + (t == 2 ? REC_TRI : 0) + tri_step(k), 128), tc::desc_hi(256, false)),
                 tc::idesc_f16(128, 64 - 16 * k, 1, 1, false, false, kNeg, false), (t | k) == 0 && first ? 0u : 1u);
}
// D (+)= H B^T over the 64 features of group g, H as hi and lo image, B the K-major [64][128] tile at `tile` in the stage; group 0 overwrites D
template <int tile, int g>
__device__ __forceinline__ void issue_state(uint32_t d_tmem, uint32_t tm, uint32_t at) {
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      tc::mma_ts(d_tmem, tm + (t ? TC_HLO : TC_HHI) + 32 * g + 8 * k, tc::smem_desc(at + tc::desc_lo(tile + 8192 * g + 32 * k, 16), tc::desc_hi(1024, true)),
                 tc::idesc_f16(128, 64, 1, 1, false, false), (g | t | k) != 0 ? 1u : 0u);
}

// kMulti: built with the parallel-parts machinery (ScanPlan::parts > 1).
template <bool kMulti>
__global__ void __launch_bounds__(SCAN_THREADS, 1)
chunk_scan_kernel(const AveGdnArgs a, const __grid_constant__ GdnMaps maps, const int32_t* chunk_start,
                     const uint8_t* recs, float* o_f32, uint8_t* qt_img,
                     float* carry, uint8_t* m0_pack, const int32_t* seq_order,
                     const __grid_constant__ ScanPlan plan) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = tc::align1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + CS_BARS);
  uint64_t* full = bars;          // [3] tiles and record of the stage landed
  uint64_t* empty = bars + 3;     // [3] everything that reads the stage is complete
  uint64_t* vn_full = bars + 6;   // [2] Vn = Tu (V - X) accumulated, for the tokens of each chain-epilogue group
  uint64_t* dh_full = bars + 8;   // [2] state increment accumulated, for the features of each group
  uint64_t* kh_full = bars + 10;  // H K^T accumulated
  uint64_t* vn_ready = bars + 11; // Vn hi+lo written to TMEM
  uint64_t* o_full = bars + 12;   // both output accumulators complete
  uint64_t* o1_empty = bars + 13; // O1 accumulator drained (the output warps take it first, whole, so O1 of the next chunk can run early)
  uint64_t* o2_empty = bars + 14; // O2 accumulator drained
  uint64_t* o1_done = bars + 15;  // O1 complete: the bf16 image of H may be overwritten
  // From a chain-epilogue group to the chain's issuer: bf16 image of its features of the state, X hi+lo and Vd hi+lo of its tokens are in TMEM.  The chain
  // waits for these, so they are hardware barriers, and their waits have no limit of their own.  A warp that arrives does not wait, so it may only come
  // back to a barrier when the issuer has gone through: its waits for what the issuer commits behind the barrier see to that as long as they end with the phase
  // complete (`alive`, one answer for a warp).  After a wait that has expired a warp meets the issuer in every hand-over instead of passing it, and an issuer
  // whose own wait has expired goes through the hand-overs that are left without a product or a commit: both sides take part 3 NG times a chunk.
  constexpr int HAND_OVERS = 3 * NG;  // of a chunk, in the issuer's order
  auto hand_over = [](int i) { return tc::NamedBar{1u + i, 32 * (4 + 1)}; };
  auto h_ready = [&](int g) { return hand_over(g); };
  auto x_ready = [&](int g) { return hand_over(NG + g); };
  auto vd_ready = [&](int g) { return hand_over(2 * NG + g); };
  auto all = [](bool done) { return __all_sync(0xffffffffu, done) != 0; };
  // A wait sees only the parity of a barrier's phase, so no barrier may complete twice before each of its waiters has seen the first
  // time.  Most are ordered by the arrivals they need.  dh_full is waited for by warp 2 as well, which no increment needs: so warp 1 issues an
  // increment only behind o_full of the chunk before, which warp 2 commits when it has seen dh_full of that chunk.
  uint64_t* tail_full = bars + 16;  // tiles and record of a ragged last chunk landed: warp 0 clears what lies behind the sequence, then completes `full`
  uint64_t* mma_end = bars + 17;    // [2] the MMAs of warps 1 and 2 complete, when a wait has expired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  // (a shuffle, so that the compiler knows a role's code to be uniform)
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // what reads nothing that a launch before wrote comes in front of the wait for it
  if (threadIdx.x == 0) {
    for (int i = 0; i < CS_STAGES; ++i) { tc::mbar_init(&full[i], 1); tc::mbar_init(&empty[i], 6); }
    for (int i = 0; i < NG; ++i) { tc::mbar_init(&vn_full[i], 1); tc::mbar_init(&dh_full[i], 1); tc::mbar_init(&mma_end[i], 1); }
    tc::mbar_init(vn_ready, 4 * NG);
    for (uint64_t* b : {kh_full, o_full, o1_done, tail_full}) tc::mbar_init(b, 1);
    tc::mbar_init(o1_empty, 4); tc::mbar_init(o2_empty, 4);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 2 && lane == 0) {
    tc::prefetch_tmap(&maps.q); tc::prefetch_tmap(&maps.k); tc::prefetch_tmap(&maps.v);
  }
  pdl_wait();
  // One CTA per (sequence, chain, value head).  Chain 0 is part 0; chains 2p-1 and 2p are the local and the transition
  // chain of part p >= 1 (see ScanPlan).
  const int chains = kMulti ? 2 * plan.parts - 1 : 1;
  const int h = blockIdx.x % a.Hv;
  const int unit = blockIdx.x / a.Hv;
  const int chain = kMulti ? unit % chains : 0;
  const int n = seq_order ? seq_order[unit / chains] : unit / chains;  // varlen: longest sequences first
  const int part = (chain + 1) >> 1;
  const bool phi = kMulti && chain > 0 && (chain & 1) == 0;
  const int hk = h / (a.Hv / a.Hk);
  if (batch_rejected(a, chunk_start)) return;
  SeqSpan sp = seq_span(a.cu_seqlens, n, a.T, a.status);
  // longer than the caller's bound: the launch schedule was sized from that bound, so the sequence is skipped (zero
  // output, no state access, like a negative slot) and flagged
  const bool too_long = a.cu_seqlens != nullptr && a.max_seqlen > 0 && sp.len > a.max_seqlen;
  if (too_long && a.status != nullptr && threadIdx.x == 0) atomicOr(a.status, AVE_GDN_DEV_BAD_SEQLEN);
  if (!sp.ok || sp.len == 0) {
    if (plan.r0 > 0 || chain > 0) return;
    // zero-length sequence: the final state is the initial state
    if (sp.ok && a.final_state != nullptr && a.final_state != a.initial_state) {
      const int slot0 = a.state_indices ? a.state_indices[n] : n;
      if (slot0 >= 0 && slot0 < a.num_slots) {
        const int64_t tile0 = ((int64_t)slot0 * a.Hv + h) * (int64_t)(D * D);
        for (int e = threadIdx.x; e < D * D; e += SCAN_THREADS)
          a.final_state[tile0 + e] = a.initial_state ? a.initial_state[tile0 + e] : 0.f;
      }
    }
    return;
  }
  const int seq_chunks = (sp.len + C - 1) / C;
  // a sequence that ends inside part 0 is one plain chain: outputs and the final state leave directly
  const bool multi = kMulti && plan.parts > 1 && seq_chunks > plan.part_begin[1] && !too_long;
  if (chain > 0 && (!multi || plan.part_begin[part] >= seq_chunks)) return;
  int slot = n;
  if (a.state_indices != nullptr) {
    slot = a.state_indices[n];
    if (slot >= a.num_slots) {
      if (a.status != nullptr && threadIdx.x == 0) atomicOr(a.status, AVE_GDN_DEV_BAD_SLOT);
      slot = -1;
    }
  }
  if (too_long) slot = -1;
  __nv_bfloat16* og = reinterpret_cast<__nv_bfloat16*>(a.o) + sp.b * a.o_stride_b + (int64_t)h * a.o_stride_h;
  // where this chain's per-token rows go: the local rows of later parts wait in fp32 scratch for the fix-up, and so do those of a
  // gated call for the norm; the transition chain's rows leave as the bf16 hi/lo operand images the fix-up's MMAs read;
  // all others are the result
  float* const out_f32 = (!phi && (a.z != nullptr || part > 0)) ? o_f32 : nullptr;
  if (slot < 0) {  // skipped sequence: zero output, no state access (chain 0 clears the whole sequence once)
    if (chain > 0 || plan.r0 > 0) return;
    float* zf = a.z != nullptr ? o_f32 : nullptr;
    for (int e = threadIdx.x; e < sp.len * D; e += SCAN_THREADS) {
      const int64_t tok = sp.t0 + e / D;
      if (zf != nullptr) zf[(((int64_t)sp.b * a.T + tok) * a.Hv + h) * D + e % D] = 0.f;
      else og[tok * a.o_stride_t + e % D] = __float2bfloat16(0.f);
    }
    return;
  }
  // This launch covers chunks [c_lo, c_hi) of the chain's part; the state enters from / leaves to the carry buffer
  // unless this is the first / last launch of a plain chain.
  const int part_end = min(plan.part_begin[part + 1], seq_chunks);
  const int c_lo = plan.part_begin[part] + plan.r0;
  const int c_hi = min(c_lo + plan.rn, part_end);
  if (c_lo >= c_hi) return;  // finished in an earlier launch, or not reached yet
  const bool seg_first = plan.r0 == 0;
  const bool seg_last = c_hi == part_end && !multi;
  const int c_first = first_record(a, chunk_start, n) + c_lo;
  sp.t0 += c_lo * C;
  sp.len = min(sp.len - c_lo * C, (c_hi - c_lo) * C);
  const int n_chunks = c_hi - c_lo;
  const int64_t carry_tile = (((int64_t)n * chains + chain) * a.Hv + h) * (int64_t)(D * D);

  if (warp == 1) tc::tmem_alloc(tmem_slot, 512);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  constexpr uint32_t tm = 0;  // all 512 columns are this CTA's, so the first is column 0
  const bool ragged = a.cu_seqlens != nullptr && sp.len < n_chunks * C;

  if (warp < 4) {
  tc::reg_set<REGS_CTRL, REGS_LAUNCH>();
  if (warp == 0) {
    // ------------------------------------------------------------------ loader: a stage is {Q, K, V, record}, three of them
    int issued = 0;  // chunks asked for
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 1;  // parity of "chunk c - 3 is done with the stage"; the first round waits for nothing
      auto load = [&](int c, uint64_t* when_full) {
        if (c == n_chunks - 1) pdl_trigger();
        if (c >= CS_STAGES && !tc::mbar_wait(&empty[s], ph, abort_flag)) return false;
        uint8_t* st = smem + s * CS_STAGE;
        const int tok = sp.t0 + c * C;
        tc::mbar_expect_tx(when_full, phi ? CS_STAGE - 16384u : (uint32_t)CS_STAGE);  // the transition chain has no V
        tc::tma_load_4d(st + CS_K, &maps.k, when_full, 0, hk, tok, sp.b);
        tc::tma_load_4d(st + CS_K + 8192, &maps.k, when_full, 64, hk, tok, sp.b);
        tc::bulk_load(st + CS_REC, recs + ((int64_t)(c_first + c) * a.Hv + h) * REC_BYTES, REC_BYTES, when_full);
        if (!phi) {
          tc::tma_load_4d(st + CS_V, &maps.v, when_full, 0, h, tok, sp.b);
          tc::tma_load_4d(st + CS_V + 8192, &maps.v, when_full, 64, h, tok, sp.b);
        }
        tc::tma_load_4d(st + CS_Q, &maps.q, when_full, 0, hk, tok, sp.b);
        tc::tma_load_4d(st + CS_Q + 8192, &maps.q, when_full, 64, hk, tok, sp.b);
        ++issued;
        if (++s == CS_STAGES) { s = 0; ph ^= 1u; }
        return true;
      };
      const int whole = ragged ? n_chunks - 1 : n_chunks;
      bool ok = true;
      for (int c = 0; c < whole && ok; ++c) ok = load(c, &full[s]);
      if (ragged && ok) load(whole, tail_full);
    }
    // The tiles of a packed sequence's last chunk go on with the rows of whatever lies behind it.  Their factors are zero, but a product is
    // not where such a row holds a NaN or an infinity, so K and V are cleared there, by the whole warp, which has nothing else to do, up to two chunks
    // before they are read.  (Q only reaches columns that are not stored; behind the end of a dense batch row the copy itself fills with zeros.)
    // 203 tokens: 29.4 us, 29.2 without; by warp 1 in front of U 29.9, and with the contractions over tokens cut at the last token instead, a
    // branch around each MMA, 30.1 (8192 tokens 318, 316, 318 and 326; by warp 3 320).
    __syncwarp();
    if (ragged && all(tc::mbar_wait_warp(tail_full, 0u, abort_flag))) {
      const int last = (n_chunks - 1) % CS_STAGES;
      uint4* st = reinterpret_cast<uint4*>(smem + last * CS_STAGE + CS_K);
      // 16-byte pieces of the halves (64 features) of K and of V; whole rows, so the swizzle does not matter.  (Not unrolled: the code
      // runs once and is fetched while it runs.)
#pragma unroll 1
      for (int i = 8 * (sp.len - (n_chunks - 1) * C) + lane; i < 8 * C; i += 32)
        st[i] = st[i + 512] = st[i + 1024] = st[i + 1536] = make_uint4(0u, 0u, 0u, 0u);
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&full[last]);
    }
    if (lane == 0) {  // nothing is on its way into the shared memory of a CTA that ends, whatever became of those who wait for it
#pragma unroll 1
      for (int c = max(0, issued - CS_STAGES); c < issued; ++c) {
        const bool tail = ragged && c == n_chunks - 1;
        tc::drain(tail ? tail_full : &full[c % CS_STAGES], tail ? 0u : (uint32_t)(c / CS_STAGES) & 1u);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ chain MMA issuer (whole warp runs the loop, one
    // elected lane issues): the MMAs the recurrence waits for.  One thread needs 20 to 60 cycles per MMA instruction, so
    // the instructions of a chunk are shared between two warps; this one keeps the state-dependent ones short:
    //   U^T(c+1) -> [state published] H K^T(c) -> [X written] Vn^T(c) -> [Vd written] dH(c)
    constexpr uint32_t id_dh = tc::idesc_f16(128, 128, 1, 1, false, true), id_dh_half = tc::idesc_f16(128, 64, 1, 1, false, true);  // B MN-major
    // U^T = V^T (Tu_hi + Tu_lo)^T opens the Vn^T accumulator of a chunk.  It does not depend on the state, so it is
    // issued a chunk ahead, right behind the previous chunk's state-increment MMAs (which read the Vd images in the
    // same columns and, issued earlier by this thread, complete first): the tensor pipe runs it while the chain
    // epilogue re-packs H.
    auto issue_u = [&](uint32_t at) {
      if (phi) return;  // v = 0: U^T = 0, the first Vn MMA overwrites the accumulator instead
      if (tc::elect_one()) {
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int k = 0; k < 4; ++k)  // 16 tokens per step: V rows 2048 bytes apart, feature halves 8192 bytes apart
            tc::mma_ss(tm + TC_VN + 16 * k, tc::smem_desc(at + tc::desc_lo(CS_V + k * 2048, 8192), tc::desc_hi(1024, true)),
                       tc::smem_desc(at + tc::desc_lo(CS_REC + REC_TU + t * REC_TRI + tri_step(k), 128), tc::desc_hi(256, false)),
                       tc::idesc_f16(128, 64 - 16 * k, 1, 1, true, false), (t | k) != 0 ? 1u : 0u);
      }
      __syncwarp();
    };
    int s = 0, s_next = 1;
    uint32_t ph_next = 0;
    const uint32_t smem0 = tc::smem_u32(smem) >> 4;
    int met = HAND_OVERS * n_chunks;  // hand-overs behind which this role leaves its loop
    const bool landed = all(tc::mbar_wait_warp(&full[0], 0u, abort_flag));
    if (!landed) met = 0;
    tc::tc_fence_after_sync();
    if (landed) issue_u(smem0);
    // what the chain waits for, step by step
    auto state_product = [&](int c, uint32_t at, int s) {
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        tc::mbar_wait_warp(h_ready(g), (uint32_t)c & 1u, abort_flag);
        tc::tc_fence_after_sync();
        if (tc::elect_one()) {
          if (g == 0) issue_state<CS_K, 0>(tm + TC_X, tm, at);
          else issue_state<CS_K, 1>(tm + TC_X, tm, at);
          if (g == NG - 1) {
            tc::mma_commit(kh_full);
            // the MMAs of the chunk before are complete with these, and the epilogue, which has published a state, is through with its scale vectors
            if (c > 0) tc::mma_commit(&empty[s == 0 ? CS_STAGES - 1 : s - 1]);
          }
        }
        __syncwarp();
      }
    };
    auto new_values = [&](int c, uint32_t at) {  // Vn^T -= X Tu^T; the tokens of a group need those before them only
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        tc::mbar_wait_warp(x_ready(g), (uint32_t)c & 1u, abort_flag);
        tc::tc_fence_after_sync();
        if (tc::elect_one()) {
          if (g == 0) issue_tri<true, 0, 2, CS_REC + REC_TU>(tm + TC_VN, tm + TC_X, at, phi);
          else issue_tri<true, 2, 4, CS_REC + REC_TU>(tm + TC_VN, tm + TC_X, at, phi);
          tc::mma_commit(&vn_full[g]);
        }
        __syncwarp();
      }
    };
    auto outputs_before = [&](int c) {  // warp 2 has seen dh_full of the chunk before (and O2 is long complete)
      return all(tc::mbar_wait_warp(o_full, (uint32_t)(c + 1) & 1u, abort_flag));
    };
    auto increment = [&](int c, uint32_t at) {
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        tc::mbar_wait_warp(vd_ready(g), (uint32_t)c & 1u, abort_flag);
        tc::tc_fence_after_sync();
        if (tc::elect_one()) {
          // dH = (Vd_hi + Vd_lo) contracted with K over the group's tokens (K tile read MN-major: 16 token rows per step); the last
          // tokens for half of the features at a time, so that one group takes its half while the other's is formed
#pragma unroll
          for (int f = 0; f <= g; ++f) {
#pragma unroll
            for (int i = 0; i < 4; ++i)  // hi, lo x two steps
              tc::mma_ts(tm + TC_DH + 64 * f, img_col(tm + TC_VN, 2 * g + (i & 1), i >> 1),
                         tc::smem_desc(at + tc::desc_lo(CS_K + 8192 * f + 2048 * (2 * g + (i & 1)), 8192), tc::desc_hi(1024, true)),
                         g == 0 ? id_dh : id_dh_half, (g | i) != 0 ? 1u : 0u);
            if (g == NG - 1) tc::mma_commit(&dh_full[f]);
          }
        }
        __syncwarp();
      }
    };
    auto values_of = [&](int stage, uint32_t parity) {
      if (!all(tc::mbar_wait_warp(&full[stage], parity, abort_flag))) return false;
      tc::tc_fence_after_sync();
      issue_u(smem0 + stage * (CS_STAGE >> 4));
      return true;
    };
    for (int c = 0; c < n_chunks && landed; ++c) {
      const uint32_t at = smem0 + s * (CS_STAGE >> 4);  // the stage has landed: this warp waited for it a chunk ago
      state_product(c, at, s);
      // (for the increment, but here the wait is hidden behind the conversion of X; a wait for what is complete takes 130 to 250 cycles)
      if (!outputs_before(c)) { met = HAND_OVERS * c + NG; break; }
      new_values(c, at);
      increment(c, at);
      if (c + 1 < n_chunks) {
        if (!values_of(s_next, ph_next)) { met = HAND_OVERS * (c + 1); break; }
        s = s_next;
        if (++s_next == CS_STAGES) { s_next = 0; ph_next ^= 1u; }
      }
    }
#pragma unroll 1
    for (; met < HAND_OVERS * n_chunks; ++met) tc::named_sync(hand_over(met % HAND_OVERS));
  } else if (warp == 2) {
    // ------------------------------------------------------------------ output MMA issuer: O1 = H Q^T once H K^T is
    // complete (so that it runs behind it, while the chain epilogue converts X), O2 = Vn P^T once Vn hi/lo are back
    const uint32_t smem0 = tc::smem_u32(smem) >> 4;
    int s = 0;
    uint32_t ph = 0;
    for (int c = 0; c < n_chunks; ++c) {
      const uint32_t cp = (uint32_t)c & 1u;
      const uint32_t at = smem0 + s * (CS_STAGE >> 4);
      if (!all(tc::mbar_wait3(kh_full, cp, o1_empty, cp ^ 1u, &full[s], ph, abort_flag))) break;
      tc::tc_fence_after_sync();
      if (tc::elect_one()) {
        issue_state<CS_Q, 0>(tm + TC_O1, tm, at);
        issue_state<CS_Q, 1>(tm + TC_O1, tm, at);  // the chain epilogue waits for its completion before it overwrites the bf16 image of H
        tc::mma_commit(o1_done);
      }
      __syncwarp();
      // behind the state increment, which the recurrence waits for: side by side they would share the tensor pipe
      if (!all(tc::mbar_wait3(vn_ready, cp, o2_empty, cp ^ 1u, &dh_full[1], cp, abort_flag))) break;
      tc::tc_fence_after_sync();
      if (tc::elect_one()) {
        issue_tri<false, 0, 4, CS_REC + REC_PT>(tm + TC_O2, tm + TC_VI, at, true);  // O2 = Vn P^T
        tc::mma_commit(o_full);
        tc::mma_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == CS_STAGES) { s = 0; ph ^= 1u; }
    }
  }
  } else if (warp < 4 + 4 * NG) {
    tc::reg_set<REGS_CHAIN, REGS_LAUNCH>();
    // ------------------------------------------------------------------ chain epilogue: Vn/Vd conversion and state update
    const int grp = (warp - 4) >> 2;    // column group
    const int quarter = warp & 3;       // TMEM lane quarter this warp may touch
    const int d = quarter * 32 + lane;  // row of H (d_v index)
    const uint32_t lane_addr = tm + ((uint32_t)(quarter * 32) << 16);
    const int64_t tile = ((int64_t)slot * a.Hv + h) * (int64_t)(D * D);
    bool alive = true;  // every wait so far has ended with its phase complete

    float2 Hreg[HC / 2];  // H[d][HC*grp + 2w .. +1] = M[HC*grp + 2w .. +1][d]
    // first launch of a chain: part 0 starts from the caller's state, a later part's local chain from zero and its
    // transition chain from the identity
    const float* state_in = !seg_first ? carry + carry_tile : (part == 0 && a.initial_state ? a.initial_state + tile : nullptr);
    float* state_out = seg_last ? (a.final_state ? a.final_state + tile : nullptr) : carry + carry_tile;
    if (phi && seg_first) {
#pragma unroll
      for (int w = 0; w < HC / 2; ++w)
        Hreg[w] = make_float2(HC * grp + 2 * w == d ? 1.f : 0.f, HC * grp + 2 * w + 1 == d ? 1.f : 0.f);
    } else if (state_in != nullptr) {
#pragma unroll
      for (int w = 0; w < HC / 2; ++w)
        Hreg[w] = make_float2(state_in[(int64_t)(HC * grp + 2 * w) * D + d], state_in[(int64_t)(HC * grp + 2 * w + 1) * D + d]);
    } else {
#pragma unroll
      for (int w = 0; w < HC / 2; ++w) Hreg[w] = make_float2(0.f, 0.f);
    }
    auto publish_h = [&]() {
#pragma unroll
      for (int part16 = 0; part16 < HC / 32; ++part16) {  // 16 packed words (32 columns of H) at a time
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int w = 0; w < 16; ++w) split_pair(Hreg[16 * part16 + w], hi[w], lo[w]);
        tc::tmem_st16(lane_addr + TC_HHI + (HC / 2) * grp + 16 * part16, hi);
        tc::tmem_st16(lane_addr + TC_HLO + (HC / 2) * grp + 16 * part16, lo);
      }
      tc::tmem_st_wait();
      tc::tc_fence_before_sync();
      __syncwarp();
      tc::mbar_arrive(h_ready(grp), alive);
    };
    publish_h();

    int s = 0;
    uint32_t ph = 0;
    for (int c = 0; c < n_chunks; ++c) {  // (to the end also when a wait has expired: the chain's issuer counts on the hand-overs)
      const uint32_t cp = (uint32_t)c & 1u;
      const float* scal = reinterpret_cast<const float*>(smem + s * CS_STAGE + CS_REC + REC_SCAL);
      alive = all(tc::mbar_wait2(&full[s], ph, kh_full, cp, abort_flag)) && alive;  // (the scale vectors come with the stage)
      if (++s == CS_STAGES) { s = 0; ph ^= 1u; }
      tc::tc_fence_after_sync();
      {  // X_j = kx_j H k_j
#pragma unroll
        for (int k = 0; k < VC / 16; ++k) {
          uint32_t acc[16], xh[8], xl[8];
          tc::tmem_ld16(lane_addr + TC_X + VC * grp + 16 * k, acc);
          tc::tmem_ld_wait();
#pragma unroll
          for (int w = 0; w < 8; w += 2) {
            const float4 kx = *reinterpret_cast<const float4*>(scal + 2 * C + VC * grp + 16 * k + 2 * w);
            split_pair(__fmul2_rn(make_float2(__uint_as_float(acc[2 * w]), __uint_as_float(acc[2 * w + 1])), make_float2(kx.x, kx.y)), xh[w], xl[w]);
            split_pair(__fmul2_rn(make_float2(__uint_as_float(acc[2 * w + 2]), __uint_as_float(acc[2 * w + 3])), make_float2(kx.z, kx.w)), xh[w + 1], xl[w + 1]);
          }
          tc::tmem_st8(lane_addr + TC_X + VC * grp + 16 * k, xh);  // into this warp's own accumulator columns
          tc::tmem_st8(lane_addr + TC_X + VC * grp + 16 * k + 8, xl);
        }
        tc::tmem_st_wait();
        tc::tc_fence_before_sync();
        __syncwarp();
        tc::mbar_arrive(x_ready(grp), alive);
      }
      alive = all(tc::mbar_wait_warp(&vn_full[grp], cp, abort_flag)) && alive;
      tc::tc_fence_after_sync();
      {
        uint32_t acc[VC];
        tc::tmem_ld_n<VC>(lane_addr + TC_VN + VC * grp, acc);
        float2 v[VC / 2];
        tc::tmem_ld_wait();
#pragma unroll
        for (int w = 0; w < VC / 2; ++w) v[w] = make_float2(__uint_as_float(acc[2 * w]), __uint_as_float(acc[2 * w + 1]));
        {  // Vd first: its columns alias nothing, and the state update waits only for it
          uint32_t dh[VC / 2], dl[VC / 2];
#pragma unroll
          for (int w = 0; w < VC / 2; w += 2) {
            const float4 ks = *reinterpret_cast<const float4*>(scal + C + VC * grp + 2 * w);
            split_pair(__fmul2_rn(v[w], make_float2(ks.x, ks.y)), dh[w], dl[w]);
            split_pair(__fmul2_rn(v[w + 1], make_float2(ks.z, ks.w)), dh[w + 1], dl[w + 1]);
          }
#pragma unroll
          for (int k = 0; k < VC / 16; ++k) {  // into this warp's own accumulator columns
            tc::tmem_st8(lane_addr + TC_VN + VC * grp + 16 * k, reinterpret_cast<const uint32_t(&)[8]>(dh[8 * k]));
            tc::tmem_st8(lane_addr + TC_VN + VC * grp + 16 * k + 8, reinterpret_cast<const uint32_t(&)[8]>(dl[8 * k]));
          }
          tc::tmem_st_wait();
          tc::tc_fence_before_sync();
          __syncwarp();
          tc::mbar_arrive(vd_ready(grp), alive);
        }
        // the Vn images of the chunk before have been read (long ago: its O2 ran beside its state's conversion)
        alive = all(tc::mbar_wait_warp(o_full, cp ^ 1u, abort_flag)) && alive;
        {
          uint32_t vh[VC / 2], vl[VC / 2];
#pragma unroll
          for (int w = 0; w < VC / 2; ++w) split_pair(v[w], vh[w], vl[w]);
#pragma unroll
          for (int k = 0; k < VC / 16; ++k) {  // beside them
            tc::tmem_st8(lane_addr + TC_VI + VC * grp + 16 * k, reinterpret_cast<const uint32_t(&)[8]>(vh[8 * k]));
            tc::tmem_st8(lane_addr + TC_VI + VC * grp + 16 * k + 8, reinterpret_cast<const uint32_t(&)[8]>(vl[8 * k]));
          }
          tc::tmem_st_wait();
          tc::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0 && alive) tc::mbar_arrive(vn_ready);
        }
      }
      alive = all(tc::mbar_wait2(&dh_full[grp], cp, o1_done, cp, abort_flag)) && alive;
      tc::tc_fence_after_sync();
      {
        const float decay = scal[3 * C];
#pragma unroll
        for (int part32 = 0; part32 < HC / 32; ++part32) {
          uint32_t dh[32];
          tc::tmem_ld32(lane_addr + TC_DH + HC * grp + 32 * part32, dh);
          tc::tmem_ld_wait();
#pragma unroll
          for (int w = 0; w < 16; ++w)
            Hreg[16 * part32 + w] = __ffma2_rn(make_float2(decay, decay), Hreg[16 * part32 + w],
                                               make_float2(__uint_as_float(dh[2 * w]), __uint_as_float(dh[2 * w + 1])));
        }
        if (c + 1 < n_chunks) publish_h();  // (as often as the issuer waits)
      }
    }
    if (alive && state_out != nullptr) {
#pragma unroll
      for (int w = 0; w < HC / 2; ++w) {
        state_out[(int64_t)(HC * grp + 2 * w) * D + d] = Hreg[w].x;
        state_out[(int64_t)(HC * grp + 2 * w + 1) * D + d] = Hreg[w].y;
      }
    }
    if (alive && multi && chain == 0 && c_hi == part_end) {
      // the state that enters part 1, as the fix-up's B operand image (row = d_v, K = d_k): this thread's row, HC / 8 pieces
      uint8_t* img = m0_pack + (((int64_t)n * (plan.parts - 1)) * a.Hv + h) * (int64_t)PACK_BYTES;
#pragma unroll
      for (int j = 0; j < HC / 8; ++j) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) split_pair(Hreg[4 * j + w], hi[w], lo[w]);
        const uint32_t off = kmajor_piece_off(d, (HC / 8) * grp + j);
        *reinterpret_cast<uint4*>(img + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(img + D * D * 2 + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
    }
  } else {
    tc::reg_set<REGS_OUT, REGS_LAUNCH>();
    // ------------------------------------------------------------------ output warps: o = qs_i O1 + O2, 32 features a warp, as accumulator
    // fragments of warp-level MMAs, which matrix stores transpose on their way into shared memory.  The tiles are formed there, in the place of the chunk's Q
    // and K (all MMAs that read them are complete with O2), 8 KB a warp, and leave by one asynchronous copy each: these warps run beside the
    // conversions that the chain waits for.  (With a row of d_v a thread, scalar stores, and 16-byte loads and stores on the way out, a chunk took them 2.0 to
    // 2.8 k cycles and the transition chains' steps were a fifth longer than the others': their rows went to 32 lines an instruction.)
    const int wq = warp & 3, gr = lane >> 2, t2 = 2 * (lane & 3), r8 = lane & 7, m4 = lane >> 3;
    const uint32_t lane_addr = tm + ((uint32_t)(wq * 32) << 16);
    int s = 0;
    for (int c = 0; c < n_chunks; ++c) {
      const uint32_t cp = (uint32_t)c & 1u;
      const float* scal = reinterpret_cast<const float*>(smem + s * CS_STAGE + CS_REC + REC_SCAL);
      uint8_t* stage = smem + s * CS_STAGE + wq * 8192;
      const uint32_t stage_s = tc::smem_u32(stage);
      const int len = min(C, sp.len - c * C);
      const int64_t tok0 = sp.t0 + c * C;
      // o_full is committed by the MMA warp after it saw this chunk's stage (tiles and scale vectors) land, so it also
      // orders the scale vectors; waiting on the stage barrier here would alias phases once this warp lags a chunk
      if (!all(tc::mbar_wait_warp(o_full, cp, abort_flag))) break;
      tc::tc_fence_after_sync();
      const bool whole = !(ragged && c == n_chunks - 1);  // (behind the end of a dense batch row the copies write nothing)
      // O1 is taken whole and released at once: O1 of the next chunk is the first thing the tensor pipe runs while the chain epilogue converts X, and X's
      // product must not wait for it.  o[4 g + 2 rr + e]: feature 32 wq + 16 hf + 8 rr + gr, token 8 g + t2 + e.
      uint32_t o[32], o_next[32];
      tc::tmem_ld_frags(lane_addr + TC_O1, o);
      tc::tmem_ld_frags(lane_addr + (16u << 16) + TC_O1, o_next);
      tc::tmem_ld_wait();
      tc::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(o1_empty);
      // 16 features at a time, in a loop that stays rolled: the code of all roles together has to stay small
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {
        auto pair = [&](int g, int rr) { return make_float2(__uint_as_float(o[4 * g + 2 * rr]), __uint_as_float(o[4 * g + 2 * rr + 1])); };
#pragma unroll
        for (int g0 = 0; g0 < C / 8; g0 += 4) {
          uint32_t o2[16];
          tc::tmem_ld_frags(lane_addr + ((uint32_t)hf << 20) + TC_O2 + 8 * g0, o2);
          tc::tmem_ld_wait();
          if (g0 == 4 && hf == 1) {
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(o2_empty);
          }
#pragma unroll
          for (int g = g0; g < g0 + 4; ++g) {
            const float2 qs = *reinterpret_cast<const float2*>(scal + 8 * g + t2);
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
              uint32_t* x = &o[4 * g + 2 * rr];
              const uint32_t* x2 = &o2[4 * (g - g0) + 2 * rr];
              const float2 y = __ffma2_rn(qs, pair(g, rr), make_float2(__uint_as_float(x2[0]), __uint_as_float(x2[1])));
              x[0] = __float_as_uint(y.x); x[1] = __float_as_uint(y.y);
            }
          }
        }
        if (kMulti && phi) {
          // qt^T of this chunk as bf16 hi and lo images [128 d_k rows][64 tokens] with the 128-byte swizzle: the fix-up
          // reads them, unchanged, as the MN-major A operand of its MMA.  32 rows a warp, 4 KB of each image.
          const uint32_t at = stage_s + (uint32_t)((16 * hf + 8 * (m4 & 1) + r8) * 128);
#pragma unroll
          for (int g = 0; g < C / 8; g += 2) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) split_pair(pair(g + (m >> 1), m & 1), hi[m], lo[m]);
            const uint32_t off = (uint32_t)(((g + (m4 >> 1)) ^ r8) << 4);
            stsm4(at + off, hi[0], hi[1], hi[2], hi[3]);
            stsm4(at + off + 4096, lo[0], lo[1], lo[2], lo[3]);
          }
        } else if (out_f32 != nullptr) {  // [64 tokens][32 features] of 4 bytes, 128-byte swizzle
          const int c0 = (4 * hf) ^ (gr >> 2) ^ t2;
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
              float* at = reinterpret_cast<float*>(stage + (t2 + e) * 128 + (((2 * rr) ^ c0 ^ e) << 4)) + (gr & 3);
#pragma unroll
              for (int g = 0; g < C / 8; ++g) at[256 * g] = __uint_as_float(o[4 * g + 2 * rr + e]);
            }
        } else {  // [64 tokens][32 features] of 2 bytes, 64-byte swizzle
          const uint32_t at = stage_s + (uint32_t)((8 * (m4 >> 1) + r8) * 64 + (((2 * hf + (m4 & 1)) ^ (r8 >> 1)) << 4));
#pragma unroll
          for (int g = 0; g < C / 8; g += 2) {
            uint32_t x[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) { const float2 y = pair(g + (m >> 1), m & 1); x[m] = pack_bf16x2(y.x, y.y); }
            stsm4t(at + 512 * g, x[0], x[1], x[2], x[3]);
          }
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = o_next[i];
      }
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (kMulti && phi) {
        if (lane == 0) {
          uint8_t* img = qt_img + ((int64_t)(c_first + c) * a.Hv + h) * (int64_t)QT_BYTES + wq * 4096;
          tc::bulk_store(img, stage, 4096);
          tc::bulk_store(img + C * D * 2, stage + 4096, 4096);
        }
      } else if (whole && (out_f32 != nullptr || maps.o_ok)) {
        if (lane == 0) tc::tma_store_4d(out_f32 != nullptr ? &maps.o32 : &maps.o, stage, 32 * wq, h, (int)tok0, sp.b);
      } else if (out_f32 != nullptr) {
        float* dst = out_f32 + (((int64_t)sp.b * a.T + tok0) * a.Hv + h) * D + 32 * wq + 4 * r8;
#pragma unroll 1
        for (int t = m4; t < len; t += 4) *reinterpret_cast<float4*>(dst + (int64_t)t * a.Hv * D) = *reinterpret_cast<const float4*>(stage + t * 128 + ((r8 ^ (t & 7)) << 4));
      } else {
        __nv_bfloat16* dst = og + tok0 * a.o_stride_t + 32 * wq + 8 * (lane & 3);
#pragma unroll 1
        for (int t = lane >> 2; t < len; t += 8) *reinterpret_cast<uint4*>(dst + t * a.o_stride_t) = *reinterpret_cast<const uint4*>(stage + t * 64 + (((lane & 3) ^ ((t >> 1) & 3)) << 4));
        tc::fence_proxy_async_smem();
      }
      if (lane == 0) {  // the next tiles of this stage come when it has been read
        tc::bulk_commit();
        tc::bulk_wait_read<0>();
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&empty[s]);
      if (++s == CS_STAGES) s = 0;
    }
    if (lane == 0) tc::bulk_wait_all();
  }

  tc::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {  // (the roles have ended: it stays as it is)
    if (threadIdx.x == 0 && a.status != nullptr) atomicOr(a.status, AVE_GDN_DEV_WAIT_EXPIRED);
    if (warp == 1 || warp == 2) tc::drain_mmas(&mma_end[warp - 1]);
    tc::tc_fence_before_sync();
    __syncthreads();
  }
  if (warp == 1) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tm, 512);
  }
}


}  // namespace
}  // namespace ave
