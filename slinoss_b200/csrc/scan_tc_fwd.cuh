// Forward kernel of the chunked scan on tcgen05 (included by scan_tc.cu inside its namespaces).
//
// One CTA walks the chunks of one segment of one (batch, head) stream.  NB = 64-column blocks of the state
// dimension held by the CTA (N = 64 NB); NWQ = warps per TMEM lane quadrant.  The CTA has 4 NWQ worker
// warps (4 lane quadrants x NWQ column groups), one scalar warp and one issue warp.
//
// MODE 0  full forward: Y, final state, optional 16-bit chunk-start states
//      1  states only: chunk-start states / the end state of the segment (no C, no scores, no Y)
//      2  adjoint states: the same walk backwards in time over C and dY, giving the adjoint of the segment's
//         start state from a zero end adjoint (the pre-pass of a backward sweep that is split in time)
//
// What bounds it: the phases of a chunk (rotation, score product, masking, second product, state update) form
// one dependent chain of about 5 k clocks, most of it latency; neither DRAM, the tensor pipe nor the issue
// slots are full.  Hence, when there are streams enough, two CTAs per SM for NB = 1 (NWQ = 2: 80 KB of tiles, 256 TMEM
// columns, 96 registers): the chain of one stream fills the waits of the other.  To fit twice, B and C are rotated in place in a single
// stage that is refilled while the scores are masked, Y is staged over the score tile, and the second product
// accumulates over the TMEM columns of the scores.
//
// Columns: inside every group of 16 real columns the 8 real parts precede the 8 imaginary parts (tiles K', Q,
// Zv and the saved states), so that two neighbouring columns are the same part of two oscillators: all the
// complex arithmetic of the passes and epilogues then runs on packed float32 pairs (fma.rn.f32x2).
//
// MMAs have M = 64 (rows in lanes 0..15 of every TMEM quadrant); the epilogues read them with the 16x256b shape
// (thread t: rows t/4 and t/4 + 8 of the quadrant, column pair 2 (t%4) of every 8-column block).
template <int NB, bool FULL, int NWQ>
struct FwdSmem {
  static constexpr uint32_t U = 0;                                   // two stages of U
  static constexpr uint32_t KZ = 2 * TILE;                           // 2 NB x [K' ; Zv]
  static constexpr uint32_t C = KZ + 4 * NB * TILE;                  // 2 NB x Q
  static constexpr uint32_t UE = C + (FULL ? 2 * NB * TILE : 0);     // e^{l_end - l_s} U
  static constexpr uint32_t S = UE + TILE;                           // scores, then Y
  static constexpr uint32_t SCAL = S + (FULL ? TILE : 0);
  static constexpr uint32_t BYTES = SCAL + 3 * SCW * 4 + (NWQ / 2) * 64 * 4 + 1024;
};

struct alignas(64) TcFwdParams {
  CUtensorMap tmU, tmB, tmC;   // MODE 2: dY, C, unused
  CUtensorMap tmY, tmS;        // 16-bit output and chunk-state tensors (TMA stores); unused ones stay zero
  const float* M;
  const float* K;
  const float* z0;      // (BH, 64, 2N) or null: start state of segment 0 (unless from_seg)
  const void* Bprev;
  const void* Uprev;
  void* Y;
  float* zfinal;        // (BH, 64, 2N) or null
  // or null: what a caller carries on from, in the operands' type (their conversion and two row copies were launches of 2 to
  // 2.6 us each behind a prompt of 121 us): the end state, and the last rows of B and U
  void *state_last, *B_last, *U_last;
  const void *U, *B;
  void* states16;       // optional (NB, BH, nchunks, 64, 128) 16-bit: conjugated start state of every chunk
  float* seg;           // (BH, nseg, 64, 128 NB) float32: start states (from_seg) or, MODE 1 / 2 pre-pass, results
  float2* seg_pi;       // (BH, nseg): transition product of the segment (pre-pass)
  int heads, groups, T, nchunks, cps, nseg, seg0;   // cps: chunks per segment; seg0: segment of blockIdx.y = 0
  int tail, bh0;   // MODE 2: the last segment's chunks where the others are longer (else 0); first stream of the grid
  int from_seg;   // start states: 1 given in seg, 2 to be folded from the segments' contributions in seg
  int to_seg;     // pre-pass: leave this segment's contribution in seg
  long long wait_limit;  // SM clocks a wait of the main loop may take before the kernel gives up
};

template <typename TIn, typename TY, int MODE, int NB, int NWQ>
__global__ void __launch_bounds__(128 * NWQ + 64, NWQ == 2 ? 2 : 1)
    scan_tc_fwd_kernel(const __grid_constant__ TcFwdParams p) {
  constexpr bool FULL = MODE == 0, ADJ = MODE == 2;
  using SM = FwdSmem<NB, FULL, NWQ>;
  constexpr int NT = 128 * NWQ;      // worker threads
  constexpr int SC = 64 / NWQ;       // score / output columns per warp
  constexpr int SB = SC / 8;
  constexpr int ZC = 128 * NB / NWQ; // state columns per warp
  constexpr int ZB = ZC / 8;
  constexpr int TPT = 512 * NB / NT; // tiles of B (and C) a thread rotates
  constexpr uint32_t TM_COLS = FULL ? (NB == 1 ? 256 : 512) : 128 * NB;
  constexpr uint32_t TM_INC = FULL ? 128 : 0;   // TMEM: [S, then Ydiag | Yoff] 0..127, Inc 128 NB columns
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t bar_u[2], bar_bc[2], bar_mma[3], bar_st, bar_sc[2], bar_drain;   // bar_mma: [S|Yoff] | Inc | Ydiag
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;
  constexpr bool Y_TMA = FULL && sizeof(TY) == 2;
  float* sc_tab = reinterpret_cast<float*>(smem + SM::SCAL);
  float* s_diag = sc_tab + 3 * SCW;   // [NWQ / 2][64] partial diagonal scores
  using PK = Pack2<TIn>;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool worker = warp < 4 * NWQ;
  const int quad = warp & 3, cg = worker ? (warp >> 2) : 0;
  const int rowA = 16 * quad + (lane >> 2), rowB = rowA + 8, cq = lane & 3;   // epilogue identity
  const int rrow = (tid >> 2) & 63, rk = tid & 3, rgrp = tid >> 8;   // rotation identity
  const uint32_t lane_base = (uint32_t)(32 * quad) << 16;
  const int bh = ADJ ? p.bh0 + blockIdx.x : blockIdx.x, b = bh / p.heads, h = bh % p.heads;
  const int bg = b * p.groups + h / (p.heads / p.groups);
  const int seg = p.seg0 + blockIdx.y;
  const int c0 = ADJ && p.tail ? p.nchunks - p.tail : seg * p.cps, n = min(p.cps, p.nchunks - c0);   // this CTA's chunks: c0 .. c0 + n - 1
  const int T = p.T;
  constexpr int D = 128 * NB;   // real columns of a state row
  const float* Mb = p.M + (size_t)bh * T * 2;
  const float* Kb = p.K + (size_t)bh * T * 4;
  const long long wl = p.wait_limit;
  auto chunk_of = [&](int i) { return ADJ ? c0 + n - 1 - i : c0 + i; };

  if (!FULL) grid_release();   // (a pre-pass: what follows it may start up meanwhile)
  if (tid == 0) {
    mbar_init(&bar_u[0], 1); mbar_init(&bar_u[1], 1); mbar_init(&bar_bc[0], 1); mbar_init(&bar_bc[1], 1);
    for (int i = 0; i < 3; ++i) mbar_init(&bar_mma[i], 1);
    mbar_init(&bar_st, 4 * NWQ);   // one arrival per worker warp
    mbar_init(&bar_sc[0], 1); mbar_init(&bar_sc[1], 1);
    mbar_init(&bar_drain, 1);
    fence_barrier_init();
    s_abort = 0;
  }
  auto issue_u = [&](int i) {   // one thread
    mbar_expect_tx(&bar_u[i & 1], TILE);
    tma_load_3d(smem + SM::U + (i & 1) * TILE, &p.tmU, &bar_u[i & 1], 0, chunk_of(i) * L, bh);
  };
  // B is single-buffered where the other half of the KZ tiles holds the state, double-buffered in the pre-passes,
  // which keep no state tile: there the load would otherwise be longer than the rest of a chunk's chain
  const bool keep_zv = FULL || p.states16 != nullptr;
  auto buf_of = [&](int i) { return keep_zv ? 0 : i & 1; };
  auto phase_of = [&](int i) { return (uint32_t)(keep_zv ? i & 1 : (i >> 1) & 1); };
  auto issue_bc = [&](int i) {   // one thread
    const int t0 = chunk_of(i) * L;
    uint64_t* bar = &bar_bc[buf_of(i)];
    mbar_expect_tx(bar, (FULL ? 4 : 2) * NB * TILE);
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      tma_load_3d(smem + SM::KZ + (2 * q + buf_of(i)) * TILE, &p.tmB, bar, 64 * q, t0, bg);
      if (FULL) tma_load_3d(smem + SM::C + q * TILE, &p.tmC, bar, 64 * q, t0, bg);
    }
  };
  auto prefetch_bc = [&](int i) {   // one thread
    const int t0 = chunk_of(i) * L;
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      tma_prefetch_3d(&p.tmB, 64 * q, t0, bg);
      if (FULL) tma_prefetch_3d(&p.tmC, 64 * q, t0, bg);
    }
  };
  if (warp == 0) {
    tmem_alloc(&tmem_slot, TM_COLS);
  } else if (warp == 4 * NWQ) {
    chunk_scalars<FULL>(sc_tab, load_scalars(Mb, Kb, chunk_of(0) * L, T, lane), lane);
  }
  if (tid == 0) {   // (after the barriers were initialised by this same thread)
    issue_bc(0);
    issue_u(0);
    if (n > 1) { issue_u(1); if (keep_zv) prefetch_bc(1); else issue_bc(1); }
  }

  // ---- carried state, conjugated.  zz[2 j + hh]: 8-column block j of this warp's ZC columns, row (hh ? rowB :
  // rowA), as a pair of neighbouring columns; even blocks hold real parts, odd blocks minus the imaginary parts
  f2 zz[2 * ZB];
#pragma unroll
  for (int j = 0; j < 2 * ZB; ++j) zz[j] = 0ull;
  auto n_of = [&](int m) { return ZC / 2 * cg + 8 * m + 2 * cq; };   // oscillators n, n + 1 of block pair m
  if (worker && !ADJ && !p.to_seg && p.from_seg != 1 && (p.z0 || p.Bprev)) {   // start state of the sequence
    const TIn* Bp = reinterpret_cast<const TIn*>(p.Bprev);
    const TIn* Up = reinterpret_cast<const TIn*>(p.Uprev);
    float xr = 0.f, xi = 0.f, up[2] = {0.f, 0.f};
    if (Bp) {  // pending prev-tap of the token before the sequence: u_prev (x) (kp_0 / m_0) b_prev
      pending_tap(Mb, Kb, xr, xi);
      up[0] = to_f32(Up[(size_t)bh * 64 + rowA]);
      up[1] = to_f32(Up[(size_t)bh * 64 + rowB]);
    }
#pragma unroll
    for (int m = 0; m < ZB / 2; ++m) {
      const int nn = n_of(m);
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.z0) z = *reinterpret_cast<const float4*>(p.z0 + ((size_t)bh * 64 + (hh ? rowB : rowA)) * D + 2 * nn);
        if (Bp) {
          const TIn* bp = Bp + (size_t)bg * D + 2 * nn;
          const float b0r = to_f32(bp[0]), b0i = to_f32(bp[1]), b1r = to_f32(bp[2]), b1i = to_f32(bp[3]);
          z.x += up[hh] * (xr * b0r - xi * b0i); z.y += up[hh] * (xr * b0i + xi * b0r);
          z.z += up[hh] * (xr * b1r - xi * b1i); z.w += up[hh] * (xr * b1i + xi * b1r);
        }
        zz[4 * m + hh] = mk2(z.x, z.z);
        zz[4 * m + 2 + hh] = mk2(-z.y, -z.w);
      }
    }
  }
  // start state of a later segment: given, or folded from the earlier segments' contributions
  if (worker && p.from_seg) {
    grid_wait();
    const size_t stride = (size_t)64 * 128 * NB;
    const float* src = p.seg + (size_t)bh * p.nseg * stride + ZC * cg + 2 * cq;
    const bool fold = p.from_seg == 2;
    for (int s = fold ? 0 : seg; s < (fold ? seg : seg + 1); ++s) {
      const float2 pi = fold ? p.seg_pi[(size_t)bh * p.nseg + s] : make_float2(0.f, 0.f);
      const f2 pr = dup2(pi.x), pim = dup2(pi.y), npim = dup2(-pi.y);
#pragma unroll
      for (int m = 0; m < ZB / 2; ++m)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float* f = src + s * stride + (size_t)(hh ? rowB : rowA) * 128 * NB + 16 * m;
          const float2 fr = *reinterpret_cast<const float2*>(f), fi = *reinterpret_cast<const float2*>(f + 8);
          const f2 a = zz[4 * m + hh], c = zz[4 * m + 2 + hh];   // conj(Pi_s) z + F_s
          zz[4 * m + hh] = fma2(pim, c, fma2(pr, a, mk2(fr.x, fr.y)));
          zz[4 * m + 2 + hh] = fma2(npim, a, fma2(pr, c, mk2(fi.x, fi.y)));
        }
    }
  }
  // 16-bit copy of the state: rows p, K-major along d, directly below the K' rows of the same 64 columns, so that
  // [K' ; Zv] is one 128-row operand
  auto store_zv_tile = [&]() {
    uint8_t* tile = smem + SM::KZ + (2 * (cg * ZC / 64) + 1) * TILE + 4 * cq;
    constexpr int CH = 64 / ZC;   // warps that share a tile
#pragma unroll
    for (int j = 0; j < ZB; ++j) {
      const int ch = (cg % CH) * ZB + j;
      *reinterpret_cast<uint32_t*>(tile + sw128(rowA, ch)) = PK::pack2(zz[2 * j]);
      *reinterpret_cast<uint32_t*>(tile + sw128(rowB, ch)) = PK::pack2(zz[2 * j + 1]);
    }
  };
  auto store_states = [&](int i) {   // issue lane: the state tile of chunk i is exactly what the backward wants
    const int c = chunk_of(i);
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q)
      tma_store_3d(&p.tmS, smem + SM::KZ + (2 * q + 1) * TILE, 64 * (q & 1), c * 64, (q >> 1) * (int)gridDim.x + bh);
    tma_store_commit();
  };
  if (worker && keep_zv) { store_zv_tile(); fence_async_smem(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;

  // Bounded waits.  After the first expired one every warp keeps walking the chunk loop without working (named
  // barriers have no time-out, so nobody may leave early); the other waits give up as soon as they see the flag.
  auto wait_one = [&](uint64_t* bar, uint32_t parity, int code) {   // one thread
    return mbar_try_wait(bar, parity) || wait_or_abort(bar, parity, wl, &s_abort, code);
  };
  auto wait_warp = [&](uint64_t* bar, uint32_t parity, int code) {  // a converged warp
    return __all_sync(0xffffffffu, wait_one(bar, parity, code)) != 0;
  };

  if (warp == 4 * NWQ) {
    // ---- scalar warp: three tables, two chunks ahead, their inputs one more (the shuffle scans and the way to memory
    // are longer than a chunk of a pre-pass) -----------------------------------------------------------------
    float pr = 1.f, pi = 0.f;   // transition product of the segment
    ScalarRaw raw = load_scalars(Mb, Kb, chunk_of(min(1, n - 1)) * L, T, lane);
    for (int i = -1; i < n; ++i) {
      if (i >= 0) {
        if (p.to_seg) {
          const float* tail = sc_tab + (i % 3) * SCW + SC_TAIL;
          const float mr = tail[0] * tail[1], mi = tail[0] * tail[2];
          const float nr = pr * mr - pi * mi;
          pi = pr * mi + pi * mr; pr = nr;
        }
        bar_sync(2, NT + 64);   // the workers are through chunk i - 1, whose table is overwritten now
      }
      const int j = i + 2;
      if (j < n) {
        const ScalarRaw cur = raw;
        if (j + 1 < n) raw = load_scalars(Mb, Kb, chunk_of(j + 1) * L, T, lane);
        chunk_scalars<FULL>(sc_tab + (j % 3) * SCW, cur, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_sc[j & 1]);
      }
    }
    if (p.to_seg && lane == 0) p.seg_pi[(size_t)bh * p.nseg + seg] = make_float2(pr, pi);
    if (FULL && p.state_last && seg == p.nseg - 1) {   // the last rows, in 16-byte pieces
      if (lane < D / 8 && bh % (p.heads / p.groups) == 0)
        reinterpret_cast<uint4*>(p.B_last)[(size_t)bg * (D / 8) + lane] =
            reinterpret_cast<const uint4*>(p.B)[((size_t)bg * T + T - 1) * (D / 8) + lane];
      if (lane < 8)
        reinterpret_cast<uint4*>(p.U_last)[(size_t)bh * 8 + lane] = reinterpret_cast<const uint4*>(p.U)[((size_t)bh * T + T - 1) * 8 + lane];
    }
  } else if (!worker) {
    // ---- issue warp (one lane): every TMA load and store and every MMA.  The workers never wait for it, only for
    // the commit barriers of the products they read.
    constexpr uint32_t ID_S = make_idesc(64, 128, PK::fmt, 0, 0);        // K-major x K-major   [S | Yoff]
    constexpr uint32_t ID_Y = make_idesc(64, 64, PK::fmt, 0, 1);         // K-major x MN-major  Ydiag
    constexpr uint32_t ID_Z = make_idesc(64, 128 * NB, PK::fmt, 1, 1);   // MN-major x MN-major Inc
    const uint64_t dKZ = make_desc(smem_u32(smem + SM::KZ), 16, 1024);
    const uint64_t dQ = make_desc(smem_u32(smem + SM::C), 16, 1024);
    const uint64_t dKm = make_desc(smem_u32(smem + SM::KZ), 2 * TILE, 1024);   // 64-column blocks two tiles apart
    const uint64_t dUE = make_desc(smem_u32(smem + SM::UE), TILE, 1024);
    const uint64_t dS = make_desc(smem_u32(smem + SM::S), 16, 1024);
    int req_u = min(n, 2), req_bc = keep_zv ? 1 : min(n, 2);   // loads requested so far
    // [S | Yoff] = Q [K' ; Zv]^T over the tiles of the first / second rotation step
    auto scores = [&](int step) {
#pragma unroll
      for (int q = step; q < 2 * NB; q += TPT)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma(tmem, desc_adv(dQ, q * TILE + 32 * k), desc_adv(dKZ, 2 * q * TILE + 32 * k), ID_S, q + k > 0);
    };
    if (lane == 0 && p.states16) store_states(0);
    __syncwarp();
    for (int i = 0; i < n; ++i) {
      const bool lead = elect_one();
      if (FULL) {
        bar_sync(5, NT + 32);   // the first (TPT = 1: all) tiles of Q and K' rotated
        if (lead && !s_abort) { tc_fence_after_sync(); scores(0); }
        __syncwarp();
      }
      bar_sync(2, NT + 64);     // rotation done
      if (lead && !s_abort) {
        tc_fence_after_sync();
        if (FULL) {
          if (TPT == 2) scores(1);
          tma_store_wait_read();   // the score tile still holds the previous Y, the Zv tiles the saved state
          umma_commit(&bar_mma[0]);
        }
        // Inc = (e^{l_end - l_s} U)^T K'
#pragma unroll
        for (int k = 0; k < 4; ++k) umma(tmem + TM_INC, desc_adv(dUE, 2048 * k), desc_adv(dKm, buf_of(i) * TILE + 2048 * k), ID_Z, k > 0);
        if (!FULL) tma_store_wait_read();
        umma_commit(&bar_mma[1]);
        // refill B and C as soon as their last products are done: what is left of the iteration hides the load
        const int nxt = i + (keep_zv ? 1 : 2);
        if (nxt < n && wait_one(&bar_mma[1], i & 1, 8)) {
          issue_bc(nxt); ++req_bc;
          if (i + 2 < n) {
            if (keep_zv) prefetch_bc(i + 2);   // on their way to L2 for a whole iteration
            if (!FULL) { issue_u(i + 2); ++req_u; }
          }
        }
      }
      __syncwarp();
      if (FULL) {
        bar_sync(4, NT + 32);   // S tile written
        if (lead && !s_abort) {
          tc_fence_after_sync();
          const uint64_t dU = make_desc(smem_u32(smem + SM::U + (i & 1) * TILE), TILE, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma(tmem, desc_adv(dS, 32 * k), desc_adv(dU, 2048 * k), ID_Y, k > 0);   // S U
          umma_commit(&bar_mma[2]);
        }
      }
      if (lead && !s_abort && (FULL || p.states16) && wait_one(&bar_st, i & 1, 5)) {
        if (Y_TMA) {
          tma_store_3d(&p.tmY, smem + SM::S, 0, chunk_of(i) * L, bh);
          tma_store_commit();
        }
        if (p.states16 && i + 1 < n) store_states(i + 1);
        if (FULL && i + 2 < n) { issue_u(i + 2); ++req_u; }
      }
      __syncwarp();
    }
    if (lane == 0) {
      // Unwind: nothing of this CTA may still be in flight when shared memory and TMEM are released.
      if (s_abort) {
        for (int i = max(0, req_bc - 2); i < req_bc; ++i) mbar_wait(&bar_bc[buf_of(i)], phase_of(i));
        for (int i = max(0, req_u - 2); i < req_u; ++i) mbar_wait(&bar_u[i & 1], (i >> 1) & 1);
      }
      umma_commit(&bar_drain);
      mbar_wait(&bar_drain, 0);
      tma_store_wait_all();
    }
    __syncwarp();
  } else {
    // ---- worker warps ---------------------------------------------------------------------------------------
    bool live = true;   // warp-uniform; cleared when a wait expired
    for (int i = 0; i < n; ++i) {
      const float* sc = sc_tab + (i % 3) * SCW;
      const float4* rot = reinterpret_cast<const float4*>(sc);
      const float4* kcl = reinterpret_cast<const float4*>(sc + SC_KCL);
      if (i > 0) live = live && wait_warp(&bar_sc[i & 1], ((i - 1) >> 1) & 1, 9);
      live = live && wait_warp(&bar_bc[buf_of(i)], phase_of(i), 1);

      // ---- rotation: C -> Q, B -> K' (in place), diagonal scores.  A thread owns 32 bytes (8 oscillators) of a
      // row in each of TPT tiles; the score products of the first tile start while the second is rotated.
      {
        const uint32_t o0 = sw128(rrow, 2 * rk), o1 = sw128(rrow, 2 * rk + 1);
        const float4 rt = rot[rrow];   // phi, w
        f2 dr = 0ull, di0 = 0ull, di1 = 0ull;   // sums of Re conj(c) b and of the two parts of Im conj(c) b
#pragma unroll
        for (int half = 0; half < TPT; ++half) {
          if (live) {
            uint8_t* tB = smem + SM::KZ + (2 * (TPT * rgrp + half) + buf_of(i)) * TILE;
            uint8_t* tC = smem + SM::C + (TPT * rgrp + half) * TILE;
            const uint4 b0 = *reinterpret_cast<const uint4*>(tB + o0), b1 = *reinterpret_cast<const uint4*>(tB + o1);
            uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
            if (FULL) { x0 = *reinterpret_cast<const uint4*>(tC + o0); x1 = *reinterpret_cast<const uint4*>(tC + o1); }
            const uint32_t bw[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            const uint32_t cw[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
            uint32_t kr[4], ki[4], qr[4], qi[4];
            const f2 phr = dup2(rt.x), phi = dup2(rt.y), nphr = dup2(-rt.x);
            const f2 wr = dup2(rt.z), nwr = dup2(-rt.z), nwi = dup2(-rt.w);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              f2 br, bi;
              PK::split(bw[2 * e], bw[2 * e + 1], br, bi);
              if (ADJ) {   // B is the C operand here: q = conj(c) phi
                kr[e] = PK::pack2(fma2(bi, phi, mul2(br, phr)));
                ki[e] = PK::pack2(fma2(bi, nphr, mul2(br, phi)));
              } else {     // k' = conj(w b)
                kr[e] = PK::pack2(fma2(bi, nwi, mul2(br, wr)));
                ki[e] = PK::pack2(fma2(bi, nwr, mul2(br, nwi)));
              }
              if (FULL) {
                f2 cr, ci;
                PK::split(cw[2 * e], cw[2 * e + 1], cr, ci);
                qr[e] = PK::pack2(fma2(ci, phi, mul2(cr, phr)));    // q = conj(c) phi
                qi[e] = PK::pack2(fma2(ci, nphr, mul2(cr, phi)));
                dr = fma2(cr, br, dr); dr = fma2(ci, bi, dr);
                di0 = fma2(cr, bi, di0); di1 = fma2(ci, br, di1);
              }
            }
            *reinterpret_cast<uint4*>(tB + o0) = make_uint4(kr[0], kr[1], kr[2], kr[3]);
            *reinterpret_cast<uint4*>(tB + o1) = make_uint4(ki[0], ki[1], ki[2], ki[3]);
            if (FULL) {
              *reinterpret_cast<uint4*>(tC + o0) = make_uint4(qr[0], qr[1], qr[2], qr[3]);
              *reinterpret_cast<uint4*>(tC + o1) = make_uint4(qi[0], qi[1], qi[2], qi[3]);
            }
          }
          if (FULL && half == 0) {
            fence_async_smem();
            tc_fence_before_sync();
            bar_arrive(5, NT + 32);
          }
        }
        live = live && wait_warp(&bar_u[i & 1], (i >> 1) & 1, 10);
        if (live) {   // Ue = e^{l_end - l_s} U   (MODE 2: e^{l_t} dY)
          const uint8_t* tU = smem + SM::U + (i & 1) * TILE;
#pragma unroll
          for (int j = 0; j < 512 / NT; ++j) {
            const int item = tid + NT * j, r = item >> 3;
            const uint32_t off = sw128(r, item & 7);
            const uint4 uv = *reinterpret_cast<const uint4*>(tU + off);
            const f2 ee = dup2(ADJ ? kcl[r].z : kcl[r].w);
            *reinterpret_cast<uint4*>(smem + SM::UE + off) =
                make_uint4(PK::pack2(mul2(PK::natural(uv.x), ee)), PK::pack2(mul2(PK::natural(uv.y), ee)),
                           PK::pack2(mul2(PK::natural(uv.z), ee)), PK::pack2(mul2(PK::natural(uv.w), ee)));
          }
        }
        if (FULL && live) {   // Re(conj(c) kc b) = kc_r Re(conj(c) b) - kc_i Im(conj(c) b), summed over the row
          const float4 kc = kcl[rrow];
          const float2 a = un2(dr), c = un2(di0), d = un2(di1);
          float dg = kc.x * (a.x + a.y) - kc.y * ((c.x + c.y) - (d.x + d.y));
          dg += __shfl_xor_sync(0xffffffffu, dg, 1);
          dg += __shfl_xor_sync(0xffffffffu, dg, 2);
          if (rk == 0) s_diag[rgrp * 64 + rrow] = dg;
        }
      }
      fence_async_smem();
      tc_fence_before_sync();
      bar_arrive(2, NT + 64);

      if (FULL) {
        // ---- scores epilogue: decay, causal mask, diagonal -> 16-bit S tile.  The 16 rows of a warp meet SB / 2 blocks
        // of 16 columns: left of the diagonal block (factored decays), on it, or right of it (zeros).  What does not
        // depend on the scores is fetched ahead of the wait, which is a compiler barrier.
        float fac[4 * SB];   // [k][q][hh]: factors of this thread's cells
        float dg2[2] = {0.f, 0.f};
        {
          const float rf[2] = {sc[SC_ROW + rowA], sc[SC_ROW + rowB]};
#pragma unroll
          for (int k = 0; k < SB; ++k) {
            const int blk16 = (cg * SB + k) >> 1, s0 = cg * SC + 8 * k + 2 * cq;
            if (blk16 < quad) {
              const float2 cf = *reinterpret_cast<const float2*>(sc + SC_COL + 64 * quad + s0);
              fac[4 * k] = cf.x * rf[0]; fac[4 * k + 1] = cf.x * rf[1];
              fac[4 * k + 2] = cf.y * rf[0]; fac[4 * k + 3] = cf.y * rf[1];
            } else if (blk16 == quad) {
              const float2 ls = *reinterpret_cast<const float2*>(sc + SC_L2 + s0);
#pragma unroll
              for (int hh = 0; hh < 2; ++hh) {
                const int R = hh ? rowB : rowA;
                const float lt = sc[SC_L2 + R];
                fac[4 * k + hh] = s0 < R ? ex2f(fminf(lt - ls.x, 0.f)) : 0.f;
                fac[4 * k + 2 + hh] = s0 + 1 < R ? ex2f(fminf(lt - ls.y, 0.f)) : 0.f;
              }
            } else {
              fac[4 * k] = fac[4 * k + 1] = fac[4 * k + 2] = fac[4 * k + 3] = 0.f;
            }
          }
        }
        const bool has_diag = (quad * 2) / SB == cg, empty = cg * SB > 2 * quad + 1;
        live = live && wait_warp(&bar_mma[0], i & 1, 2);
        tc_fence_after_sync();
        if (live) {
          uint32_t r[4 * SB];
          if (!empty) tmem_ld_16x256<SB>(tmem + lane_base + cg * SC, r);
          if (has_diag) {
            dg2[0] = s_diag[rowA]; dg2[1] = s_diag[rowB];
            if (NWQ == 4) { dg2[0] += s_diag[64 + rowA]; dg2[1] += s_diag[64 + rowB]; }
          }
          tmem_ld_wait();
          uint8_t* tS = smem + SM::S + 4 * cq;
#pragma unroll
          for (int k = 0; k < SB; ++k) {
            const int blk16 = (cg * SB + k) >> 1, s0 = cg * SC + 8 * k + 2 * cq;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              const int R = hh ? rowB : rowA;
              uint32_t word = 0u;
              if (blk16 <= quad) {
                float v0 = __uint_as_float(r[4 * k + 2 * hh]) * fac[4 * k + hh];
                float v1 = __uint_as_float(r[4 * k + 2 * hh + 1]) * fac[4 * k + 2 + hh];
                if (blk16 == quad) {
                  v0 = s0 == R ? dg2[hh] : v0;
                  v1 = s0 + 1 == R ? dg2[hh] : v1;
                }
                word = PK::pack(v0, v1);
              }
              *reinterpret_cast<uint32_t*>(tS + sw128(R, cg * SB + k)) = word;
            }
          }
        }
        fence_async_smem();
        tc_fence_before_sync();
        bar_arrive(4, NT + 32);
      }

      // ---- state update: zv = conj(u_end) (e^{l_end} zv + Inc);  MODE 2: dz = e^{l_end} (u_end dz) + Inc -----------
      live = live && wait_warp(&bar_mma[1], i & 1, 3);
      tc_fence_after_sync();
      if (live) {
        const float e_end = sc[SC_TAIL], ur = sc[SC_TAIL + 1], ui = sc[SC_TAIL + 2];
        const f2 E = dup2(e_end), R = dup2(ADJ ? e_end * ur : ur), I = dup2(ADJ ? e_end * ui : ui);
        const f2 NI = dup2(ADJ ? -e_end * ui : -ui);
#pragma unroll
        for (int part = 0; part < ZC / 32; ++part) {
          uint32_t inc[16];
          tmem_ld_16x256<4>(tmem + lane_base + TM_INC + ZC * cg + 32 * part, inc);
          tmem_ld_wait();
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              const int j = 8 * part + 4 * m + hh;   // zz[j]: real parts, zz[j + 2]: imaginary parts
              const f2 ir = mk2(__uint_as_float(inc[8 * m + 2 * hh]), __uint_as_float(inc[8 * m + 2 * hh + 1]));
              const f2 ii = mk2(__uint_as_float(inc[8 * m + 4 + 2 * hh]), __uint_as_float(inc[8 * m + 4 + 2 * hh + 1]));
              if (ADJ) {
                const f2 a = zz[j], c = zz[j + 2];
                zz[j] = fma2(c, NI, fma2(a, R, ir));
                zz[j + 2] = fma2(c, R, fma2(a, I, ii));
              } else {
                const f2 a = fma2(zz[j], E, ir), c = fma2(zz[j + 2], E, ii);
                zz[j] = fma2(c, I, mul2(a, R));
                zz[j + 2] = fma2(a, NI, mul2(c, R));
              }
            }
        }
        if (keep_zv) store_zv_tile();
      }

      if (FULL) {
        // ---- output: y = Y_diag + e^{l_t} Y_off ---------------------------------------------------------------
        const float et[2] = {kcl[rowA].z, kcl[rowB].z};
        live = live && wait_warp(&bar_mma[2], i & 1, 4);
        tc_fence_after_sync();
        if (live) {
          uint32_t yd[4 * SB], yo[4 * SB];
          tmem_ld_16x256<SB>(tmem + lane_base + cg * SC, yd);
          tmem_ld_16x256<SB>(tmem + lane_base + 64 + cg * SC, yo);
          tmem_ld_wait();
          const int t0 = (c0 + i) * L;
#pragma unroll
          for (int k = 0; k < SB; ++k)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              const int R = hh ? rowB : rowA;
              const float y0 = __uint_as_float(yd[4 * k + 2 * hh]) + et[hh] * __uint_as_float(yo[4 * k + 2 * hh]);
              const float y1 = __uint_as_float(yd[4 * k + 2 * hh + 1]) + et[hh] * __uint_as_float(yo[4 * k + 2 * hh + 1]);
              if constexpr (sizeof(TY) == 2) {   // over the score tile; rows beyond T are clipped by the store
                *reinterpret_cast<uint32_t*>(smem + SM::S + sw128(R, cg * SB + k) + 4 * cq) = Pack2<TY>::pack(y0, y1);
              } else if (t0 + R < T) {
                float* dst = reinterpret_cast<float*>(p.Y) + ((size_t)bh * T + t0 + R) * 64 + cg * SC + 8 * k + 2 * cq;
                *reinterpret_cast<float2*>(dst) = make_float2(y0, y1);
              }
            }
        }
      }
      fence_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_st);   // this warp's part of the Y and Zv tiles is complete
    }
    if (live && p.to_seg) {
      float* dst = p.seg + ((size_t)bh * p.nseg + seg) * 64 * 128 * NB + ZC * cg + 2 * cq;
#pragma unroll
      for (int j = 0; j < ZB; ++j) {
        *reinterpret_cast<float2*>(dst + (size_t)rowA * 128 * NB + 8 * j) = un2(zz[2 * j]);
        *reinterpret_cast<float2*>(dst + (size_t)rowB * 128 * NB + 8 * j) = un2(zz[2 * j + 1]);
      }
    } else if (live && (p.zfinal || (FULL && p.state_last)) && seg == p.nseg - 1) {
#pragma unroll
      for (int m = 0; m < ZB / 2; ++m) {
        const int nn = n_of(m);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float2 re = un2(zz[4 * m + hh]), im = un2(zz[4 * m + 2 + hh]);
          const size_t at = ((size_t)bh * 64 + (hh ? rowB : rowA)) * D + 2 * nn;
          if (p.zfinal) *reinterpret_cast<float4*>(p.zfinal + at) = make_float4(re.x, -im.x, re.y, -im.y);
          if (FULL && p.state_last)
            *reinterpret_cast<uint2*>(reinterpret_cast<TIn*>(p.state_last) + at) = make_uint2(PK::pack(re.x, -im.x), PK::pack(re.y, -im.y));
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, TM_COLS);
}

// Start state of every segment from the segments' own contributions: seg[s] <- Z_s, Z_{s+1} = Pi_s Z_s + F_s (conj
// pairs, so conj(Pi_s)), or, for adjoints, backwards in time: seg[s] <- Z_s (at the segment's END), Z_{s-1} = Pi_s Z_s + F_s.
// ``init`` = (BH, 64, 2N) start state / end adjoint or null; Bprev / Uprev add the pending tap to it.  One thread per
// (row, oscillator); the serial chain is nseg multiply-adds long and its loads are requested eight at a time.
// Used when there are more than FOLD_SEGS segments: up to there the sweeps fold the contributions of the segments
// before theirs themselves (32 KB per segment and CTA from L2), which costs less than a launch.
template <typename TIn, bool REVERSE>
__global__ void __launch_bounds__(256) scan_tc_combine_kernel(float* __restrict__ seg, const float2* __restrict__ seg_pi,
                                                              const float* __restrict__ init,
                                                              const TIn* __restrict__ Bprev,
                                                              const TIn* __restrict__ Uprev,
                                                              const float* __restrict__ M, const float* __restrict__ K,
                                                              int heads, int groups, int T, int N, int nseg) {
  const int e = blockIdx.y * 256 + threadIdx.x, bh = blockIdx.x;
  const int row = e / N, n = e % N;
  grid_release();
  if (row >= 64) return;
  float zr = 0.f, zi = 0.f;
  if (init) {
    const float2 z = *reinterpret_cast<const float2*>(init + ((size_t)bh * 64 + row) * 2 * N + 2 * n);
    zr = z.x; zi = z.y;
  }
  if (Bprev) {
    const int bg = (bh / heads) * groups + (bh % heads) / (heads / groups);
    float xr, xi;
    pending_tap(M + (size_t)bh * T * 2, K + (size_t)bh * T * 4, xr, xi);
    const float br = to_f32(Bprev[(size_t)bg * 2 * N + 2 * n]), bi = to_f32(Bprev[(size_t)bg * 2 * N + 2 * n + 1]);
    const float u = to_f32(Uprev[(size_t)bh * 64 + row]);
    zr += u * (xr * br - xi * bi);
    zi += u * (xr * bi + xi * br);
  }
  zi = -zi;
  const size_t stride = (size_t)64 * 2 * N;
  float* base = seg + (size_t)bh * nseg * stride + (size_t)row * 2 * N + (n >> 3) * 16 + (n & 7);
  const float2* pis = seg_pi + (size_t)bh * nseg;
  grid_wait();
  for (int k0 = 0; k0 < nseg; k0 += 8) {
    float fr[8], fi[8];
    float2 pi[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      fr[k] = fi[k] = 0.f; pi[k] = make_float2(0.f, 0.f);
      if (k0 + k < nseg - 1) {   // (the contribution of the last segment of the walk is not needed)
        const int s = REVERSE ? nseg - 1 - (k0 + k) : k0 + k;
        fr[k] = base[s * stride]; fi[k] = base[s * stride + 8]; pi[k] = pis[s];
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k0 + k >= nseg) break;
      const int s = REVERSE ? nseg - 1 - (k0 + k) : k0 + k;
      base[s * stride] = zr; base[s * stride + 8] = zi;
      const float pim = REVERSE ? pi[k].y : -pi[k].y;
      const float nr = pi[k].x * zr - pim * zi + fr[k];
      zi = pi[k].x * zi + pim * zr + fi[k];
      zr = nr;
    }
  }
}
