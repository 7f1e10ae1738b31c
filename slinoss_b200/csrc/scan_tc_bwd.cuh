// Backward of the chunked scan on tcgen05 (included by scan_tc.cu inside its namespaces).
//
// With V_t = m_t W_{t-1} (state after the decay, before the injection of token t):
//     y_t = Re<c_t, V_t> + u_t Re(conj(c_t) kc_t b_t),      W_t = V_t + u_t (x) (g_t b_t).
// One CTA walks the chunks of one segment of one (batch, head) and one block of 64 state columns (32 KB of dB / dC
// per chunk and block) in REVERSE order carrying dz = adjoint of the chunk-end state (conjugated pairs, float32,
// in registers).  Streams that do not fill the chip are split in time: the adjoint states at the segment ends then
// come from the MODE 2 pre-pass of scan_tc_fwd.cuh.
// Per chunk, with the same rotated operands as the forward (unit phases on the 16-bit
// operands, decays exp(<=0) on float32 accumulators):
//     P~ = Q K'^T,  dS = dY U^T      -> Pdec = mask_{s<t} e^{l_t-l_s} P~ ,  dP = mask_{s<t} e^{l_t-l_s} dS
//     dQ = dP K' + e^{l_t} (dY Zv)                     -> dC  (un-rotate, + diagonal term)
//     dX = dP^T Q + (e^{l_end-l_s} U) dWv              -> dB, dg   (dWv = dz rotated by the unit phase of Pi_end;
//                                                        the decay is folded into the 16-bit rows of U)
//     dU = Pdec^T dY + e^{l_end-l_s} (K' dWv^T)        (+ dy_s diag_s)
//     dz <- e^{l_end} dWv + (e^{l_t} dY)^T Q           (adjoint of the chunk-start state)
// Per-token scalars for dM / dK go to the workspace and are finished by
// scan_tc_bwd_post_kernel using
//     conj(m_t) dm_t = S_t,   S_t = S_{t+1} + <q_t, dq_t> - conj(g_t) dg_t,
// anchored at every chunk end by S = <dZ, Z> of the state carried across that boundary.

constexpr uint32_t B_STAGE = 8 * TILE;                 // U | B(2) | C(2) | dY | Zv(2)
constexpr uint32_t B_OFF_Q = 2 * B_STAGE;              // Q (2)
constexpr uint32_t B_OFF_KP = B_OFF_Q + 2 * TILE;      // K' (2)
constexpr uint32_t B_OFF_DYO = B_OFF_KP + 2 * TILE;    // e^{l_t} dY (1)
constexpr uint32_t B_OFF_PD = B_OFF_DYO + TILE;        // Pdec (1)
constexpr uint32_t B_OFF_DP = B_OFF_PD + TILE;         // dP (1)
constexpr uint32_t B_OFF_DW = B_OFF_DP + TILE;         // dWv (2)
constexpr uint32_t B_OFF_UE = B_OFF_DW + 2 * TILE;     // e^{l_end-l_s} U (1)
constexpr uint32_t B_OFF_SCAL = B_OFF_UE + TILE;
constexpr int B_SCAL_FLOATS = 2 * SCW_B + 64 + 4 * 64 + 32 * 64;   // tables, sigma, [2][64] c conj(b), 4 x 8 partial sums
constexpr uint32_t B_SMEM_BYTES = B_OFF_SCAL + B_SCAL_FLOATS * 4 + 1024;
// TMEM columns: P~ then dUa 0 | dS then dUb 64 | dQ 128..255 | dX 256..383 | dZ 384..511.  All products have
// M = 64 (rows in lanes 0..15 of a quadrant).  P~, dS, dUa and dUb are N = 64 and read with the 16x256b load
// shape; dQ, dX and dZ are N = 128 products (each the sum of two operand pairs but for dZ) read with the
// 16x32bx2 shape (thread t: row t % 16 of column half t / 16).  dUa and dUb reuse the columns of P~ and dS,
// which are dead after epilogue 1.
// The state columns of Q, K', Zv and dWv are in the order of the forward kernel (per 16 columns: 8 real parts, 8
// imaginary parts), so a thread's 16 accumulator columns are whole oscillators and its arithmetic runs on packed
// float32 pairs; B, C, dB and dC keep the interleaved order of the tensors.
constexpr uint32_t B_TMEM_COLS = 512;

struct alignas(64) TcBwdParams {
  CUtensorMap tmU, tmB, tmC, tmdY, tmZ;
  CUtensorMap tmdU[2], tmdB, tmdC;   // outputs, written with TMA stores from shared memory; dU per column block
  const float* M;
  const float* K;
  const float* dfinal;   // (BH, 64, 2N) or null
  const float* zfinal;   // forward final state (BH, 64, 2N), read when dfinal is given
  const float* seg;      // (BH, nseg, 64, 128 NB): see fold; unused when there is one segment
  const float2* seg_pi;
  int fold;              // 1: seg holds the segments' own contributions, 0: the adjoint at every segment's end
  float2 *dg, *sterm, *dkcd, *anchor;   // per token / per chunk scalars (workspace), one set per column block
  float* dinit;          // (BH, 64, 2N) adjoint of the carried start state, or null
  int T, N, nchunks, cps, nseg;
  int tail, whole;       // tail > 0: two segments, the last of ``tail`` chunks, for the streams from ``whole`` on; the others in one
  int heads, groups;     // B and C are shared by the heads of a group; dB / dC leave per head
  long long wait_limit;  // SM clocks a wait of the main loop may take before the kernel gives up
};

// grid (batch * heads, column blocks, segments).  NW = warps per TMEM lane quadrant.
template <typename TIn, int NW>
__global__ void __launch_bounds__(128 * NW + 64, 1) scan_tc_bwd_kernel(const __grid_constant__ TcBwdParams p) {
  static_assert(NW == 4, "a thread owns 8 oscillators of a row: 16 worker warps");
  constexpr int NT = 128 * NW;               // worker threads; two more warps: scalars, TMA + MMA issue
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t bar_tma[2], bar_mma[5];   // bar_mma: P~,dS | dX | dQ | dU | dZ (all earlier MMAs)
  __shared__ uint64_t bar_st[3], bar_drain;    // output tiles staged in shared memory: dB | dC | dU
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;
  __shared__ float s_red[8 * NW + 2];
  float* sc_tab = reinterpret_cast<float*>(smem + B_OFF_SCAL);   // two tables (chunk parity)
  float* s_sig = sc_tab + 2 * SCW_B;                               // sigma_t = <dy_t, u_t>
  float2* s_cb = reinterpret_cast<float2*>(s_sig + 64);          // [2 halves][64]: sum_n c conj(b)
  float* s_acc = s_sig + 64 + 4 * 64;   // [4 quantities][8 = column group x half][64 rows]: re/im of <q,dq>, of R
  using PK = Pack2<TIn>;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool worker = warp < 4 * NW;
  const int quad = warp & 3, cg = worker ? (warp >> 2) : 0;
  const int row = 16 * quad + (lane & 15), hf = lane >> 4;
  const int rowA = 16 * quad + (lane >> 2), rowB = rowA + 8, cq = lane & 3;   // identity for the 16x256b loads
  constexpr int WC = 64 / NW, WB = WC / 8;   // columns / 8-column blocks per warp of a 64-wide accumulator
  const int d0 = cg * 16;                    // first column (inside the half) of this thread
  const uint32_t cell0 = sw128(row, 2 * cg), cell1 = sw128(row, 2 * cg + 1);   // its 32 bytes of a tile row
  const int bh = blockIdx.x, blk = blockIdx.y, seg = blockIdx.z, nb = gridDim.y;
  const int nseg = p.tail && bh < p.whole ? 1 : p.nseg;   // of this stream
  if (seg >= nseg) return;
  const int bg = (bh / p.heads) * p.groups + (bh % p.heads) / (p.heads / p.groups);   // row of B and C
  const int T = p.T, nC = p.nchunks, D = 2 * p.N;
  // this CTA's chunks: c_lo + n - 1 down to c_lo
  const int c_lo = p.tail ? (seg ? nC - p.tail : 0) : seg * p.cps;
  const int n = p.tail ? (nseg == 1 ? nC : seg ? p.tail : nC - p.tail) : min(p.cps, nC - c_lo);
  const int osc0 = 64 * blk + 32 * hf + 8 * cg;              // first of this thread's 8 oscillators
  const size_t set = (size_t)blk * gridDim.x + bh;           // row of the scalar workspaces
  const float* Mb = p.M + (size_t)bh * T * 2;
  const float* Kb = p.K + (size_t)bh * T * 4;
  const uint32_t lane_base = (uint32_t)(32 * quad) << 16;
  const long long wl = p.wait_limit;   // limit of the main loop's waits (the drain waits keep the default)

  if (tid == 0) {
    mbar_init(&bar_tma[0], 1); mbar_init(&bar_tma[1], 1);
    for (int i = 0; i < 5; ++i) mbar_init(&bar_mma[i], 1);
    for (int i = 0; i < 3; ++i) mbar_init(&bar_st[i], 4 * NW);   // one arrival per worker warp
    mbar_init(&bar_drain, 1);
    fence_barrier_init();
    s_abort = 0;
  }
  // The stage of chunk c is requested at the top of the previous iteration, as soon as the output stores of
  // the chunk that used the stage before have read it (half an iteration ahead was not enough any more: the
  // workers were seen waiting 1000+ clk for the data).  That chunk's deferred epilogue 5 works on a register
  // copy of its Zv cells.
  auto issue_loads = [&](int it) {   // one thread
    const int c = c_lo + n - 1 - it;
    uint8_t* st = smem + (it & 1) * B_STAGE;
    uint64_t* bar = &bar_tma[it & 1];
    mbar_expect_tx(bar, B_STAGE);
    tma_load_3d(st + TILE, &p.tmB, bar, 128 * blk, c * L, bg);
    tma_load_3d(st + 2 * TILE, &p.tmB, bar, 128 * blk + 64, c * L, bg);
    tma_load_3d(st + 3 * TILE, &p.tmC, bar, 128 * blk, c * L, bg);
    tma_load_3d(st + 4 * TILE, &p.tmC, bar, 128 * blk + 64, c * L, bg);
    tma_load_3d(st, &p.tmU, bar, 0, c * L, bh);
    tma_load_3d(st + 5 * TILE, &p.tmdY, bar, 0, c * L, bh);
    tma_load_3d(st + 6 * TILE, &p.tmZ, bar, 0, c * 64, (int)set);
    tma_load_3d(st + 7 * TILE, &p.tmZ, bar, 64, c * 64, (int)set);
  };
  if (warp == 0) {
    tmem_alloc(&tmem_slot, B_TMEM_COLS);
  } else if (warp == 4 * NW) {
    chunk_scalars_at(sc_tab, Mb, Kb, (c_lo + n - 1) * L, T, lane);
  }
  if (tid == 0) issue_loads(0);   // (after the barriers were initialised by this same thread)

  auto block_sum2 = [&](float a, float b, float& oa, float& ob) {
    a = warp_sum(a); b = warp_sum(b);   // workers only
    bar_sync(1, NT);
    if (lane == 0) { s_red[2 * warp] = a; s_red[2 * warp + 1] = b; }
    bar_sync(1, NT);
    oa = 0.f; ob = 0.f;
#pragma unroll
    for (int k = 0; k < 4 * NW; ++k) { oa += s_red[2 * k]; ob += s_red[2 * k + 1]; }
  };

  // adjoint state of this thread's 8 oscillators, conjugated pairs (da, db):  dz = da - i db; pairs of neighbours
  f2 dza[4], dzb[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) { dza[e] = 0ull; dzb[e] = 0ull; }
  const bool last = seg == nseg - 1;
  if (worker && (last || p.fold)) {
    float ar = 0.f, ai = 0.f;
    if (p.dfinal) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const size_t o = ((size_t)bh * 64 + row) * D + 2 * (osc0 + 2 * e);
        const float4 g = *reinterpret_cast<const float4*>(p.dfinal + o), z = *reinterpret_cast<const float4*>(p.zfinal + o);
        ar += g.x * z.x + g.y * z.y + g.z * z.z + g.w * z.w;   // d_final * conj(z_final)
        ai += g.y * z.x - g.x * z.y + g.w * z.z - g.z * z.w;
        dza[e] = mk2(g.x, g.z); dzb[e] = mk2(-g.y, -g.w);
      }
    }
    if (last) {
      float sr, si;
      block_sum2(ar, ai, sr, si);
      if (tid == 0) p.anchor[set * nC + nC - 1] = make_float2(sr, si);
    }
  }
  if (worker && !last) {   // the adjoint at this segment's end: given, or folded from the later segments' contributions
    const size_t stride = (size_t)64 * 128 * nb;
    const float* src = p.seg + ((size_t)bh * p.nseg * 64 + row) * 128 * nb + 128 * blk + 64 * hf + d0;
    for (int s = p.fold ? p.nseg - 1 : seg; s >= (p.fold ? seg + 1 : seg); --s) {
      const float2 pi = p.fold ? p.seg_pi[(size_t)bh * p.nseg + s] : make_float2(0.f, 0.f);
      const f2 pr = dup2(pi.x), pim = dup2(pi.y), npim = dup2(-pi.y);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float4 a = reinterpret_cast<const float4*>(src + s * stride)[e];
        const float4 c = reinterpret_cast<const float4*>(src + s * stride + 8)[e];
        const f2 fa[2] = {mk2(a.x, a.y), mk2(a.z, a.w)}, fb[2] = {mk2(c.x, c.y), mk2(c.z, c.w)};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const f2 za = dza[2 * e + k], zb = dzb[2 * e + k];
          dza[2 * e + k] = fma2(npim, zb, fma2(pr, za, fa[k]));
          dzb[2 * e + k] = fma2(pim, za, fma2(pr, zb, fb[k]));
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;

  constexpr uint32_t ID_KK64 = make_idesc(64, 64, PK::fmt, 0, 0);
  constexpr uint32_t ID_MM64 = make_idesc(64, 64, PK::fmt, 1, 1);
  constexpr uint32_t ID_KM128 = make_idesc(64, 128, PK::fmt, 0, 1);
  constexpr uint32_t ID_MM128 = make_idesc(64, 128, PK::fmt, 1, 1);
  const uint32_t aQ = smem_u32(smem + B_OFF_Q), aKP = smem_u32(smem + B_OFF_KP),
                 aDYO = smem_u32(smem + B_OFF_DYO), aPD = smem_u32(smem + B_OFF_PD),
                 aDP = smem_u32(smem + B_OFF_DP), aDW = smem_u32(smem + B_OFF_DW),
                 aUE = smem_u32(smem + B_OFF_UE);
  bool ok = true;
  int issued_it = 0;   // issue lane: the last iteration whose loads were requested (iteration 0 by thread 0 above)
  auto wait_warp = [&](uint64_t* bar, uint32_t parity, int code) {  // a converged warp
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity) || wait_or_abort(bar, parity, wl, &s_abort, code)) != 0;
  };

  // ---- epilogue 5 of the chunk of iteration itp (run one iteration late): dz <- e^{l_end} dWv + dZ,
  // and the anchor S = <dz, z> of the boundary below that chunk ------------------------------------------
  float em_keep = 0.f;    // e^{l_end} of the chunk whose epilogue 5 is pending
  uint4 zv_keep[2];       // and this thread's cells of its Zv tiles (real parts, minus imaginary parts)
  zv_keep[0] = zv_keep[1] = make_uint4(0u, 0u, 0u, 0u);
  auto epilogue5 = [&](int itp, bool live) {
    live = live && wait_warp(&bar_mma[4], itp & 1, 16);
    tc_fence_after_sync();
    const f2 em = dup2(em_keep);
    f2 sr = 0ull, sa = 0ull, sb = 0ull;
    if (live) {
      uint32_t zi[16];
      tmem_ld_16x32bx2<16, 64>(tmem + lane_base + 384 + d0, zi);
      tmem_ld_wait();
      const uint32_t za[4] = {zv_keep[0].x, zv_keep[0].y, zv_keep[0].z, zv_keep[0].w};
      const uint32_t zb[4] = {zv_keep[1].x, zv_keep[1].y, zv_keep[1].z, zv_keep[1].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const f2 da = fma2(em, dza[e], mk2(__uint_as_float(zi[2 * e]), __uint_as_float(zi[2 * e + 1])));
        const f2 db = fma2(em, dzb[e], mk2(__uint_as_float(zi[8 + 2 * e]), __uint_as_float(zi[9 + 2 * e])));
        dza[e] = da; dzb[e] = db;
        const f2 a = PK::natural(za[e]), bq = PK::natural(zb[e]);   // z = a - i b ; dz = da - i db
        sr = fma2(da, a, sr); sr = fma2(db, bq, sr);                // dz conj(z)
        sa = fma2(da, bq, sa); sb = fma2(db, a, sb);
      }
    }
    const float2 r2 = un2(sr), a2 = un2(sa), b2 = un2(sb);
    // per-warp partial sums of the anchor; they are added up by finish_anchor() on the scalar warp after
    // named barrier 7 (no CTA-wide reduction here)
    const float ar = warp_sum(r2.x + r2.y), ai = warp_sum((a2.x + a2.y) - (b2.x + b2.y));
    if (lane == 0) { s_red[2 * warp] = live ? ar : 0.f; s_red[2 * warp + 1] = live ? ai : 0.f; }
  };
  auto finish_anchor = [&](int itp) {   // one thread of the scalar warp, after the barrier that follows epilogue5(itp)
    const int cp = c_lo + n - 1 - itp;
    if (cp <= 0) return;
    float sr = 0.f, si = 0.f;
#pragma unroll
    for (int k = 0; k < 4 * NW; ++k) { sr += s_red[2 * k]; si += s_red[2 * k + 1]; }
    p.anchor[set * nC + cp - 1] = make_float2(sr, si);
  };
  // ---- dWv tile of a chunk: dz rotated by the unit phase of Pi_end: (a,b) -> (ur a - ui b, ui a + ur b) ---------
  auto make_dwv = [&](const float* sc) {
    const f2 ur = dup2(sc[SC_TAIL + 1]), ui = dup2(sc[SC_TAIL + 2]), nui = dup2(-sc[SC_TAIL + 2]);
    uint8_t* dw = smem + B_OFF_DW + hf * TILE;
    uint32_t wa[4], wb[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const f2 a = dza[e], bq = dzb[e];
      dza[e] = fma2(nui, bq, mul2(ur, a));
      dzb[e] = fma2(ur, bq, mul2(ui, a));
      wa[e] = PK::pack2(dza[e]); wb[e] = PK::pack2(dzb[e]);
    }
    *reinterpret_cast<uint4*>(dw + cell0) = make_uint4(wa[0], wa[1], wa[2], wa[3]);
    *reinterpret_cast<uint4*>(dw + cell1) = make_uint4(wb[0], wb[1], wb[2], wb[3]);
  };

  for (int it = 0; it < n && ok; ++it) {
    const int t0 = (c_lo + n - 1 - it) * L;
    uint8_t* st = smem + (it & 1) * B_STAGE;
    uint8_t *tU = st, *tB = st + TILE, *tC = st + 3 * TILE, *tDY = st + 5 * TILE, *tZ = st + 6 * TILE;
    const float* sc = sc_tab + (it & 1) * SCW_B;
    const float4* rot = reinterpret_cast<const float4*>(sc);
    const float4* kcl = reinterpret_cast<const float4*>(sc + SC_KCL);
    if (warp == 4 * NW) {
      // scalars of the next (earlier) chunk; this warp meets the others only at the barrier that
      // ends the iteration
      // (it starts after the workers' first passes: global loads issued while every worker warp
      // bursts shared-memory traffic at the top of the iteration stalled the whole SM for about a
      // DRAM round trip; computing the table at the top from inputs requested an iteration ahead measured 10 %
      // slower for the same reason)
      bar_sync(2, NT + 64);   // the workers only arrive here (bar_arrive): they never wait for this warp
      if (it + 1 < n) chunk_scalars_at(sc_tab + ((it + 1) & 1) * SCW_B, Mb, Kb, t0 - L, T, lane);
      // the anchor of the previous chunk: a global store by a worker thread here would make that
      // thread's next proxy fence (epilogue 1) wait for the store, and every worker for that thread
      bar_sync(7, NT + 32);
      if (lane == 0 && it > 0 && s_abort == 0) finish_anchor(it - 1);
      __syncwarp();
    } else if (!worker) {
      // Issue warp (one lane): every MMA of this chunk, the TMA loads of the next (earlier) chunk and
      // the TMA stores of this chunk's outputs.  The workers never wait for this warp, only for the
      // commit barriers of the products they read: they arrive on named barriers 2 ("passes done")
      // and 4 ("epilogue 1 done") without waiting and move on.
      // K-major (kX) and MN-major (mX) base descriptors of every operand tile of this chunk
      const uint64_t kQ = make_desc(aQ, 16, 1024), mQ = make_desc(aQ, 8192, 1024);
      const uint64_t kKP = make_desc(aKP, 16, 1024), mKP = make_desc(aKP, 8192, 1024);
      const uint64_t kU = make_desc(smem_u32(tU), 16, 1024);
      const uint64_t kDY = make_desc(smem_u32(tDY), 16, 1024), mDY = make_desc(smem_u32(tDY), 8192, 1024);
      const uint64_t mZ = make_desc(smem_u32(tZ), 8192, 1024);
      const uint64_t kDP = make_desc(aDP, 16, 1024), mDP = make_desc(aDP, 8192, 1024);
      const uint64_t mPD = make_desc(aPD, 8192, 1024), mDYO = make_desc(aDYO, 8192, 1024), kDYO = make_desc(aDYO, 16, 1024);
      const uint64_t kDW = make_desc(aDW, 16, 1024), mDW = make_desc(aDW, 8192, 1024);
      const uint64_t kUE = make_desc(aUE, 16, 1024);
      bool go = elect_one() && s_abort == 0;
      if (go) do {
        // (1) products of raw tiles, as soon as the stage has landed
        if (!mbar_wait(&bar_tma[it & 1], (it >> 1) & 1, wl)) { report_timeout(20); s_abort = 1; go = false; break; }
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          // dS[t][s] = sum_p dY[t][p] U[s][p]            A: dY K-major, B: U K-major rows s
          umma(tmem + 64, desc_adv(kDY, 32 * k), desc_adv(kU, 32 * k), ID_KK64, k > 0);
        if (it + 1 < n) {   // next chunk's input tiles
          tma_store_wait_read();   // the stores of the previous chunk read the stage being refilled
          issue_loads(it + 1);
          issued_it = it + 1;
        }
      } while (false);
      __syncwarp();
      // (1b) P~, once Q and K' are rotated (the pass over dY and U is still running)
      bar_sync(5, NT + 32);
      if (go && s_abort == 0) {
        tc_fence_after_sync();
        // P~[t][s] = sum_d Q[t][d] K'[s][d]              A: Q K-major, B: K' K-major rows s
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t ko = (k >> 2) * TILE + (k & 3) * 32;
          umma(tmem + 0, desc_adv(kQ, ko), desc_adv(kKP, ko), ID_KK64, k > 0);
        }
        umma_commit(&bar_mma[0]);   // P~ and dS: epilogue 1 may start
      }
      __syncwarp();
      // (2) products of scaled tiles, once the workers' passes are done
      bar_sync(2, NT + 64);
      if (go && s_abort == 0) {
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          // dQ[t][d] = sum_p dYoff[t][p] Zv[p][d] (+ dP K' below)   A: dYoff K-major, B: Zv MN-major (rows = p)
          umma(tmem + 128, desc_adv(kDYO, 32 * k), desc_adv(mZ, 2048 * k), ID_KM128, k > 0);
      }
      __syncwarp();
      // (2b) once the workers have finished epilogue 5 of the previous chunk (the Zv tiles of the other
      // stage are free) and written this chunk's dWv
      bar_sync(6, NT + 32);
      if (go && s_abort == 0) {
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          // dX[s][d] = sum_p (e^{l_end-l_s} U[s][p]) dWv[p][d] (+ dP^T Q below)   A: Uee K-major, B: dWv MN-major
          umma(tmem + 256, desc_adv(kUE, 32 * k), desc_adv(mDW, 2048 * k), ID_KM128, k > 0);
      }
      __syncwarp();
      // (3) products of the masked tiles, once epilogue 1 has written Pdec and dP; ordered by the
      // epilogue that consumes them (dX, dQ, dU, dZ)
      bar_sync(4, NT + 32);
      if (go && s_abort == 0) do {
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          // dX[s][d] += sum_t dP[t][s] Q[t][d]         A: dP MN-major (rows = t), B: Q MN-major
          umma(tmem + 256, desc_adv(mDP, 2048 * k), desc_adv(mQ, 2048 * k), ID_MM128, 1);
        umma_commit(&bar_mma[1]);   // dX
#pragma unroll
        for (int k = 0; k < 4; ++k)
          // dQa[t][d] = sum_s dP[t][s] K'[s][d]        A: dP K-major, B: K' MN-major (rows = s)
          umma(tmem + 128, desc_adv(kDP, 32 * k), desc_adv(mKP, 2048 * k), ID_KM128, 1);
        umma_commit(&bar_mma[2]);   // dQ
#pragma unroll
        for (int k = 0; k < 4; ++k)
          // dUa[s][p] = sum_t Pdec[t][s] dY[t][p]        A: Pdec MN-major, B: dY MN-major
          umma(tmem + 0, desc_adv(mPD, 2048 * k), desc_adv(mDY, 2048 * k), ID_MM64, k > 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          // dUb[s][p] = sum_d K'[s][d] dWv[p][d]         A: K' K-major, B: dWv K-major rows p
          const uint32_t ko = (k >> 2) * TILE + (k & 3) * 32;
          umma(tmem + 64, desc_adv(kKP, ko), desc_adv(kDW, ko), ID_KK64, k > 0);
        }
        umma_commit(&bar_mma[3]);   // dU
#pragma unroll
        for (int k = 0; k < 4; ++k)
          // dZ[p][d]  = sum_t dYoff[t][p] Q[t][d]      A: dYoff MN-major, B: Q MN-major
          umma(tmem + 384, desc_adv(mDYO, 2048 * k), desc_adv(mQ, 2048 * k), ID_MM128, k > 0);
        umma_commit(&bar_mma[4]);   // dZ
        // (4) output tiles: the workers overwrite dead operand tiles of this stage in place (C with dB,
        // B with dC, dY with dU) and signal; one TMA store per tile writes full 128-byte rows.
        if (!mbar_wait(&bar_st[0], it & 1, wl)) { report_timeout(17); s_abort = 1; break; }
        tma_store_3d(&p.tmdB, tC, 128 * blk, t0, bh);
        tma_store_3d(&p.tmdB, tC + TILE, 128 * blk + 64, t0, bh);
        tma_store_commit();
        if (!mbar_wait(&bar_st[1], it & 1, wl)) { report_timeout(18); s_abort = 1; break; }
        tma_store_3d(&p.tmdC, tB, 128 * blk, t0, bh);
        tma_store_3d(&p.tmdC, tB + TILE, 128 * blk + 64, t0, bh);
        tma_store_commit();
        if (!mbar_wait(&bar_st[2], it & 1, wl)) { report_timeout(19); s_abort = 1; break; }
        tma_store_3d(&p.tmdU[blk], tDY, 0, t0, bh);
        tma_store_commit();
        // The next iteration's passes overwrite the dYoff and Q tiles that the dZ products (issued after
        // everything the workers wait for in this iteration) read: this lane sees them complete before it
        // joins the barrier that ends the iteration.
        if (!mbar_wait(&bar_mma[4], it & 1, wl)) { report_timeout(21); s_abort = 1; break; }
      } while (false);
      __syncwarp();
    } else {
    bool live = true;   // warp-uniform; cleared when a bounded wait expired: the rest of the chunk is skipped
    live = wait_warp(&bar_tma[it & 1], (it >> 1) & 1, 11);

    // ---- pass over B, C: Q, K', sum_n c conj(b).  A thread owns 8 oscillators of a row.
    if (live) {
      const int r = (tid >> 2) & 63, k = tid & 3, half = tid >> 8;
      const uint32_t o0 = half * TILE + sw128(r, 2 * k), o1 = half * TILE + sw128(r, 2 * k + 1);
      const uint4 b0 = *reinterpret_cast<const uint4*>(tB + o0), b1 = *reinterpret_cast<const uint4*>(tB + o1);
      const uint4 x0 = *reinterpret_cast<const uint4*>(tC + o0), x1 = *reinterpret_cast<const uint4*>(tC + o1);
      const float4 rt = rot[r];
      const uint32_t bw[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      const uint32_t cw[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
      uint32_t kr[4], ki[4], qr[4], qi[4];
      const f2 phr = dup2(rt.x), phi = dup2(rt.y), nphr = dup2(-rt.x);
      const f2 wr = dup2(rt.z), nwr = dup2(-rt.z), nwi = dup2(-rt.w);
      f2 sr = 0ull, sa = 0ull, sb = 0ull;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        f2 br, bi, cr, ci;
        PK::split(bw[2 * e], bw[2 * e + 1], br, bi);
        PK::split(cw[2 * e], cw[2 * e + 1], cr, ci);
        kr[e] = PK::pack2(fma2(bi, nwi, mul2(br, wr)));     // k' = conj(w b)
        ki[e] = PK::pack2(fma2(bi, nwr, mul2(br, nwi)));
        qr[e] = PK::pack2(fma2(ci, phi, mul2(cr, phr)));    // q = conj(c) phi
        qi[e] = PK::pack2(fma2(ci, nphr, mul2(cr, phi)));
        sr = fma2(cr, br, sr); sr = fma2(ci, bi, sr);       // c conj(b)
        sa = fma2(ci, br, sa); sb = fma2(cr, bi, sb);
      }
      *reinterpret_cast<uint4*>(smem + B_OFF_KP + o0) = make_uint4(kr[0], kr[1], kr[2], kr[3]);
      *reinterpret_cast<uint4*>(smem + B_OFF_KP + o1) = make_uint4(ki[0], ki[1], ki[2], ki[3]);
      *reinterpret_cast<uint4*>(smem + B_OFF_Q + o0) = make_uint4(qr[0], qr[1], qr[2], qr[3]);
      *reinterpret_cast<uint4*>(smem + B_OFF_Q + o1) = make_uint4(qi[0], qi[1], qi[2], qi[3]);
      const float2 r2 = un2(sr), a2 = un2(sa), b2 = un2(sb);
      float cbr = r2.x + r2.y, cbi = (a2.x + a2.y) - (b2.x + b2.y);
      cbr += __shfl_xor_sync(0xffffffffu, cbr, 1); cbi += __shfl_xor_sync(0xffffffffu, cbi, 1);
      cbr += __shfl_xor_sync(0xffffffffu, cbr, 2); cbi += __shfl_xor_sync(0xffffffffu, cbi, 2);
      if (k == 0) s_cb[half * 64 + r] = make_float2(cbr, cbi);
    }
    fence_async_smem();
    tc_fence_before_sync();
    bar_arrive(5, NT + 32);
    // ---- pass over dY, U: sigma_t = <dy_t, u_t>, dYoff = e^{l_t} dY, Ue = e^{l_end - l_t} U --------------
    if (live) {
      const int r = tid >> 3, ch = tid & 7;
      const uint32_t off = sw128(r, ch);
      const uint4 dv = *reinterpret_cast<const uint4*>(tDY + off);
      const uint4 uv = *reinterpret_cast<const uint4*>(tU + off);
      const uint32_t dw_[4] = {dv.x, dv.y, dv.z, dv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
      const float4 kc = kcl[r];
      const f2 et = dup2(kc.z), ee = dup2(kc.w);
      uint32_t o[4], ue[4];
      f2 s2 = 0ull;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const f2 dy2 = PK::natural(dw_[e]), u2 = PK::natural(uw[e]);
        s2 = fma2(dy2, u2, s2);
        o[e] = PK::pack2(mul2(et, dy2));
        ue[e] = PK::pack2(mul2(ee, u2));
      }
      *reinterpret_cast<uint4*>(smem + B_OFF_DYO + off) = make_uint4(o[0], o[1], o[2], o[3]);
      *reinterpret_cast<uint4*>(smem + B_OFF_UE + off) = make_uint4(ue[0], ue[1], ue[2], ue[3]);
      const float2 sg2 = un2(s2);
      float sg = sg2.x + sg2.y;
      sg += __shfl_xor_sync(0xffffffffu, sg, 4);
      sg += __shfl_xor_sync(0xffffffffu, sg, 2);
      sg += __shfl_xor_sync(0xffffffffu, sg, 1);
      if (ch == 0) s_sig[r] = sg;
    }
    fence_async_smem();
    tc_fence_before_sync();
    // no barrier among the workers here or at the end of the gap below: what a warp does next (epilogue 5
    // of the previous chunk, dWv, the decay factors) touches nothing the passes of another warp read or
    // write; the workers meet at the end of epilogue 1
    bar_arrive(2, NT + 64);      // the scalar and issue warps are told without being waited for
    live = live && s_abort == 0;
    live = __all_sync(0xffffffffu, live) != 0;
    // ---- in the shadow of the P~ MMAs: epilogue 5 of the previous iteration, then this chunk's dWv ------
    if (it > 0) epilogue5(it - 1, live);
    if (live) make_dwv(sc);
    em_keep = sc[SC_TAIL];
    fence_async_smem();
    tc_fence_before_sync();
    bar_arrive(6, NT + 32);      // dWv written, the previous dZ accumulator and Zv tiles released
    bar_arrive(7, NT + 32);      // anchor partial sums written: the scalar warp adds them up and stores

    // ---- MMA group 1 (issued by the look-ahead warp): P~ = Q K'^T, dS = dY U^T ------------------------
    // The waits and TMEM loads below are compiler barriers, so everything an epilogue reads from shared
    // memory is fetched by hand BEFORE the wait it would otherwise queue behind.
    float dec[4 * WB];   // causal decay factors of this thread's (row, column) cells, [hh][i][0..1]
    {
      // loads and exponentials are unconditional (a load under a condition is not speculated by the
      // compiler: eight serial branches, each with its own load-to-exp latency); the mask is a select
      float ls[2 * WB];
#pragma unroll
      for (int i = 0; i < WB; ++i) {
        const float2 l2 = *reinterpret_cast<const float2*>(sc + SC_L2 + cg * WC + 8 * i + 2 * cq);
        ls[2 * i] = l2.x; ls[2 * i + 1] = l2.y;
      }
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int R = hh ? rowB : rowA;
        const float lt = sc[SC_L2 + R];
#pragma unroll
        for (int i = 0; i < WB; ++i) {
          const int s0 = cg * WC + 8 * i + 2 * cq;
          const float e0 = ex2f(fminf(lt - ls[2 * i], 0.f)), e1 = ex2f(fminf(lt - ls[2 * i + 1], 0.f));
          dec[(hh * WB + i) * 2 + 0] = s0 < R ? e0 : 0.f;
          dec[(hh * WB + i) * 2 + 1] = s0 + 1 < R ? e1 : 0.f;
        }
      }
    }
    live = live && wait_warp(&bar_mma[0], it & 1, 12);
    tc_fence_after_sync();

    // ---- epilogue 1: decayed, strictly causal Pdec and dP as 16-bit tiles -------------------------------
    if (live) {
      uint32_t pr[4 * WB], ds[4 * WB];
      if (cg <= quad) {
        tmem_ld_16x256<WB>(tmem + lane_base + 0 + cg * WC, pr);
        tmem_ld_16x256<WB>(tmem + lane_base + 64 + cg * WC, ds);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int k = 0; k < 4 * WB; ++k) pr[k] = ds[k] = 0u;
      }
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int R = hh ? rowB : rowA;
#pragma unroll
        for (int i = 0; i < WB; ++i) {
          const float dec0 = dec[(hh * WB + i) * 2 + 0], dec1 = dec[(hh * WB + i) * 2 + 1];
          const uint32_t off = sw128(R, cg * WB + i) + 4 * cq;
          *reinterpret_cast<uint32_t*>(smem + B_OFF_PD + off) =
              PK::pack(dec0 * __uint_as_float(pr[4 * i + 2 * hh]), dec1 * __uint_as_float(pr[4 * i + 2 * hh + 1]));
          *reinterpret_cast<uint32_t*>(smem + B_OFF_DP + off) =
              PK::pack(dec0 * __uint_as_float(ds[4 * i + 2 * hh]), dec1 * __uint_as_float(ds[4 * i + 2 * hh + 1]));
        }
      }
    }
    fence_async_smem();
    tc_fence_before_sync();
    bar_sync(3, NT);
    bar_arrive(4, NT + 32);
    live = __all_sync(0xffffffffu, live && s_abort == 0) != 0;

    // ---- MMA group 2 (issued by the look-ahead warp, one commit per accumulator set) ------------------
    // operands of epilogues 3 and 2 (this thread's cells of the C, B and Q tiles and its row's scalars),
    // fetched while the products are still running
    uint4 cvv[2], bvv[2], qvv[2];
    cvv[0] = *reinterpret_cast<const uint4*>(tC + hf * TILE + cell0);
    cvv[1] = *reinterpret_cast<const uint4*>(tC + hf * TILE + cell1);
    bvv[0] = *reinterpret_cast<const uint4*>(tB + hf * TILE + cell0);
    bvv[1] = *reinterpret_cast<const uint4*>(tB + hf * TILE + cell1);
    qvv[0] = *reinterpret_cast<const uint4*>(smem + B_OFF_Q + hf * TILE + cell0);
    qvv[1] = *reinterpret_cast<const uint4*>(smem + B_OFF_Q + hf * TILE + cell1);
    const float sig = s_sig[row];
    const float4 rt = rot[row], kc4 = kcl[row];
    const f2 skr = dup2(sig * kc4.x), ski = dup2(sig * kc4.y), nski = dup2(-sig * kc4.y);   // sigma kc
    const uint32_t bw[8] = {bvv[0].x, bvv[0].y, bvv[0].z, bvv[0].w, bvv[1].x, bvv[1].y, bvv[1].z, bvv[1].w};
    live = live && wait_warp(&bar_mma[1], it & 1, 13);
    tc_fence_after_sync();

    // ---- epilogue 3 (first): dX -> dB, R = sum conj(b) dX ---------------------------------------------------------
    if (live) {
      uint32_t x[16];
      tmem_ld_16x32bx2<16, 64>(tmem + lane_base + 256 + d0, x);
      tmem_ld_wait();
      const uint32_t cw[8] = {cvv[0].x, cvv[0].y, cvv[0].z, cvv[0].w, cvv[1].x, cvv[1].y, cvv[1].z, cvv[1].w};
      const f2 wr = dup2(rt.z), nwr = dup2(-rt.z), nwi = dup2(-rt.w);
      f2 ra = 0ull, rb = 0ull, rc = 0ull, rd = 0ull;
      uint32_t o[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const f2 ga = mk2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1]));        // dX = ga - i gb
        const f2 gb = mk2(__uint_as_float(x[8 + 2 * e]), __uint_as_float(x[9 + 2 * e]));
        f2 cr, ci, br, bi;
        PK::split(cw[2 * e], cw[2 * e + 1], cr, ci);
        PK::split(bw[2 * e], bw[2 * e + 1], br, bi);
        ra = fma2(br, ga, ra); rb = fma2(bi, gb, rb);     // R += conj(b) dX = (br ga - bi gb) - i (br gb + bi ga)
        rc = fma2(br, gb, rc); rc = fma2(bi, ga, rc);
        // db = conj(w) dX + sigma conj(kc) c
        const f2 dbr = fma2(ci, ski, fma2(cr, skr, fma2(gb, nwi, mul2(ga, wr))));
        const f2 dbi = fma2(ci, skr, fma2(cr, nski, fma2(ga, nwi, mul2(gb, nwr))));
        PK::join(dbr, dbi, o[2 * e], o[2 * e + 1]);
      }
      rd = rb;
      *reinterpret_cast<uint4*>(tC + hf * TILE + cell0) = make_uint4(o[0], o[1], o[2], o[3]);   // dB over C, in place
      *reinterpret_cast<uint4*>(tC + hf * TILE + cell1) = make_uint4(o[4], o[5], o[6], o[7]);
      const float2 va = un2(ra), vb = un2(rd), vc = un2(rc);
      s_acc[(2 * 8 + 2 * cg + hf) * 64 + row] = (va.x + va.y) - (vb.x + vb.y);
      s_acc[(3 * 8 + 2 * cg + hf) * 64 + row] = -(vc.x + vc.y);
    }
    // the tile is complete once every worker warp has arrived; the issue warp then stores it
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar_st[0]);
    live = live && wait_warp(&bar_mma[2], it & 1, 14);
    tc_fence_after_sync();
    // ---- epilogue 2: dQ -> dC, <q,dq> ------------------------------------------------------------------
    if (live) {
      uint32_t x[16];
      tmem_ld_16x32bx2<16, 64>(tmem + lane_base + 128 + d0, x);
      tmem_ld_wait();
      const uint32_t qa[4] = {qvv[0].x, qvv[0].y, qvv[0].z, qvv[0].w}, qb[4] = {qvv[1].x, qvv[1].y, qvv[1].z, qvv[1].w};
      const f2 phr = dup2(rt.x), phi = dup2(rt.y), nphr = dup2(-rt.x);
      f2 ar = 0ull, aa = 0ull, ab = 0ull;
      uint32_t o[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const f2 dqr = mk2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1]));
        const f2 dqi = mk2(__uint_as_float(x[8 + 2 * e]), __uint_as_float(x[9 + 2 * e]));
        const f2 qr = PK::natural(qa[e]), qi = PK::natural(qb[e]);
        f2 br, bi;
        PK::split(bw[2 * e], bw[2 * e + 1], br, bi);
        ar = fma2(qr, dqr, ar); ar = fma2(qi, dqi, ar);       // conj(q) dq
        aa = fma2(qr, dqi, aa); ab = fma2(qi, dqr, ab);
        // dc = conj(dq) phi + sigma kc b
        const f2 dcr = fma2(bi, nski, fma2(br, skr, fma2(dqi, phi, mul2(dqr, phr))));
        const f2 dci = fma2(bi, skr, fma2(br, ski, fma2(dqi, nphr, mul2(dqr, phi))));
        PK::join(dcr, dci, o[2 * e], o[2 * e + 1]);
      }
      *reinterpret_cast<uint4*>(tB + hf * TILE + cell0) = make_uint4(o[0], o[1], o[2], o[3]);   // dC over B, in place
      *reinterpret_cast<uint4*>(tB + hf * TILE + cell1) = make_uint4(o[4], o[5], o[6], o[7]);
      const float2 va = un2(ar), vb = un2(aa), vc = un2(ab);
      s_acc[(0 * 8 + 2 * cg + hf) * 64 + row] = va.x + va.y;
      s_acc[(1 * 8 + 2 * cg + hf) * 64 + row] = (vb.x + vb.y) - (vc.x + vc.y);
    }
    // the tile is complete once every worker warp has arrived; the issue warp then stores it
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar_st[1]);
    // operands of epilogue 4: this thread's cells of the dY tile and its rows' scalars
    uint32_t dyc[2 * WB];
    float e4s[4];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int R = hh ? rowB : rowA;
      const float4 kc = kcl[R];
      const float2 cb0 = s_cb[R], cb1 = s_cb[64 + R];
      // diagonal term Re sum conj(c) kc b = Re(kc conj(sum c conj(b))); dU belongs to the whole row, so every column
      // block contributes the diagonal of its own columns
      e4s[2 * hh] = kc.w; e4s[2 * hh + 1] = kc.x * (cb0.x + cb1.x) + kc.y * (cb0.y + cb1.y);
#pragma unroll
      for (int i = 0; i < WB; ++i)
        dyc[hh * WB + i] = *reinterpret_cast<const uint32_t*>(tDY + sw128(R, cg * WB + i) + 4 * cq);
    }
    live = live && wait_warp(&bar_mma[3], it & 1, 15);
    tc_fence_after_sync();
    // ---- epilogue 4: dU ---------------------------------------------------------------------------------------
    if (live) {
      uint32_t ua[4 * WB], ub[4 * WB];
      tmem_ld_16x256<WB>(tmem + lane_base + 0 + cg * WC, ua);
      tmem_ld_16x256<WB>(tmem + lane_base + 64 + cg * WC, ub);
      tmem_ld_wait();
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int R = hh ? rowB : rowA;
        const float ee = e4s[2 * hh], dgv = e4s[2 * hh + 1];
#pragma unroll
        for (int i = 0; i < WB; ++i) {
          uint32_t* cell = reinterpret_cast<uint32_t*>(tDY + sw128(R, cg * WB + i) + 4 * cq);
          const float2 d2 = PK::unpack(dyc[hh * WB + i]);
          *cell = PK::pack(__uint_as_float(ua[4 * i + 2 * hh]) + ee * __uint_as_float(ub[4 * i + 2 * hh]) + dgv * d2.x,
                           __uint_as_float(ua[4 * i + 2 * hh + 1]) + ee * __uint_as_float(ub[4 * i + 2 * hh + 1]) + dgv * d2.y);   // dU over dY, in place
        }
      }
    }
    // the tile is complete once every worker warp has arrived; the issue warp then stores it
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar_st[2]);
    // (epilogue 5 of this chunk - the update of dz - runs in the next iteration, in the shadow of the
    // P~ MMAs; its inputs, the dZ accumulator and the Zv tiles of this stage, stay untouched until then)
    zv_keep[0] = *reinterpret_cast<const uint4*>(tZ + hf * TILE + cell0);   // for the deferred epilogue 5 of this chunk
    zv_keep[1] = *reinterpret_cast<const uint4*>(tZ + hf * TILE + cell1);
    bar_sync(1, NT);   // the partial sums written by epilogues 2 and 3 are read by other threads below
    // the proxy fence for this iteration's shared-memory accesses goes BEFORE the global stores
    // below (the code after them touches no tile)
    fence_async_smem();
    // ---- per-token scalars of this chunk ---------------------------------------------------------------------
    if (live && tid < 64 && t0 + tid < T) {
      const int t = tid;
      float Ar = 0.f, Ai = 0.f, Rr = 0.f, Ri = 0.f;
#pragma unroll
      for (int k = 0; k < 2 * NW; ++k) {
        Ar += s_acc[(0 * 8 + k) * 64 + t]; Ai += s_acc[(1 * 8 + k) * 64 + t];
        Rr += s_acc[(2 * 8 + k) * 64 + t]; Ri += s_acc[(3 * 8 + k) * 64 + t];
      }
      const float4 r4 = rot[t];
      const size_t o = set * T + t0 + t;
      p.dg[o] = make_float2(r4.x * Rr - r4.y * Ri, r4.x * Ri + r4.y * Rr);              // phi R
      p.sterm[o] = make_float2(Ar - (r4.z * Rr + r4.w * Ri), Ai - (r4.z * Ri - r4.w * Rr));   // A - conj(w) R
      const float sg = s_sig[t];
      p.dkcd[o] = make_float2(sg * (s_cb[t].x + s_cb[64 + t].x), sg * (s_cb[t].y + s_cb[64 + t].y));
    }
    tc_fence_before_sync();
    }  // worker
    __syncthreads();
    if (s_abort) { ok = false; break; }
  }

  if (ok && worker) epilogue5(n - 1, true);
  __syncthreads();
  ok = ok && s_abort == 0;
  if (ok && tid == 128 * NW) finish_anchor(n - 1);   // (of the segment before this one)
  if (ok && p.dinit && worker && c_lo == 0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = un2(dza[e]), c = un2(dzb[e]);
      *reinterpret_cast<float4*>(p.dinit + ((size_t)bh * 64 + row) * D + 2 * (osc0 + 2 * e)) = make_float4(a.x, -c.x, a.y, -c.y);
    }
  }
  // Unwind: nothing of this CTA may still be in flight when shared memory and TMEM are released.  The
  // issue lane started every asynchronous operation (but for the loads of the first iteration), so it
  // drains them: after an expired wait the loads of the last two requested iterations (their barriers,
  // default long limit) and, always, every tcgen05.mma issued so far (one more commit) and its TMA stores.
  if (warp == 4 * NW + 1 && lane == 0) {
    if (s_abort)
      for (int ii = issued_it > 0 ? issued_it - 1 : 0; ii <= issued_it; ++ii) mbar_wait(&bar_tma[ii & 1], (ii >> 1) & 1);
    umma_commit(&bar_drain);
    mbar_wait(&bar_drain, 0);
    tma_store_wait_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, B_TMEM_COLS);
}

// What follows the sweep, in one launch: the blocks are dealt out to three independent jobs.
struct TcPostParams {
  const float *M, *K;
  const float2 *dg, *sterm, *dkcd, *anchor, *dg_boundary;
  float *dM, *dK;
  const void *per_head_b, *per_head_c;   // grouped B / C: dB and dC per head, or null
  void *dB, *dC;
  void* dU;
  const void* dU2;                       // two column blocks: the second one's part of dU, or null
  int BH, heads, groups, T, nC, D;
  unsigned fin_blocks, red_blocks;       // job 1, job 2; the rest is job 3
};

// Job 1: dM and dK from the per-token scalars.  One warp per chunk (two tokens per lane); chunks are
// independent given the anchors.  The scalars are linear in the state columns: with two column blocks the sets of
// both are added up.
template <int NB>
__device__ __forceinline__ void post_scalars(const TcPostParams& p, unsigned block) {
  const float2 *dg = p.dg, *sterm = p.sterm, *dkcd = p.dkcd, *anchor = p.anchor, *dg_boundary = p.dg_boundary;
  const float *M = p.M, *K = p.K;
  const int T = p.T, nC = p.nC, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned per = (nC + 3) / 4;
  const size_t bh = block / per, BH = p.BH;
  const int c = (int)(block % per) * 4 + warp;
  if (c >= nC) return;
  auto sum_at = [&](const float2* a, size_t len, size_t i) {
    float2 v = a[bh * len + i];
    if (NB == 2) { const float2 w = a[(BH + bh) * len + i]; v.x += w.x; v.y += w.y; }
    return v;
  };
  const int tA = c * 64 + 2 * lane, tB = tA + 1;
  float2 sA = make_float2(0.f, 0.f), sB = sA, gA = sA, gB = sA, gP = sA, kA = sA, kB = sA;
  float2 mA = make_float2(1.f, 0.f), mB = mA;
  float4 k4A = make_float4(0.f, 0.f, 0.f, 0.f), k4B = k4A;
  if (tA < T) {
    sA = sum_at(sterm, T, tA); gA = sum_at(dg, T, tA); kA = sum_at(dkcd, T, tA);
    mA = reinterpret_cast<const float2*>(M)[bh * T + tA];
    k4A = reinterpret_cast<const float4*>(K)[bh * T + tA];
    // the prev-tap of token t belongs to the merged coefficient of token t-1; for t = 0 that is the
    // pending tap of the token before the sequence (carried B_prev / U_prev), if there is one
    if (tA > 0) gP = sum_at(dg, T, tA - 1);
    else if (dg_boundary) gP = dg_boundary[bh];
  }
  if (tB < T) {
    sB = sum_at(sterm, T, tB); gB = sum_at(dg, T, tB); kB = sum_at(dkcd, T, tB);
    mB = reinterpret_cast<const float2*>(M)[bh * T + tB];
    k4B = reinterpret_cast<const float4*>(K)[bh * T + tB];
  }
  const float2 an = sum_at(anchor, nC, c);
  // inclusive suffix sums over the chunk
  float xr = sA.x + sB.x, xi = sA.y + sB.y;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float yr = __shfl_down_sync(0xffffffffu, xr, o), yi = __shfl_down_sync(0xffffffffu, xi, o);
    if (lane + o < 32) { xr += yr; xi += yi; }
  }
  const float SAr = an.x + xr, SAi = an.y + xi;            // S at token tA
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int t = q ? tB : tA;
    if (t >= T) continue;
    const float Sr = q ? SAr - sA.x : SAr, Si = q ? SAi - sA.y : SAi;
    const float mr = q ? mB.x : mA.x, mi = q ? mB.y : mA.y;
    const float den = mr * mr + mi * mi;
    const float4 k4 = q ? k4B : k4A;
    const float2 gp = q ? gA : gP, gc = q ? gB : gA, kd = q ? kB : kA;
    // x / conj(m) = x m / |m|^2
    const float dmr = (Sr * mr - Si * mi) / den, dmi = (Sr * mi + Si * mr) / den;
    const float dkpr = (gp.x * mr - gp.y * mi) / den, dkpi = (gp.x * mi + gp.y * mr) / den;
    // q = kp / m ; dm -= conj(q) dkp
    const float qr = (k4.x * mr + k4.y * mi) / den, qi = (k4.y * mr - k4.x * mi) / den;
    float2* dMo = reinterpret_cast<float2*>(p.dM) + bh * T + t;
    *dMo = make_float2(dmr - (qr * dkpr + qi * dkpi), dmi - (qr * dkpi - qi * dkpr));
    *reinterpret_cast<float4*>(p.dK + (bh * T + t) * 4) = make_float4(dkpr, dkpi, gc.x + kd.x, gc.y + kd.y);
  }
}

// Job 2, grouped B / C: the sweep leaves dB and dC per head (16-bit); here the heads of a group are added up in
// float32 and cast once (the reference reduces in float32 as well:
// slinoss/ops/v2x2ssd/cute/kernels/bwd/__init__.py:548-563).  One thread per 16-byte piece of an output row.
template <typename TIn>
__device__ __forceinline__ void post_group_reduce(const TcPostParams& p, unsigned block) {
  const int hpg = p.heads / p.groups, ppr = p.D / 8;
  const size_t pieces = (size_t)(p.BH / p.heads) * p.groups * p.T * ppr;
  const size_t i = (size_t)block * 128 + threadIdx.x;   // piece index over (batch*groups, T, D / 8)
  if (i >= pieces) return;
  const size_t row = i / ppr, piece = i % ppr;
  const size_t bgi = row / p.T, t = row % p.T;
  const size_t bh0 = bgi / p.groups * p.heads + bgi % p.groups * hpg;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const TIn* src = reinterpret_cast<const TIn*>(which ? p.per_head_c : p.per_head_b) + (bh0 * p.T + t) * p.D + piece * 8;
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
#pragma unroll 4
    for (int hh = 0; hh < hpg; ++hh) {
      float v[8];
      load16<TIn>(src + (size_t)hh * p.T * p.D, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += v[k];
    }
    store16<TIn>(reinterpret_cast<TIn*>(which ? p.dC : p.dB) + (bgi * p.T + t) * p.D + piece * 8, acc);
  }
}

// Job 3, two column blocks: dU += the second block's part (summed in float32)
template <typename TIn>
__device__ __forceinline__ void post_add_du(const TcPostParams& p, unsigned block) {
  const size_t i = ((size_t)block * 128 + threadIdx.x) * 8;
  if (i >= (size_t)p.BH * p.T * 64) return;
  TIn* a = reinterpret_cast<TIn*>(p.dU) + i;
  float x[8], y[8];
  load16<TIn>(a, x);
  load16<TIn>(reinterpret_cast<const TIn*>(p.dU2) + i, y);
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] += y[k];
  store16<TIn>(a, x);
}

template <typename TIn, int NB>
__global__ void __launch_bounds__(128) scan_tc_bwd_post_kernel(TcPostParams p) {
  const unsigned b = blockIdx.x;
  if (b < p.fin_blocks) post_scalars<NB>(p, b);
  else if (b < p.fin_blocks + p.red_blocks) post_group_reduce<TIn>(p, b - p.fin_blocks);
  else if (NB == 2) post_add_du<TIn>(p, b - p.fin_blocks - p.red_blocks);
}

// Carried taps: the sequence starts from  W_{-1} = z_{-1} + u_prev (x) (X b_prev),  X = kp_0 / m_0.  Given
// D = the adjoint of W_{-1} (what the sweep leaves as d_initial), per (batch, head):
//     v[n]      = sum_p u_prev[p] D[p,n]
//     dB_prev  += conj(X) v            (summed over the heads of a group, float32, cast once)
//     dU_prev[p] = Re sum_n conj(X b_prev[n]) D[p,n]
//     dX        = sum_n conj(b_prev[n]) v[n]     -> scan_tc_bwd_post_kernel turns it into dkp_0 and its part of dm_0
// (reference: slinoss/ops/v2x2ssd/cute/autograd.py:269-276 returns these as dB_prev / dU_prev).
// One CTA of 256 threads per (batch, group); thread j < 2N owns the interleaved lane j of B_prev.
template <typename TIn>
__global__ void __launch_bounds__(256) scan_tc_bwd_boundary_kernel(const float* __restrict__ D,
                                                                   const TIn* __restrict__ Bprev,
                                                                   const TIn* __restrict__ Uprev,
                                                                   const float* __restrict__ M,
                                                                   const float* __restrict__ K,
                                                                   TIn* __restrict__ dBprev, TIn* __restrict__ dUprev,
                                                                   float2* __restrict__ dg_boundary, int heads,
                                                                   int groups, int T, int N) {
  __shared__ float s_v[256], s_b[256], s_u[64], s_red[16];
  const int bg = blockIdx.x, b = bg / groups, g = bg % groups, hpg = heads / groups;
  const int j = threadIdx.x, lane = j & 31, warp = j >> 5, W = 2 * N;
  s_b[j] = j < W ? to_f32(Bprev[(size_t)bg * W + j]) : 0.f;
  float acc_db = 0.f;   // this lane of dB_prev, summed over the heads of the group
  for (int hh = 0; hh < hpg; ++hh) {
    const size_t bh = (size_t)b * heads + g * hpg + hh;
    const float* Dh = D + bh * 64 * W;
    float xr, xi;   // X = kp_0 / m_0
    pending_tap(M + bh * T * 2, K + bh * T * 4, xr, xi);
    __syncthreads();   // s_u, s_v of the previous head are no longer read
    if (j < 64) s_u[j] = to_f32(Uprev[bh * 64 + j]);
    __syncthreads();
    float v = 0.f;
    if (j < W) {
#pragma unroll 8
      for (int p = 0; p < 64; ++p) v += s_u[p] * Dh[p * W + j];
    }
    s_v[j] = v;
    __syncthreads();
    // conj(X) v on the (re, im) pair this lane belongs to
    const float vr = s_v[j & ~1], vi = s_v[j | 1];
    acc_db += (j & 1) ? (xr * vi - xi * vr) : (xr * vr + xi * vi);
    // dX = sum_n conj(b[n]) v[n]: lane pairs contribute (re: br vr + bi vi, im: br vi - bi vr)
    float cr = 0.f, ci = 0.f;
    if (!(j & 1)) {
      const float br = s_b[j], bi = s_b[j + 1];
      cr = br * vr + bi * vi;
      ci = br * vi - bi * vr;
    }
    cr = warp_sum(cr); ci = warp_sum(ci);
    if (lane == 0) { s_red[2 * warp] = cr; s_red[2 * warp + 1] = ci; }
    // dU_prev[p] = Re sum_n conj(X b[n]) D[p,n]   (a warp takes eight rows)
    if (dUprev) {
      for (int p = warp; p < 64; p += 8) {
        float du = 0.f;
        for (int n = lane; n < N; n += 32) {
          const float yr = xr * s_b[2 * n] - xi * s_b[2 * n + 1], yi = xr * s_b[2 * n + 1] + xi * s_b[2 * n];   // X b
          const float2 d2 = *reinterpret_cast<const float2*>(Dh + p * W + 2 * n);
          du += yr * d2.x + yi * d2.y;
        }
        du = warp_sum(du);
        if (lane == 0) dUprev[bh * 64 + p] = from_f32<TIn>(du);
      }
    }
    __syncthreads();
    if (j == 0) {
      float sr = 0.f, si = 0.f;
      for (int k = 0; k < 8; ++k) { sr += s_red[2 * k]; si += s_red[2 * k + 1]; }
      dg_boundary[bh] = make_float2(sr, si);
    }
  }
  if (dBprev && j < W) dBprev[(size_t)bg * W + j] = from_f32<TIn>(acc_db);
}
