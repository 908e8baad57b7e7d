// The GEMM of fb_vtc.cuh with one work item per CTA and K split over a cluster: trees, and short prompts, whose tiles alone would leave most
// SMs without work.
//
// One tile of up to 64 tokens (tree verification) is sized so that TWO CTAs share an SM: at most 113 KB of shared memory, 256 tensor-memory
// columns and 72 registers a thread. A verify pass is a chain of short dependent launches (4 to 6 us of work each); with programmatic
// dependent launch the next GEMM's CTAs become resident while the previous kernel still runs, so barrier set-up, the tensor-memory
// allocation, the weight ring and the first dequantised stages are done before the activations exist. The 200 KB form left every launch to
// ramp up after its predecessor had gone: QKV / O / gate-up / down took 9.7 / 9.4 / 11.1 / 12.1 us at 26 tokens of the 3B shape. The 128-token
// tiles of a prompt take a whole SM; what their long K needs is the split (64 groups of the down projection in a row are 22 us).
//
// One work item (row block of a token tile) per CTA, K split over a cluster of up to eight CTAs (four at 128 tokens). Warps: 0 weight
// producer, 1 MMA issue, 2..4 activations (tensor copies, or the fp16 conversion of the attention output), 5 code warm-up (trees), 6..13
// dequantise, then epilogue.
#pragma once
#include "fb_vtc.cuh"

namespace fb {

constexpr int kTlThreads = 448;
template <int NT, bool HZ>
struct VtlSmem {
  static constexpr int REC = tc_rec_bytes(HZ);
  static constexpr int NS = NT == 128 ? (HZ ? 5 : 6) : (NT == 64 && HZ ? 2 : 3);      // dequantised groups (64 tensor-memory columns each)
  static constexpr int NB = NT == 16 ? 8 : (NT == 32 ? 5 : (NT == 64 ? 3 : 4));       // activation stages
  static constexpr int NRAW = NT == 16 ? 7 : (NT == 32 ? 5 : (NT == 64 || HZ ? 3 : 4)); // raw int4 groups
  static constexpr int BSTAGE = NT * 256;
  static constexpr int B = 0;
  static constexpr int RAW = B + NB * BSTAGE;
  static constexpr int ND = 8;                                     // barriers that retire groups: see VtcSmem::ND
  static_assert(ND >= NB && ND >= NS, "a retired group must not be overtaken by the next one on its barrier");
  static constexpr int YS = RAW + NRAW * REC;                      // K splits: [source rank][tokens][128 rows] fp32
  static constexpr int BAR = YS + NT * 512;
  static constexpr int TOTAL = BAR + 512 + 1024;
  static constexpr int CTAS = NT == 128 ? 1 : 2;                   // per SM
  static_assert(TOTAL <= (CTAS == 2 ? 113 : 227) * 1024, "shared memory of an SM");
  static_assert(NT < 128 || 8 * kTcEpiBytes <= NB * BSTAGE, "the epilogue of 128 tokens stages in the dead activation ring");
  static constexpr int T_A = NT, T_AZ = T_A + NS * 64, TCOLS = 512 / CTAS;
  static_assert(T_AZ + (HZ ? NS * 8 : 0) <= TCOLS, "tensor memory columns");
};

// after a failure: the copies and MMAs in flight (see drain_phase); out of line, a healthy launch never comes here
template <int NRAW, int NS, int NB, int ND>
inline __device__ __noinline__ void tl_drain(uint64_t* bars, volatile int* s_issued, bool exchange) {
  uint64_t *raw_full = bars, *b_full = bars + 2 * NRAW + NS, *done = b_full + NB, *acc_full = done + ND;
  const int n = s_issued[1];
  drain_ring<NRAW>(raw_full, s_issued[0]);
  drain_ring<NB>(b_full, s_issued[2]);
  if (n) drain_phase(n > 0 ? &done[(n - 1) % ND] : acc_full, n > 0 ? ((n - 1) / ND) & 1 : 0);
  // sums on their way here or from here: a neighbour that gave up before it sent any leaves the barrier open, and every neighbour is behind the
  // cluster barrier by now, so what is under way lands within microseconds
  if (exchange)
#pragma unroll 1
    for (int i = 0; i < 200 && !mbar_test(acc_full + 1, 0); i++) __nanosleep(1000);
  __syncwarp();
}

template <int NT, int EPI, bool HZ>
__global__ void __launch_bounds__(kTlThreads, NT == 128 ? 1 : 2) v_gemm_tl(const __grid_constant__ VtcParams P) {
  using S = VtlSmem<NT, HZ>;
  constexpr bool ASYNC = NT < 64;                                // how a split's sums travel, see below
  constexpr int NRAW = S::NRAW, NS = S::NS, NB = S::NB, ND = S::ND, REC = S::REC, HC = NT / 2;
  extern __shared__ __align__(1024) uint8_t tsm_raw[];
  uint8_t* tsm = tsm_raw + ((1024u - (smem_u32(tsm_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(tsm + S::BAR);
  uint64_t *raw_full = bars, *raw_empty = bars + NRAW, *a_full = bars + 2 * NRAW, *b_full = a_full + NS, *done = b_full + NB,
           *acc_full = done + ND;
  uint64_t* xbar = acc_full + 1;                                // K splits: the cluster's sums of this CTA's tokens have arrived
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(xbar + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  volatile int* s_issued = s_abort + 1;                          // [3] copies or MMA groups (-1: all) that warps 0, 1, 2 have issued
  float* ys = reinterpret_cast<float*>(tsm + S::YS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < NRAW; i++) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 8); }
    for (int i = 0; i < NS; i++) mbar_init(&a_full[i], 8);
    for (int i = 0; i < NB; i++) mbar_init(&b_full[i], 1);
    for (int i = 0; i < ND; i++) mbar_init(&done[i], 1);
    mbar_init(acc_full, 1);
    mbar_init(xbar, 1);
    *s_abort = s_issued[2] = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(S::TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  pdl_trigger();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  WaitCtl wc{P.status, s_abort, P.spin_limit};
  const int ns = P.nsplit, lg = 31 - __clz(ns), rank = (int)blockIdx.x & (ns - 1), item = (int)blockIdx.x >> lg, G = P.K / 128;
  // a prompt may have several token tiles (NT = 128 only)
  const int nrb = (P.rows + kTcRowBlock - 1) / kTcRowBlock, rb = NT == 128 ? item % nrb : item, tok0 = NT == 128 ? item / nrb * P.ntok : 0,
            tend = NT == 128 ? min(P.M, tok0 + P.ntok) : P.M;
  const int g0 = G * rank >> lg, ng = (G * (rank + 1) >> lg) - g0;           // this CTA's groups (ng >= 1)
  const bool split = NT == 128 || ns > 1;                        // 128-token tiles come here only to be split
  const int TPR = NT >> lg;                                      // splits: this CTA finishes tokens [rank * TPR, (rank + 1) * TPR) of the tile
  if (split) {
    if (ASYNC && tid == 0) mbar_expect_tx(xbar, (uint32_t)(max(0, min(TPR, P.M - rank * TPR)) * ns * 512));
    cluster_arrive();                                            // the neighbours' shared memory exists, and expects, from here on
    cluster_wait();
  }
  const uint8_t* blk = P.w + (size_t)rb * tc_block_bytes(P.K, HZ);
  bool ok = true;

  if (warp == 0) {
    // ---------------- producer: the groups' records (weights do not depend on the previous kernel)
    if (lane == 0) {
      Ring<NRAW> r;
      int gi = 0;
      for (; gi < ng; gi++, r.next()) {
        ok = mbar_wait(&raw_empty[r.i], r.lap ^ 1u, wc, W_EMPTY, 2);
        if (!ok) break;
        mbar_expect_tx(&raw_full[r.i], REC);
        bulk_g2s(tsm + S::RAW + r.i * REC, blk + (size_t)(g0 + gi) * REC, REC, &raw_full[r.i]);
      }
      s_issued[0] = gi;
    }
  } else if (warp == 1) {
    // ---------------- MMA issue
    const uint32_t idesc = (1u << 4) | ((uint32_t)(P.ntok >> 3) << 17) | ((128u >> 4) << 24);      // fp16 x fp16 -> fp32
    Ring<NS> rs;
    Ring<NB> rb_;
    Ring<ND> rd;
    int gi = 0;
    for (; gi < ng; gi++, rs.next(), rb_.next(), rd.next()) {
      bool now = mbar_try(&a_full[rs.i], rs.lap);
      now = mbar_try(&b_full[rb_.i], rb_.lap) && now;
      if (!now) ok = mbar_wait(&a_full[rs.i], rs.lap, wc, W_FULL, 4) && mbar_wait(&b_full[rb_.i], rb_.lap, wc, W_FULL, 4);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t ta = tmem + S::T_A + rs.i * 64, tz = tmem + S::T_AZ + rs.i * 8;
        const uint64_t db0 = tc_desc(smem_u32(tsm + S::B + rb_.i * S::BSTAGE));
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint64_t db = db0 + (uint64_t)(((k >> 2) * (NT * 128) + (k & 3) * 32) >> 4);
          tc_mma_ts(tmem, ta + k * 8, db, idesc, (gi || k) ? 1u : 0u);
          if (HZ) tc_mma_ts(tmem, tz, db, idesc, 1u);
        }
        tc_commit(gi == ng - 1 ? acc_full : &done[rd.i]);         // nobody waits for the last group's stages
      }
      __syncwarp();
    }
    if (lane == 0) s_issued[1] = gi < ng ? gi : -1;
  } else if (warp < 5) {
    // ---------------- activations (the previous kernel's output). Token rows past M only feed accumulator columns that nobody reads.
    if (NT < 128 && EPI == EPI_RESID && P.xbf) {
      // the attention output in bf16: each of the three warps converts every third group to fp16 times the token's power of two
      pdl_wait();
      float fm[2];
#pragma unroll
      for (int k = 0; k < 2; k++) fm[k] = 32 * k + lane < P.M ? pow2_for(__uint_as_float(__ldcg(P.amax + 32 * k + lane))).x : 0.f;
      const int c16 = lane & 15;
      for (int li = warp - 2; li < ng; li += 3) {
        ok = li < NB || __all_sync(0xffffffffu, mbar_wait(&done[(li - NB) % ND], ((li - NB) / ND) & 1, wc, W_EMPTY, 8));
        if (!ok) break;
        uint8_t* dst = tsm + S::B + (li % NB) * S::BSTAGE + (c16 >> 3) * (NT * 128);
        const uint16_t* src = P.xbf + (size_t)(g0 + li) * 128 + c16 * 8;
#pragma unroll 1                                               // unrolled, the loads of all tokens at once spill: 26 / 61 tokens 2116 / 2735 us, so 2079 / 2637
        for (int k0 = 0; k0 < NT / 2; k0 += 8) {
          uint4 v[8];
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const int m = (lane >> 4) + 2 * (k0 + k);
            v[k] = m < P.M ? __ldcg(reinterpret_cast<const uint4*>(src + (size_t)m * P.K)) : make_uint4(0, 0, 0, 0);
          }
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const int m = (lane >> 4) + 2 * (k0 + k);
            const float f = __shfl_sync(0xffffffffu, k0 + k < 16 ? fm[0] : fm[1], m & 31);
            *reinterpret_cast<uint4*>(dst + m * 128 + (((c16 & 7) ^ (m & 7)) << 4)) =
                make_uint4(f16x2_scaled(v[k].x, f), f16x2_scaled(v[k].y, f), f16x2_scaled(v[k].z, f), f16x2_scaled(v[k].w, f));
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_full[li % NB]);
      }
    } else if (warp == 2) {
      pdl_wait();
      if (lane == 0) {
        Ring<NB> r;
        int gi = 0;
        for (; gi < ng; gi++, r.next()) {
          ok = gi < NB || mbar_wait(&done[(gi - NB) % ND], ((gi - NB) / ND) & 1, wc, W_EMPTY, 8);    // group gi - NB has retired
          if (!ok) break;
          mbar_expect_tx(&b_full[r.i], S::BSTAGE);
          uint8_t* dst = tsm + S::B + r.i * S::BSTAGE;
          tma_load_2d(dst, &P.xmap, (g0 + gi) * 128, tok0, &b_full[r.i]);
          tma_load_2d(dst + NT * 128, &P.xmap, (g0 + gi) * 128 + 64, tok0, &b_full[r.i]);
        }
        s_issued[2] = gi;
      }
    }
  } else if (NT < 128 || warp > 5) {
    // ---------------- dequantise: thread = (row of the block = TMEM lane, half of the group's columns), then epilogue: thread = (row,
    // half of the tokens). Warp 5 walks through the epilogue first, with every store and remote write switched off, so that its
    // instructions are in the cache when the sums arrive: the code of a dozen kernels passes through that cache every layer, and cold
    // the QKV epilogue took 3.3 us for what is 0.4 us of work.
    constexpr bool STAGED = NT == 128 && (EPI == EPI_RESID || EPI == EPI_SWIGLU);
    constexpr int CH = STAGED ? 16 : 4;
    const int quad = warp & 3, row = quad * 32 + lane, half = warp >= 10;
    const uint32_t tq = tmem + ((uint32_t)(quad * 32) << 16);
    const int* trailer = reinterpret_cast<const int*>(blk + (size_t)G * REC);
    const bool fast = !HZ && __ldg(trailer + kTcRowBlock) != 0;
    const int lgT = 31 - __clz(TPR), HT = split ? TPR >> 1 : HC;
    const int srow = rb * 128 + row, th0 = tok0 + (split ? rank * TPR : 0) + half * HT, the = min(tend, th0 + HT);
    TcOperands<EPI, STAGED ? 1 : CH> pre;
    TcStaged<EPI> staged;
    TcFactors<EPI> fac;
    auto fetch = [&]() {                                         // what the epilogue reads, requested while the last groups run
      pdl_wait();
      if constexpr (STAGED) staged.fetch(P, srow - lane, th0, the, lane);
      else pre.fetch(P, srow, th0, the);
      fac.fetch(P, th0, the, lane);
    };
    pre.fetch(P, srow, 0, 0);                                    // nothing: defined values for the walk-through
    fac.fetch(P, 0, 0, lane);
    const float rf = __int_as_float(__ldg(trailer + row));
    const uint32_t tlane = tq + half * HC, mine = smem_u32(ys) + (uint32_t)(rank * TPR * 128 + row) * 4;
    const float* yw = ys + half * HT * 128 + row;
    Ring<NRAW> rr;
    Ring<NS> rs;
    int gi = 0;
    const bool real = warp > 5;
    const int gend = real ? ng : 0, tlast = real ? the : th0, push_end = real ? tend - tok0 : 0;
#pragma unroll 1
    for (; gi < gend; gi++, rr.next(), rs.next()) {
      if (gi == NS) fetch();                                   // the first groups are ready; everything later needs the activations
      uint64_t* freed = &done[(gi - NS) & (ND - 1)];             // the stage's previous group has retired
      const uint32_t fpar = ((gi - NS) / ND) & 1;
      bool now = mbar_try(&raw_full[rr.i], rr.lap);
      if (gi >= NS) now = mbar_try(freed, fpar) && now;
      if (!now) ok = mbar_wait(&raw_full[rr.i], rr.lap, wc, W_FULL, 5) && (gi < NS || mbar_wait(freed, fpar, wc, W_EMPTY, 6));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint8_t* rec = tsm + S::RAW + rr.i * REC;
      const uint32_t raw = smem_u32(rec) + (uint32_t)row * 4 + half * 4096;
      const __half2 sc = __half2half2(reinterpret_cast<const __half*>(rec + 8192)[row]);
      uint32_t v[32];
      if (!HZ && fast) {
        const __half2 sh = __hmul2(sc, tc_as_h2(0x2C002C00u)), off = __hmul2(sc, tc_as_h2(0x80088008u));      // S / 16, -8 S 2^-24
#pragma unroll
        for (int q8 = 0; q8 < 8; q8++) {
          const uint32_t wv = lds32(raw + q8 * 512), wh = wv >> 8;
          v[4 * q8] = tc_cvt_fast(wv & 0x000F000Fu, sc, off); v[4 * q8 + 1] = tc_cvt_fast(wv & 0x00F000F0u, sh, off);
          v[4 * q8 + 2] = tc_cvt_fast(wh & 0x000F000Fu, sc, off); v[4 * q8 + 3] = tc_cvt_fast(wh & 0x00F000F0u, sh, off);
        }
      } else {
#pragma unroll
        for (int q8 = 0; q8 < 8; q8++) {
          const uint32_t wv = lds32(raw + q8 * 512);
          v[4 * q8] = tc_cvt_lo(wv, sc); v[4 * q8 + 1] = tc_cvt_hi(wv, sc);
          v[4 * q8 + 2] = tc_cvt_lo(wv >> 8, sc); v[4 * q8 + 3] = tc_cvt_hi(wv >> 8, sc);
        }
      }
      tc_st32(tq + S::T_A + rs.i * 64 + half * 32, v);
      if (HZ && half == 0) {
        const uint16_t z = reinterpret_cast<const uint16_t*>(rec + 8448)[row];       // one k16 step: A_z = z for every column
        tc_st8(tq + S::T_AZ + rs.i * 8, (uint32_t)z | ((uint32_t)z << 16));
      }
      tc_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(&a_full[rs.i]); mbar_arrive(&raw_empty[rr.i]); }
    }
    if (real) {
      if (ng <= NS) fetch();
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, wc, W_FULL, 10));
      tc_fence_after();
    }
    // K splits: token t's sums go to the CTA that finishes it. Few tokens: an asynchronous store per value, counted on that CTA's barrier, so that
    // nobody waits for a round trip (4 / 14 / 26 tokens of the 3B shape 1647 / 1802 / 2080 -> 1602 / 1749 / 2046 us against a cluster barrier
    // behind plain stores). From 64 tokens on the plain stores and the barrier are faster: 61 tokens 2637, asynchronous stores 2658, one bulk
    // copy per neighbour 2670; a prompt of 100 tokens 2667, 2731, 2767.
    if (split) {
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < HC; c += 8) {
          uint32_t u[8];
          tc_ld8(tlane + c, u);
          tc_ld_wait();
#pragma unroll
          for (int e = 0; e < 8; e++) {
            const int tk = half * HC + c + e;
            if (tk < push_end) {
              const uint32_t to = cluster_map(mine + (uint32_t)(tk & (TPR - 1)) * 512, tk >> lgT);
              if (ASYNC) st_async(to, u[e], cluster_map(smem_u32(xbar), tk >> lgT));
              else st_cluster(to, u[e]);
            }
          }
        }
      }
      if (real) {                                              // every rank's sums are in
        if (ASYNC) {
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait<true>(xbar, 0, wc, W_FULL, 11));
        } else {
          __syncwarp();
          cluster_arrive();
          cluster_wait();
          ok = __all_sync(0xffffffffu, ok && *s_abort == 0);
        }
      }
    }
    int t0 = 0;
    if (ok) do {
      float v[CH];
      if (split) {
        if (!STAGED && t0) pre.fetch(P, srow, th0 + t0, tlast);
#pragma unroll
        for (int e = 0; e < CH; e++) {
          v[e] = 0.f;
          if (t0 + e < HT) {
            if constexpr (NT < 64) {                           // four ranks' sums requested together; 64 tokens keep enough loads in flight
#pragma unroll 1
              for (int r0 = 0; r0 < ns; r0 += 4) {
                float y[4];
#pragma unroll
                for (int r = 0; r < 4; r++) y[r] = r0 + r < ns ? yw[((r0 + r) * TPR + t0 + e) * 128] : 0.f;
#pragma unroll
                for (int r = 0; r < 4; r++) v[e] += y[r];
              }
            } else {
#pragma unroll 4
              for (int r = 0; r < ns; r++) v[e] += yw[(r * TPR + t0 + e) * 128];
            }
          }
        }
      } else if constexpr (!STAGED) {
        uint32_t u[8];
        tc_ld8(tlane + t0, u);
        if (t0) pre.fetch(P, srow, th0 + t0, tlast);
        tc_ld_wait();
#pragma unroll
        for (int e = 0; e < CH; e++) v[e] = __uint_as_float(u[e]);
      }
      if constexpr (STAGED) {
        uint8_t* area = tsm + S::B + (warp - 6) * kTcEpiBytes;
        TcFactorTable tab{reinterpret_cast<float*>(area), reinterpret_cast<float*>(area) + kTcTable};
        if (t0 == 0) tab.put<EPI, 2>(fac, lane);
        else staged.fetch(P, srow - lane, th0 + t0, tlast, lane);
        staged.run(P, area + 2 * kTcTable * 4, srow - lane, th0 + t0, tlast, v, rf, tab, t0, lane);
      } else {
        vtc_epilogue<EPI, CH>(P, srow, th0 + t0, tlast, v, rf, fac, t0, pre, lane);
      }
      t0 += CH;
    } while (th0 + t0 < tlast);
  }
  if (split && (ASYNC || warp < 6)) {                            // nobody leaves before its neighbours have sent what they will send
    __syncwarp();
    if (ASYNC) cluster_arrive_relaxed();
    else cluster_arrive();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*s_abort) tl_drain<NRAW, NS, NB, ND>(bars, s_issued, ASYNC && split);
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::TCOLS));
  }
}

}  // namespace fb
