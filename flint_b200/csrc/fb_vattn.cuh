// Attention of the M-token passes (tree verification, prompts) on the tensor pipe: flash attention over the cache, one launch.
//
// A CTA of eight warps takes, for one kv head, RT row tiles of 16 query rows (row = token * R + head of the group: the R query
// heads share every K/V row) and one span of positions; its warps are RT tiles x PG = 8 / RT position groups, a group taking every
// PG-th unit of UP positions. K/V stages come by cp.async. Spans are the CTAs of a CLUSTER: all warps leave their un-normalised
// partials (acc, running max, denominator) in shared memory, the CTA's position groups are merged, and every row's result goes to the CTA of
// the cluster that finishes it, so there is no merge kernel and no trip of the partials through L2. That pair of kernels took 12.3 + 8.3 us
// for 26 tokens over 1024 positions (3B shape), mostly latency: one 64-position chunk per CTA, then 4.6 MB of partials written and read
// back. The partials are pushed: read from the neighbours' memory between two cluster barriers, passes of 4 / 14 / 26 tokens (3B) and 5 / 26 / 61
// (8B) took 1587 / 1741 / 2020 and 2078 / 2354 / 3370 us, so 1537 / 1727 / 2029 and 2053 / 2339 / 3342.
// Bound by latency for trees; by instruction issue for prompts (softmax around 16 x 8 MMAs), hence ldmatrix for both operands, packed
// conversions, base-2 exponentials, and masks only in the units that need one.
#pragma once
#include "fb_common.cuh"
#include "fb_verify.cuh"

namespace fb {

template <int HD, int RT>
struct VaCfg {
  static constexpr int SP = RT == 4 ? 64 : 128;         // positions of a stage: every warp finds a unit in it
  static constexpr int NSTG = RT == 4 ? 3 : 2;          // stages in flight
  static constexpr int UP = RT == 1 ? 16 : 32, PG = 8 / RT;
  static constexpr int STR = HD * 2 + 16;               // bytes per K / V row: padded, conflict-free for ldmatrix
  static constexpr int STAGE = 2 * SP * STR;
  static constexpr int PW = HD + 4;                     // floats per partial row: acc[HD], max, denominator
  static constexpr int PART = 8 * 16 * PW * 4;          // partials (over the dead stages)
  static constexpr int RING = NSTG * STAGE > PART ? NSTG * STAGE : PART;
  static constexpr int INBOX = RING;                    // the spans' partials of this CTA's rows: [span][row][PW]
  static constexpr int BAR = INBOX + 16 * RT * PW * 4;
  static constexpr int TOTAL = BAR + 16;
  static_assert(SP / UP == PG || RT == 4, "one unit per warp and stage");
};

__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans_a(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

struct VattnParams {
  const uint16_t* q;       // bf16 [M][n_head * HD]
  const uint16_t *kc, *vc; // layer base of the caches, bf16 [max_seq][nkv][HD]
  const uint8_t* amask;    // [M][M] or nullptr: causal chain
  uint16_t* ao;            // bf16 [M][n_head * HD]
  unsigned* amax;          // [M] largest |output| of each token as float bits (cleared by the token's norm), or nullptr
  int n_head, nkv, pos, M, span;
  float scale;             // times log2(e)
  DevStatus* status;
  unsigned spin_limit;
};

// grid (spans = CTAs of a cluster, kv heads, row groups of RT tiles), 256 threads
template <int HD, int R, int RT>
__global__ void __launch_bounds__(256) v_attn(const VattnParams P) {
  using S = VaCfg<HD, RT>;
  constexpr int KSTEPS = HD / 16, NTD = HD / 8, STR = S::STR, PW = S::PW, SP = S::SP, UP = S::UP, NU = SP / UP, NT = UP / 8, PG = S::PG,
                NSTG = S::NSTG;
  static_assert(HD % 16 == 0 && UP % 16 == 0, "head_dim and units are multiples of 16");
  extern __shared__ __align__(16) uint8_t va_sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x, nspan = gridDim.x, kvh = blockIdx.y;
  const int zg = P.amask ? (int)blockIdx.z : (int)gridDim.z - 1 - (int)blockIdx.z;     // causal: the longest rows first
  const int pg = warp / RT, tile = zg * RT + warp % RT;
  const int M = P.M, T = P.pos + M, QD = P.n_head * HD, rows = M * R, ntile = (rows + 15) / 16;
  const int m_last = min(M - 1, ((zg * RT + RT) * 16 - 1) / R);                        // the CTA's last token
  const int t_begin = rank * P.span, t_end = min(P.amask ? T : P.pos + m_last + 1, t_begin + P.span);
  const int nst = t_end > t_begin ? (t_end - t_begin + SP - 1) / SP : 0;
  pdl_trigger();
  uint64_t* xbar = reinterpret_cast<uint64_t*>(va_sm + S::BAR);                        // spans: all partials of this CTA's rows have arrived
  volatile int* s_abort = reinterpret_cast<volatile int*>(xbar + 1);
  constexpr bool ASYNC = RT == 1;                                // how the partials are known to have arrived, see below
  const bool alone = nspan == 1;
  if (!alone) {
    if (ASYNC && tid == 0) {
      *s_abort = 0;
      mbar_init(xbar, 1);
      mbar_fence_init();
      mbar_expect_tx(xbar, 16 * RT * (HD + 4) * 4);
    }
    cluster_arrive();                                            // partials are sent once every neighbour is known to run
  }
  auto issue = [&](int s) {
    if (s < nst) {
      uint8_t* k_s = va_sm + (s % NSTG) * S::STAGE;
      uint8_t* v_s = k_s + SP * STR;
      const int c0 = t_begin + s * SP;
      for (int i = tid; i < SP * NTD; i += 256) {
        const int row = i / NTD, pc = i % NTD, tp = c0 + row;
        const bool ok = tp < t_end;                              // rows past the end: zeros (0 * garbage could be NaN)
        const size_t off = ((size_t)(ok ? tp : t_begin) * P.nkv + kvh) * HD + pc * 8;
        cp_async16_zfill(k_s + row * STR + pc * 16, P.kc + off, ok);
        cp_async16_zfill(v_s + row * STR + pc * 16, P.vc + off, ok);
      }
    }
    cp_async_commit();
  };
  // Rows below `pos` do not depend on the previous kernel: the first stages that hold no others are requested while it runs, and the rest of
  // the span is brought into L2 (with all of it only brought into L2, 26 / 61 tokens over 1024 positions took 2049 / 2640 us a pass, so
  // 2020 / 2617).
  for (int s = 0, waited = 0;; s++) {
    if (!waited && (s == NSTG - 1 || min(t_end, t_begin + (s + 1) * SP) > P.pos)) {
      if (nspan > 1) {
        constexpr int PER = (HD * 2 + 127) / 128 + 1;
        const int p0 = t_begin + s * SP, n = max(0, min(t_end, P.pos) - p0) * 2 * PER;
        for (int i = tid; i < n; i += 256) {
          const int tp = p0 + i / (2 * PER), k = i % (2 * PER);
          const uint16_t* base = (k < PER ? P.kc : P.vc) + ((size_t)tp * P.nkv + kvh) * HD;
          const int off = min((k % PER) * 128, HD * 2 - 2);
          asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(base) + off));
        }
      }
      pdl_wait();
      waited = 1;
    }
    if (s == NSTG - 1) break;
    issue(s);
  }
  const bool live = tile < ntile;
  const int r_lo = min(tile * 16 + g, rows - 1), r_hi = min(tile * 16 + g + 8, rows - 1);
  const int m_lo = r_lo / R, m_hi = r_hi / R;
  const int m_bot = min(rows - 1, tile * 16) / R, m_top = min(rows - 1, tile * 16 + 15) / R;   // the tile's first and last token
  uint32_t aq[KSTEPS][4];
  {
    const uint16_t* q_lo = P.q + (size_t)m_lo * QD + (size_t)(kvh * R + r_lo % R) * HD;
    const uint16_t* q_hi = P.q + (size_t)m_hi * QD + (size_t)(kvh * R + r_hi % R) * HD;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ks++) {
      aq[ks][0] = *reinterpret_cast<const uint32_t*>(q_lo + 16 * ks + 2 * t);
      aq[ks][1] = *reinterpret_cast<const uint32_t*>(q_hi + 16 * ks + 2 * t);
      aq[ks][2] = *reinterpret_cast<const uint32_t*>(q_lo + 16 * ks + 2 * t + 8);
      aq[ks][3] = *reinterpret_cast<const uint32_t*>(q_hi + 16 * ks + 2 * t + 8);
    }
  }
  float o[NTD][4];
#pragma unroll
  for (int j = 0; j < NTD; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[j][e] = 0.f;
  float mrun[2] = {-1e30f, -1e30f}, lrun[2] = {0.f, 0.f};
  // this lane's row of the 8 x 8 matrices: K as 16 positions x 16 dims (n-major), V as 16 positions x 16 dims (transposed on the way)
  const uint32_t k_lane = smem_u32(va_sm) + (uint32_t)(((lane & 7) + ((lane >> 4) & 1) * 8) * STR + ((lane >> 3) & 1) * 16);
  const uint32_t v_lane = smem_u32(va_sm) + (uint32_t)((SP + (lane & 7) + ((lane >> 3) & 1) * 8) * STR + ((lane >> 4) & 1) * 16);
  for (int s = 0; s < nst; s++) {
    cp_async_wait<NSTG - 2>();
    __syncthreads();
    issue(s + NSTG - 1);
#pragma unroll 1
    for (int u = pg; u < NU; u += PG) {
      const int c0 = t_begin + s * SP + u * UP;
      if (!live || c0 >= t_end || (!P.amask && c0 > P.pos + m_top)) break;      // past the end, or beyond this tile's last token
      const uint32_t so = (uint32_t)((s % NSTG) * S::STAGE + u * UP * STR);
      float sc[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; nt++) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ks++)
#pragma unroll
        for (int n2 = 0; n2 < NT / 2; n2++) {
          uint32_t b[4];
          ldmatrix_x4(b, k_lane + so + n2 * 16 * STR + ks * 32);
          mma_bf16(sc[2 * n2], aq[ks], b[0], b[1]);
          mma_bf16(sc[2 * n2 + 1], aq[ks], b[2], b[3]);
        }
      if (c0 + UP > t_end || c0 + UP - 1 > P.pos + (P.amask ? -1 : m_bot)) {     // the unit needs a mask
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int tp = c0 + nt * 8 + 2 * t + (e & 1), mq = e < 2 ? m_lo : m_hi;
            bool ok = tp < t_end;
            if (ok && tp >= P.pos) ok = P.amask ? P.amask[mq * M + (tp - P.pos)] != 0 : tp - P.pos <= mq;
            if (!ok) sc[nt][e] = -INFINITY;
          }
      }
      // row maxima (rows g and g + 8; a row's scores live in the 4 lanes of a quad)
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) mx[e >> 1] = fmaxf(mx[e >> 1], sc[nt][e]);
      float corr[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
        const float mn = fmaxf(mrun[h], mx[h] * P.scale);       // finite: the running maximum starts at -1e30
        corr[h] = ex2(mrun[h] - mn);
        mrun[h] = mn;
      }
      if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
        lrun[0] *= corr[0]; lrun[1] *= corr[1];
#pragma unroll
        for (int j = 0; j < NTD; j++) { o[j][0] *= corr[0]; o[j][1] *= corr[0]; o[j][2] *= corr[1]; o[j][3] *= corr[1]; }
      }
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float pv = ex2(fmaf(sc[nt][e], P.scale, -mrun[e >> 1]));
          sc[nt][e] = pv;
          lrun[e >> 1] += pv;                                   // this lane's columns; the quad is summed at the end
        }
      // O += P V, 16 positions per step; P = hi + lo in bf16 keeps the probabilities to ~2^-17
#pragma unroll
      for (int kk = 0; kk < UP / 16; kk++) {
        uint32_t ah[4], al[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float p0 = sc[2 * kk + (e >> 1)][(e & 1) * 2], p1 = sc[2 * kk + (e >> 1)][(e & 1) * 2 + 1];
          ah[e] = cvt_bf16x2(p0, p1);
          al[e] = cvt_bf16x2(p0 - bflo(ah[e]), p1 - bfhi(ah[e]));
        }
#pragma unroll
        for (int j = 0; j < NTD; j += 2) {
          uint32_t b[4];
          ldmatrix_x4_trans_a(b, v_lane + so + kk * 16 * STR + j * 16);
          mma_bf16(o[j], ah, b[0], b[1]);
          mma_bf16(o[j + 1], ah, b[2], b[3]);
          mma_bf16(o[j], al, b[0], b[1]);
          mma_bf16(o[j + 1], al, b[2], b[3]);
        }
      }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int h = 0; h < 2; h++) {
    lrun[h] += __shfl_xor_sync(0xffffffffu, lrun[h], 1);
    lrun[h] += __shfl_xor_sync(0xffffffffu, lrun[h], 2);
  }
  __syncthreads();                                              // every warp has left the stages
  float* part = reinterpret_cast<float*>(va_sm);
  {
    float* mine = part + (size_t)warp * 16 * PW;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float* pr = mine + (g + 8 * h) * PW;
#pragma unroll
      for (int j = 0; j < NTD; j++) *reinterpret_cast<float2*>(pr + j * 8 + 2 * t) = make_float2(o[j][2 * h], o[j][2 * h + 1]);
      if (t == 0) *reinterpret_cast<float2*>(pr + HD) = make_float2(mrun[h], lrun[h]);
    }
  }
  __syncthreads();
  const int nown = RT * 16 / nspan;                              // this CTA finishes local rows rank, rank + nspan, ...
  if (!alone) cluster_wait();
  // the position groups of the CTA meet first: a warp merges 2 RT rows (in place of position group 0's partials), so that the cluster
  // exchanges one partial per row and span
  auto finish = [&](int lr, float4 acc, float den) {             // local row lr, lane = 4 dims: normalise and write
    const int row = zg * RT * 16 + lr;
    if (row < rows) {
      const float inv = 1.0f / den;
      const uint32_t w0 = cvt_bf16x2(acc.x * inv, acc.y * inv), w1 = cvt_bf16x2(acc.z * inv, acc.w * inv);
      if (lane < HD / 4)
        *reinterpret_cast<uint2*>(P.ao + (size_t)(row / R) * QD + (size_t)(kvh * R + row % R) * HD + lane * 4) = make_uint2(w0, w1);
      if (P.amax) {
        const float bm = lane < HD / 4 ? fmaxf(fmaxf(fabsf(bflo(w0)), fabsf(bfhi(w0))), fmaxf(fabsf(bflo(w1)), fabsf(bfhi(w1)))) : 0.f;
        const uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(bm));   // non-negative floats order like their bits
        if (lane == 0) atomicMax(P.amax + row / R, bits);
      }
    }
  };
  // eight rows a warp as a loop (less code to fetch: 61 tokens over 3000 positions, 8B shape, 3340 -> 3325 us, a prompt of 180 tokens 3558 -> 3537),
  // two or four unrolled (26 tokens, 8B, rolled 2363 instead of 2344)
  constexpr int MERGE_UNROLL = RT == 4 ? 1 : 2 * RT;
#pragma unroll MERGE_UNROLL
  for (int i = 0; i < 2 * RT; i++) {
    const int lr = warp * 2 * RT + i;
    float* p0 = part + ((lr >> 4) * 16 + (lr & 15)) * PW;        // position group 0; group k is k * RT tiles further
    float2 ml[PG];
    float4 v[PG];
#pragma unroll
    for (int k = 0; k < PG; k++) {
      ml[k] = *reinterpret_cast<const float2*>(p0 + k * RT * 16 * PW + HD);
      v[k] = lane < HD / 4 ? *reinterpret_cast<const float4*>(p0 + k * RT * 16 * PW + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float gm = ml[0].x, den = 0.f;
#pragma unroll
    for (int k = 1; k < PG; k++) gm = fmaxf(gm, ml[k].x);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < PG; k++) {
      const float e = ex2(ml[k].x - gm);
      den = fmaf(ml[k].y, e, den);
      acc.x = fmaf(v[k].x, e, acc.x); acc.y = fmaf(v[k].y, e, acc.y); acc.z = fmaf(v[k].z, e, acc.z); acc.w = fmaf(v[k].w, e, acc.w);
    }
    if (alone) {
      finish(lr, acc, den);
    } else {                                                     // to the CTA that finishes the row
      const uint32_t to = lr & (nspan - 1), a = cluster_map(smem_u32(va_sm + S::INBOX) + (uint32_t)((rank * nown + lr / nspan) * PW) * 4, to),
                     xb = cluster_map(smem_u32(xbar), to);
      const float4 md = make_float4(gm, den, 0.f, 0.f);
      if (ASYNC) {
        if (lane < HD / 4) st_async(a + lane * 16, acc, xb);
        if (lane == 0) st_async(a + HD * 4, md, xb);
      } else {
        if (lane < HD / 4) st_cluster(a + lane * 16, acc);
        if (lane == 0) st_cluster(a + HD * 4, md);
      }
    }
  }
  if (!alone) {
    // One row tile a CTA: asynchronous stores that count on the receiver's barrier, which leaves its neighbours' pace out of it. More: plain
    // stores and a cluster barrier (26 tokens of the 3B shape 2038 asynchronous, 2029 plain).
    bool ok = true;
    if (ASYNC) {
      const WaitCtl wc{P.status, s_abort, P.spin_limit};
      ok = __all_sync(0xffffffffu, mbar_wait<true>(xbar, 0, wc, W_FULL, 12));
    } else {
      cluster_arrive();
      cluster_wait();
    }
    const float* in = reinterpret_cast<const float*>(va_sm + S::INBOX);
    for (int ri = warp; ok && ri < nown; ri += 8) {
      float2 ml[8];
      float4 v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        ml[k] = make_float2(-1e30f, 0.f);
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < nspan) {
          const float* a = in + (k * nown + ri) * PW;
          ml[k] = *reinterpret_cast<const float2*>(a + HD);
          if (lane < HD / 4) v[k] = *reinterpret_cast<const float4*>(a + lane * 4);
        }
      }
      float gm = ml[0].x, den = 0.f;
#pragma unroll
      for (int k = 1; k < 8; k++) gm = fmaxf(gm, ml[k].x);
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const float e = ex2(ml[k].x - gm);
        den = fmaf(ml[k].y, e, den);
        acc.x = fmaf(v[k].x, e, acc.x); acc.y = fmaf(v[k].y, e, acc.y); acc.z = fmaf(v[k].z, e, acc.z); acc.w = fmaf(v[k].w, e, acc.w);
      }
      finish(rank + ri * nspan, acc, den);
    }
    // Nobody leaves before its neighbours have sent what they will send; after a failure (somebody gave up before it sent), not before what is
    // under way has landed, which takes microseconds.
    if (ASYNC) {
      __syncwarp();
      cluster_arrive_relaxed();
      cluster_wait();
      if (!ok && tid == 0)
#pragma unroll 1
        for (int i = 0; i < 200 && !mbar_test(xbar, 0); i++) __nanosleep(1000);
    }
  }
}

}  // namespace fb
