// Attention of the M-token passes (tree verification, prompts) on the tensor pipe: flash attention over the cache, one launch.
//
// A CTA of eight warps takes, for one kv head, `rt` row tiles of 16 query rows (row = token * R + head of the group: the R query
// heads share every K/V row) and one span of positions; its warps are rt tiles x 8 / rt position groups, a group taking every
// (8 / rt)-th unit of UP positions. K/V stages of 64 positions come by cp.async, three in flight. Spans are the CTAs of a CLUSTER:
// all warps leave their un-normalised partials (acc, running max, denominator) in shared memory and every CTA finishes a share of
// the rows from its neighbours' shared memory, so there is no merge kernel and no trip of the partials through L2. That pair of
// kernels took 12.3 + 8.3 us for 26 tokens over 1024 positions (3B shape), mostly latency: one 64-position chunk per CTA, then
// 4.6 MB of partials written and read back.
// Bound by latency for trees (K/V of a span are 20 KB); by the tensor pipe and the exponentials for prompts, where a CTA takes 128
// query rows so that a K/V stage is read once per 128 rows (direct: no spans, the CTA writes its rows itself).
#pragma once
#include "fb_common.cuh"
#include "fb_verify.cuh"

namespace fb {

constexpr int kVaStages = 3;                    // K/V stages in flight
constexpr int kVaPos = 64;                      // positions of a stage
template <int HD>
struct VaSmem {
  static constexpr int STR = HD * 2 + 16;       // bytes per K / V row: padded, conflict-free for ldmatrix
  static constexpr int STAGE = 2 * kVaPos * STR;
  static constexpr int PW = HD + 4;             // floats per partial row: acc[HD], max, denominator
  static constexpr int PART = 8 * 16 * PW * 4;  // partials (over the dead stages)
  static constexpr int RING = kVaStages * STAGE > PART ? kVaStages * STAGE : PART;
  static constexpr int TOTAL = RING + 2 * 128 * 4;      // + (max, denominator) of the rows that this CTA finishes
};

__device__ __forceinline__ uint32_t cluster_map(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

struct VattnParams {
  const uint16_t* q;       // bf16 [M][n_head * HD]
  const uint16_t *kc, *vc; // layer base of the caches, bf16 [max_seq][nkv][HD]
  const uint8_t* amask;    // [M][M] or nullptr: causal chain
  uint16_t* ao;            // bf16 [M][n_head * HD]
  unsigned* amax;          // [M] largest |output| of each token as float bits (cleared by the token's norm), or nullptr
  int n_head, nkv, pos, M, rt, span;
  float scale;
};

// grid (spans = CTAs of a cluster, kv heads, row groups), 256 threads
template <int HD, int R, int UP, bool DIRECT>
__global__ void __launch_bounds__(256) v_attn(const VattnParams P) {
  using S = VaSmem<HD>;
  constexpr int KSTEPS = HD / 16, NTD = HD / 8, STR = S::STR, PW = S::PW, NU = kVaPos / UP, NT = UP / 8;
  static_assert(HD % 16 == 0 && UP % 16 == 0, "head_dim and units are multiples of 16");
  extern __shared__ __align__(16) uint8_t va_sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x, nspan = gridDim.x, kvh = blockIdx.y;
  const int zg = DIRECT ? (int)gridDim.z - 1 - (int)blockIdx.z : (int)blockIdx.z;      // prompts: the longest rows first
  const int rt = DIRECT ? 8 : P.rt, PG = 8 / rt, pg = warp / rt, tile = zg * rt + warp % rt;
  const int M = P.M, T = P.pos + M, QD = P.n_head * HD, rows = M * R, ntile = (rows + 15) / 16;
  const int m_last = min(M - 1, ((zg * rt + rt) * 16 - 1) / R);                        // the CTA's last token
  const int t_begin = rank * P.span, t_end = min(P.amask ? T : P.pos + m_last + 1, t_begin + P.span);
  const int nst = t_end > t_begin ? (t_end - t_begin + kVaPos - 1) / kVaPos : 0;
  pdl_trigger();
  // the span's old rows do not depend on the previous kernel: bring them into L2 while it runs
  {
    constexpr int PER = (HD * 2 + 127) / 128 + 1;
    const int old_end = min(t_end, P.pos), n = max(0, old_end - t_begin) * 2 * PER;
    for (int i = tid; i < n; i += 256) {
      const int tp = t_begin + i / (2 * PER), k = i % (2 * PER);
      const uint16_t* base = (k < PER ? P.kc : P.vc) + ((size_t)tp * P.nkv + kvh) * HD;
      const int off = min((k % PER) * 128, HD * 2 - 2);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(base) + off));
    }
  }
  pdl_wait();
  auto issue = [&](int s) {
    if (s < nst) {
      uint8_t* k_s = va_sm + (s % kVaStages) * S::STAGE;
      uint8_t* v_s = k_s + kVaPos * STR;
      const int c0 = t_begin + s * kVaPos;
      for (int i = tid; i < kVaPos * NTD; i += 256) {
        const int row = i / NTD, pc = i % NTD, tp = c0 + row;
        const bool ok = tp < t_end;                              // rows past the end: zeros (0 * garbage could be NaN)
        const size_t off = ((size_t)(ok ? tp : t_begin) * P.nkv + kvh) * HD + pc * 8;
        cp_async16_zfill(k_s + row * STR + pc * 16, P.kc + off, ok);
        cp_async16_zfill(v_s + row * STR + pc * 16, P.vc + off, ok);
      }
    }
    cp_async_commit();
  };
  for (int s = 0; s < kVaStages - 1; s++) issue(s);
  const bool live = tile < ntile;
  const int r_lo = min(tile * 16 + g, rows - 1), r_hi = min(tile * 16 + g + 8, rows - 1);
  const int m_lo = r_lo / R, m_hi = r_hi / R, m_top = min(rows - 1, tile * 16 + 15) / R;
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
  const int mat = lane >> 3;
  for (int s = 0; s < nst; s++) {
    cp_async_wait<kVaStages - 2>();
    __syncthreads();
    issue(s + kVaStages - 1);
    const uint8_t* k_s = va_sm + (s % kVaStages) * S::STAGE;
    const uint8_t* v_s = k_s + kVaPos * STR;
#pragma unroll 1
    for (int u = 0; u < NU; u++) {
      const int c0 = t_begin + s * kVaPos + u * UP;
      if (!live || c0 >= t_end || ((s * NU + u) & (PG - 1)) != pg) continue;
      if (!P.amask && c0 > P.pos + m_top) continue;             // beyond this tile's last token
      float sc[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; nt++) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ks++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          const uint8_t* kr = k_s + (u * UP + nt * 8 + g) * STR + (16 * ks + 2 * t) * 2;
          mma_bf16(sc[nt], aq[ks], *reinterpret_cast<const uint32_t*>(kr), *reinterpret_cast<const uint32_t*>(kr + 16));
        }
      // scale, mask, row maxima (rows g and g + 8; a row's scores live in the 4 lanes of a quad)
      float mx[2] = {-INFINITY, -INFINITY};
      const bool edge = c0 + UP > P.pos || c0 + UP > t_end;      // the unit reaches into the M new slots or past the end
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          bool ok = true;
          if (edge) {
            const int tp = c0 + nt * 8 + 2 * t + (e & 1), mq = e < 2 ? m_lo : m_hi;
            ok = tp < t_end;
            if (ok && tp >= P.pos) ok = P.amask ? P.amask[mq * M + (tp - P.pos)] != 0 : tp - P.pos <= mq;
          }
          const float v = ok ? sc[nt][e] * P.scale : -INFINITY;
          sc[nt][e] = v;
          mx[e >> 1] = fmaxf(mx[e >> 1], v);
        }
      float corr[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
        const float mn = fmaxf(mrun[h], mx[h]);                 // finite: the running maximum starts at -1e30
        corr[h] = __expf(mrun[h] - mn);
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
          const float pv = __expf(sc[nt][e] - mrun[e >> 1]);
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
          const float h0 = rbf(p0), h1 = rbf(p1);
          ah[e] = pack_bf16(h0, h1);
          al[e] = pack_bf16(p0 - h0, p1 - h1);
        }
#pragma unroll
        for (int j = 0; j < NTD; j += 2) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, v_s + (u * UP + kk * 16 + (mat & 1) * 8 + (lane & 7)) * STR + (j + (mat >> 1)) * 16);
          mma_bf16(o[j], ah, b[0], b[1]);
          mma_bf16(o[j], al, b[0], b[1]);
          mma_bf16(o[j + 1], ah, b[2], b[3]);
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
  if constexpr (DIRECT) {
    if (live) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int row = tile * 16 + g + 8 * h;
        if (row < rows) {
          const float inv = 1.0f / lrun[h];
          uint16_t* dst = P.ao + (size_t)(row / R) * QD + (size_t)(kvh * R + row % R) * HD;
#pragma unroll
          for (int j = 0; j < NTD; j++)
            *reinterpret_cast<uint32_t*>(dst + j * 8 + 2 * t) = pack_bf16(o[j][2 * h] * inv, o[j][2 * h + 1] * inv);
        }
      }
    }
  } else {
    __syncthreads();                                            // every warp has left the stages
    float* part = reinterpret_cast<float*>(va_sm) + (size_t)warp * 16 * PW;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float* pr = part + (g + 8 * h) * PW;
#pragma unroll
      for (int j = 0; j < NTD; j++) *reinterpret_cast<float2*>(pr + j * 8 + 2 * t) = make_float2(o[j][2 * h], o[j][2 * h + 1]);
      if (t == 0) *reinterpret_cast<float2*>(pr + HD) = make_float2(mrun[h], lrun[h]);
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    // this CTA finishes local rows rank, rank + nspan, ...; a row has nspan * PG partials
    const int nown = rt * 16 / nspan, nsrc = nspan * PG;         // nown * nsrc == 128
    float* wm = reinterpret_cast<float*>(va_sm + S::RING);
    float* wl = wm + 128;
    const uint32_t base = smem_u32(va_sm);
    auto src_addr = [&](int lr, int src) {                       // partial row of local row lr from source (cta, position group)
      const int cta = src / PG, w = lr / 16 + rt * (src % PG);
      return cluster_map(base + (uint32_t)((w * 16 + (lr & 15)) * PW) * 4, cta);
    };
    if (tid < 128) {
      const float2 ml = ld_cluster_f2(src_addr(rank + (tid / nsrc) * nspan, tid % nsrc) + HD * 4);
      wm[tid] = ml.x;
      wl[tid] = ml.y;
    }
    __syncthreads();
    for (int ri = warp; ri < nown; ri += 8) {
      const int lr = rank + ri * nspan, row = zg * rt * 16 + lr;
      const float* pm = wm + ri * nsrc;
      const float* pl = wl + ri * nsrc;
      float gm = -1e30f, den = 0.f;
      for (int s2 = 0; s2 < nsrc; s2++) gm = fmaxf(gm, pm[s2]);
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int s2 = 0; s2 < nsrc; s2++) {
        const float e = __expf(pm[s2] - gm);
        den = fmaf(pl[s2], e, den);
        if (lane < HD / 4) {
          const float4 v = ld_cluster_f4(src_addr(lr, s2) + lane * 16);
          acc.x = fmaf(v.x, e, acc.x); acc.y = fmaf(v.y, e, acc.y); acc.z = fmaf(v.z, e, acc.z); acc.w = fmaf(v.w, e, acc.w);
        }
      }
      if (row < rows) {
        const float a0 = rbf(acc.x / den), a1 = rbf(acc.y / den), a2 = rbf(acc.z / den), a3 = rbf(acc.w / den);
        float bm = lane < HD / 4 ? fmaxf(fmaxf(fabsf(a0), fabsf(a1)), fmaxf(fabsf(a2), fabsf(a3))) : 0.f;
        if (lane < HD / 4)
          *reinterpret_cast<uint2*>(P.ao + (size_t)(row / R) * QD + (size_t)(kvh * R + row % R) * HD + lane * 4) =
              make_uint2(pack_bf16(a0, a1), pack_bf16(a2, a3));
        if (P.amax) {
#pragma unroll
          for (int of = 16; of > 0; of >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, of));
          if (lane == 0) atomicMax(P.amax + row / R, __float_as_uint(bm));
        }
      }
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // nobody leaves while a neighbour reads its shared memory
  }
}

}  // namespace fb
