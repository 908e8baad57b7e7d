// Decode megakernel, data-flow synchronisation.
//
// Phases of one token are chained by DATA, not by grid barriers: every vector that crosses CTAs (residual h, q / new
// k / new v, attention output, SwiGLU activations, arg-max candidates) lives in global memory as 8-byte words that
// carry their payload (two bf16 values or one fp32/int32) together with a 32-bit tag unique to (launch, layer,
// phase). A producer publishes the word once; a consumer polls the word itself until the tag matches, so the value
// arrives with the same L2 round trip that a barrier would only have announced. Each hop costs about one L2 round
// trip instead of three (barrier arrive, barrier poll, data fetch). (Arrival flags that were waited for ahead of the words gained as long as words were
// stored, see ll_store; with exchanges they cost 847 us a token of the 3B-class shape at 200 positions against 808 without.)
//
// Why single buffers are enough: a CTA publishes words only behind its own reads of the phase's input, a phase's words are made from all words of the phase before
// (of the attention: of the queries of all heads), so whoever publishes a buffer's next words knows, through the phases in between, that all readers of the last ones
// are done. That holds for words whose writer has waited, and only for those: nobody publishes anything else (columns that nobody computes are not
// published as zeros but left out of the reading, see o_words). A CTA without rows of a phase skips its input: nothing of its own would hold the next words
// back, and it might find the input overwritten. tests/test_decode_order.py follows all shapes through.
#pragma once
#include <cuda.h>

#include "fb_pipe.cuh"

namespace fb {

// K/V rows travel through the weight ring: NPS positions per stage, K rows first, then V rows. Head dimensions that are whole
// multiples of 64 are cut into column blocks of 64 (128 bytes, the swizzle width), [block][position][64] each, so that the eight
// rows of an 8x8 matrix load lie in different banks (unswizzled rows of 128 or 256 bytes all start in the same bank: 8 times
// the shared-memory cycles); other head dimensions keep whole rows (160 bytes for 80: two rows per bank group).
template <int HD, int STG>
struct AttnCfg {
  static constexpr int NPS = 2 * 64 * HD * 2 <= STG ? 64 : 32;
  static constexpr int MATRIX_BYTES = NPS * HD * 2, KV_STAGE_BYTES = 2 * MATRIX_BYTES;
  static constexpr bool SPLIT = HD % 64 == 0;
  static constexpr int BLKS = SPLIT ? HD / 64 : 1, BCOLS = SPLIT ? 64 : HD, ROWB = BCOLS * 2;
  static_assert(HD % 8 == 0 && HD <= 128, "head_dim must be a multiple of 8 and <= 128");
  static_assert(KV_STAGE_BYTES <= STG && MATRIX_BYTES % 128 == 0, "a ring stage holds one sweep of K and V rows");
};

// ------------------------------------------------------------------------------------------------ tagged words
// Words are published by atomic exchanges, whose result nobody wants: an exchange is performed at L2 at once, a store waits in the SM's store path until
// something pushes it out (200 cached positions of the 3B-class shape: 882 us a token with stores, 784 with exchanges; with stores and an exchange per
// CTA and phase behind them, the arrival flags that this kernel once had, 809).
__device__ __forceinline__ void ll_store(uint64_t* p, uint32_t payload, uint32_t tag) {
  const uint64_t v = ((uint64_t)tag << 32) | payload;
  asm volatile("{ .reg .b64 old;\n atom.relaxed.gpu.global.exch.b64 old, [%0], %1; }" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void ll_load2(const uint64_t* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

// words exchanged between GPUs (peer stores over NVLink, polled in local memory): system scope
__device__ __forceinline__ void ll_store_sys(uint64_t* p, uint32_t payload, uint32_t tag) {
  const uint64_t v = ((uint64_t)tag << 32) | payload;
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t ll_load_sys(const uint64_t* p) {
  uint64_t a;
  asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  return a;
}
__device__ __forceinline__ void ll_store2_sys(uint64_t* p, uint32_t pay0, uint32_t pay1, uint32_t tag) {
  const uint64_t a = ((uint64_t)tag << 32) | pay0, b = ((uint64_t)tag << 32) | pay1;
  asm volatile("st.relaxed.sys.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ll_load2_sys(const uint64_t* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.sys.global.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
// bounded poll of one word written by another GPU; returns the payload (0 after a failure)
__device__ __forceinline__ uint32_t ll_poll_sys(const uint64_t* p, uint32_t tag, const WaitCtl& wc, int layer) {
#pragma unroll 1
  for (unsigned spin = 0;; spin++) {
    const uint64_t v = ll_load_sys(p);
    if ((uint32_t)(v >> 32) == tag) return (uint32_t)v;
    if (*wc.s_abort) return 0;
    if ((spin & 255) == 255 && ld_volatile_s32(&wc.st->abort)) { *wc.s_abort = 1; return 0; }
    if (spin >= wc.limit) { report_fail_far(wc, W_FLAG, layer, (int)tag, -3); return 0; }
  }
}

// 16 bytes = two tagged words in one store (each word carries its own tag)
__device__ __forceinline__ void ll_store2(uint64_t* p, uint32_t pay0, uint32_t pay1, uint32_t tag) {
  const uint64_t a = ((uint64_t)tag << 32) | pay0, b = ((uint64_t)tag << 32) | pay1;
  asm volatile("{ .reg .b128 v, old;\n mov.b128 v, {%1, %2};\n atom.relaxed.gpu.global.exch.b128 old, [%0], v; }" ::"l"(p), "l"(a), "l"(b) : "memory");
}
// one round of a bounded poll went by without the word: true = give up (abort seen or limit reached)
inline __device__ __noinline__ bool poll_again(unsigned spin, const WaitCtl wc, int layer, int expected, int seen) {
  if (*wc.s_abort) return true;
  if ((spin & 255) == 255 && ld_volatile_s32(&wc.st->abort)) { *wc.s_abort = 1; return true; }
  if (spin >= wc.limit) { report_fail_far(wc, W_FLAG, layer, expected, seen); return true; }
  return false;
}

// Poll tagged words, 16-byte aligned: pair k of a thread is words 2 (tid + k * nthreads) and the one behind it, pairs [first, end) in all; their payloads go to
// v[k] (zero where there is no such pair). All of a thread's loads are issued before any is checked.
template <int MAXP>
__device__ __forceinline__ void ll_gather(const uint64_t* src, int end, uint32_t tag, uint2 (&v)[MAXP], int tid, int nthreads,
                                          const WaitCtl& wc, int layer, int first = 0) {
  uint32_t pending = 0;
#pragma unroll
  for (int k = 0; k < MAXP; k++) {
    v[k] = make_uint2(0, 0);
    if (tid + k * nthreads >= first && tid + k * nthreads < end) pending |= 1u << k;
  }
#pragma unroll 1
  for (unsigned spin = 0; pending; spin++) {
    uint64_t a[MAXP], b[MAXP];
#pragma unroll
    for (int k = 0; k < MAXP; k++)
      if (pending & (1u << k)) ll_load2(src + 2 * (size_t)(tid + k * nthreads), a[k], b[k]);
#pragma unroll
    for (int k = 0; k < MAXP; k++)
      if (pending & (1u << k)) {
        if ((uint32_t)(a[k] >> 32) == tag && (uint32_t)(b[k] >> 32) == tag) {
          v[k] = make_uint2((uint32_t)a[k], (uint32_t)b[k]);
          pending &= ~(1u << k);
        }
      }
    if (pending && poll_again(spin, wc, layer, (int)tag, -1)) break;
  }
}

// ------------------------------------------------------------------------------------------------ staging from tagged vectors
// Both are real functions, one instance per kernel, not inlined at their five call sites: every kilobyte of the layer loop shortens all phases (inlined
// copies of one generic staging function 1187 us a token of the 3B-class shape; one shared copy 1051; templated on the widths and shared
// as here 1001). Both plain phases share the instance of the wider one. The tile products stay inlined per phase: one shared product costs more in
// calls than it saves (1125).
// Both leave the phase's activations in sm.x8 / sm.xf (digits + per-group factors) and end with a consumer-wide barrier. A thread owns the 4
// elements 4*pr .. 4*pr+3 for pr = tid_c, tid_c + kConsumerThreads, ... and keeps them in registers, so a warp owns whole groups of 128.
// xn = bf16( (float(h) * r) * float(w) ) from the tagged residual vector (dim/2 words)
template <int MAXP, bool SUM>
inline __device__ __noinline__ void stage_norm_ll(const uint64_t* hll, uint32_t tag, const uint16_t* gw, int D, float eps, DevStatus* status, unsigned limit, int layer,
                                                  bool have_h, long long* dbg = nullptr) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const Smem sm = carve_smem(smem_raw);
  const WaitCtl wc{status, sm.s_abort, limit};
  const int tid_c = threadIdx.x;
  float* red = sm.red;
  const int npairs = D / 4, lane = tid_c & 31;
  uint2 wv[MAXP];                       // norm weights do not depend on the wait: fetch them first
#pragma unroll
  for (int k = 0; k < MAXP; k++) {
    const int pr = tid_c + k * kConsumerThreads;
    wv[k] = pr < npairs ? __ldg(reinterpret_cast<const uint2*>(gw) + pr) : make_uint2(0, 0);
  }
  uint2 raw[MAXP];
  if (!have_h) {
    // Every warp has left the phase before (and whose activations it read): polling that starts while slow warps still multiply costs them
    // more than it gains.
    named_bar_sync(kBarConsumers, kConsumerThreads);
    ll_gather<MAXP>(hll, npairs, tag, raw, tid_c, kConsumerThreads, wc, layer);
    if (dbg && tid_c == 0) dbg[11] = (long long)globaltimer_ns();
  } else {            // layer 0 finds the raw residual (bf16, natural order) in place; the barrier below comes before anybody overwrites it
    const uint2* h0 = reinterpret_cast<const uint2*>(sm.x8);
#pragma unroll
    for (int k = 0; k < MAXP; k++) {
      const int pr = tid_c + k * kConsumerThreads;
      raw[k] = pr < npairs ? h0[pr] : make_uint2(0, 0);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < MAXP; k++) {
    const uint32_t a = raw[k].x, b = raw[k].y;
    ss = fmaf(bflo(a), bflo(a), ss); ss = fmaf(bfhi(a), bfhi(a), ss);
    ss = fmaf(bflo(b), bflo(b), ss); ss = fmaf(bfhi(b), bfhi(b), ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (lane == 0) red[tid_c >> 5] = ss;
  named_bar_sync(kBarConsumers, kConsumerThreads);
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < kConsumerWarps; w += 2) {
    const float2 v = *reinterpret_cast<const float2*>(red + w);
    tot += v.x;
    tot += v.y;
  }
  const float r = 1.0f / sqrtf(tot / (float)D + eps);
#pragma unroll
  for (int k = 0; k < MAXP; k++) {
    const uint32_t a = raw[k].x, b = raw[k].y;
    raw[k].x = (uint32_t)f2bf(bflo(a) * r * bflo(wv[k].x)) | ((uint32_t)f2bf(bfhi(a) * r * bfhi(wv[k].x)) << 16);
    raw[k].y = (uint32_t)f2bf(bflo(b) * r * bflo(wv[k].y)) | ((uint32_t)f2bf(bfhi(b) * r * bfhi(wv[k].y)) << 16);
  }
  stage_groups<SUM, MAXP>(raw, tid_c >> 5, kConsumerWarps, D / 128, sm.x8, sm.xf, lane);
  named_bar_sync(kBarConsumers, kConsumerThreads);
}

// `only`, in the kernels of ranks: first and end pair of the words that somebody publishes; the other elements are zero. (A parameter pack: the kernels of one GPU
// have no such argument.)
template <int MAXP, bool SUM, class... Only>
inline __device__ __noinline__ void stage_plain_ll(const uint64_t* src, uint32_t tag, int K,
                                                   DevStatus* status, unsigned limit, int layer, Only... only) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const Smem sm = carve_smem(smem_raw);
  const WaitCtl wc{status, sm.s_abort, limit};
  const int tid_c = threadIdx.x;
  const int npairs = K / 4, lane = tid_c & 31;
  named_bar_sync(kBarConsumers, kConsumerThreads);            // every warp has left the phase that read the activations
  uint2 raw[MAXP];
  if constexpr (sizeof...(Only) > 0) {
    const WordPairs w{only...};
    ll_gather<MAXP>(src, w.end, tag, raw, tid_c, kConsumerThreads, wc, layer, w.first);
  } else {
    ll_gather<MAXP>(src, npairs, tag, raw, tid_c, kConsumerThreads, wc, layer);
  }
  stage_groups<SUM, MAXP>(raw, tid_c >> 5, kConsumerWarps, K / 128, sm.x8, sm.xf, lane);
  named_bar_sync(kBarConsumers, kConsumerThreads);
}

// ------------------------------------------------------------------------------------------------ attention (tagged in/out)
// q and the new k live in "pair-major" tagged words: word (head*HD/2 + p) = (x[p], x[p + HD/2]), which is what one
// RoPE thread produces; v words are (v[2w], v[2w+1]).
struct AttnArgs {
  const uint64_t* q_ll;     // [NH * HD/2]
  const uint64_t* k_ll;     // [NKV * HD/2] new key of this step, pair-major
  const uint64_t* v_ll;     // [NKV * HD/2] new value, natural order
  uint64_t* ao_ll;          // [NH * HD/2] natural order
  uint64_t* part_ll;        // [NKV][maxchunks][R*HD + 2R] tagged chunk partials (acc, then m, then d per head)
  int nkv, pos, nchunks, maxchunks;
  float scale;              // times log2(e)
  uint32_t tag_in, tag_part, tag_out;
};

// byte offset of 8-column block `c` of row `row` of a K or V matrix in a ring stage at shared address `base`
template <int HD, int STG>
__device__ __forceinline__ uint32_t kv_addr(uint32_t base, int row, int c) {
  using C = AttnCfg<HD, STG>;
  if constexpr (!C::SPLIT) return base + (uint32_t)(row * C::ROWB + c * 16);
  const uint32_t a = base + (uint32_t)((c >> 3) * (C::NPS * 128) + row * 128);
  return a + ((((uint32_t)c & 7) ^ ((a >> 7) & 7)) << 4);       // the tensor copy's 128-byte swizzle: address bits 4..6 ^ 7..9
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ int count_unit(int* n) {
  int old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.s32 %0, [%1], 1;" : "=r"(old) : "r"(smem_u32(n)) : "memory");
  return old;
}

// Flash-decode of this CTA's (kv head, chunk) items on the tensor pipe, K/V from the ring, at every cached length. Warp w takes units
// of 16 positions w, w + 14, ...: the R query heads of the group are the rows of a 16-row MMA tile, the positions the N dimension of
// Q K^T and the K dimension of P V. Probabilities enter P V as three bf16 terms (24 bits: fp32 precision). What bounds it is latency:
// the wait for q, one pass of the warps, the merge of the warps, the round trip of the merge of the chunks. Against dot products on the CUDA cores
// with K/V loaded by the warps themselves: 40 / 8 heads of 64, 604 positions 1240 -> 1014 us a token (24 us a layer in all), 32 / 8 heads
// of 64, 22 positions 433 -> 397. Against the earlier ring form (unswizzled 256-byte rows, 8-way bank conflicts on K and V, all 14 warps
// merged whether they had a unit or not) heads of 128, 1778 positions: attention 9.8 -> 7.9 us a layer.
template <int HD, int R, int STG>
__device__ __forceinline__ void attention_phase(const AttnArgs& a, uint8_t* scratch, int cw, int lane, int tid_c, const WaitCtl& wc, int layer,
                                                Pipe& pipe, int* tdone) {
  using C = AttnCfg<HD, STG>;
  constexpr int HP = HD / 2, KSTEPS = (HD + 15) / 16, NTD = HD / 8, NPS = C::NPS, UP = 16, SPLIT = NPS / UP, RH = R > 8 ? 2 : 1;
  static_assert(R <= 16 && NPS % UP == 0, "the query heads of a group are the rows of one MMA tile");
  static_assert(kConsumerWarps * R * (HD + 2) * 4 + (R + 2) * HD * 2 <= kAttnScratch, "attention scratch");
  float* wacc = reinterpret_cast<float*>(scratch);                 // [CW][R][HD]
  float* wm = wacc + kConsumerWarps * R * HD;                      // [CW][R]
  float* wd = wm + kConsumerWarps * R;                             // [CW][R]
  uint32_t* qs = reinterpret_cast<uint32_t*>(wd + kConsumerWarps * R);   // bf16 [R][HD] q, [HD] new k, [HD] new v
  const int T = a.pos + 1;
  const int items = a.nkv * a.nchunks;
  const int chunk_len = (T + a.nchunks - 1) / a.nchunks;
  const int g = lane >> 2, t = lane & 3, mat = lane >> 3;
#pragma unroll 1
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int kvh = item / a.nchunks, c = item - kvh * a.nchunks;
    const int t0 = c * chunk_len, t1 = min(T, t0 + chunk_len);
    const bool has_new = (a.pos >= t0 && a.pos < t1);     // the chunk that contains this step's own position
    // ---- gather q (R heads) and, for the last chunk, the new k / v: at most one word pair per thread ----
    {
      constexpr int NQ = R * HP;
      static_assert(NQ + 2 * HP <= 2 * kConsumerThreads, "one word pair per thread");
      const int w = 2 * tid_c;
      if (w < NQ + (has_new ? 2 * HP : 0)) {
        const uint64_t* src = w < NQ ? a.q_ll + (size_t)kvh * NQ + w
                            : (w < NQ + HP ? a.k_ll + (size_t)kvh * HP + (w - NQ) : a.v_ll + (size_t)kvh * HP + (w - NQ - HP));
#pragma unroll 1
        for (unsigned spin = 0;; spin++) {
          uint64_t u, v;
          ll_load2(src, u, v);
          if ((uint32_t)(u >> 32) == a.tag_in && (uint32_t)(v >> 32) == a.tag_in) {
            const uint32_t x = (uint32_t)u, y = (uint32_t)v;
            if (w < NQ + HP) {                                     // pairs p, p + 1 -> dims p, p + 1 and HP + p, HP + p + 1
              const int row = w / HP, p = w - row * HP;
              qs[row * HP + (p >> 1)] = (x & 0xffffu) | (y << 16);
              qs[row * HP + (HP >> 1) + (p >> 1)] = (x >> 16) | (y & 0xffff0000u);
            } else {
              qs[w] = x; qs[w + 1] = y;
            }
            break;
          }
          if (poll_again(spin, wc, layer, (int)a.tag_in, -2)) break;
        }
      }
    }
    named_bar_sync(kBarConsumers, kConsumerThreads);
    const int nst = t1 > t0 ? (t1 - t0 + NPS - 1) / NPS : 0, units = t1 > t0 ? (t1 - t0 + UP - 1) / UP : 0;
    if (cw < nst * SPLIT) {
      uint32_t aq[KSTEPS][4];
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ks++)
#pragma unroll
        for (int e = 0; e < 4; e++) {                              // rows g, g + 8; columns 2t, 2t + 8
          const int row = g + 8 * (e & 1), d2 = 8 * ks + t + 4 * (e >> 1);
          aq[ks][e] = (e & 1) && RH == 1 ? 0u : (row < R && d2 < HP ? qs[row * HP + d2] : 0u);
        }
      float o[NTD][4];
#pragma unroll
      for (int j = 0; j < NTD; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) o[j][e] = 0.f;
      float mrun[RH], lrun[RH];
#pragma unroll
      for (int h = 0; h < RH; h++) { mrun[h] = -1e30f; lrun[h] = 0.f; }
      // a stage is cut into units of 16 positions that different warps take: a chunk of a few stages keeps most warps busy
#pragma unroll 1
      for (int u = cw; u < nst * SPLIT; u += kConsumerWarps) {
        const int st = u / SPLIT, part = u % SPLIT;
        const uint32_t it = pipe.it + st;
        const int sslot = it % kStages;
        if (!wait_stage(pipe, it, wc, layer)) break;
        uint8_t* stage = pipe.stages + (size_t)sslot * STG;
        const uint32_t k_s = smem_u32(stage), v_s = k_s + C::MATRIX_BYTES;
        const int row0 = part * UP, base = t0 + st * NPS + row0, nvalid = min(UP, t1 - base);
        if (nvalid > 0) {
          const int own = a.pos - base;
          if (own >= 0 && own < UP && lane < NTD) {                // this step's own row: from the tagged words, not the cache
            const uint4 kn = reinterpret_cast<const uint4*>(qs + R * HP)[lane], vn = reinterpret_cast<const uint4*>(qs + (R + 1) * HP)[lane];
            *reinterpret_cast<uint4*>(stage + (kv_addr<HD, STG>(k_s, row0 + own, lane) - k_s)) = kn;
            *reinterpret_cast<uint4*>(stage + (kv_addr<HD, STG>(v_s, row0 + own, lane) - k_s)) = vn;
          }
          // rows past the chunk are other cache rows (or never written): their V must not meet a zero probability as NaN
#pragma unroll 1
          for (int i = lane; i < (UP - nvalid) * NTD; i += 32)
            *reinterpret_cast<uint4*>(stage + (kv_addr<HD, STG>(v_s, row0 + nvalid + i / NTD, i % NTD) - k_s)) = make_uint4(0, 0, 0, 0);
          __syncwarp();
          float sc[2][4];
#pragma unroll
          for (int nt = 0; nt < 2; nt++) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
          for (int ks = 0; ks < KSTEPS; ks++) {
            uint32_t bk[4];                                        // (positions 0..7, columns 0..7), (.., 8..15), (8..15, 0..7), (8..15, 8..15)
            ldmatrix_x4(bk, kv_addr<HD, STG>(k_s, row0 + (mat >> 1) * 8 + (lane & 7), min(2 * ks + (mat & 1), NTD - 1)));
            mma_bf16(sc[0], aq[ks], bk[0], bk[1]);
            mma_bf16(sc[1], aq[ks], bk[2], bk[3]);
          }
          uint32_t ap[3][4];
#pragma unroll
          for (int h = 0; h < RH; h++) {                           // rows g + 8h
            float mx = mrun[h];                                    // finite: the running maximum starts at -1e30
#pragma unroll
            for (int nt = 0; nt < 2; nt++)
#pragma unroll
              for (int e = 0; e < 2; e++) {
                float& v = sc[nt][2 * h + e];
                v = (nt * 8 + 2 * t + e) < nvalid ? v * a.scale : -INFINITY;
                mx = fmaxf(mx, v);
              }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float corr = ex2(mrun[h] - mx);
            mrun[h] = mx;
            lrun[h] *= corr;
#pragma unroll
            for (int j = 0; j < NTD; j++) { o[j][2 * h] *= corr; o[j][2 * h + 1] *= corr; }
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {                       // A columns 2t (+ 1) of positions 8 nt ..
              float p0 = ex2(sc[nt][2 * h] - mx), p1 = ex2(sc[nt][2 * h + 1] - mx);
              lrun[h] += p0 + p1;                                  // this lane's columns; the quad is summed at the end
#pragma unroll
              for (int e = 0; e < 3; e++) {
                const float h0 = rbf(p0), h1 = rbf(p1);
                ap[e][2 * nt + h] = pack_bf16(h0, h1);
                p0 -= h0; p1 -= h1;
              }
            }
          }
          if (RH == 1)
#pragma unroll
            for (int e = 0; e < 3; e++) ap[e][1] = ap[e][3] = 0u;
#pragma unroll
          for (int j = 0; j < NTD; j += 2) {
            uint32_t bv[4];
            ldmatrix_x4_t(bv, kv_addr<HD, STG>(v_s, row0 + (mat & 1) * 8 + (lane & 7), min(j + (mat >> 1), NTD - 1)));
#pragma unroll
            for (int e = 0; e < 3; e++) {
              mma_bf16(o[j], ap[e], bv[0], bv[1]);
              if (j + 1 < NTD) mma_bf16(o[j + 1 < NTD ? j + 1 : j], ap[e], bv[2], bv[3]);
            }
          }
        }
        __syncwarp();
        // The stage's last unit hands it back. Stores of other units (the step's own row, the zeroed rows) must not land after the next
        // copy into the stage: the counter's release and acquire order them before this lane, its proxy fence before the copy.
        if (lane == 0 && count_unit(tdone + sslot) == SPLIT - 1) {
          tdone[sslot] = 0;
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          mbar_arrive(&pipe.empty[sslot]);
        }
      }
#pragma unroll
      for (int h = 0; h < RH; h++) {
        lrun[h] += __shfl_xor_sync(0xffffffffu, lrun[h], 1);
        lrun[h] += __shfl_xor_sync(0xffffffffu, lrun[h], 2);
        const int row = g + 8 * h;
        if (cw < units && row < R) {
          float* dst = wacc + (cw * R + row) * HD + 2 * t;
#pragma unroll
          for (int j = 0; j < NTD; j++) *reinterpret_cast<float2*>(dst + j * 8) = make_float2(o[j][2 * h], o[j][2 * h + 1]);
          if (t == 0) { wm[cw * R + row] = mrun[h]; wd[cw * R + row] = lrun[h]; }
        }
      }
    }
    pipe.it += (uint32_t)nst;                                 // producer and consumers count alike
    named_bar_sync(kBarConsumers, kConsumerThreads);
    // ---- merge the CTA's warps that had a unit; one thread per (head, dim pair) ----
    constexpr int WPC = R * HD + 2 * R;                       // words of one chunk partial
    const int nact = min(units, kConsumerWarps);
    uint64_t* mine = a.part_ll + ((size_t)kvh * a.maxchunks + c) * WPC;
#pragma unroll 1
    for (int o = tid_c; o < R * HP; o += kConsumerThreads) {
      const int r = o / HP, d = 2 * (o - r * HP);
      // The units of a chunk of two stages side by side: one after the other they are a chain of shared-memory round trips (8 / 4 at a time for heads
      // below / of 128: 200 positions at 3B 797 -> 785 us, 1B 284 -> 280, 40 heads 790 -> 787, 8B 1423 -> 1412; 8 at 8B 1443).
      constexpr int WU = 2 * SPLIT;
      float gm = -1e30f;
#pragma unroll 1
      for (int w0 = 0; w0 < nact; w0 += WU)
#pragma unroll
        for (int w = 0; w < WU; w++) gm = fmaxf(gm, w0 + w < nact ? wm[(w0 + w) * R + r] : -1e30f);
      float Dn = 0.f, A0 = 0.f, A1 = 0.f;
#pragma unroll 1
      for (int w0 = 0; w0 < nact; w0 += WU) {
        float m[WU], dn[WU];
        float2 v[WU];
#pragma unroll
        for (int w = 0; w < WU; w++) {
          const bool on = w0 + w < nact;
          m[w] = on ? wm[(w0 + w) * R + r] : -INFINITY;
          dn[w] = on ? wd[(w0 + w) * R + r] : 0.f;
          v[w] = on ? *reinterpret_cast<const float2*>(wacc + ((w0 + w) * R + r) * HD + d) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int w = 0; w < WU; w++) {
          const float e = ex2(m[w] - gm);
          Dn += dn[w] * e;
          A0 += v[w].x * e;
          A1 += v[w].y * e;
        }
      }
      if (a.nchunks == 1) {
        ll_store(a.ao_ll + (size_t)(kvh * R + r) * HP + (d >> 1), (uint32_t)f2bf(A0 / Dn) | ((uint32_t)f2bf(A1 / Dn) << 16), a.tag_out);
      } else {
        ll_store2(mine + r * HD + d, __float_as_uint(A0), __float_as_uint(A1), a.tag_part);
        if (d == 0) {
          ll_store(mine + R * HD + r, __float_as_uint(gm), a.tag_part);
          ll_store(mine + R * HD + R + r, __float_as_uint(Dn), a.tag_part);
        }
      }
    }
    if (a.nchunks > 1) {
      // Every chunk CTA of the kv head merges its share of the output: dim pairs c, c + nchunks, ... From each chunk's
      // partial it needs the 2R words (max, denominator) and its own pairs only: one 16-byte tagged load per thread,
      // no counter, no fence, a single round trip.
      named_bar_sync(kBarConsumers, kConsumerThreads);        // wacc / wm / wd are dead: scratch is free
      constexpr int npairs = R * HP;
      const int nown = (npairs - c + a.nchunks - 1) / a.nchunks;
      const int per = R + nown;                                // loads per source chunk
      uint32_t* pg = reinterpret_cast<uint32_t*>(scratch);     // [nchunks][per][2] payloads
      const int total = a.nchunks * per;                       // <= kConsumerThreads (host checks the shape)
      if (tid_c < total) {
        const int cc = tid_c / per, sl2 = tid_c - cc * per;
        int w;
        if (sl2 < R) {
          w = R * HD + 2 * sl2;
        } else {
          const int o = c + (sl2 - R) * a.nchunks;
          w = (o / HP) * HD + 2 * (o % HP);
        }
        const uint64_t* src = a.part_ll + ((size_t)kvh * a.maxchunks + cc) * WPC + w;
#pragma unroll 1
        for (unsigned spin = 0;; spin++) {
          uint64_t u, v;
          ll_load2(src, u, v);
          if ((uint32_t)(u >> 32) == a.tag_part && (uint32_t)(v >> 32) == a.tag_part) {
            *reinterpret_cast<uint2*>(pg + 2 * tid_c) = make_uint2((uint32_t)u, (uint32_t)v);
            break;
          }
          if (poll_again(spin, wc, layer, (int)a.tag_part, -4)) break;
        }
      }
      named_bar_sync(kBarConsumers, kConsumerThreads);
      if (tid_c < nown) {
        const float* pf = reinterpret_cast<const float*>(pg);
        const int o = c + tid_c * a.nchunks, r = o / HP, d = 2 * (o % HP);
        // words 0..R-1 of a chunk's (max, denominator) area are the maxima, R..2R-1 the denominators
        float gm = -1e30f;
#pragma unroll 4
        for (int cc = 0; cc < a.nchunks; cc++) gm = fmaxf(gm, pf[cc * per * 2 + r]);
        float Dn = 0.f, A0 = 0.f, A1 = 0.f;
#pragma unroll 4
        for (int cc = 0; cc < a.nchunks; cc++) {
          const float e = ex2(pf[cc * per * 2 + r] - gm);
          const float2 v = *reinterpret_cast<const float2*>(pf + (cc * per + R + tid_c) * 2);
          Dn += pf[cc * per * 2 + R + r] * e;
          A0 += v.x * e;
          A1 += v.y * e;
        }
        ll_store(a.ao_ll + (size_t)(kvh * R + r) * HP + (d >> 1), (uint32_t)f2bf(A0 / Dn) | ((uint32_t)f2bf(A1 / Dn) << 16), a.tag_out);
      }
    }
    named_bar_sync(kBarConsumers, kConsumerThreads);          // the scratch is free for the next item
  }
}

// Producer side of the attention: the K and V rows of this CTA's chunk(s), NPS positions per ring stage. The caches are
// [layer * max_seq + position][kv head][HD]: 4-D tensors (column, column block, kv head, row), one copy per matrix, stage and
// column block brings the strided rows in one request. Rows past the chunk (the last stage) are real cache rows that
// nobody reads; past the end of the cache the copy fills zeros. Called by the producer lane.
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int w, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar)) : "memory");
}
template <int HD, int STG>
__device__ __forceinline__ bool produce_kv(Pipe& p, const CUtensorMap* kmap, const CUtensorMap* vmap, int row0, int nkv, int nchunks,
                                           int T, int b, int G, const WaitCtl& wc, int layer) {
  using C = AttnCfg<HD, STG>;
  const int items = nkv * nchunks, chunk_len = (T + nchunks - 1) / nchunks;
#pragma unroll 1
  for (int item = b; item < items; item += G) {
    const int kvh = item / nchunks, c = item - kvh * nchunks, t0 = c * chunk_len, t1 = min(T, t0 + chunk_len);
#pragma unroll 1
    for (int ts = t0; ts < t1; ts += C::NPS) {
      if (!stage_slot(p, wc, layer)) return false;
      const int s = (int)(p.it % kStages);
      mbar_expect_tx(&p.full[s], (uint32_t)C::KV_STAGE_BYTES);
      uint8_t* dst = p.stages + (size_t)s * STG;
#pragma unroll
      for (int bl = 0; bl < C::BLKS; bl++) {
        tma_load_4d(dst + bl * (C::NPS * C::ROWB), kmap, 0, bl, kvh, row0 + ts, &p.full[s]);
        tma_load_4d(dst + C::MATRIX_BYTES + bl * (C::NPS * C::ROWB), vmap, 0, bl, kvh, row0 + ts, &p.full[s]);
      }
      if (!stage_issued(p, wc, layer)) return false;
    }
  }
  return true;
}

// ------------------------------------------------------------------------------------------------ kernel
struct Decode2Params {
  CUtensorMap kmap, vmap;     // the K / V caches as (column, column block, kv head, n_layer * max_seq rows) tensors
  const uint8_t *w_qkv, *w_o, *w_gu, *w_d, *w_lm;
  const uint16_t *n1, *n2, *nf, *embed;
  const float* invf;
  uint16_t *kc, *vc;
  uint64_t *h_ll, *q_ll, *k_ll, *v_ll, *ao_ll, *act_ll, *cand_ll;   // tagged vectors
  uint64_t* part_ll;
  DevStatus* status;
  const int32_t* d_token;
  uint16_t* d_h;
  float* d_logits;
  int32_t* d_next;
  int32_t token, pos, max_seq;
  int32_t n_layer, dim, n_head, n_kv, ffn, vocab, nchunks, maxchunks;
  unsigned tag_base, spin_limit;
  float eps, attn_scale, resid, emb_mult, logits_scaling;
  long long* prof;
  unsigned max_fly, lm_fly;   // bulk copies in flight per CTA while the layers run, and for the LM head
  // tensor parallelism: this GPU holds a slice of every matrix (heads, FFN columns, vocabulary rows); the partial sums
  // of the K-sharded O and down projections are exchanged by peer stores into every rank's inbox
  int32_t tp_size, tp_rank, vocab_base;
  int32_t ao_off;             // columns between the start of this rank's O window and its own attention output (0 or 64)
  uint64_t* inbox;            // local: [2 parities][tp_size][dim] tagged fp32 partials, then [tp_size][2] arg-max candidates
  uint64_t* peer_inbox[8];    // the same buffer of every rank (peer-mapped); own entry = inbox
};

// tags: phase ids inside a layer
enum { PH_QKV = 1, PH_ATT = 2, PH_O = 3, PH_GU = 4, PH_DOWN = 5, PH_LM = 6, PH_PART = 7 };
__device__ __forceinline__ uint32_t mk_tag(unsigned base, int layer, int ph) { return base + (unsigned)(layer * 8 + ph); }

__host__ __device__ constexpr int imax(int a, int b) { return a > b ? a : b; }

// the ring stage of a kernel of these widths
template <int KDIM, int KOUT, int KFFN>
using DecodePlan = SmemPlan<imax(KDIM, imax(KOUT, KFFN))>;

// TP: the kernel of a rank of several (the exchange's code, even where it never runs, costs a single GPU 1 to 7 %: 3B / 1B / 8B-class 821 / 298 / 1545 us a token
// with it, 794 / 280 / 1442 without)
template <int KDIM, int KOUT, int KFFN, int HD, int R, bool HZ, bool TP>
__global__ void __launch_bounds__(kThreads, 1) decode_mega2(const __grid_constant__ Decode2Params P) {
  using S = DecodePlan<KDIM, KOUT, KFFN>;
  constexpr int STG = S::STAGE;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  Smem sm = carve_smem(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = gridDim.x, b = blockIdx.x;
  // (cos, sin) of this step's position for every rotation pair: once per launch instead of a full-range sincosf in every
  // QKV epilogue of every layer
  __shared__ float2 s_rope[64];
  if (tid == 0) pipe_init(sm);
  if (tid < HD / 2) {
    float sn, cs;
    sincosf((float)P.pos * __ldg(P.invf + tid), &sn, &cs);
    s_rope[tid] = make_float2(cs, sn);
  }
  __syncthreads();
  WaitCtl wc{P.status, sm.s_abort, P.spin_limit};
  Pipe pipe{smem_raw + S::RING, sm.full, sm.empty, sm.landed, 0u, P.max_fly, STG};
  constexpr int HP = HD / 2;
  using CD = TCfg<KDIM, STG>;                 // QKV, gate/up, LM head
  using CO = TCfg<KOUT, STG>;                 // O projection (K = this rank's attention output width)
  using CF = TCfg<KFFN, STG>;                 // down projection
  constexpr int UO = imax(CO::RT, CF::RT);    // O and down give a CTA the same rows of the residual stream
  const int D = P.dim, FF = P.ffn, L = P.n_layer, V = P.vocab;
  const int QKV = (P.n_head + 2 * P.n_kv) * HD;
  constexpr int recD = rec_bytes_of(KDIM, HZ), recO = rec_bytes_of(KOUT, HZ), recF = rec_bytes_of(KFFN, HZ);
  const size_t strQ = (size_t)pad_rows(QKV, KDIM) * recD, strO = (size_t)pad_rows(D, KOUT) * recO,
               strG = (size_t)pad_rows(2 * FF, KDIM) * recD, strF = (size_t)pad_rows(D, KFFN) * recF;
  const int N = TP ? P.tp_size : 1, me = TP ? P.tp_rank : 0;
  int q0, q1, o0, o1, g0, g1, l0, l1;
  cta_rows(QKV, CD::RT, b, G, q0, q1);
  cta_rows(D, UO, b, G, o0, o1);         // the same rows of h belong to this CTA in the O and the down phase
  cta_rows(2 * FF, CD::RT, b, G, g0, g1);   // (g_i, u_i, g_i+1, u_i+1) stay together: one tagged word of activations
  cta_rows(V, CD::RT, b, G, l0, l1);

  if (warp == kConsumerWarps) {
    if (lane == 0) {
      bool ok = true;
#pragma unroll 1
      for (int l = 0; l < L && ok; l++) {
        ok = produce_rows<CD, HZ>(pipe, P.w_qkv + l * strQ, q0, q1, wc, l);
        ok = ok && produce_kv<HD, STG>(pipe, &P.kmap, &P.vmap, l * P.max_seq, P.n_kv, P.nchunks, P.pos + 1, b, G, wc, l);
        ok = ok && produce_rows<CO, HZ>(pipe, P.w_o + l * strO, o0, o1, wc, l) && produce_rows<CD, HZ>(pipe, P.w_gu + l * strG, g0, g1, wc, l) &&
             produce_rows<CF, HZ>(pipe, P.w_d + l * strF, o0, o1, wc, l);
      }
      pipe.max_fly = P.lm_fly;
      if (ok) produce_rows<CD, HZ>(pipe, P.w_lm, l0, l1, wc, L);
    }
  } else {
    const int cw = warp, tid_c = tid;
    float* hown = sm.hown;                                      // this CTA's rows of the residual stream (exact bf16 values)
    // what this warp takes of every phase (its own entries: no barrier needed beyond the warp)
    uint32_t* units = sm.units + cw;
    if (lane == 0) {
      units[0] = unit_entry_far((q1 - q0 + CD::RT - 1) / CD::RT * CD::NC, CD::RPC, cw);
      units[16] = unit_entry_far((o1 - o0 + CO::RT - 1) / CO::RT * CO::NC, CO::RPC, cw);
      units[32] = unit_entry_far((g1 - g0 + CD::RT - 1) / CD::RT * CD::NC, CD::RPC, cw);
      units[48] = unit_entry_far((o1 - o0 + CF::RT - 1) / CF::RT * CF::NC, CF::RPC, cw);
    }
    __syncwarp();
    const QueueState qs_{sm.qpart, sm.tdone, sm.bcnt};
    const XStage xs_{sm.x8, sm.xf};
    float* ypart = sm.hown + kMaxOwnRows;                       // tensor parallel: this rank's partial sums of its rows
    constexpr int MAXP_O = (KOUT / 4 + kConsumerThreads - 1) / kConsumerThreads;
    // O / down epilogue. One GPU: h = bf16(h + y * resid) at once. Tensor parallel: y is a partial sum over this
    // rank's K slice: keep it, push it to every peer's inbox, finish in resid_finish once all rows are done.
    auto resid_epi = [&](int row0, float c, int nvalid, uint32_t tag, int par) {
      const int r = row0 + (lane >> 2);
      if (N > 1) {
        // quad r holds the partial sum of row row0 + r; lane j < N-1 pushes all eight to one peer, 16 bytes a store, so the N-1 transfers of a tile
        // leave the SM side by side instead of one after the other
        if ((lane & 3) == 0 && (lane >> 2) < nvalid) ypart[r] = c;
        const int p = lane >= me ? lane + 1 : lane;
        uint64_t* dst = P.peer_inbox[lane < N - 1 ? p : me] + ((size_t)(par * N + me)) * D + o0 + row0;     // 64-byte aligned: row0 % 8 == 0
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          const float c0 = __shfl_sync(0xffffffffu, c, 4 * i), c1 = __shfl_sync(0xffffffffu, c, 4 * i + 4);
          if (lane < N - 1 && i < nvalid) ll_store2_sys(dst + i, __float_as_uint(c0), __float_as_uint(c1), tag);      // whole pairs: dim is even
        }
        return;
      }
      float hn = 0.f;
      if ((lane & 3) == 0 && (lane >> 2) < nvalid) {
        hn = rbf(hown[r] + c * P.resid);
        hown[r] = hn;
      }
      const float hn1 = __shfl_down_sync(0xffffffffu, hn, 4);
      if ((lane & 7) == 0 && (lane >> 2) < nvalid)
        ll_store(P.h_ll + ((o0 + r) >> 1), (uint32_t)f2bf(hn) | ((uint32_t)f2bf(hn1) << 16), tag);
    };
    // tensor parallel only: collect the peers' partials of this CTA's rows (one 16-byte load per thread and poll round,
    // all peers and row pairs in flight together), sum in rank order (identical on every rank), update h, publish
    float* yin = sm.yin;                                      // [N-1][kMaxOwnRows]
    auto resid_finish = [&](uint32_t tag, int par, int layer) {
      const int npair = (o1 - o0) / 2, nitem = npair * (N - 1);
#pragma unroll 1
      for (int it = tid_c; it < nitem; it += kConsumerThreads) {
        const int j = it / npair, pr = it % npair, s2 = j >= me ? j + 1 : j;
        const uint64_t* src = P.inbox + ((size_t)(par * N + s2)) * D + o0 + 2 * pr;
#pragma unroll 1
        for (unsigned spin = 0;; spin++) {
          uint64_t u, v;
          ll_load2_sys(src, u, v);
          if ((uint32_t)(u >> 32) == tag && (uint32_t)(v >> 32) == tag) {
            yin[j * kMaxOwnRows + 2 * pr] = __uint_as_float((uint32_t)u);
            yin[j * kMaxOwnRows + 2 * pr + 1] = __uint_as_float((uint32_t)v);
            break;
          }
          if (*wc.s_abort) break;
          if ((spin & 255) == 255 && ld_volatile_s32(&wc.st->abort)) { *wc.s_abort = 1; break; }
          if (spin >= wc.limit) { report_fail_far(wc, W_FLAG, layer, (int)tag, -3); break; }
        }
      }
      named_bar_sync(kBarConsumers, kConsumerThreads);        // every row's own partial and every peer's are in shared memory
#pragma unroll 1
      for (int pr = tid_c; pr < npair; pr += kConsumerThreads) {
        float tot0 = 0.f, tot1 = 0.f;
#pragma unroll 1
        for (int s2 = 0; s2 < N; s2++) {
          const float* src = s2 == me ? ypart : yin + (s2 > me ? s2 - 1 : s2) * kMaxOwnRows;
          tot0 += src[2 * pr]; tot1 += src[2 * pr + 1];
        }
        const float h0 = rbf(hown[2 * pr] + tot0 * P.resid), h1 = rbf(hown[2 * pr + 1] + tot1 * P.resid);
        hown[2 * pr] = h0; hown[2 * pr + 1] = h1;
        ll_store(P.h_ll + ((o0 >> 1) + pr), (uint32_t)f2bf(h0) | ((uint32_t)f2bf(h1) << 16), tag);
      }
      named_bar_sync(kBarConsumers, kConsumerThreads);
    };
    constexpr int MAXP_D = (KDIM / 4 + kConsumerThreads - 1) / kConsumerThreads;
    constexpr int MAXP_F = (KFFN / 4 + kConsumerThreads - 1) / kConsumerThreads;
    // ---- residual stream at layer 0: every CTA reads the embedding row (or the caller's h) itself ----
    {
      int tok = P.d_token ? (int)ld_cg_u32(P.d_token) : P.token;
      if ((unsigned)tok >= (unsigned)(V * N)) {                 // V is this rank's slice of the vocabulary
        tok = 0;
        if (tid_c == 0 && b == 0) atomicCAS(&P.status->code, 0, 6 /*FB_ERR_RANGE*/);
      }
#pragma unroll 1
      for (int i = tid_c; i < D; i += kConsumerThreads) {
        const uint16_t v = P.d_h ? ld_cg_u16(P.d_h + i) : f2bf(bf2f(__ldg(P.embed + (size_t)tok * D + i)) * P.emb_mult);
        reinterpret_cast<uint16_t*>(sm.x8)[i] = v;
        if (i >= o0 && i < o1) hown[i - o0] = bf2f(v);
      }
      named_bar_sync(kBarConsumers, kConsumerThreads);
    }
#define FB_STAMP(i) do { if (P.prof && tid_c == 0) P.prof[((size_t)b * L + l) * 16 + (i)] = (long long)globaltimer_ns(); } while (0)
#pragma unroll 1
    for (int l = 0; l < L; l++) {
      uint16_t* kcl = P.kc + (size_t)l * P.max_seq * P.n_kv * HD;
      uint16_t* vcl = P.vc + (size_t)l * P.max_seq * P.n_kv * HD;
      const uint32_t tg_qkv = mk_tag(P.tag_base, l, PH_QKV), tg_att = mk_tag(P.tag_base, l, PH_ATT),
                     tg_o = mk_tag(P.tag_base, l, PH_O), tg_gu = mk_tag(P.tag_base, l, PH_GU),
                     tg_dn = mk_tag(P.tag_base, l, PH_DOWN);
      // ================= QKV: norm1 -> GEMV -> RoPE -> tagged q / new k / new v, cache append =================
      FB_STAMP(0);
      if (q1 > q0) stage_norm_ll<MAXP_D, HZ>(P.h_ll, mk_tag(P.tag_base, l - 1, PH_DOWN), P.n1 + (size_t)l * D, D, P.eps,
                            P.status, P.spin_limit, l, l == 0, P.prof ? P.prof + ((size_t)b * L + l) * 16 : nullptr);
      FB_STAMP(1);
      consume_tiles<CD, HZ>(pipe, q1 - q0, units[0], xs_, qs_, cw, lane, wc, l, [&](int row0, float c, int nvalid) {
        // quad r holds row row0 + r: four RoPE pairs (or eight v dims)
        const float c1 = __shfl_down_sync(0xffffffffu, c, 4);
        if ((lane & 7) == 0 && (lane >> 2) < nvalid) {
          const int rs = q0 + row0 + (lane >> 2);              // stream row of the pair's first element (even)
          const int head = rs / HD, within = rs % HD;
          if (head < P.n_head + P.n_kv) {
            const int i = within >> 1;
            const float x0 = rbf(c), x1 = rbf(c1);
            const float cs = s_rope[i].x, sn = s_rope[i].y;
            const uint32_t y0 = f2bf(x0 * cs - x1 * sn), y1 = f2bf(x1 * cs + x0 * sn);
            if (head < P.n_head) {
              ll_store(P.q_ll + (size_t)head * HP + i, y0 | (y1 << 16), tg_qkv);
            } else {
              const int kvh = head - P.n_head;
              ll_store(P.k_ll + (size_t)kvh * HP + i, y0 | (y1 << 16), tg_qkv);
              uint16_t* kr = kcl + ((size_t)P.pos * P.n_kv + kvh) * HD;
              kr[i] = (uint16_t)y0;
              kr[i + HP] = (uint16_t)y1;
            }
          } else {
            const int kvh = head - P.n_head - P.n_kv;
            const uint32_t pv = (uint32_t)f2bf(c) | ((uint32_t)f2bf(c1) << 16);
            ll_store(P.v_ll + (size_t)kvh * HP + (within >> 1), pv, tg_qkv);
            *reinterpret_cast<uint32_t*>(vcl + ((size_t)P.pos * P.n_kv + kvh) * HD + within) = pv;
          }
        }
      }, P.prof ? P.prof + ((size_t)b * L + l) * 16 : nullptr);
      FB_STAMP(2);
      // ================= attention =================
      {
        const AttnArgs aa{P.q_ll, P.k_ll, P.v_ll, TP ? P.ao_ll + (P.ao_off >> 1) : P.ao_ll, P.part_ll, P.n_kv, P.pos, P.nchunks,
                     P.maxchunks, P.attn_scale, tg_qkv, mk_tag(P.tag_base, l, PH_PART), tg_att};
        named_bar_sync(kBarConsumers, kConsumerThreads);        // scratch (the activations) is free: every warp left the GEMV
        attention_phase<HD, R, STG>(aa, sm.scratch, cw, lane, tid_c, wc, l, pipe, sm.tdone);
      }
      FB_STAMP(3);
      // ================= O projection + residual =================
      {
        // a rank of several: the window's other columns belong to a neighbour, whose O projection sees them; this one sees zeros there
        if constexpr (TP) {
          const WordPairs own = o_words(P.n_head * HD, P.ao_off);
          if (o1 > o0) stage_plain_ll<imax(MAXP_O, MAXP_F), HZ>(P.ao_ll, tg_att, KOUT, P.status, P.spin_limit, l, own.first, own.end);
        } else {
          if (o1 > o0) stage_plain_ll<imax(MAXP_O, MAXP_F), HZ>(P.ao_ll, tg_att, KOUT, P.status, P.spin_limit, l);
        }
        FB_STAMP(4);
        consume_tiles<CO, HZ>(pipe, o1 - o0, units[16], xs_, qs_, cw, lane, wc, l,
                                  [&](int row0, float c, int nvalid) { resid_epi(row0, c, nvalid, tg_o, 0); });
        if (N > 1) resid_finish(tg_o, 0, l);
      }
      FB_STAMP(5);
      // ================= gate/up + SwiGLU =================
      if (g1 > g0) stage_norm_ll<MAXP_D, HZ>(P.h_ll, tg_o, P.n2 + (size_t)l * D, D, P.eps, P.status, P.spin_limit, l, false);
      FB_STAMP(6);
      consume_tiles<CD, HZ>(pipe, g1 - g0, units[32], xs_, qs_, cw, lane, wc, l, [&](int row0, float c, int nvalid) {
        // rows (g_i, u_i, ...) -> act[i] .. act[i + 3] -> two tagged words
        const float u = __shfl_down_sync(0xffffffffu, c, 4);
        float av = 0.f;
        if ((lane & 7) == 0 && (lane >> 2) < nvalid) {
          const float gg = rbf(c), uu = rbf(u);
          av = rbf((gg / (1.0f + __expf(-gg))) * uu);
        }
        const float av1 = __shfl_down_sync(0xffffffffu, av, 8);
        if ((lane & 15) == 0 && (lane >> 2) + 4 <= nvalid)
          ll_store(P.act_ll + ((g0 + row0) >> 2) + (lane >> 4), (uint32_t)f2bf(av) | ((uint32_t)f2bf(av1) << 16), tg_gu);
      });
      FB_STAMP(7);
      // ================= down projection + residual =================
      {
        if constexpr (TP) {
          if (o1 > o0) stage_plain_ll<imax(MAXP_O, MAXP_F), HZ>(P.act_ll, tg_gu, FF, P.status, P.spin_limit, l, 0, FF / 4);
        } else {
          if (o1 > o0) stage_plain_ll<imax(MAXP_O, MAXP_F), HZ>(P.act_ll, tg_gu, FF, P.status, P.spin_limit, l);
        }
        FB_STAMP(8);
        consume_tiles<CF, HZ>(pipe, o1 - o0, units[48], xs_, qs_, cw, lane, wc, l,
                                  [&](int row0, float c, int nvalid) { resid_epi(row0, c, nvalid, tg_dn, 1); });
        if (N > 1) resid_finish(tg_dn, 1, l);
      }
      FB_STAMP(9);
    }
#undef FB_STAMP
    // ================= final norm + LM head + arg-max =================
    stage_norm_ll<MAXP_D, HZ>(P.h_ll, mk_tag(P.tag_base, L - 1, PH_DOWN), P.nf, D, P.eps, P.status, P.spin_limit, L, false);
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    consume_tiles<CD, HZ>(pipe, l1 - l0, unit_entry_far((l1 - l0 + CD::RT - 1) / CD::RT * CD::NC, CD::RPC, cw), xs_, qs_, cw, lane, wc, L, [&](int row0, float c, int nvalid) {
      if ((lane & 3) == 0 && (lane >> 2) < nvalid) {
        const int row = P.vocab_base + l0 + row0 + (lane >> 2);     // index in the full vocabulary
        const float y = c / P.logits_scaling;
        if (P.d_logits) P.d_logits[row] = y;
        if (y > bv || (y == bv && row < bi)) { bv = y; bi = row; }
      }
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { sm.red[cw] = bv; sm.misc[cw] = bi; }
    named_bar_sync(kBarConsumers, kConsumerThreads);
    const uint32_t tg_lm = mk_tag(P.tag_base, L, PH_LM);
    if (tid_c == 0) {
#pragma unroll 1
      for (int w = 1; w < kConsumerWarps; w++)
        if (sm.red[w] > bv || (sm.red[w] == bv && sm.misc[w] < bi)) { bv = sm.red[w]; bi = sm.misc[w]; }
      ll_store(P.cand_ll + 2 * b, __float_as_uint(bv), tg_lm);
      ll_store(P.cand_ll + 2 * b + 1, (uint32_t)bi, tg_lm);
    }
    if (b == 0) {
      uint32_t* cs = reinterpret_cast<uint32_t*>(sm.x8);
      named_bar_sync(kBarConsumers, kConsumerThreads);
      uint2 cand[1];
      ll_gather<1>(P.cand_ll, G, tg_lm, cand, tid_c, kConsumerThreads, wc, L);
      if (tid_c < G) *reinterpret_cast<uint2*>(cs + 2 * tid_c) = cand[0];
      named_bar_sync(kBarConsumers, kConsumerThreads);
      if (cw == 0) {
        float v = -INFINITY;
        int ix = 0x7fffffff;
#pragma unroll 1
        for (int c = lane; c < G; c += 32) {
          const float ov = __uint_as_float(cs[2 * c]);
          const int oi = (int)cs[2 * c + 1];
          if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, v, o);
          const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
          if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
        }
        if (N > 1 && lane == 0) {
          // every rank holds a slice of the vocabulary: exchange the N (value, index) candidates, reduce in rank order
          uint64_t* mine = P.inbox + (size_t)2 * N * D;
#pragma unroll 1
          for (int p = 0; p < N; p++) {
            uint64_t* dst = (p == me ? mine : P.peer_inbox[p] + (size_t)2 * N * D) + 2 * me;
            ll_store_sys(dst, __float_as_uint(v), tg_lm);
            ll_store_sys(dst + 1, (uint32_t)ix, tg_lm);
          }
          v = -INFINITY; ix = 0x7fffffff;
#pragma unroll 1
          for (int s2 = 0; s2 < N; s2++) {
            const float ov = __uint_as_float(ll_poll_sys(mine + 2 * s2, tg_lm, wc, L));
            const int oi = (int)ll_poll_sys(mine + 2 * s2 + 1, tg_lm, wc, L);
            if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
          }
        }
        if (lane == 0 && P.d_next) *P.d_next = ix;
      }
    }
    // final residual back to the caller (the reference clobbers its h argument): every CTA writes its own rows
    if (P.d_h)
#pragma unroll 1
      for (int r = tid_c; r < o1 - o0; r += kConsumerThreads) P.d_h[o0 + r] = f2bf(hown[r]);
  }
  __syncthreads();
  if (*sm.s_abort && tid == kConsumerThreads) drain_ring<kStages>(pipe.full, pipe.it);
}

}  // namespace fb
