// The weight pipeline every streaming kernel of this library shares, the stand-alone GEMV built on it and the kernels
// that convert between the caller's weight layout and the tiled streaming layout.
//
// One CTA per SM: the last warp (lane 0) is the producer; it walks the CTA's static list of weight tiles and issues
// 1-D bulk copies into an 8-stage shared-memory ring. It never waits for activations, so the weights of the next
// phase stream in while the consumers are still waiting for their inputs. The other warps are consumers: warp w takes
// tiles w, w + n, ... straight off the ring; there are no warp groups and no block-wide barriers in the steady state.
#pragma once
#include "fb_common.cuh"

namespace fb {

struct Pipe {
  uint8_t* stages;
  uint64_t* full;
  uint64_t* empty;
  volatile int* landed;  // stage loads that are known to be complete (written by the producer, read by consumers)
  uint32_t it;           // running stage-load counter; producer and consumers walk the same sequence
  uint32_t max_fly;      // producer only: bulk copies allowed in flight at once (1..kStages/2)
  uint32_t stage_bytes;  // SmemPlan::STAGE
};

struct Smem {
  uint8_t* scratch;
  uint8_t* x8;         // activations of the current phase (see XStage)
  uint64_t* full;
  uint64_t* empty;
  volatile int* s_abort;
  volatile int* landed;
  float* red;          // 32 floats for block reductions
  int* misc;           // 32 ints
  float* hown;         // [2 * kMaxOwnRows] this CTA's rows of the residual stream, then tensor-parallel partial sums
  uint32_t* units;     // [4 phases][16] unit_entry of every warp
  int* tdone;          // [kStages] units finished per stage in flight
  int* bcnt;           // [32] units finished per tile in flight
  float4* xf;          // [112] per-group activation factors
  float* yin;          // [7][kMaxOwnRows] tensor parallel: the peers' partial sums of this CTA's rows
  float* qpart;        // slice partials
};

__device__ __forceinline__ Smem carve_smem(uint8_t* base) {
  Smem s;
  s.full = reinterpret_cast<uint64_t*>(base);
  s.empty = s.full + kStages;
  s.s_abort = reinterpret_cast<volatile int*>(base + 128);
  s.landed = reinterpret_cast<volatile int*>(base + 132);
  s.red = reinterpret_cast<float*>(base + 256);
  s.misc = reinterpret_cast<int*>(base + 384);
  s.hown = reinterpret_cast<float*>(base + 512);
  s.units = reinterpret_cast<uint32_t*>(base + 1024);
  s.tdone = reinterpret_cast<int*>(base + 1280);
  s.bcnt = reinterpret_cast<int*>(base + 1312);
  s.xf = reinterpret_cast<float4*>(base + 1536);
  s.yin = reinterpret_cast<float*>(base + 3328);
  s.qpart = reinterpret_cast<float*>(base + 5120);
  s.scratch = base + kTailBytes;
  s.x8 = s.scratch;
  return s;
}
static_assert(2 * kMaxOwnRows * 4 <= 512 && 3328 + 7 * kMaxOwnRows * 4 <= 5120 && 5120 + kPartBytes <= kTailBytes, "tail layout");

// called by one thread before the CTA-wide barrier that opens the kernel
__device__ __forceinline__ void pipe_init(const Smem& sm) {
  for (int s = 0; s < kStages; s++) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); sm.tdone[s] = 0; }
  for (int i = 0; i < 32; i++) sm.bcnt[i] = 0;
  *sm.s_abort = 0;
  *sm.landed = 0;
  mbar_fence_init();
}

// rows [r0, r1) of a phase that CTA b of G owns; `unit` rows stay together (the tile height of the matrix)
__device__ __forceinline__ void cta_rows(int rows, int unit, int b, int G, int& r0, int& r1) {
  r0 = cta_first_row(rows, unit, b, G);
  r1 = cta_first_row(rows, unit, b + 1, G);
}

// ------------------------------------------------------------------------------------------------ producer side
// The number of copies in flight is kept short: with the whole ring in flight (27 MB over 148 SMs) every small
// latency-critical access of the consumers (tagged words) waits microseconds behind bulk weight traffic. The trailing
// wait of stage_issued also tells the consumers which loads have landed: one may only wait for load i on a stage's
// one-bit phase once load i - kStages is known to be complete.
__device__ __forceinline__ bool stage_slot(const Pipe& p, const WaitCtl& wc, int layer) {
  return mbar_wait_far(&p.empty[p.it % kStages], ((p.it / kStages) & 1) ^ 1, wc, W_EMPTY, layer);     // p.it counts issued loads only
}
__device__ __forceinline__ bool stage_issued(Pipe& p, const WaitCtl& wc, int layer) {
  p.it++;
  if (p.it > p.max_fly) {
    const uint32_t j = p.it - 1 - p.max_fly;
    if (!mbar_wait_far(&p.full[j % kStages], (j / kStages) & 1, wc, W_FULL, layer)) return false;
    *p.landed = (int)(j + 1);
  }
  return true;
}
// `src`: the first of `nch` chunks of `bytes` each, `cps` of them per stage
__device__ __forceinline__ bool produce_chunks(Pipe& p, const uint8_t* src, int nch, int cps, uint32_t bytes, const WaitCtl& wc, int layer) {
#pragma unroll 1
  for (int c = 0; c < nch; c += cps) {
    const uint32_t n = (uint32_t)min(cps, nch - c) * bytes;
    if (!stage_slot(p, wc, layer)) return false;
    const int s = p.it % kStages;
    mbar_expect_tx(&p.full[s], n);
    bulk_g2s(p.stages + (size_t)s * p.stage_bytes, src + (size_t)c * bytes, n, &p.full[s]);
    if (!stage_issued(p, wc, layer)) return false;
  }
  return true;
}
// the whole tiles (the last may be partly padding) of a CTA's rows [r0, r1)
template <class C, bool HZ>
__device__ __forceinline__ bool produce_rows(Pipe& p, const uint8_t* w, int r0, int r1, const WaitCtl& wc, int layer) {
  constexpr int CH = C::chunk(HZ);
  return produce_chunks(p, w + (size_t)(r0 / C::RT) * (C::NC * CH), (r1 - r0 + C::RT - 1) / C::RT * C::NC, C::CPS, CH, wc, layer);
}

// ------------------------------------------------------------------------------------------------ consumer side
struct QueueState {
  float* qpart;
  int* tdone;
  int* bcnt;
};

// wait until stage load `it` has landed: on the stage's one-bit phase, once the stage's previous load is known to be complete
__device__ __forceinline__ bool wait_stage(const Pipe& p, uint32_t it, const WaitCtl& wc, int layer) {
  if (it >= (uint32_t)kStages) {
    bool ok = false;
#pragma unroll 1
    for (unsigned i = 0; i < wc.limit; i++) {
      if ((uint32_t)*p.landed > it - kStages) { ok = true; break; }
      if ((i & 63) == 63 && *wc.s_abort) break;
    }
    if (!ok) {
      if (*wc.s_abort == 0) report_fail_far(wc, W_LANDED, layer, (int)it, *p.landed);
      return false;
    }
  }
  return mbar_wait_far(&p.full[it % kStages], (it / kStages) & 1, wc, W_FULL, layer);
}

// GEMV over this CTA's `nrows` rows of one phase (they start on a tile boundary); `entry`: the warp's unit_entry. Every finished group of up to 8 rows is
// handed to `epi(row0_local, c, nvalid)` by the whole warp, the lanes of quad r holding the total of row row0_local + r, so results leave the
// CTA as soon as they exist. A stage goes back to the producer when its last unit finishes (shared-memory counter); the warp that finishes the
// last unit of a tile of several adds their sums in order and runs the epilogue.
template <class C, bool HZ, class Epi>
__device__ __forceinline__ void consume_tiles(Pipe& p, int nrows, uint32_t entry, const XStage& x, const QueueState& q, int cw, int lane,
                                              const WaitCtl& wc, int layer, Epi epi, long long* dbg = nullptr) {
  constexpr int RT = C::RT, NC = C::NC, CPS = C::CPS, SLOTS = C::SLOTS;
  const int nch = (nrows + RT - 1) / RT * NC, nst = (nch + CPS - 1) / CPS;
  const int r0 = (entry >> 8) & 255, nr = (entry >> 16) & 255, ks = entry >> 24;
#pragma unroll 1
  for (int ch = entry & 255; ch < nch; ch += ks > 1 ? nch : kConsumerWarps) {
    const int st = ch / CPS, tl = ch / NC;
    const uint32_t it = p.it + st;
    const int s = it % kStages;
    if (!wait_stage(p, it, wc, layer)) break;
    if (dbg && cw == 0 && lane == 0 && ch == 0) dbg[13] = (long long)globaltimer_ns();
    float lo, hi;
    chunk_dot<C, HZ>(p.stages + (size_t)s * p.stage_bytes + (size_t)(ch % CPS) * C::chunk(HZ), ch % NC, r0, nr, x, lane, lo, hi);
    if (dbg && cw == 0 && lane == 0 && ch == 0) dbg[14] = (long long)globaltimer_ns();
    const int nvalid = min(RT, nrows - tl * RT);
    bool last = true;
    if (NC * ks > 1) {
      const int u = ks > 1 ? cw : ch;                            // units of a phase in order; sliced ones are the warps
      float* part = q.qpart + (u % SLOTS) * RT;
      if ((lane & 3) == 0) {
        part[lane >> 2] = lo;
        if (RT == 16) part[8 + (lane >> 2)] = hi;
      }
      __syncwarp();
      int fin = 0;
      if (lane == 0) {
        __threadfence_block();
        fin = atomicAdd(q.bcnt + tl % 32, 1) == NC * ks - 1;
        if (fin) q.bcnt[tl % 32] = 0;
      }
      last = __shfl_sync(0xffffffffu, fin, 0) != 0;
      if (last) {                                                // every unit of this tile is in
        __threadfence_block();
        lo = hi = 0.f;
        const int u0 = tl * NC * ks;
#pragma unroll 4
        for (int i = 0; i < NC * ks; i++) {
          const float* src = q.qpart + ((u0 + i) % SLOTS) * RT + (lane >> 2);
          lo += src[0];
          if (RT == 16) hi += src[8];
        }
      }
    }
    if (last) {
      epi(tl * RT, lo, min(8, nvalid));
      if (RT == 16) epi(tl * RT + 8, hi, min(8, nvalid - 8));
    }
    __syncwarp();
    if (lane == 0) {                                             // the stage's last unit hands the slot back
      const int units = min(CPS, nch - st * CPS) * ks;
      const int old = atomicAdd(q.tdone + s, 1);
      if (old == units - 1) {
        q.tdone[s] = 0;
        mbar_arrive(&p.empty[s]);
      }
    }
  }
  p.it += nst;
}

// ------------------------------------------------------------------------------------------------ stand-alone GEMV
struct GemvParams {
  const uint8_t* w;        // streaming layout
  const uint16_t* x;       // bf16 [K]
  float* y;                // f32 [rows], original row order
  DevStatus* status;
  int32_t rows, order, order_arg, order_rows;
  unsigned spin_limit;
};

// every consumer thread calls; ends with a consumer-wide barrier. A warp's groups are loaded and converted side by side (one after the other 2560 rows of K =
// 8192 / 14336 5.5 / 8.6 us a launch instead of 5.0 / 7.6).
template <int K, bool HZ>
__device__ __forceinline__ void stage_x_global(const uint16_t* gx, const Smem& sm, int tid_c) {
  constexpr int G = K / 128, N = (G + kConsumerWarps - 1) / kConsumerWarps;
  const int warp = tid_c >> 5, lane = tid_c & 31;
  uint2 v[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    const int grp = warp + k * kConsumerWarps;
    v[k] = grp < G ? __ldg(reinterpret_cast<const uint2*>(gx + grp * 128) + lane) : make_uint2(0, 0);
  }
  stage_groups<HZ, N>(v, warp, kConsumerWarps, G, sm.x8, sm.xf, lane);
  named_bar_sync(kBarConsumers, kConsumerThreads);
}

// Row r of `n` plain rows times x: what a thread's columns add, summed over its warp. All consumer threads of a CTA share a row, 32 columns (16 bytes) each: up to K =
// 14336 one load of weights and four of x a thread, side by side.
inline __device__ __noinline__ float plain_row_part(const uint8_t* base, int n, int r, int k, bool hz, const uint16_t* x, int tid_c) {
  const int G = k / 128;
  const uint4* q = reinterpret_cast<const uint4*>(base + (size_t)r * (k / 2));
  const uint16_t *sc = reinterpret_cast<const uint16_t*>(base + (size_t)n * (k / 2)) + (size_t)r * G, *zr = sc + (size_t)n * G;
  float acc = 0.f;
#pragma unroll 1
  for (int c = tid_c; c < k / 32; c += kConsumerThreads) {
    const uint4 w = __ldg(q + c);
    const uint4* xp = reinterpret_cast<const uint4*>(x) + 4 * c;
    const uint4 x0 = __ldg(xp), x1 = __ldg(xp + 1), x2 = __ldg(xp + 2), x3 = __ldg(xp + 3);
    const float s = bf2f(__ldg(sc + (c >> 2))), z = hz ? bf2f(__ldg(zr + (c >> 2))) : 0.f;
    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
    const uint4 xs[4] = {x0, x1, x2, x3};
    float dot = 0.f, sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t p[4] = {xs[i].x, xs[i].y, xs[i].z, xs[i].w};
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const float v = e & 1 ? bfhi(p[e >> 1]) : bflo(p[e >> 1]);
        dot = fmaf((float)(ws[i] >> (4 * e) & 15u) - 8.0f, v, dot);
        sum += v;
      }
    }
    acc = fmaf(s, dot, acc);
    if (hz) acc = fmaf(z, sum, acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

template <int K, bool HZ>
__global__ void __launch_bounds__(kThreads, 1) gemv_stream(const GemvParams P) {
  using S = SmemPlan<K>;
  using C = TCfg<K, S::STAGE>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  Smem sm = carve_smem(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) pipe_init(sm);
  __syncthreads();
  WaitCtl wc{P.status, sm.s_abort, P.spin_limit};
  Pipe pipe{smem_raw + S::RING, sm.full, sm.empty, sm.landed, 0u, 4u, S::STAGE};
  int r0, r1;
  const int full = P.rows / C::RT * C::RT;
  cta_rows(full, C::RT, blockIdx.x, gridDim.x, r0, r1);
  if (warp == kConsumerWarps) {
    if (lane == 0) produce_rows<C, HZ>(pipe, P.w, r0, r1, wc, 0);
  } else {
    // The rows behind the last whole tile, a CTA each from the first one on (cta_rows gives the first CTAs the fewest tiles), ahead of the staging: the tiles are on
    // their way meanwhile. 37 / 2567 / 16389 rows of K = 14336, 300 / 2563 / 16389 of K = 2560, a launch of a graph: 5.2 / 8.4 / 23.6 and 3.9 / 4.0 / 5.2 us; as scalar
    // loops of a warp each in one CTA 18.9 / 21.9 / 55.9 and 5.8 / 6.0 / 7.4. (Loading them beside the activations and multiplying behind the staging: no faster.)
    const int plain = P.rows - full;
    float* part = sm.yin;                                       // [row of this CTA][warp]
    int mine = 0;
    for (int r = blockIdx.x; r < plain; r += gridDim.x, mine++) {
      const float v = plain_row_part(P.w + (size_t)full * rec_bytes_of(K, HZ), plain, r, K, HZ, P.x, tid);
      if (lane == 0) part[16 * mine + warp] = v;
    }
    stage_x_global<K, HZ>(P.x, sm, tid);
    for (int i = warp; i < mine; i += kConsumerWarps) {
      float v = lane < kConsumerWarps ? part[16 * i + lane] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) P.y[perm_row(full + (int)blockIdx.x + i * (int)gridDim.x, P.order, P.order_arg, P.order_rows)] = v;
    }
    const XStage xs{sm.x8, sm.xf};
    const QueueState qs{sm.qpart, sm.tdone, sm.bcnt};
    const uint32_t entry = unit_entry((r1 - r0 + C::RT - 1) / C::RT * C::NC, C::RPC, warp);
    consume_tiles<C, HZ>(pipe, r1 - r0, entry, xs, qs, warp, lane, wc, 0, [&](int row0, float c, int nvalid) {
      if ((lane & 3) == 0 && (lane >> 2) < nvalid) P.y[perm_row(r0 + row0 + (lane >> 2), P.order, P.order_arg, P.order_rows)] = c;
    });
  }
  __syncthreads();
  if (*sm.s_abort && tid == kConsumerThreads) drain_ring<kStages>(pipe.full, pipe.it);
}

// ------------------------------------------------------------------------------------------------ layout kernels
// Caller layout -> tiles. One CTA per tile; blockIdx.y = layer (the matrices of all layers are stacked; every layer
// starts on a tile boundary and repeats the row order). Rows beyond `rows` are padding: nibble 8 (value 0), scale 0.
template <int K>
__global__ void repack_tiles(const uint32_t* q, const uint16_t* sc, const uint16_t* zr, int rows, int order, int order_arg,
                             int order_rows, uint8_t* out) {
  using C = TCfg<K, SmemPlan<K>::STAGE>;
  constexpr int RT = C::RT, KC = C::KC;
  const bool hz = zr != nullptr;
  const int T = blockIdx.x, tiles = (rows + RT - 1) / RT;
  uint8_t* tile = out + ((size_t)blockIdx.y * tiles + T) * tile_bytes(K, hz);
  __shared__ int src_row[16];
  if (threadIdx.x < RT) {
    const int j = T * RT + threadIdx.x;
    src_row[threadIdx.x] = j < rows ? (int)blockIdx.y * rows + perm_row(j, order, order_arg, order_rows) : -1;
  }
  __syncthreads();
  auto nib = [&](int r, int col) -> uint32_t {
    const int row = src_row[r];
    if (row < 0) return 8u;
    return (__ldg(q + (size_t)row * (K / 8) + (col >> 3)) >> (4 * (col & 7))) & 15u;
  };
  for (int wi = threadIdx.x; wi < C::NC * (C::NIB / 4); wi += blockDim.x) {
    const int k = wi / (C::NIB / 4), w0 = wi % (C::NIB / 4);     // chunk and word in it
    const int i = w0 & 3, lane = (w0 >> 2) & 31, bq = w0 >> 7, g = lane >> 2, t = lane & 3;
    const int rl = g % RT, rh = (g + 8) % RT, jl = g / RT, jh = (g + 8) / RT;
    const int c0 = k * KC + 64 * bq + 16 * t + 4 * i, cl = jl * (KC / C::NJ) + c0, ch = jh * (KC / C::NJ) + c0;
    uint32_t w = 0;
    for (int b = 0; b < 4; b++) w |= (nib(rh, ch + b) ^ 8u) << (8 * b) | (nib(rl, cl + b) ^ 8u) << (8 * b + 4);
    reinterpret_cast<uint32_t*>(tile + (size_t)k * C::chunk(hz))[w0] = w;
  }
  for (int i = threadIdx.x; i < RT * (K / 128); i += blockDim.x) {
    const int grp = i / RT, row = src_row[i % RT], k = grp / C::G, at = (grp % C::G) * RT + i % RT;
    uint16_t* meta = reinterpret_cast<uint16_t*>(tile + (size_t)k * C::chunk(hz) + C::NIB);
    meta[at] = row >= 0 ? sc[(size_t)row * (K / 128) + grp] : 0;
    if (hz) meta[RT * C::G + at] = row >= 0 ? zr[(size_t)row * (K / 128) + grp] : 0;
  }
}

// The rows from `full` on, plainly (see stream_row_unit). One CTA per row.
template <int UNIT = 0>      // (a template so that several translation units may include it)
__global__ void repack_plain(const uint32_t* q, const uint16_t* sc, const uint16_t* zr, int full, int k, int order, int order_arg, int order_rows, uint8_t* out) {
  const int n = gridDim.x, r = blockIdx.x, nw = k / 8, G = k / 128, row = perm_row(full + r, order, order_arg, order_rows);
  uint32_t* dq = reinterpret_cast<uint32_t*>(out) + (size_t)r * nw;
  uint16_t *ds = reinterpret_cast<uint16_t*>(out + (size_t)n * nw * 4) + (size_t)r * G, *dz = ds + (size_t)n * G;
  for (int w = threadIdx.x; w < nw; w += blockDim.x) dq[w] = q[(size_t)row * nw + w];
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    ds[g] = sc[(size_t)row * G + g];
    if (zr) dz[g] = zr[(size_t)row * G + g];
  }
}
template <int UNIT = 0>
__global__ void dequant_plain(const uint8_t* in, int full, int k, int has_zeros, int order, int order_arg, int order_rows, float* out) {
  const int n = gridDim.x, r = blockIdx.x, nw = k / 8, G = k / 128, row = perm_row(full + r, order, order_arg, order_rows);
  const uint32_t* q = reinterpret_cast<const uint32_t*>(in) + (size_t)r * nw;
  const uint16_t *sc = reinterpret_cast<const uint16_t*>(in + (size_t)n * nw * 4) + (size_t)r * G, *zr = sc + (size_t)n * G;
  for (int c = threadIdx.x; c < k; c += blockDim.x) {
    float v = ((float)(q[c >> 3] >> (4 * (c & 7)) & 15u) - 8.0f) * bf2f(sc[c >> 7]);
    if (has_zeros) v = v + bf2f(zr[c >> 7]);
    out[(size_t)row * k + c] = v;
  }
}

// tiles -> f32 [rows][K] in the caller's row order: (nib - 8) * scale (+ zero). One CTA per stream row.
template <int K>
__global__ void dequant_tiles(const uint8_t* in, int rows, int has_zeros, int order, int order_arg, int order_rows, float* out) {
  using C = TCfg<K, SmemPlan<K>::STAGE>;
  constexpr int RT = C::RT, KC = C::KC;
  const int j = blockIdx.x, T = j / RT, r = j % RT;
  const int dstrow = perm_row(j, order, order_arg, order_rows);
  const uint8_t* tile = in + (size_t)T * tile_bytes(K, has_zeros);
  for (int c = threadIdx.x; c < K; c += blockDim.x) {
    const uint8_t* chunk = tile + (size_t)(c / KC) * C::chunk(has_zeros);
    const uint16_t* meta = reinterpret_cast<const uint16_t*>(chunk + C::NIB);
    const int cc = c % KC, jr = cc / (KC / C::NJ), cl = cc % (KC / C::NJ), mrow = r + RT * jr;      // MMA row
    const int lane = 4 * (mrow & 7) + ((cl & 63) >> 4), i = (cl >> 2) & 3;
    const uint32_t w = reinterpret_cast<const uint32_t*>(chunk)[(((cl >> 6) * 32 + lane) << 2) + i];
    const float nibv = (float)(((w >> (8 * (cl & 3) + 4 * (1 - (mrow >> 3)))) & 0xF) ^ 8u) - 8.0f;
    const int at = (cc >> 7) * RT + r;
    float v = nibv * bf2f(meta[at]);
    if (has_zeros) v = v + bf2f(meta[RT * C::G + at]);
    out[(size_t)dstrow * K + c] = v;
  }
}

}  // namespace fb
