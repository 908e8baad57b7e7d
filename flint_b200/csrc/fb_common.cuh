// Shared device-side building blocks of the sm_100a decode path: PTX wrappers (mbarrier, 1-D bulk copies,
// coherent loads), bounded waits that report instead of hanging, the tiled streaming weight layout and the int4 tile x
// vector product (integer mma.sync) that every GEMV phase uses.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fb_geometry.hpp"

namespace fb {

// ------------------------------------------------------------------------------------------------ constants
#ifndef FB_CW
#define FB_CW 14      // 14 consumers + 1 producer = 15 warps -> at most 4 per scheduler -> 128 registers per thread
#endif
constexpr int kConsumerWarps = FB_CW;
constexpr int kConsumerThreads = kConsumerWarps * 32;
constexpr int kThreads = kConsumerThreads + 32;    // + one producer warp (lane 0 issues the bulk copies)
constexpr int kStages = 8;                         // ring depth
constexpr int kTailBytes = 6144;                   // mbarriers, flags, reductions, unit table, slice partials, owned rows, group factors
constexpr int kSmemBytes = 231424;                 // 226 KB: with the static variables what a CTA may have
constexpr int kAttnScratch = 40960;                // attention scratch, which shares its place with the activations
constexpr int kMaxOwnRows = 64;                    // rows of the residual stream one CTA may own
constexpr int kMaxGroups = 112;                    // K <= 14336

// named barriers (0 is __syncthreads)
constexpr int kBarConsumers = 1;                   // all consumer threads

// device status words (global memory, owned by the context)
struct DevStatus {
  int code;        // 0 ok, else FB_ERR_TIMEOUT
  int where;       // phase id of the wait that gave up
  int layer, block, expected, seen;
  int abort;       // set with the first failure; every other wait polls it and leaves
  int pad;
};

enum Where { W_FULL = 2, W_EMPTY = 3, W_FLAG = 5, W_LANDED = 6 };

// ------------------------------------------------------------------------------------------------ small helpers
__device__ __forceinline__ float bf2f(uint16_t b) { return __uint_as_float(((uint32_t)b) << 16); }
__device__ __forceinline__ float bflo(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float bfhi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
__device__ __forceinline__ uint16_t f2bf(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }
__device__ __forceinline__ float rbf(float f) { return bf2f(f2bf(f)); }   // round an fp32 value to bf16 precision

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// loads that must see data written by other SMs during this launch: L2 is the point of coherence
__device__ __forceinline__ uint32_t ld_cg_u32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint16_t ld_cg_u16(const void* p) {
  uint16_t v;
  asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_volatile_s32(const int* p) {
  int v;
  asm volatile("ld.volatile.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// ------------------------------------------------------------------------------------------------ mbarrier + bulk copy
__device__ __forceinline__ void mbar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// REMOTE: the phase is completed by stores of other CTAs of the cluster (st.async), whose data the waiter reads: acquire at cluster scope
// (the default is the CTA's own).
template <bool REMOTE = false>
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  if (REMOTE)
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok) : "r"(smem_u32(b)), "r"(parity) : "memory");
  else
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok) : "r"(smem_u32(b)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok) : "r"(smem_u32(b)), "r"(parity) : "memory");
  return ok != 0;
}
// global -> this CTA's shared memory, size and both addresses multiples of 16; completion counted on `bar`
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst_smem)), "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// ------------------------------------------------------------------------------------------------ clusters
// Barrier over all threads of all CTAs of a cluster (release / acquire unless said otherwise), and a neighbour's shared memory: the address of the
// same place there, stores, and stores that count as bytes on a barrier of that CTA.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() { cluster_arrive(); cluster_wait(); }
__device__ __forceinline__ uint32_t cluster_map(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, float4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];"
               ::"r"(addr), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar)
               : "memory");
}

// ------------------------------------------------------------------------------------------------ bounded waits
// Every wait in this library has an iteration limit. When it runs out the waiter records where it gave up and
// raises the abort word; every other waiter polls that word and leaves too, so the launch always ends.
struct WaitCtl {
  DevStatus* st;        // global
  volatile int* s_abort;  // shared: this CTA saw a failure
  unsigned limit;       // spin limit per wait
};

__device__ __forceinline__ void report_fail(const WaitCtl& c, int where, int layer, int expected, int seen) {
  if (atomicCAS(&c.st->code, 0, 5 /*FB_ERR_TIMEOUT*/) == 0) {
    c.st->where = where; c.st->layer = layer; c.st->block = (int)blockIdx.x; c.st->expected = expected; c.st->seen = seen;
  }
  atomicExch(&c.st->abort, 1);
  *c.s_abort = 1;
  __threadfence();
}

template <bool REMOTE = false>
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, const WaitCtl& c, int where, int layer) {
  if (mbar_try<REMOTE>(b, parity)) return true;
  for (unsigned i = 0; i < c.limit; i++) {
    if (mbar_try<REMOTE>(b, parity)) return true;
    if ((i & 63) == 63) {
      if (*c.s_abort) return false;
      if ((i & 1023) == 1023) {
        if (ld_volatile_s32(&c.st->abort)) { *c.s_abort = 1; return false; }
        __nanosleep(64);
      }
    }
  }
  report_fail(c, where, layer, (int)parity, -1);
  return false;
}

// Before a CTA may exit, every copy and MMA that it issued has to have completed its barrier phase. In a healthy launch somebody has waited for
// each of them; after a failure of any role (known for sure only behind the CTA's last barrier) whoever issued them does, with a limit of its
// own, because a caller may set the limit of the other waits to nothing.
constexpr unsigned kDrainLimit = 1u << 20;
__device__ __forceinline__ void drain_phase(uint64_t* b, uint32_t parity) {
#pragma unroll 1
  for (unsigned i = 0; i < kDrainLimit; i++) {
    if (mbar_try(b, parity)) return;
    if ((i & 1023) == 1023) __nanosleep(64);
  }
}

// the same for the last (up to) N of `issued` copies into a ring of N stages
template <int N>
__device__ __forceinline__ void drain_ring(uint64_t* full, uint32_t issued) {
  const uint32_t n = issued < (uint32_t)N ? issued : (uint32_t)N;
#pragma unroll 1
  for (uint32_t k = 1; k <= n; k++) drain_phase(&full[(issued - k) % N], ((issued - k) / N) & 1);
}

// mbar_wait and report_fail out of line, for the decode kernel, whose per-layer code does not fit the instruction cache: what a healthy step
// never executes stays out of the way.
inline __device__ __noinline__ void report_fail_far(const WaitCtl c, int where, int layer, int expected, int seen) {
  report_fail(c, where, layer, expected, seen);
}
inline __device__ __noinline__ bool mbar_wait_slow(uint64_t* b, uint32_t parity, const WaitCtl c, int where, int layer) {
  return mbar_wait(b, parity, c, where, layer);
}
__device__ __forceinline__ bool mbar_wait_far(uint64_t* b, uint32_t parity, const WaitCtl& c, int where, int layer) {
  return mbar_try(b, parity) || mbar_wait_slow(b, parity, c, where, layer);
}

// ------------------------------------------------------------------------------------------------ streaming layout
// Weights are stored as TILES of RT consecutive stream rows x all K columns, cut into CHUNKS of KC columns (tiles of long rows do not fit a ring stage), and
// a chunk is laid out for the tensor pipe. Batch-1 decode has no second matrix dimension to fill the 16 rows of an mma.m16n8k32 with, so
// these are RT weight rows x NJ = 16/RT column ranges of KC/NJ columns each: MMA row i = (tile row i % RT, range i / RT).
//
// The product is exact integer arithmetic: weights as s8 16 (nib - 8), activations as s8 digits. A group of 128 activations is brought by a power of two to
// [2^28, 2^29) and rounded to integers (exact for every bf16 element down to 2^-21 of the group's largest magnitude, off by at most 2^-29 of
// that magnitude below), and four signed digits of a number, of weights 2^23, 2^15, 2^8 and 1, go to four COLUMNS of the B operand, which a
// matrix-vector product leaves idle anyway: with two ranges all eight are in use. Lane t of a quad holds columns 2t and 2t + 1, two digits of one range.
// The group's flush joins them and multiplies by the power of two and the bf16 scale in fp32: the reference's sum (nib - 8) * s * x in
// another order of summation.
//
// A block of 64 columns of every range is 512 bytes: 16 per lane (g = lane / 4, t = lane % 4). Byte b of word i holds columns 16t + 4i + b of MMA row g (high
// nibble) and row g + 8 (low nibble), as nib - 8 in two's complement: words 2s and 2s + 1 are the A operand of MMA step s after w & 0xF0F0F0F0 and
// (w << 4) & 0xF0F0F0F0. The columns of a step are not the ones that the instruction numbers so, but B is read in the same order. After a chunk's
// nibble area come its scales as bf16 [KC/128][RT], then (asymmetric layout) its zeros in the same shape.
//
// This replaced fp16 operands (m16n8k16, nibbles as fp16 subnormals, four ranges of four rows): five ALU operations and one MMA per eight weights of a lane
// against three and a half, half the shared-memory reads of activations, and a flush per group of eight rows instead of four. (e4m3 operands need
// the same operations, but sm_100a runs mma.sync on them at less than half of the integer rate: 7.2 against 3.0 cycles an instruction and SM, operands
// from shared memory.) Gate/up of the 3B / 1B / 8B-class shapes, 16384 x 2560, 16384 x 2048, 28672 x 4096, in the decode kernel: 4.4 / 3.9 / 11.8 us before,
// 2.5 / 2.2 / 7.3 now; the stand-alone product over 400000 x 2560 5.3 -> 5.8 TB/s. The products are off from 64-bit ones by 3.4e-7
// (normal activations) to 1.5e-5 (outliers, SwiGLU outputs) before and by 5e-8 to 9.4e-8 now, whatever the activations: they round only in the flush. Elements below
// 2^-21 of their group's largest, which the fp16 form held exactly, were lost there to the fp32 sums of nibble times the largest.
__host__ __device__ constexpr int chunk_bytes(int rt, int kc, int has_zeros) { return rt * (kc / 2 + (kc / 128) * 2 * (has_zeros ? 2 : 1)); }
constexpr int kChunkFit = 20992;                   // the smallest ring stage (SmemPlan of K = 14336)
// Columns of a chunk: all of K where that fits a stage; else 4096 or 2048 where they divide K (8192 in 2, 14336 in 7: with 28 rows a CTA two chunks a warp), else
// the longest whole number of groups per range that divides K and fits.
__host__ __device__ constexpr int chunk_k(int k) {
  const int rt = tile_rt(k), unit = 128 * (16 / rt);
  if (chunk_bytes(rt, k, 1) <= kChunkFit) return k;
  if (k % 4096 == 0) return 4096;
  if (k % 2048 == 0) return 2048;
  int best = unit;
  for (int c = unit; c < k; c += unit)
    if (k % c == 0 && chunk_bytes(rt, c, 1) <= kChunkFit) best = c;
  return best;
}
__host__ __device__ constexpr int tile_bytes(int k, int has_zeros) { return k / chunk_k(k) * chunk_bytes(tile_rt(k), chunk_k(k), has_zeros); }
// bytes per stream row (a tile is RT of these; only whole tiles are addressable)
__host__ __device__ constexpr int rec_bytes_of(int k, int has_zeros) { return tile_bytes(k, has_zeros) / tile_rt(k); }
__host__ __device__ constexpr int pad_rows(int rows, int k) { return (rows + tile_rt(k) - 1) / tile_rt(k) * tile_rt(k); }

// A matrix on its own (fb_repack, fb_gemv, fb_dequant) holds whole tiles only; the rows behind the last one follow plainly, [rows][K/8] words in the caller's
// order, then their scales [rows][K/128] (and zeros), so that a matrix of few rows is not padded to a tile. Its buffer: rows in multiples of these.
__host__ __device__ constexpr int stream_row_unit(int k) {
  const int g = k / 128;
  return g % 4 == 0 && 4 * (k / 2 + g * 4) <= 23040 ? 4 : (g % 8 == 0 ? 2 : (g % 2 == 0 ? 8 : 16));
}

// Shared memory of a kernel whose longest K is MAXK: the tail (fixed offsets), the activations (4 bytes each) or the attention's scratch, and what is left
// in eight ring stages.
template <int MAXK>
struct SmemPlan {
  static constexpr int SCRATCH = 4 * MAXK > kAttnScratch ? 4 * MAXK : kAttnScratch;
  static constexpr int RING = kTailBytes + SCRATCH;
  static constexpr int STAGE = (kSmemBytes - RING) / kStages / 128 * 128;
  static_assert(MAXK / 128 <= 112, "group factors");
};

// stream row j of a matrix holds source row perm(j)
//   order 0: identity
//   order 1: rows [0, order_rows) are heads of `arg` rows; inside a head stream rows (2p, 2p+1) hold dims (p, p+arg/2),
//            so one thread gets both halves of a RoPE pair; rows beyond order_rows (V) keep their order
//   order 2: stream rows (2i, 2i+1) hold (gate_i, up_i) = source rows (i, i+arg)
__host__ __device__ __forceinline__ int perm_row(int j, int order, int arg, int order_rows) {
  if (order == 1) {
    if (j >= order_rows) return j;
    const int head = j / arg, w = j % arg;
    return head * arg + (w >> 1) + (w & 1) * (arg >> 1);
  }
  if (order == 2) return (j >> 1) + (j & 1) * arg;
  return j;
}

constexpr int kPartBytes = 1024;                   // partial sums of units: [32][8 rows] or [16][16 rows]
// Compile-time schedule of one matrix shape over ring stages of STAGE bytes: CPS chunks travel in one bulk copy. A chunk is RPC rounds (one group of every
// range, two blocks); the warps of a CTA that has few chunks share one by rounds (unit_entry).
template <int K_, int STAGE>
struct TCfg {
  static constexpr int K = K_, RT = tile_rt(K_), NJ = 16 / RT, KC = chunk_k(K_), NC = K / KC;
  static constexpr int G = KC / 128, RPC = G / NJ;
  static constexpr int NIB = RT * KC / 2;
  static constexpr int chunk(bool hz) { return chunk_bytes(RT, KC, hz); }
  static constexpr int FIT = STAGE / chunk_bytes(RT, KC, 1), CPS = NC > 1 ? (RT == 8 && FIT > 1 ? 2 : 1) : (FIT > 8 ? 8 : FIT);
  static_assert(K % KC == 0 && G % NJ == 0, "columns must split into chunks and whole groups per range");
  static_assert(CPS >= 1 && CPS * chunk_bytes(RT, KC, 1) <= STAGE, "a stage holds whole chunks");
  // partial sums are kept in a ring of SLOTS units: the oldest unfinished chunk holds its stage, so younger ones are at most a ring ahead
  static constexpr int SLOTS = kPartBytes / (RT * 4);
  static_assert(FIT >= 1 && (NC == 1 || (kStages + 1) * CPS + NC <= SLOTS) && SLOTS >= kConsumerWarps, "partial sums");
  static_assert(chunk_bytes(RT, KC, 0) % 16 == 0, "bulk copies move multiples of 16 bytes");
};
// Which chunks of a phase a warp takes: chunk, first round, rounds, slices per chunk, a byte each. Few chunks: each is cut in `ks` slices so that as
// many warps as possible have one; else the warps take whole chunks w, w + 14, ...
__device__ __forceinline__ uint32_t unit_entry(int nch, int rpc, int warp) {
  int ks = nch > 0 && nch <= kConsumerWarps / 2 ? kConsumerWarps / nch : 1;
  if (ks > rpc) ks = rpc;
  const int ci = warp / ks, sl = warp - ci * ks, r0 = rpc * sl / ks, r1 = rpc * (sl + 1) / ks;
  return (uint32_t)(ci < nch ? ci : 255) | (uint32_t)r0 << 8 | (uint32_t)(r1 - r0) << 16 | (uint32_t)ks << 24;
}
// ... out of line, for the decode kernel, which asks once per phase and launch: five copies with their divisions are code that its layer loop has to share the
// instruction cache with (3B-class 794 -> 784 us a token, 8B 1409 -> 1417, others as before)
inline __device__ __noinline__ uint32_t unit_entry_far(int nch, int rpc, int warp) { return unit_entry(nch, rpc, warp); }

// activations of the current phase in shared memory: per 64 columns their lowest digits [64], then the next ones, in column order; and per group of
// 128 columns {2^-e, sum x} for the lanes that hold the two low digits, {2^15 2^-e, 0} for those of the two high ones (sum x: asymmetric layout only)
struct XStage {
  const uint8_t* x8;
  const float4* xf;
};

// Convert bf16 activations for the tensor pipe: v[k] holds elements 4 lane .. 4 lane + 3 of group first + k * step, which a warp converts together if it is
// below `groups`. Every CTA converts the whole vector in every phase, and the phase waits for it: no branch but the stores' predicates, so that
// the groups of a thread run side by side. The two halves of a number come out of the mantissas of sums with 1.5 * 2^23 + 128 (the 128 makes the
// low byte's digit signed), on the FMA pipe.
template <bool SUM, int N>
__device__ __forceinline__ void stage_groups(const uint2 (&v)[N], int first, int step, int groups, uint8_t* x8, float4* xf, int lane) {
  uint32_t em[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    const uint32_t mm = __vmaxu2(v[k].x & 0x7fff7fffu, v[k].y & 0x7fff7fffu);
    em[k] = __reduce_max_sync(0xffffffffu, max(mm >> 16, mm & 0xffffu)) >> 7;
  }
  float sx[N];
#pragma unroll
  for (int k = 0; k < N; k++) sx[k] = SUM ? (bflo(v[k].x) + bfhi(v[k].x)) + (bflo(v[k].y) + bfhi(v[k].y)) : 0.f;
  if (SUM)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < N; k++) sx[k] += __shfl_xor_sync(0xffffffffu, sx[k], o);
#pragma unroll
  for (int k = 0; k < N; k++) {
    const uint32_t mf = min(267u - em[k], 253u);                // exponent field of the multiplier: largest magnitude in [2^13, 2^14)
    const float mult = __uint_as_float(mf << 23), magic = 12583040.f;
    const float x[4] = {bflo(v[k].x), bfhi(v[k].x), bflo(v[k].y), bfhi(v[k].y)};
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float h = fmaf(x[i], mult, magic);                  // the nearest integer, in the low bits
      const float r = fmaf(x[i], mult, magic - h);              // exact: what is left, |r| <= 1/2
      hi[i] = __float_as_uint(h);
      lo[i] = __float_as_uint(fmaf(r, 32768.f, magic));
    }
    // 4 x 4 bytes transposed: a word holds one digit of the four elements
    const uint32_t a = __byte_perm(lo[0], lo[1], 0x5140), b = __byte_perm(lo[2], lo[3], 0x5140), c = __byte_perm(hi[0], hi[1], 0x5140),
                   d = __byte_perm(hi[2], hi[3], 0x5140);
    const int grp = first + k * step;
    const float inv = em[k] == 255u ? __uint_as_float(0x7fc00000u) : __uint_as_float((254u - mf) << 23);      // infinities and NaN: the group's products are NaN
    if (grp < groups) {
      uint32_t* dst = reinterpret_cast<uint32_t*>(x8 + grp * 512 + (lane >> 4) * 256) + (lane & 15);
      dst[0] = __byte_perm(a, b, 0x5410) ^ 0x80808080u;
      dst[16] = __byte_perm(a, b, 0x7632);
      dst[32] = __byte_perm(c, d, 0x5410) ^ 0x80808080u;
      dst[48] = __byte_perm(c, d, 0x7632);
      if (lane == 0) xf[grp] = make_float4(inv * 0.0625f * (1.f / 32768.f), sx[k], inv * 0.0625f, 0.f);
    }
  }
}

// ------------------------------------------------------------------------------------------------ tile x vector
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 lds64f(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ float lds_bf16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return __uint_as_float(((uint32_t)v) << 16);
}
__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Programmatic dependent launch: every kernel of the verify chain is launched with the stream-serialisation attribute.
// pdl_trigger() lets the next kernel's CTAs start (and prefetch what does not depend on this kernel) once every CTA of
// this kernel has called it; pdl_wait() returns when the previous kernel has completed and its writes are visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The kernels of a call read weights before they wait for their predecessor. Those are the caller's tensors, and whatever ran before the
// call may have written them: the FIRST kernel of a call waits before it lets the next ones start. A draft step (two calls) with early
// reads from the first kernel on 123.3 us, so 126.2; the first kernel launched in plain stream order instead 128.5, its first weights
// requested into L2 ahead of the wait 133.8.
__device__ __forceinline__ void pdl_begin(bool first) {
  if (first) pdl_wait();
  pdl_trigger();
}

// launch with programmatic stream serialisation: the kernel may start while its predecessor drains (see pdl_wait)
// (`cluster` consecutive CTAs form a thread-block cluster)
template <class... KArgs, class... Args>
cudaError_t launch_pdl_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, unsigned cluster,
                               const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}
template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const Args&... args) {
  return launch_pdl_cluster(kern, grid, block, smem, st, 1u, args...);
}

// bf16 tensor-core helpers shared by the attention kernels and the draft head
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the attention kernels' softmax is in base 2: scores are multiplied by scale * log2(e)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) { return (uint32_t)f2bf(lo) | ((uint32_t)f2bf(hi) << 16); }

// Rounds [r0, r0 + n) of a chunk (its `ci`-th of the tile) against the staged activations. RT 8: on return every lane of quad g holds the total of tile
// row g in out_lo. RT 16: row g in out_lo and row g + 8 in out_hi.
// The loop is ROLLED (two rounds per iteration): every phase of the decode kernel has its own copy of it, and they share the instruction cache. Per round of 2048
// weights a warp issues 24 half-rate ALU operations, 4 MMAs and 4 loads of 16 bytes a lane (16 cycles of an SM's shared memory); on its own the loop
// streams at 0.99 of the copy bandwidth.
template <class C, bool HZ>
__device__ __forceinline__ void chunk_dot(const uint8_t* chunk, int ci, int r0, int n, const XStage& x, int lane, float& out_lo, float& out_hi) {
  constexpr int RT = C::RT, NJ = C::NJ;
  constexpr uint32_t META = RT * 2;                              // bytes of a group's scales
  const int g = lane >> 2, t = lane & 3;
  const int j = NJ == 2 ? t >> 1 : 0;                            // the range of this lane's accumulator columns
  const bool up = NJ == 2 && t >= 2;                             // ... and with two ranges the MMA rows: g or g + 8
  const uint32_t tb = smem_u32(chunk);
  uint32_t wa = tb + (uint32_t)(r0 * 64 + lane) * 16;
  // B: lane (g, t) reads column g, digit g & 3 of range g >> 2 (one range: again). Eight lanes read 128 bytes in a row: no bank twice.
  uint32_t xa = smem_u32(x.x8) + (uint32_t)(ci * C::KC + (NJ == 2 ? (g >> 2) * (C::KC / NJ) : 0)) * 4 + (uint32_t)(r0 * 512 + (g & 3) * 64 + 16 * t);
  uint32_t ma = tb + C::NIB + (uint32_t)(j * C::RPC + r0) * META + (uint32_t)g * 2;
  uint32_t fa = smem_u32(x.xf) + (uint32_t)(ci * C::G + j * C::RPC + r0) * 16 + (t & 1) * 8;
  float ct = 0.f, ct2 = 0.f;
  uint4 w0 = lds128(wa), w1 = lds128(wa + 512), x0 = lds128(xa), x1 = lds128(xa + 256);
  auto round = [&](bool more) {
    const uint32_t wstep = more ? 1024u : 0u, xstep = more ? 512u : 0u;      // the last round reads its own operands again
    wa += wstep;
    xa += xstep;
    const uint4 wn0 = lds128(wa), wn1 = lds128(wa + 512), xn0 = lds128(xa), xn1 = lds128(xa + 256);
    const float2 F = lds64f(fa);
    const float s = lds_bf16(ma);
    int c[4] = {0, 0, 0, 0};
    const uint32_t ws[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w}, xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const uint32_t a[4] = {ws[k] & 0xF0F0F0F0u, (ws[k] << 4) & 0xF0F0F0F0u, ws[k + 1] & 0xF0F0F0F0u, (ws[k + 1] << 4) & 0xF0F0F0F0u};
      mma_s8(c, a, xs[k], xs[k + 1]);
    }
    const float v = __int2float_rn((up ? c[2] : c[0]) + 256 * (up ? c[3] : c[1]));
    ct = fmaf(s, F.x * v, ct);                                  // in this order: F.x alone may be subnormal
    if (HZ) ct = fmaf(lds_bf16(ma + C::G * META), F.y, ct);
    if (RT == 16) {
      ct2 = fmaf(lds_bf16(ma + 16), F.x * __int2float_rn(c[2] + 256 * c[3]), ct2);
      if (HZ) ct2 = fmaf(lds_bf16(ma + C::G * META + 16), F.y, ct2);
    }
    ma += META;
    fa += 16;
    w0 = wn0; w1 = wn1; x0 = xn0; x1 = xn1;
  };
#pragma unroll 1
  for (; n >= 2; n -= 2) {
    round(true);
    round(n > 2);
  }
  if (n) round(false);
  if (RT == 8) {
    ct += __shfl_xor_sync(0xffffffffu, ct, 1);
    ct += __shfl_xor_sync(0xffffffffu, ct, 2);
    out_lo = ct;
    out_hi = 0.f;
  } else {                                                       // lanes 2 and 3 of a quad hold nothing
    ct += __shfl_xor_sync(0xffffffffu, ct, 1);
    ct2 += __shfl_xor_sync(0xffffffffu, ct2, 1);
    out_lo = __shfl_sync(0xffffffffu, ct, lane & 28);
    out_hi = __shfl_sync(0xffffffffu, ct2, lane & 28);
  }
}

}  // namespace fb
