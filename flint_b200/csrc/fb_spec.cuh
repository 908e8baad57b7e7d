// Speculative-decoding side of the decode path, all on the device: token sampling from logits (temperature / top-k,
// Gumbel-max with a counter-based generator, no host sync), chain and tree acceptance, KV compaction of an accepted
// tree path, and the EAGLE draft head (one decoder block over [target feature ; token embedding], bf16 weights as the
// reference trains and runs it).
//
// The draft head's arithmetic follows the rounding sites of bf16 PyTorch modules: every linear layer, norm, rotation,
// activation and residual addition rounds its result to bf16; accumulation inside a layer is fp32.
#pragma once
#include "fb_common.cuh"
#include "fb_geometry.hpp"

namespace fb {

// ------------------------------------------------------------------------------------------------ random numbers
// splitmix64 finaliser over (seed, counter, index): independent streams per call (counter) and per vocabulary entry
__device__ __forceinline__ uint32_t mix32(unsigned long long seed, unsigned long long ctr, uint32_t idx) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (ctr + 1) + (((unsigned long long)idx << 1) | 1ull) * 0xD1B54A32D192ED03ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return (uint32_t)(z >> 32);
}
// standard Gumbel variate from 23 random bits: u in (0, 1) exactly representable, never 0 or 1
__device__ __forceinline__ float gumbel(uint32_t bits) {
  const float u = ((float)(bits >> 9) + 0.5f) * (1.0f / 8388608.0f);
  return -logf(-logf(u));
}
// order-preserving map float -> uint32 (larger float = larger key)
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_value(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k); }

// ------------------------------------------------------------------------------------------------ sampling
struct SampleParams {
  const float* logits;          // [rows] vectors of `vocab` floats, `row_stride` elements apart (0: every row samples the same vector)
  long long row_stride;
  int32_t vocab, top_k;         // top_k <= 0: the whole vocabulary
  float temperature;            // <= 0: arg-max (first index of the maximum)
  unsigned long long seed, counter;   // row r draws from stream (seed, counter + r)
  int32_t* out;                 // [rows] token ids
  int32_t ctas;                 // CTAs (one cluster) of a row
};

// One cluster of CTAs per row: a CTA keeps its slice of the row in registers (up to 16 values a thread; longer slices are read again),
// so a row is read once, by several SMs. top-k keeps every entry >= the k-th largest value (ties included, as `logits < v[-1] -> -inf`
// does, reference: engine/generate.py:41-45). The draw is arg-max of logit / T + Gumbel noise, which is a sample of softmax(logits / T) over the kept
// entries: the same distribution as arg-max(p / Exponential(1)) (reference: engine/generate.py:37-39).
// Up to 4/5 as many kept entries as the row has warps (256 for a row of 8 CTAs): the k-th largest of the warps' maxima bounds the k-th largest value from
// below, and few values lie above it (about 60 for k = 50 of 128256 normal values, 400 for k = 200). They go to the first CTA's list, where an entry
// is kept if fewer than k entries are larger: two cluster barriers and no histogram. More kept entries, or so many ties that the list is
// full: radix select on order-preserving keys in three digits of 11, 11 and 10 bits; every CTA counts its own slice and reads the others'
// counts from their shared memory: four cluster barriers, three scans, and most of the first digit's atomics on a handful of bins.
// Logits of 128256 entries, one row, k = 50: 16.4 us with the radix select, 7.5 with the list (a call back to back: 10, the host's part); 16 rows of k = 50 / 200 33.6 / 34.4
// -> 14.4 / 17.9, 64 rows 87 / 89 -> 37 / 42. Without top-k, in a kernel without the selection: 64 rows arg-max 24.2 -> 19.3, draw 53 -> 47. (One CTA per row and five passes took 83 us for one row.)
constexpr int kSampleRegs = 16;
// Another CTA's shared memory may be touched only once that CTA is known to run. Every CTA of the cluster arrives at the start of the kernel
// and waits before its first remote access: the row's loads lie in between and hide the barrier.
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t add_cluster(uint32_t a, uint32_t n) {
  uint32_t old;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(n) : "memory");
  return old;
}
__device__ __forceinline__ uint2 ld_cluster(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared::cluster.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
// the better of two (value, index) pairs: larger value, then smaller index
__device__ __forceinline__ void take_best(float& bv, int& bi, float ov, int oi) {
  if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
}
__device__ __forceinline__ void warp_best(float& bv, int& bi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    take_best(bv, bi, ov, oi);
  }
}

// grid (rows * CTAs per row), clusters of one row's CTAs, 1024 threads. Rows lie on grid.x: grid.y ends at 65535, and a program may
// draw any number of rows from one vector (stride 0).
constexpr int kSampleList = 1024;                 // candidates of the short selection: one per thread
// SELECT: a draw with top-k
template <bool REG, bool SELECT>
__global__ void __launch_bounds__(1024) sample_rows(const SampleParams P) {
  __shared__ __align__(16) unsigned hist[SELECT ? 3 : 1][SELECT ? 2048 : 4];                 // radix select; the short selection: keys of the warps' maxima, of the list, indices of the list
  __shared__ unsigned s_warp[32], s_bin, s_k, s_cnt;
  __shared__ float s_v[32];
  __shared__ int s_i[32];
  __shared__ float c_v[16];                       // the CTAs' candidates, in the first CTA
  __shared__ int c_i[16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = P.ctas, row = blockIdx.x / C, rank = blockIdx.x % C;
  const float* lg = P.logits + (long long)row * P.row_stride;
  const int per = (P.vocab + C - 1) / C, i0 = rank * per, i1 = min(P.vocab, i0 + per);
  const bool draw = SELECT || P.temperature > 0.f, brief = SELECT && P.top_k <= C * 32 * 4 / 5;
  if (tid == 0) s_cnt = 0u;
  if (!SELECT || brief) cluster_arrive();         // the radix select's own barriers come before its first remote read
  pdl_trigger();
  pdl_wait();
  float v[REG ? kSampleRegs : 1];
  if constexpr (REG) {
#pragma unroll
    for (int j = 0; j < kSampleRegs; j++) v[j] = i0 + tid + j * 1024 < i1 ? lg[i0 + tid + j * 1024] : 0.f;
  }
  auto each = [&](auto f) {
    if constexpr (REG) {
#pragma unroll
      for (int j = 0; j < kSampleRegs; j++)
        if (i0 + tid + j * 1024 < i1) f(i0 + tid + j * 1024, v[j]);
    } else {
      for (int i = i0 + tid; i < i1; i += 1024) f(i, lg[i]);
    }
  };
  const float inv_t = draw ? 1.0f / P.temperature : 1.0f;
  auto score = [&](int i, float x) { return draw ? x * inv_t + gumbel(mix32(P.seed, P.counter + (unsigned long long)row, (uint32_t)i)) : x; };
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  if constexpr (SELECT) if (brief) {
    unsigned *wkey = hist[0], *lkey = hist[1], *lidx = hist[1] + kSampleList;
    uint32_t top = 0u;
    each([&](int, float x) { top = max(top, fkey(x)); });
    top = __reduce_max_sync(0xffffffffu, top);
    cluster_wait();
    if (lane < C) st_cluster(cluster_map((uint32_t)__cvta_generic_to_shared(wkey + rank * 32 + warp), lane), top);
    cluster_sync();
    if (warp == 0) {
      // the largest 16-bit prefix that at least k of the maxima reach
      uint32_t w[8], lo = 0xffffu, hi = 0u;
#pragma unroll
      for (int c = 0; c < 8; c++) {
        w[c] = c < C ? wkey[c * 32 + lane] >> 16 : 0u;
        if (c < C) { lo = min(lo, w[c]); hi = max(hi, w[c]); }
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      while (lo < hi) {                                          // at least k reach lo
        const uint32_t mid = (lo + hi + 1) / 2;
        unsigned n = 0;
#pragma unroll
        for (int c = 0; c < 8; c++) n += w[c] >= mid;
        if (__reduce_add_sync(0xffffffffu, n) >= (unsigned)P.top_k) lo = mid;
        else hi = mid - 1;
      }
      if (lane == 0) s_bin = lo << 16;
    }
    __syncthreads();
    const uint32_t floor = s_bin;
    unsigned own = 0;
    each([&](int, float x) { own += fkey(x) >= floor; });
    const unsigned all = __reduce_add_sync(0xffffffffu, own);
    if (all) {
      unsigned at = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += u;
      }
      unsigned base = 0;
      if (lane == 0) base = add_cluster(cluster_map((uint32_t)__cvta_generic_to_shared(&s_cnt), 0), all);
      at += __shfl_sync(0xffffffffu, base, 0) - own;
      if (own) {
        const uint32_t k0 = cluster_map((uint32_t)__cvta_generic_to_shared(lkey), 0), x0 = cluster_map((uint32_t)__cvta_generic_to_shared(lidx), 0);
        each([&](int i, float x) {
          if (fkey(x) >= floor) {
            if (at < kSampleList) {
              st_cluster(k0 + at * 4, fkey(x));
              st_cluster(x0 + at * 4, (uint32_t)i);
            }
            at++;
          }
        });
      }
    }
    cluster_sync();
    const unsigned n = ld_cluster_u32(cluster_map((uint32_t)__cvta_generic_to_shared(&s_cnt), 0));
    cluster_arrive();                             // the first CTA stays until the others have read its count
    if (n <= kSampleList) {
      if (rank == 0) {
        const unsigned n4 = (n + 3) / 4 * 4;
        if (tid >= (int)n && tid < (int)n4) lkey[tid] = 0u;
        __syncthreads();
        if (tid < (int)n) {
          const uint32_t mine = lkey[tid];
          unsigned larger = 0;
#pragma unroll 4
          for (unsigned c = 0; c < n4; c += 4) {
            const uint4 o = *reinterpret_cast<const uint4*>(lkey + c);
            larger += (o.x > mine) + (o.y > mine) + (o.z > mine) + (o.w > mine);
          }
          if (larger < (unsigned)P.top_k) {
            const int i = (int)lidx[tid];
            take_best(bv, bi, score(i, fkey_value(mine)), i);
          }
        }
        warp_best(bv, bi);
        if (lane == 0) { s_v[warp] = bv; s_i[warp] = bi; }
        __syncthreads();
        if (warp == 0) {
          bv = s_v[lane]; bi = s_i[lane];
          warp_best(bv, bi);
          if (lane == 0) P.out[row] = bi == 0x7fffffff ? 0 : bi;
        }
      }
      cluster_wait();
      return;
    }
    cluster_wait();
  }
  uint32_t thr = 0u;
  if constexpr (SELECT) {
    for (int i = tid; i < 2048; i += 1024) { hist[0][i] = hist[1][i] = hist[2][i] = 0u; }
    __syncthreads();
    uint32_t prefix = 0u, mask = 0u;
    unsigned k = (unsigned)P.top_k;
#pragma unroll 1
    for (int d = 0; d < 3; d++) {
      const int shift = d == 0 ? 21 : (d == 1 ? 10 : 0);
      const uint32_t dmask = d == 2 ? 1023u : 2047u;
      each([&](int, float x) {
        const uint32_t key = fkey(x);
        if ((key & mask) == prefix) atomicAdd(&hist[d][(key >> shift) & dmask], 1u);
      });
      cluster_sync();
      // thread t holds bins 2047 - 2t and 2046 - 2t: an inclusive scan in thread order counts from the largest key down
      const uint32_t h = (uint32_t)__cvta_generic_to_shared(&hist[d][2046 - 2 * tid]);
      unsigned b0 = 0u, b1 = 0u;
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (c < C) {
          const uint2 u = ld_cluster(cluster_map(h, c));
          b0 += u.x;
          b1 += u.y;
        }
      unsigned s = b1 + b0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += u;
      }
      if (lane == 31) s_warp[warp] = s;
      __syncthreads();
      if (warp == 0) {
        unsigned w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned u = __shfl_up_sync(0xffffffffu, w, o);
          if (lane >= o) w += u;
        }
        s_warp[lane] = w;
      }
      __syncthreads();
      const unsigned before = s - b1 - b0 + (warp ? s_warp[warp - 1] : 0u);      // entries in larger bins
      if (before < k && before + b1 >= k) { s_bin = 2047 - 2 * tid; s_k = k - before; }
      else if (before + b1 < k && before + b1 + b0 >= k) { s_bin = 2046 - 2 * tid; s_k = k - before - b1; }
      __syncthreads();
      prefix |= s_bin << shift;
      mask |= dmask << shift;
      k = s_k;
    }
    thr = prefix;                                 // key of the k-th largest value
  }
  each([&](int i, float x) {
    if (!SELECT || fkey(x) >= thr) take_best(bv, bi, score(i, x), i);
  });
  warp_best(bv, bi);
  if (lane == 0) { s_v[warp] = bv; s_i[warp] = bi; }
  __syncthreads();
  if (!SELECT) cluster_wait();
  if (warp == 0) {
    bv = s_v[lane]; bi = s_i[lane];
    warp_best(bv, bi);
    if (lane == 0) {
      st_cluster(cluster_map((uint32_t)__cvta_generic_to_shared(c_v + rank), 0), __float_as_uint(bv));
      st_cluster(cluster_map((uint32_t)__cvta_generic_to_shared(c_i + rank), 0), (uint32_t)bi);
    }
  }
  cluster_sync();
  if (rank == 0 && warp == 0) {
    bv = lane < C ? c_v[lane] : -INFINITY;
    bi = lane < C ? c_i[lane] : 0x7fffffff;
    warp_best(bv, bi);
    if (lane == 0) P.out[row] = bi == 0x7fffffff ? 0 : bi;
  }
}

// The B best entries of every row in order (value descending, first index on ties). One cluster per row: every CTA picks the B best of
// its slice in B rounds of a block arg-max over registers, the first CTA picks the B best of the candidates. grid (cluster, rows)
template <bool REG>
__global__ void __launch_bounds__(1024) topb_rows(const float* logits, long long row_stride, int vocab, int B, int32_t* out_idx,
                                                  float* out_val) {
  __shared__ float s_v[32];
  __shared__ int s_i[32], s_pick;
  __shared__ float c_v[16 * 16];
  __shared__ int c_i[16 * 16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = blockIdx.y, C = gridDim.x, rank = blockIdx.x;
  const float* lg = logits + (long long)row * row_stride;
  const int per = (vocab + C - 1) / C, i0 = rank * per, i1 = min(vocab, i0 + per);
  cluster_arrive();
  pdl_trigger();
  pdl_wait();
  float v[REG ? kSampleRegs : 1];
  unsigned taken = 0u;                            // this thread's entries that were picked already
  if constexpr (REG) {
#pragma unroll
    for (int j = 0; j < kSampleRegs; j++) {
      const int i = i0 + tid + j * 1024;
      v[j] = i < i1 ? lg[i] : 0.f;
      if (i >= i1) taken |= 1u << j;
    }
  }
  float pv = INFINITY;                            // longer slices: the pick of the last round; later picks come after it in order
  int pi = -1;
  for (int r = 0; r < B; r++) {
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    if constexpr (REG) {
#pragma unroll
      for (int j = 0; j < kSampleRegs; j++)
        if (!(taken >> j & 1u)) take_best(bv, bi, v[j], i0 + tid + j * 1024);
    } else {
      for (int i = i0 + tid; i < i1; i += 1024) {
        const float x = lg[i];
        if (x < pv || (x == pv && i > pi)) take_best(bv, bi, x, i);
      }
    }
    warp_best(bv, bi);
    if (lane == 0) { s_v[warp] = bv; s_i[warp] = bi; }
    __syncthreads();
    if (r == 0) cluster_wait();
    if (warp == 0) {
      bv = s_v[lane]; bi = s_i[lane];
      warp_best(bv, bi);
      if (lane == 0) {
        s_pick = bi;
        s_v[0] = bv;
        st_cluster(cluster_map((uint32_t)__cvta_generic_to_shared(c_v + rank * B + r), 0), __float_as_uint(bv));
        st_cluster(cluster_map((uint32_t)__cvta_generic_to_shared(c_i + rank * B + r), 0), (uint32_t)bi);
      }
    }
    __syncthreads();
    pi = s_pick;
    pv = s_v[0];
    const int loc = pi - i0 - tid;
    if (REG && pi != 0x7fffffff && loc >= 0 && (loc & 1023) == 0) taken |= 1u << (loc >> 10);
    __syncthreads();
  }
  cluster_sync();
  if (rank == 0 && warp == 0) {
    unsigned used = 0u;                           // lane l looks at candidates l, l + 32, ... (at most 256: 8 each)
    for (int r = 0; r < B; r++) {
      float bv = -INFINITY;
      int bi = 0x7fffffff, bc = 0;
      for (int c = lane, j = 0; c < C * B; c += 32, j++)
        if (!(used >> j & 1u) && (c_v[c] > bv || (c_v[c] == bv && c_i[c] < bi))) { bv = c_v[c]; bi = c_i[c]; bc = j; }
      const int own = bi;
      warp_best(bv, bi);
      if (own == bi && bi != 0x7fffffff) used |= 1u << bc;
      if (lane == 0) {
        out_idx[(size_t)row * B + r] = bi == 0x7fffffff ? 0 : bi;
        if (out_val) out_val[(size_t)row * B + r] = bv;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ acceptance
// chain: longest prefix of the K drafted tokens the target's greedy choices agree with
// (reference: spec_mega.py:106-113). out[0] = accepted count, out[1] = the target's token after the accepted prefix.
__global__ void accept_chain(const int32_t* tgt, const int32_t* draft, int K, int32_t* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    int acc = 0;
    while (acc < K && tgt[acc] == draft[acc]) acc++;
    out[0] = acc;
    out[1] = tgt[acc];
  }
}
// tree: walk from the root along the first child (lowest node index) whose token equals the target's choice at the
// current node (reference: spec_tree.py:108-118). out[0] = nodes on the path (root included), out[1] = the target's
// token at the last node, out[2 + i] = node index of path step i.
__global__ void accept_tree(const int32_t* cand, const int32_t* parent, const int32_t* tgt, int M, int32_t* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    int cur = 0, len = 1;
    out[2] = 0;
    for (;;) {
      int nxt = -1;
      for (int ch = cur + 1; ch < M; ch++)
        if (parent[ch] == cur && cand[ch] == tgt[cur]) { nxt = ch; break; }
      if (nxt < 0) break;
      out[2 + len] = nxt;
      len++;
      cur = nxt;
    }
    out[0] = len;
    out[1] = tgt[cur];
  }
}
// cache row pos + step <- row pos + path[step] for step = 1 .. len-1, K and V, every layer (reference:
// spec_tree.py:124-128). path indices grow strictly, so no row is read after it was overwritten.
// grid (n_layer, 2); `acc` is accept_tree's output.
__global__ void kv_compact(uint16_t* kc, uint16_t* vc, const int32_t* acc, int pos, size_t layer_elems, int row_elems, int max_seq) {
  uint16_t* base = (blockIdx.y ? vc : kc) + (size_t)blockIdx.x * layer_elems;
  const int len = acc[0];
  for (int step = 1; step < len; step++) {
    const int src = pos + acc[2 + step], dst = pos + step;
    if (src == dst || src >= max_seq || dst >= max_seq || src < 0) continue;
    const uint4* s = reinterpret_cast<const uint4*>(base + (size_t)src * row_elems);
    uint4* d = reinterpret_cast<uint4*>(base + (size_t)dst * row_elems);
    for (int i = threadIdx.x; i < row_elems / 8; i += blockDim.x) d[i] = s[i];
  }
}

// ------------------------------------------------------------------------------------------------ draft head
enum { DL_STORE = 0, DL_RESID = 1, DL_SWIGLU = 2, DL_LOGITS = 3 };

struct DLin {
  const uint16_t* W[3];         // bf16 [N, K] (torch Linear layout), K = k0 + k1; up to three matrices over the same input (q, k, v)
  const uint16_t* W2;           // DL_SWIGLU: the `up` matrix, same shape as W[0]
  const uint16_t* x0;           // first input segment: bf16 rows of k0 elements, ldx0 apart
  const uint16_t* x1;           // second segment (k1 elements, ldx1 apart) or nullptr: the input is cat(x0, x1)
  const int32_t* x1_tokens;     // when set, segment 1 of token t is row x1_tokens[t] of x1, an embedding table of x1_rows rows; outside: zeros
  int x1_rows;
  int ldx0, ldx1, k0, k1;
  int N[3], T;
  uint16_t* y[3];               // bf16 [T, N] rows ldy apart (STORE / RESID / SWIGLU)
  const uint16_t* resid;        // DL_RESID: y = bf16(resid + bf16(acc)), rows ldr apart
  float* yf;                    // DL_LOGITS: f32 [T, N] = bf16(bf16(acc) / scale), rows ldy apart
  int ldy[3], ldr;
  float scale;
  bool first;                   // the first kernel of a call
  int ks;                       // CTAs of a cluster that share K
  const uint16_t* norm_w;       // when set (draft_folds_norm): x0 is normalised by every CTA (d_norm_row), weights bf16 [k0]
  float norm_eps;
};
// RMSNorm inside the linear behind it, for a single token whose row fits the registers: every CTA normalises it (an L2 round trip and a block reduction) instead
// of waiting for a kernel that does (one row, step and token head, with d_attn_one: 120.4 -> 118.5 us at 3B, 140.0 -> 136.6 at 1B, 157.7 -> 155.3 with 40 heads).
constexpr int kNormRegs = 16;                     // elements of a thread
__host__ __device__ constexpr bool draft_folds_norm(int T, int D) { return T == 1 && D <= kNormRegs * 256; }

// d_rmsnorm's arithmetic, in its order, with the row in registers (D <= kNormRegs * 256), by a CTA of 256 threads that has yet to wait for the row.
__device__ __forceinline__ void d_norm_row(const uint16_t* xr, const uint16_t* w, uint16_t* y, int D, float eps, float* red) {
  const int tid = threadIdx.x;
  uint16_t wv[kNormRegs], xv[kNormRegs];
#pragma unroll
  for (int k = 0; k < kNormRegs; k++) wv[k] = tid + 256 * k < D ? w[tid + 256 * k] : (uint16_t)0;
  pdl_wait();
#pragma unroll
  for (int k = 0; k < kNormRegs; k++) xv[k] = tid + 256 * k < D ? xr[tid + 256 * k] : (uint16_t)0;
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < kNormRegs; k++) ss += rbf(bf2f(xv[k]) * bf2f(xv[k]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) tot += red[i];
  const float r = rbf(rsqrtf(rbf(rbf(tot / (float)D) + eps)));
#pragma unroll
  for (int k = 0; k < kNormRegs; k++)
    if (tid + 256 * k < D) y[tid + 256 * k] = f2bf(rbf(bf2f(xv[k]) * r) * bf2f(wv[k]));
  __syncthreads();
}

// y[t, n] = sum_k W[n, k] x[t, k] for up to 8 NT tokens (t0 ...) on the tensor pipe, weights read once. A CTA takes 16 MT rows of W and
// its WARPS warps share K: warp w takes the 32-column chunks w, w + WARPS, ... A lane loads 16 bytes of row g (and g + 8) straight into
// the A fragments of two MMA steps -- the order of columns inside a chunk does not matter as long as x is read the same way, 16 bytes of
// token g at the same columns -- so nothing goes through shared memory but the warps' partial sums. HBM-bound: a warp keeps AH chunks of
// weights and activations in flight; the first weights are requested before the previous kernel is waited for (see pdl_begin). (The CUDA-core form
// read the weights once per 8 or 16 tokens and took 62 us for a 13 to 50 MB matrix at 32 tokens.)
// A matrix whose rows give less than the GPU's worth of CTAs is also cut in K over a cluster of ks: the CTAs push their sums into the shared
// memory of the one that finishes the token, which adds them in rank order. (With 16 warps and no split a 2560-row matrix ran on 80
// SMs: block over 32 rows 130.6 -> 105.9 us, 48 rows 202 -> 167; one row, three CTAs an SM, 77.2 without the split, 74.0 with it.)
template <int NT, int MT, int MODE, bool CAT, bool FOLD>
__global__ void __launch_bounds__(kDraftWarps * 32, NT == 1 ? 3 : 2) d_gemm(const DLin P, int t0) {
  constexpr int WARPS = kDraftWarps;
  constexpr int NW = MODE == DL_SWIGLU ? 2 : 1, AH = NT == 1 && NW == 1 ? 4 : 2, ROWS = 16 * MT * NW;      // weight matrices per row, chunks in flight
  __shared__ float red[8][ROWS][8 * NT + 1];
  __shared__ float part[kDraftSplits][8 * NT][ROWS];             // split K: [source rank][token][row]
  __shared__ __align__(16) uint16_t xs[FOLD ? kNormRegs * 256 : 8];      // FOLD: the normalised row
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int K = P.k0 + P.k1, nch = (K + 31) >> 5;
  // the token head has CTAs enough
  const int ks = MODE == DL_LOGITS ? 1 : P.ks, rank = MODE == DL_LOGITS ? 0 : (int)blockIdx.x % ks;
  int blk = (int)blockIdx.x / ks, which = 0;
  if (MODE == DL_STORE) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int nb = (P.N[which] + 16 * MT - 1) / (16 * MT);
      if (P.W[which + 1] && blk >= nb) { blk -= nb; which++; }
      else break;
    }
  }
  const int N = P.N[which], r0 = blk * 16 * MT;
  // rows of this lane as 32-bit offsets in units of 8 elements (both matrices of a SwiGLU pair have the same shape)
  uint32_t wr[MT][2];
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int h = 0; h < 2; h++) wr[m][h] = (uint32_t)min(r0 + m * 16 + h * 8 + g, N - 1) * (uint32_t)(K >> 3) + t;
  const uint4* wb[NW];
  wb[0] = reinterpret_cast<const uint4*>(P.W[which]);
  if (NW > 1) wb[NW - 1] = reinterpret_cast<const uint4*>(P.W2);
  uint4 wv[AH][NW][MT][2], xv[AH][NT];
  auto load_w = [&](int c, uint4 (&d)[NW][MT][2]) {
    const bool ok = c < nch && c * 32 + 8 * t < K;
#pragma unroll
    for (int i = 0; i < NW; i++)
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) d[i][m][h] = ok ? __ldcs(wb[i] + (wr[m][h] + c * 4)) : make_uint4(0, 0, 0, 0);
  };
  if (ks > 1) cluster_arrive();                      // remote stores wait for it below
  const int c1 = rank * WARPS + warp, step = WARPS * ks;         // this warp's chunks
  pdl_begin(P.first && t0 == 0);
#pragma unroll
  for (int a = 0; a < AH; a++) load_w(c1 + step * a, wv[a]);
  if constexpr (FOLD) d_norm_row(P.x0, P.norm_w, xs, P.k0, P.norm_eps, &red[0][0][0]);
  else pdl_wait();
  const uint16_t* x0 = FOLD ? xs : P.x0;
  int x1[CAT ? NT : 1];                              // second segment: row of each token, or -1
  if (CAT) {
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const int tok = t0 + j * 8 + g, id = tok < P.T ? (P.x1_tokens ? P.x1_tokens[tok] : tok) : -1;
      x1[j] = P.x1_tokens && id >= P.x1_rows ? -1 : id;
    }
  }
  // The token head's CTAs are short (ten chunks a warp at 2560 columns), and what each does before its first MMA counts: with the split's divisions and an
  // address per chunk it took 58.0 / 97 / 92 us for one row of the 3B, 40-head and 1B shapes, so 56.0 / 94 / 89.5. In the longer linears a
  // pointer per token costs more than it saves (one row, whole block 74.2 -> 75.2).
  const uint16_t* xrow = MODE == DL_LOGITS && NT == 1 && t0 + g < P.T ? P.x0 + (size_t)(t0 + g) * P.ldx0 + 8 * t : nullptr;
  auto load_x = [&](int c, uint4 (&d)[NT]) {
    const int col = c * 32 + 8 * t;
    if (MODE == DL_LOGITS && NT == 1) {
      d[0] = xrow && col < K ? *reinterpret_cast<const uint4*>(xrow + c * 32) : make_uint4(0, 0, 0, 0);
      return;
    }
    const bool second = CAT && col >= P.k0;
    const uint16_t* base = second ? P.x1 + (col - P.k0) : x0 + col;
    const int ld = second ? P.ldx1 : P.ldx0;
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const int tok = t0 + j * 8 + g, row = second ? x1[CAT ? j : 0] : (tok < P.T ? tok : -1);
      d[j] = row >= 0 && col < K ? *reinterpret_cast<const uint4*>(base + (size_t)row * ld) : make_uint4(0, 0, 0, 0);
    }
  };
#pragma unroll
  for (int a = 0; a < AH; a++) load_x(c1 + step * a, xv[a]);
  float acc[NW][MT][NT][4];
#pragma unroll
  for (int i = 0; i < NW; i++)
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int j = 0; j < NT; j++) acc[i][m][j][0] = acc[i][m][j][1] = acc[i][m][j][2] = acc[i][m][j][3] = 0.f;
  for (int c0 = c1; c0 < nch; c0 += step * AH) {
#pragma unroll
    for (int a = 0; a < AH; a++) {                   // chunks past the end multiply zeros
      const int c = c0 + step * a;
#pragma unroll
      for (int i = 0; i < NW; i++)
#pragma unroll
        for (int m = 0; m < MT; m++) {
          const uint4 lo = wv[a][i][m][0], hi = wv[a][i][m][1];
          const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
          for (int j = 0; j < NT; j++) {
            mma_bf16(acc[i][m][j], a0, xv[a][j].x, xv[a][j].y);
            mma_bf16(acc[i][m][j], a1, xv[a][j].z, xv[a][j].w);
          }
        }
      load_w(c + step * AH, wv[a]);
      load_x(c + step * AH, xv[a]);
    }
  }
  auto at = [&](int i, int m, int j, int e) -> float& {
    return red[warp][(i * MT + m) * 16 + g + 8 * (e >> 1)][j * 8 + 2 * t + (e & 1)];
  };
  auto each_acc = [&](auto f) {
#pragma unroll
    for (int i = 0; i < NW; i++)
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
          for (int e = 0; e < 4; e++) f(i, m, j, e);
  };
  each_acc([&](int i, int m, int j, int e) { at(i, m, j, e) = acc[i][m][j][e]; });
  __syncthreads();
  constexpr int NO = 16 * MT * 8 * NT;
  if (ks > 1) {
    cluster_wait();
    for (int o = tid; o < NO * NW; o += WARPS * 32) {
      const int r = o % ROWS, tk = o / ROWS;
      if (t0 + tk >= P.T) break;
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; w++) s += red[w][r][tk];
      st_cluster(cluster_map(smem_u32(&part[rank][tk][r]), tk % ks), __float_as_uint(s));
    }
    cluster_sync();
  }
  for (int o = tid; o < NO; o += WARPS * 32) {
    const int r = o % (16 * MT), tk = o / (16 * MT), n = r0 + r, tok = t0 + tk;
    if (n >= N || tok >= P.T || (ks > 1 && tk % ks != rank)) continue;
    float s = 0.f, s2 = 0.f;
    if (ks > 1) {
      for (int q = 0; q < ks; q++) {
        s += part[q][tk][r];
        if (NW > 1) s2 += part[q][tk][16 * MT * (NW - 1) + r];
      }
    } else {
#pragma unroll
      for (int w = 0; w < 8; w++) {
        s += red[w][r][tk];
        if (NW > 1) s2 += red[w][16 * MT * (NW - 1) + r][tk];
      }
    }
    if (MODE == DL_LOGITS) {
      P.yf[(size_t)tok * P.ldy[0] + n] = rbf(rbf(s) / P.scale);
      continue;
    }
    uint16_t* y = P.y[which] + (size_t)tok * P.ldy[which] + n;
    if (MODE == DL_STORE) {
      *y = f2bf(s);
    } else if (MODE == DL_RESID) {
      *y = f2bf(bf2f(P.resid[(size_t)tok * P.ldr + n]) + rbf(s));
    } else {
      const float gg = rbf(s), u = rbf(s2);
      *y = f2bf(rbf(gg / (1.0f + expf(-gg))) * u);
    }
  }
}

// y = bf16(bf16(x * r) * w), r = bf16(rsqrt(bf16(bf16(mean(bf16(x^2))) + eps))): RMSNorm as a bf16 PyTorch expression
// evaluates it (reference: train/draft_model.py:9-10). One CTA of 256 threads per row.
__global__ void __launch_bounds__(256) d_rmsnorm(const uint16_t* x, int ldx, const uint16_t* w, uint16_t* y, int ldy, int D, float eps,
                                                 bool first) {
  __shared__ float red[8];
  const int tid = threadIdx.x;
  pdl_begin(first);
  pdl_wait();
  const uint16_t* xr = x + (size_t)blockIdx.x * ldx;
  float ss = 0.f;
  for (int i = tid; i < D; i += 256) {
    const float v = bf2f(xr[i]);
    ss += rbf(v * v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) tot += red[i];
  const float r = rbf(rsqrtf(rbf(rbf(tot / (float)D) + eps)));
  for (int i = tid; i < D; i += 256)
    y[(size_t)blockIdx.x * ldy + i] = f2bf(rbf(bf2f(xr[i]) * r) * bf2f(w[i]));
}

// The same with the row in registers
__global__ void __launch_bounds__(256) d_rmsnorm_regs(const uint16_t* x, int ldx, const uint16_t* w, uint16_t* y, int ldy, int D, float eps, bool first) {
  __shared__ float red[8];
  pdl_begin(first);
  d_norm_row(x + (size_t)blockIdx.x * ldx, w, y + (size_t)blockIdx.x * ldy, D, eps, red);
}

// Half-split rotation of q and k (bf16 cos / sin tables as the reference casts them, reference:
// train/draft_model.py:12-22) and the cache write: token t's rotated k and its v go to cache slot slots[t].
// grid (T, n_head + n_kv), 64 threads: one CTA per (token, head), a thread per rotation pair (the angle's powf / cosf / sinf are the
// slow part: one per thread). q is rotated in place; a kv-head CTA also copies its v row.
__global__ void d_rope_store(uint16_t* q, const uint16_t* k, const uint16_t* v, const int32_t* positions, const int32_t* slots,
                             uint16_t* kc, uint16_t* vc, int nh, int nkv, int hd, float rope_base, int max_roll) {
  const int t = blockIdx.x, head = blockIdx.y, half = hd >> 1;
  pdl_trigger();
  pdl_wait();
  const float pos = (float)positions[t];
  const int slot = slots ? slots[t] : t;
  if (slot < 0 || slot >= max_roll) return;
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    const float inv = 1.0f / powf(rope_base, (float)(2 * i) / (float)hd);
    const float ang = pos * inv;
    const float c = rbf(cosf(ang)), s = rbf(sinf(ang));
    if (head < nh) {
      uint16_t* p = q + ((size_t)t * nh + head) * hd;
      const float a = bf2f(p[i]), b = bf2f(p[i + half]);
      p[i] = f2bf(rbf(a * c) + rbf(-b * s));
      p[i + half] = f2bf(rbf(b * c) + rbf(a * s));
    } else {
      const int kh = head - nh;
      const uint16_t* p = k + ((size_t)t * nkv + kh) * hd;
      uint16_t* d = kc + ((size_t)slot * nkv + kh) * hd;
      const float a = bf2f(p[i]), b = bf2f(p[i + half]);
      d[i] = f2bf(rbf(a * c) + rbf(-b * s));
      d[i + half] = f2bf(rbf(b * c) + rbf(a * s));
    }
  }
  if (head >= nh) {
    const int kh = head - nh;
    for (int o = threadIdx.x; o < hd; o += blockDim.x)
      vc[((size_t)slot * nkv + kh) * hd + o] = v[((size_t)t * nkv + kh) * hd + o];
  }
}

// Causal attention of token t over cache slots 0 .. slots[t] (the rows of a lower-triangular mask, reference:
// train/draft_model.py:43,57-59). grid (T, nh), 128 threads; softmax in fp32, output bf16.
__global__ void __launch_bounds__(128) d_attn(const uint16_t* q, const int32_t* slots, const uint16_t* kc, const uint16_t* vc,
                                              uint16_t* out, int nh, int nkv, int hd, int max_roll) {
  extern __shared__ float d_sc[];                  // [max_roll] scores, then [hd] the query
  __shared__ float red[4];
  float* qs = d_sc + max_roll;
  const int t = blockIdx.x, head = blockIdx.y, kh = head / (nh / nkv), tid = threadIdx.x;
  pdl_trigger();
  pdl_wait();
  const int last = min(slots ? slots[t] : t, max_roll - 1);
  if (last < 0) return;
  for (int i = tid; i < hd; i += 128) qs[i] = bf2f(q[((size_t)t * nh + head) * hd + i]);
  __syncthreads();
  const float scale = rsqrtf((float)hd);
  float mx = -INFINITY;
  for (int s = tid; s <= last; s += 128) {
    const uint16_t* kr = kc + ((size_t)s * nkv + kh) * hd;
    float d = 0.f;
    if (hd % 8 == 0) {                               // rows start on 16-byte boundaries
#pragma unroll 4
      for (int i = 0; i < hd; i += 8) {
        const uint4 kv = *reinterpret_cast<const uint4*>(kr + i);
        const uint32_t p[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
        for (int e = 0; e < 4; e++) { d = fmaf(qs[i + 2 * e], bflo(p[e]), d); d = fmaf(qs[i + 2 * e + 1], bfhi(p[e]), d); }
      }
    } else {
      for (int i = 0; i < hd; i++) d = fmaf(qs[i], bf2f(kr[i]), d);
    }
    d *= scale;
    d_sc[s] = d;
    mx = fmaxf(mx, d);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) red[tid >> 5] = mx;
  __syncthreads();
  mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  __syncthreads();
  float den = 0.f;
  for (int s = tid; s <= last; s += 128) {
    const float e = expf(d_sc[s] - mx);
    d_sc[s] = e;
    den += e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
  if ((tid & 31) == 0) red[tid >> 5] = den;
  __syncthreads();
  den = red[0] + red[1] + red[2] + red[3];
  for (int i = tid; i < hd; i += 128) {
    float a = 0.f;
#pragma unroll 8
    for (int s = 0; s <= last; s++) a = fmaf(d_sc[s], bf2f(vc[((size_t)s * nkv + kh) * hd + i]), a);
    out[((size_t)t * nh + head) * hd + i] = f2bf(a / den);
  }
}

// d_rope_store and d_attn of a single token in one launch: every query head's CTA rotates its own q and the group's new k, the first of the group
// writes k and v to the cache, and nobody reads the new rows from there. The same operations in the same order. grid (nh), 128 threads.
__global__ void __launch_bounds__(128) d_attn_one(const uint16_t* q, const uint16_t* k, const uint16_t* v, const int32_t* positions, const int32_t* slots,
                                                  uint16_t* kc, uint16_t* vc, uint16_t* out, int nh, int nkv, int hd, float rope_base, int max_roll) {
  extern __shared__ float d_sc[];                  // [max_roll] scores, [hd] the query, [hd] the new k, [hd] the new v
  __shared__ float red[4];
  float *qs = d_sc + max_roll, *ks = qs + hd, *vs = ks + hd;
  const int head = blockIdx.x, kh = head / (nh / nkv), tid = threadIdx.x;
  pdl_trigger();
  pdl_wait();
  const int slot = slots ? slots[0] : 0, last = min(slot, max_roll - 1);
  if (last < 0) return;
  const bool fresh = slot < max_roll;              // else the cache keeps its rows and q stays as it is, as in d_rope_store
  const uint16_t* qh = q + (size_t)head * hd;
  if (fresh) {
    const float pos = (float)positions[0];
    const bool writes = head % (nh / nkv) == 0;
    const size_t row = ((size_t)slot * nkv + kh) * hd;
    const int half = hd >> 1;
    for (int i = tid; i < half; i += 128) {
      const float ang = pos * (1.0f / powf(rope_base, (float)(2 * i) / (float)hd));
      const float c = rbf(cosf(ang)), s = rbf(sinf(ang));
      const float a = bf2f(qh[i]), b = bf2f(qh[i + half]), e = bf2f(k[kh * hd + i]), f = bf2f(k[kh * hd + i + half]);
      qs[i] = rbf(rbf(a * c) + rbf(-b * s));
      qs[i + half] = rbf(rbf(b * c) + rbf(a * s));
      const uint16_t k0 = f2bf(rbf(e * c) + rbf(-f * s)), k1 = f2bf(rbf(f * c) + rbf(e * s));
      ks[i] = bf2f(k0);
      ks[i + half] = bf2f(k1);
      if (writes) { kc[row + i] = k0; kc[row + i + half] = k1; }
    }
    for (int i = tid; i < hd; i += 128) {
      const uint16_t x = v[kh * hd + i];
      vs[i] = bf2f(x);
      if (writes) vc[row + i] = x;
    }
  } else {
    for (int i = tid; i < hd; i += 128) qs[i] = bf2f(qh[i]);
  }
  __syncthreads();
  const float scale = rsqrtf((float)hd);
  const int cached = fresh ? slot : last + 1;      // rows that come from the cache
  float mx = -INFINITY;
  for (int s = tid; s <= last; s += 128) {
    float d = 0.f;
    if (s == cached) {
      for (int i = 0; i < hd; i++) d = fmaf(qs[i], ks[i], d);
    } else if (hd % 8 == 0) {                        // rows start on 16-byte boundaries
      const uint16_t* kr = kc + ((size_t)s * nkv + kh) * hd;
#pragma unroll 4
      for (int i = 0; i < hd; i += 8) {
        const uint4 kv = *reinterpret_cast<const uint4*>(kr + i);
        const uint32_t p[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
        for (int e = 0; e < 4; e++) { d = fmaf(qs[i + 2 * e], bflo(p[e]), d); d = fmaf(qs[i + 2 * e + 1], bfhi(p[e]), d); }
      }
    } else {
      for (int i = 0; i < hd; i++) d = fmaf(qs[i], bf2f(kc[((size_t)s * nkv + kh) * hd + i]), d);
    }
    d *= scale;
    d_sc[s] = d;
    mx = fmaxf(mx, d);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) red[tid >> 5] = mx;
  __syncthreads();
  mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  __syncthreads();
  float den = 0.f;
  for (int s = tid; s <= last; s += 128) {
    const float e = expf(d_sc[s] - mx);
    d_sc[s] = e;
    den += e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
  if ((tid & 31) == 0) red[tid >> 5] = den;
  __syncthreads();
  den = red[0] + red[1] + red[2] + red[3];
  for (int i = tid; i < hd; i += 128) {
    float a = 0.f;
#pragma unroll 8
    for (int s = 0; s < cached; s++) a = fmaf(d_sc[s], bf2f(vc[((size_t)s * nkv + kh) * hd + i]), a);
    if (fresh) a = fmaf(d_sc[slot], vs[i], a);
    out[(size_t)head * hd + i] = f2bf(a / den);
  }
}

}  // namespace fb
