// int4 GEMM of the M-token passes on the 5th-generation tensor cores (tcgen05): a weight row is read once and multiplied with a tile of
// up to NT tokens. This file: the layout, the arithmetic, the epilogues, and the kernel for prompts (tiles of up to 128 or 192 tokens);
// fb_vtl.cuh: the kernel with one work item per CTA and K split over clusters, for trees (one tile of 16 / 32 / 64) and short prompts (tiles of 128).
//
// D[128 weight rows][NT tokens] (fp32, in TENSOR MEMORY) += A[128][128] * B[NT][128]^T per group of 128 columns, issued as
// eight tcgen05.mma (K = 16 each) into ONE accumulator for the whole K range. A is the group's weights with their scale,
// (nib - 8) * s * 2^er, in fp16: the product of a 4-bit and an 8-bit significand fits fp16's 11 bits, and the row's power of two
// 2^er (chosen from the row's largest scale) keeps it in range, so it is EXACT (up to group scales 2^29 apart within a row). B is
// the tokens' bf16-rounded activations as fp16, multiplied by one power of two per token: exact as well for elements down to 2^-31
// of the token's bound. The powers of two come out in the epilogue. The arithmetic is the reference's sum (nib - 8) * s * x with fp32
// accumulation (reference: kernels/verify_mega.cu:18-75), only the order of summation differs. The asymmetric layout's zero points
// are a second MMA per step with A = z * 2^er into the same accumulator.
// What this replaced: bf16 operands (nib - 8) with one accumulator per group, folded with the scale by eight warps that read every
// group back from tensor memory. That costs a load and an fma per (row, token, group) and two more barrier hand-overs per group: 1000
// clocks a group for 128 tokens against 512 for its MMAs.
//
// A is dequantised by 128-thread sets, thread = weight row = TMEM lane, and stored with tcgen05.st straight into tensor memory (a
// ring of 64-column stages): routing A through shared memory would cost 8 bytes of shared-memory traffic per int4 byte. B comes by
// tensor copies (box 64 columns x NT tokens) in the K-major 128-byte-swizzle layout the MMA reads.
//
// Weight layout ("TC layout", a library-owned copy made by tc_repack): per block of 128 rows, one record per group of 128
// columns: two 4 KB chunks [8 words][128 rows] -- word (w, r) holds columns 8w .. 8w+7 of row r with the nibbles ordered so
// that the four mask conversions yield ADJACENT column pairs -- then the group's fp16 scales s * 2^er [128 rows] (and zeros);
// after the last record the rows' factors 2^-er, fp32 [128]. One 1-D bulk copy brings a record; the dequantising thread of row r
// reads its words without bank conflicts.
//
// Work item = (token tile, row block), round-robin over persistent CTAs; two accumulators, so an item's epilogue overlaps the MMAs of
// the next. Trees and short prompts split K over a CLUSTER instead (fb_vtl.cuh): every CTA sends the sums of a share of the tokens to each CTA
// of its cluster through distributed shared memory, and each finishes its own tokens (sum in split order: deterministic), so the split costs
// no round trip through global memory. Every wait is bounded.
#pragma once
#include <cuda.h>

#include "fb_common.cuh"
#include "fb_geometry.hpp"
#include "fb_verify.cuh"

namespace fb {

constexpr int kTcThreads = 640;   // warps: 0 weights, 1 MMA issue, 2 activations, 4..11 dequantise, 12..19 epilogue
constexpr int kTcTable = 96;      // tokens of an epilogue warp, at most
constexpr int kTcEpiBytes = 2 * kTcTable * 4 + 16 * 64;
constexpr int kTcTrailer = kTcRowBlock * 4 + 16;      // a block's row factors, then its flag

__host__ __device__ constexpr int tc_rec_bytes(int has_zeros) { return 8192 + 256 * (has_zeros ? 2 : 1); }
__host__ __device__ constexpr size_t tc_block_bytes(int k, int has_zeros) {
  return (size_t)(k / 128) * tc_rec_bytes(has_zeros) + kTcTrailer;
}
__host__ __device__ constexpr size_t tc_matrix_bytes(int rows, int k, int has_zeros) {
  return (size_t)((rows + kTcRowBlock - 1) / kTcRowBlock) * tc_block_bytes(k, has_zeros);
}

__device__ __forceinline__ uint32_t f16x2_scaled(uint32_t bf16_pair, float f) {
  const __half2 hh = __floats2half2_rn(bflo(bf16_pair) * f, bfhi(bf16_pair) * f);
  return *reinterpret_cast<const uint32_t*>(&hh);
}

// caller layout (word c of a row = columns 8c .. 8c+7, column 8c+m in bits [4m, 4m+4)) -> TC layout.
// grid (row blocks, layers), 256 threads. norms (gate/up only): [layer][2] largest squared row norm of the gate and the up rows,
// as the bits of non-negative floats (zero before the launch).
__global__ void __launch_bounds__(256) tc_repack(const uint32_t* q, const uint16_t* sc, const uint16_t* zr, int rows, int K,
                                                 int order, int order_arg, int order_rows, uint8_t* out, unsigned* norms) {
  const bool hz = zr != nullptr;
  const int rb = blockIdx.x, nrb = gridDim.x, G = K / 128, nw = K / 8, rec = tc_rec_bytes(hz), r = threadIdx.x & 127,
            part = threadIdx.x >> 7;                            // two threads per row
  uint8_t* blk = out + ((size_t)blockIdx.y * nrb + rb) * tc_block_bytes(K, hz);
  __shared__ float s_max[256], s_min[256], s_sq[256];
  const int j = rb * 128 + r;
  const int row = j < rows ? (int)blockIdx.y * rows + perm_row(j, order, order_arg, order_rows) : -1;
  float mx = 0.f, mn = INFINITY;
  if (row >= 0)
    for (int g = part; g < G; g += 2) {
      const float a = fabsf(bf2f(sc[(size_t)row * G + g]));
      mx = fmaxf(mx, 8.0f * a);
      if (a > 0.f) mn = fminf(mn, a);
      if (hz) mx = fmaxf(mx, fabsf(bf2f(zr[(size_t)row * G + g])));
    }
  s_max[threadIdx.x] = mx;
  s_min[threadIdx.x] = mn;
  __syncthreads();
  const float rmax = fmaxf(s_max[r], s_max[r + 128]);
  float2 f = rmax > 0.f ? pow2_for(rmax) : make_float2(1.f, 1.f);      // 8 s in [2^14, 2^15)
  // the block's scales are stored for the one-fma conversion (S = 16 s 2^er, then in [2^15, 2^16), and 2^24 in the factor) when that
  // is exact in every row: no scale of a row below S = 128
  const bool fits = fminf(s_min[r], s_min[r + 128]) * f.x * 16.0f >= 128.0f;
  const bool fast = __syncthreads_and(!hz && fits && f.x < 1e30f && f.y < 1e25f);
  if (fast) f = make_float2(f.x * 16.0f, f.y * (16777216.0f / 16.0f));
  float sq = 0.f;
  for (int wq = part; wq < nw; wq += 2) {                      // word wq of the row
    const int g = wq >> 4;
    uint32_t d = 0x88888888u;                                  // padding rows: value 0
    if (row >= 0) {
      const uint32_t s = __ldg(q + (size_t)row * nw + wq);
      // column offset e goes to nibble slot [0, 4, 1, 5, 2, 6, 3, 7][e]: (w & 0x000F000F) is then columns (0, 1),
      // (w & 0x00F000F0) columns (2, 3), and the same two masks on w >> 8 columns (4, 5) and (6, 7)
      d = (s & 0xFu) | ((s >> 4 & 0xFu) << 16) | ((s >> 8 & 0xFu) << 4) | ((s >> 12 & 0xFu) << 20) | ((s >> 16 & 0xFu) << 8) |
          ((s >> 20 & 0xFu) << 24) | ((s >> 24 & 0xFu) << 12) | ((s >> 28 & 0xFu) << 28);
      if (norms) {
        const float sv = bf2f(sc[(size_t)row * G + g]), zv = hz ? bf2f(zr[(size_t)row * G + g]) : 0.f;
        for (int e = 0; e < 8; e++) {
          const float w = ((float)(s >> (4 * e) & 0xFu) - 8.0f) * sv + zv;
          sq = fmaf(w, w, sq);
        }
      }
    }
    reinterpret_cast<uint32_t*>(blk + (size_t)g * rec)[(wq & 15) * 128 + r] = d;
  }
  for (int g = part; g < G; g += 2) {
    __half* meta = reinterpret_cast<__half*>(blk + (size_t)g * rec + 8192);
    meta[r] = __float2half_rn(row >= 0 ? bf2f(sc[(size_t)row * G + g]) * f.x : 0.f);
    if (hz) meta[128 + r] = __float2half_rn(row >= 0 ? bf2f(zr[(size_t)row * G + g]) * f.x : 0.f);
  }
  if (part == 0) reinterpret_cast<float*>(blk + (size_t)G * rec)[r] = f.y;
  if (threadIdx.x < 4) reinterpret_cast<int*>(blk + (size_t)G * rec)[kTcRowBlock + threadIdx.x] = fast;
  if (norms) {
    s_sq[threadIdx.x] = sq;
    __syncthreads();
    if (part == 0 && row >= 0)
      atomicMax(norms + blockIdx.y * 2 + (j & 1), __float_as_uint(s_sq[r] + s_sq[r + 128]));
  }
}

// xn[m] = bf16((float(h) * r) * float(w)) of one token, as fp16 times a power of two for the GEMM, and as it is for the caller
// (feat). Leaves the token's factors: fx[m] = inverse of xn's power of two; with `norms` (the following gate/up matrix' largest
// squared row norms) also the power of two of the SwiGLU output and its inverse: |silu(g) u| <= |g| |u| <= |xn|^2 |Wg| |Wu|.
// Clears the token's attention bound. One CTA per token; D <= 8 * 256 * NV.
template <int NV>
__global__ void __launch_bounds__(256) v_norm_f16(const uint16_t* h, const uint16_t* w, uint16_t* xn, uint16_t* feat, float* fx,
                                                  const unsigned* norms, float* fa, float* fa_inv, unsigned* amax, int D, float eps) {
  const int m = blockIdx.x, tid = threadIdx.x;
  const uint4* hm = reinterpret_cast<const uint4*>(h + (size_t)m * D);
  const uint4* wv = reinterpret_cast<const uint4*>(w);
  const int nvec = D / 8;
  __shared__ float red[8], red2[8], red3[8];
  uint4 hv[NV], ww[NV];
  float ss = 0.f;
  pdl_trigger();
#pragma unroll
  for (int k = 0; k < NV; k++) {       // the norm weights do not depend on the previous kernel
    const int i = tid + k * 256;
    ww[k] = make_uint4(0, 0, 0, 0);
    if (i < nvec) ww[k] = __ldg(wv + i);
  }
  pdl_wait();
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const int i = tid + k * 256;
    hv[k] = make_uint4(0, 0, 0, 0);
    if (i < nvec) hv[k] = hm[i];
    const uint32_t p[4] = {hv[k].x, hv[k].y, hv[k].z, hv[k].w};
#pragma unroll
    for (int e = 0; e < 4; e++) { ss = fmaf(bflo(p[e]), bflo(p[e]), ss); ss = fmaf(bfhi(p[e]), bfhi(p[e]), ss); }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) tot += red[i];
  const float r = 1.0f / sqrtf(tot / (float)D + eps);
  float mx = 0.f, sq = 0.f;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const uint32_t p[4] = {hv[k].x, hv[k].y, hv[k].z, hv[k].w}, q[4] = {ww[k].x, ww[k].y, ww[k].z, ww[k].w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      o[e] = (uint32_t)f2bf(bflo(p[e]) * r * bflo(q[e])) | ((uint32_t)f2bf(bfhi(p[e]) * r * bfhi(q[e])) << 16);
      mx = fmaxf(mx, fmaxf(fabsf(bflo(o[e])), fabsf(bfhi(o[e]))));
      sq = fmaf(bflo(o[e]), bflo(o[e]), fmaf(bfhi(o[e]), bfhi(o[e]), sq));
    }
    hv[k] = make_uint4(o[0], o[1], o[2], o[3]);
    const int i = tid + k * 256;
    if (feat && i < nvec) reinterpret_cast<uint4*>(feat + (size_t)m * D)[i] = hv[k];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
  }
  if ((tid & 31) == 0) { red2[tid >> 5] = mx; red3[tid >> 5] = sq; }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; i++) mx = fmaxf(mx, red2[i]);
  const float2 f = pow2_for(mx);
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const int i = tid + k * 256;
    if (i < nvec)
      reinterpret_cast<uint4*>(xn + (size_t)m * D)[i] = make_uint4(f16x2_scaled(hv[k].x, f.x), f16x2_scaled(hv[k].y, f.x),
                                                                  f16x2_scaled(hv[k].z, f.x), f16x2_scaled(hv[k].w, f.x));
  }
  if (tid == 0) {
    fx[m] = f.y;
    amax[m] = 0u;
    if (norms) {
      float n2 = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i++) n2 += red3[i];
      const float2 a = pow2_for(n2 * sqrtf(__uint_as_float(norms[0])) * sqrtf(__uint_as_float(norms[1])));
      fa[m] = a.x;
      fa_inv[m] = a.y;
    }
  }
}

// Attention output of one token, bf16 -> fp16 times a power of two, in place: prompts, whose GEMM brings its activations by tensor copies (the
// tree GEMM converts them on the way in). One CTA of 256 threads per token.
__global__ void __launch_bounds__(256) v_row_f16(uint16_t* x, float* fx, int D) {
  const int m = blockIdx.x, tid = threadIdx.x, nvec = D / 8;
  __shared__ float red[8];
  uint4* xm = reinterpret_cast<uint4*>(x + (size_t)m * D);
  pdl_trigger();
  pdl_wait();
  float mx = 0.f;
  for (int i = tid; i < nvec; i += 256) {
    const uint4 v = xm[i];
    const uint32_t p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; e++) mx = fmaxf(mx, fmaxf(fabsf(bflo(p[e])), fabsf(bfhi(p[e]))));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) red[tid >> 5] = mx;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; i++) mx = fmaxf(mx, red[i]);
  const float2 f = pow2_for(mx);
  for (int i = tid; i < nvec; i += 256) {
    const uint4 v = xm[i];
    xm[i] = make_uint4(f16x2_scaled(v.x, f.x), f16x2_scaled(v.y, f.x), f16x2_scaled(v.z, f.x), f16x2_scaled(v.w, f.x));
  }
  if (tid == 0) fx[m] = f.y;
}

// cos / sin of every (token, rotation pair): the QKV epilogue reads them instead of evaluating sincosf per output.
// depth == nullptr: a chain, token m sits at position pos + m
__global__ void v_rope_table(const int32_t* depth, const float* invf, int pos, int half, float2* out) {
  const int m = blockIdx.x;
  pdl_trigger();
  pdl_wait();
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    float sn, cs;
    sincosf((float)(pos + (depth ? depth[m] : m)) * invf[i], &sn, &cs);
    out[(size_t)m * half + i] = make_float2(cs, sn);
  }
}

struct alignas(64) VtcParams {
  CUtensorMap xmap;          // activations fp16 [rows >= M][K] as a 2-D tensor, box 64 columns x NT tokens, 128-byte swizzle
  const uint8_t* w;          // TC layout of this matrix
  int rows, K, M;
  int nsplit;                // v_gemm_tl: CTAs of a cluster that share one item's K (1, 2, 4 or 8)
  int ntok, ntile;           // tokens of one tile (a multiple of 16, <= NT; one tile unless this is a prompt) and tiles
  DevStatus* status;
  unsigned spin_limit;
  const float* fx;           // [M] inverse of the power of two in each token's activations
  const uint16_t* xbf;       // O of a tree: the attention output as bf16 [M][K]; this kernel converts it on the way in (xmap unused),
  const unsigned* amax;      // with the power of two of the token's largest magnitude (float bits), fx unused. One item per CTA.
  // epilogue operands
  uint16_t* h;               // RESID: bf16 [M][out_ld] in/out
  uint16_t* q;               // QKV: bf16 [M][n_head * HD]
  uint16_t *kc, *vc;         // QKV: layer base of the caches [max_seq][nkv][HD]
  uint16_t* act;             // SWIGLU: fp16 [M][out_ld], times the token's fa
  const float* fa;           // SWIGLU: [M]
  float* logits;             // LOGITS: f32 [M][out_ld]
  const float2* rope;        // QKV: [M][HD / 2] (cos, sin)
  int n_head, nkv, pos, out_ld, head_dim;
  float resid, logits_scaling;
};

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
// nibble pairs in bits (0..3, 16..19) / (4..7, 20..23) -> fp16 pair (nib - 8) * s, the magic-exponent conversion that is published for int4
// weights (Kim et al., "Who Says Elephants Can't Run", 2022): OR-ing in the exponent of 1024 makes 1024 + nib
// (1024 + 16 nib); taking 1032 off (or a sixteenth minus 72) is exact, and so is the product
__device__ __forceinline__ uint32_t tc_h2(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ __half2 tc_as_h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t tc_cvt_lo(uint32_t w, __half2 s) {
  return tc_h2(__hmul2(__hsub2(tc_as_h2((w & 0x000F000Fu) | 0x64006400u), tc_as_h2(0x64086408u)), s));
}
__device__ __forceinline__ uint32_t tc_cvt_hi(uint32_t w, __half2 s) {
  return tc_h2(__hmul2(__hfma2(tc_as_h2((w & 0x00F000F0u) | 0x64006400u), tc_as_h2(0x2C002C00u), tc_as_h2(0xD480D480u)), s));
}
// The same in one fma, for row blocks whose scales are not more than 2^8 apart in any row (the trailer's flag): the masked bits are
// the fp16 subnormals nib * 2^-24 (16 nib * 2^-24); times S = s * 2^24 * 2^er (or S / 16) minus 8 S 2^-24 is exact as long as the
// result's last bit, that of s, is not below 2^-24
__device__ __forceinline__ uint32_t tc_cvt_fast(uint32_t bits, __half2 s, __half2 c) { return tc_h2(__hfma2(tc_as_h2(bits), s, c)); }
// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}
// 32 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
        "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
        "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// one lane of a converged warp; unlike `lane == 0` the compiler knows that the rest of the warp does the same uniform work
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, uint32_t z) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
// Shared-memory plan (bytes). The raw ring keeps HBM busy; a stage of activations is a group's two 64-column tiles.
// Tiles of 128 tokens, or of 192: an item's groups then take about 4/3 of the time for 3/2 of the tokens (680 cycles a group at 128, 950
// at 192), because dequantising a group and storing it to tensor memory (which keeps the MMAs out meanwhile) is a cost per item. What is
// left of tensor memory allows two A stages, and none for zero points.
template <bool HZ, int NT_>
struct VtcSmem {
  static constexpr int NT = NT_, REC = tc_rec_bytes(HZ);
  static constexpr int NS = NT == 192 ? 2 : (HZ ? 3 : 4);          // A stages (64 columns): what two accumulators leave
  static constexpr int NB = NT == 192 ? 3 : 5, NRAW = 6;           // activation stages, raw int4 groups
  static constexpr int BSTAGE = NT * 256;                          // two [NT rows x 128 bytes] swizzled tiles
  static constexpr int B = 0;
  static constexpr int RAW = B + NB * BSTAGE;
  // Barriers that the MMAs of a group complete (one commit per group): group g's is done[g % ND]. Everybody who waits for a
  // group to retire (its A stage, its activation stage) waits there; nobody is ND groups behind.
  static constexpr int ND = 16;
  static_assert(ND >= NB && ND >= NS, "a retired group must not be overtaken by the next one on its barrier");
  static constexpr int BAR = RAW + NRAW * REC;
  static constexpr int EPI = BAR + 512;                            // per epilogue warp: token factors, then 16 tokens x 32 rows of 16 bits
  static constexpr int TOTAL = EPI + 8 * kTcEpiBytes + 1024;       // + slack to align the base
  static_assert(TOTAL <= 227 * 1024, "prompt GEMM shared memory");
  // tensor memory columns: two accumulators, A stages, A_z (8 columns = one k16 step of the row's zero point, the same for every
  // step of the group)
  static constexpr int T_A = 2 * NT, T_AZ = T_A + NS * 64;
  static_assert(T_AZ + (HZ ? NS * 8 : 0) <= 512, "tensor memory columns");
};

// position in a ring of N: index and the parity of its current lap
template <int N>
struct Ring {
  int i = 0;
  uint32_t lap = 0;
  __device__ __forceinline__ void next() { if (++i == N) { i = 0; lap ^= 1u; } }
};

// work items of this CTA in order (token tile by token tile: the tile's activations stay in L2); every role walks the same
// sequence
struct TcWalk {
  int item, nitems, nrb, step, G, rb, tt;
  __device__ __forceinline__ TcWalk(const VtcParams& P) {
    G = P.K / 128;
    nrb = (P.rows + kTcRowBlock - 1) / kTcRowBlock;
    nitems = nrb * P.ntile;
    item = (int)blockIdx.x;
    step = (int)gridDim.x;
    set();
  }
  __device__ __forceinline__ bool valid() const { return item < nitems; }
  __device__ __forceinline__ void set() { tt = item / nrb; rb = item % nrb; }
  __device__ __forceinline__ void next() { item += step; set(); }
};

// What one chunk of the epilogue reads from global memory (issued early: it does not depend on the GEMM)
template <int EPI, int CH>
struct TcOperands {
  uint16_t h[EPI == EPI_RESID ? CH : 1];
  float2 cs[EPI == EPI_QKV ? CH : 1];
  __device__ __forceinline__ void fetch(const VtcParams& P, int srow, int t0, int tend) {
    if constexpr (EPI == EPI_RESID) {
#pragma unroll
      for (int e = 0; e < CH; e++)
        h[e] = (srow < P.rows && t0 + e < tend) ? ld_cg_u16(P.h + (size_t)(t0 + e) * P.out_ld + srow) : (uint16_t)0;
    } else if constexpr (EPI == EPI_QKV) {
      const int HP = P.head_dim >> 1, head = srow / P.head_dim, i = (srow % P.head_dim) >> 1;
      const bool rot = head < P.n_head + P.nkv;
#pragma unroll
      for (int e = 0; e < CH; e++)
        cs[e] = (rot && t0 + e < tend) ? __ldg(P.rope + (size_t)(t0 + e) * HP + i) : make_float2(1.f, 0.f);
    }
  }
};
// The token factors of a warp's (up to 32 NF) tokens, spread over its lanes: one load per item instead of an L2 round trip per chunk
template <int EPI, int NF = 2>
struct TcFactors {
  float fx[NF], fa[NF];
  __device__ __forceinline__ void fetch(const VtcParams& P, int t0, int tend, int lane) {
#pragma unroll
    for (int k = 0; k < NF; k++) {
      const int t = t0 + 32 * k + lane;
      fx[k] = t >= tend ? 0.f : (EPI == EPI_RESID && P.amax) ? pow2_for(__uint_as_float(__ldcg(P.amax + t))).y : __ldcg(P.fx + t);
      if (EPI == EPI_SWIGLU) fa[k] = t < tend ? __ldcg(P.fa + t) : 0.f;
    }
  }
  __device__ __forceinline__ float x(int i) const { return __shfl_sync(0xffffffffu, i < 32 ? fx[0] : fx[1], i & 31); }
  __device__ __forceinline__ float a(int i) const { return __shfl_sync(0xffffffffu, i < 32 ? fa[0] : fa[1], i & 31); }
};
// The same from a table that the warp keeps in shared memory (prompts: up to 96 tokens of an item; a shuffle per token and factor costs more)
struct TcFactorTable {
  float *fx, *fa;
  template <int EPI, int NF>
  __device__ __forceinline__ void put(const TcFactors<EPI, NF>& f, int lane) {
#pragma unroll
    for (int k = 0; k < NF; k++) {
      fx[32 * k + lane] = f.fx[k];
      if (EPI == EPI_SWIGLU) fa[32 * k + lane] = f.fa[k];
    }
    __syncwarp();
  }
  __device__ __forceinline__ float x(int i) const { return fx[i]; }
  __device__ __forceinline__ float a(int i) const { return fa[i]; }
};
// silu(g) = g / (1 + e^-g) with the exact division, the decode kernel's expression. (The approximate one, off by up to 2 ulp and zero where 1 + e^-g is
// above 2^126, rounds bf16(silu(g) u) the other way at 386 of the 65280 x 128 pairs of a finite bf16 g and a mantissa of u, all but two of them
// at g = -87.5 .. -88.5. Without its branches a prompt of 725 tokens of the 3B shape takes 6185 us instead of 6349, engine calls back to back, a
// 26-node tree 0.5 % less.)
__device__ __forceinline__ float tc_silu(float g) { return g / (1.0f + __expf(-g)); }
// v[e] = accumulator of (stream row srow, token t0 + e), the i0 + e-th of the warp's tokens; rf = the row's factor. The whole warp
// calls this together: lanes 2i, 2i + 1 hold the two rows of a RoPE or gate/up pair.
template <int EPI, int CH, class F>
__device__ __forceinline__ void vtc_epilogue(const VtcParams& P, int srow, int t0, int tend, float (&v)[CH], float rf,
                                             const F& f, int i0, const TcOperands<EPI, CH>& o, int lane) {
  const bool live = srow < P.rows, odd = lane & 1;
#pragma unroll
  for (int e = 0; e < CH; e++) v[e] = v[e] * rf * f.x(i0 + e);
  if constexpr (EPI == EPI_RESID) {
#pragma unroll
    for (int e = 0; e < CH; e++)
      if (live && t0 + e < tend) P.h[(size_t)(t0 + e) * P.out_ld + srow] = f2bf(bf2f(o.h[e]) + v[e] * P.resid);
  } else if constexpr (EPI == EPI_LOGITS) {
#pragma unroll
    for (int e = 0; e < CH; e++)
      if (live && t0 + e < tend) P.logits[(size_t)(t0 + e) * P.out_ld + srow] = v[e] / P.logits_scaling;
  } else if constexpr (EPI == EPI_SWIGLU) {
    // stream rows (2i, 2i+1) = (gate_i, up_i): the even lane takes the even tokens of the pair, the odd lane the odd ones
#pragma unroll
    for (int e = 0; e < CH; e += 2) {
      const float got = __shfl_xor_sync(0xffffffffu, odd ? v[e] : v[e + 1], 1);
      const float gg = rbf(odd ? got : v[e]), uu = rbf(odd ? v[e + 1] : got);
      const float f0 = f.a(i0 + e), f1 = f.a(i0 + e + 1);
      const int t = t0 + e + (odd ? 1 : 0);
      const __half a = __float2half_rn(rbf(tc_silu(gg) * uu) * (odd ? f1 : f0));
      if (live && t < tend) P.act[(size_t)t * P.out_ld + (srow >> 1)] = __half_as_ushort(a);
    }
  } else {
    // QKV: stream rows (2p, 2p+1) of a q / k head are dims (p, p + HD/2); v rows keep their order
    const int HD = P.head_dim, HP = HD >> 1, QD = P.n_head * HD, head = srow / HD, within = srow % HD;
    const bool rot = head < P.n_head + P.nkv;
    uint16_t* base;
    size_t ld;
    if (head < P.n_head) {
      base = P.q + head * HD + (within >> 1) + (odd ? HP : 0);
      ld = QD;
    } else {
      const int kvh = rot ? head - P.n_head : head - P.n_head - P.nkv;
      ld = (size_t)P.nkv * HD;
      base = (rot ? P.kc : P.vc) + (size_t)P.pos * ld + kvh * HD + (rot ? (within >> 1) + (odd ? HP : 0) : within);
    }
#pragma unroll
    for (int e = 0; e < CH; e++) {
      const float x = rbf(v[e]), y = __shfl_xor_sync(0xffffffffu, x, 1);
      const float r = odd ? x * o.cs[e].x + y * o.cs[e].y : x * o.cs[e].x - y * o.cs[e].y;
      if (live && t0 + e < tend) base[(size_t)(t0 + e) * ld] = f2bf(rot ? r : v[e]);
    }
  }
}

// RESID and SWIGLU of 16 tokens by a warp (32 weight rows), through 1 KB of shared memory: the outputs of a token are adjacent there and
// leave 16 bytes at a time (the residual comes the same way). Thread by thread they are 2-byte accesses, an address and a predicate per
// value, and with them the epilogue of a 128 x 128 item took as long as its MMAs left idle: prompts of 100 / 250 / 725 tokens of the 3B
// shape 3710 / 4465 / 7200 us, without any epilogue 3100 / 3630 / 6270, staged (with the approximate silu) 3380 / 4062 / 6840.
template <int EPI>
struct TcStaged {
  static constexpr int NV = EPI == EPI_RESID ? 2 : 1;           // 16-byte vectors of a lane: 16 tokens x 64 bytes, or x 32 (SWIGLU halves the rows)
  static constexpr int LPT = NV * 2;                            // lanes per token
  uint4 h[NV];
  __device__ __forceinline__ uint16_t* at(const VtcParams& P, int wrow, int tok, int lane) const {
    uint16_t* base = EPI == EPI_RESID ? P.h + wrow : P.act + (wrow >> 1);
    return base + (size_t)tok * P.out_ld + (lane % LPT) * 8;
  }
  __device__ __forceinline__ void fetch(const VtcParams& P, int wrow, int t0, int tend, int lane) {
    if (EPI == EPI_RESID) {
#pragma unroll
      for (int i = 0; i < NV; i++) {
        const int tok = t0 + i * (32 / LPT) + lane / LPT;
        h[i] = tok < tend ? __ldcg(reinterpret_cast<const uint4*>(at(P, wrow, tok, lane))) : make_uint4(0, 0, 0, 0);
      }
    }
  }
  // v[e]: accumulator of row wrow + lane and token t0 + e, the i0 + e-th of the warp's tokens
  __device__ __forceinline__ void run(const VtcParams& P, uint8_t* stage, int wrow, int t0, int tend, float (&v)[16], float rf,
                                      const TcFactorTable& f, int i0, int lane) {
    uint16_t* s16 = reinterpret_cast<uint16_t*>(stage);
    const bool odd = lane & 1;
    if (EPI == EPI_RESID) {
#pragma unroll
      for (int i = 0; i < NV; i++) reinterpret_cast<uint4*>(stage)[i * 32 + lane] = h[i];
      __syncwarp();
    }
#pragma unroll
    for (int e4 = 0; e4 < 16; e4 += 4) {
      const float4 fx = *reinterpret_cast<const float4*>(f.fx + i0 + e4);
      v[e4] = v[e4] * rf * fx.x; v[e4 + 1] = v[e4 + 1] * rf * fx.y; v[e4 + 2] = v[e4 + 2] * rf * fx.z; v[e4 + 3] = v[e4 + 3] * rf * fx.w;
      if (EPI == EPI_RESID) {
#pragma unroll
        for (int e = e4; e < e4 + 4; e++) s16[e * 32 + lane] = f2bf(bf2f(s16[e * 32 + lane]) + v[e] * P.resid);
      } else {
        const float4 fa = *reinterpret_cast<const float4*>(f.fa + i0 + e4);
        // rows (2i, 2i + 1) = (gate_i, up_i): the even lane takes the even tokens of the pair, the odd lane the odd ones
#pragma unroll
        for (int e = e4; e < e4 + 4; e += 2) {
          const float got = __shfl_xor_sync(0xffffffffu, odd ? v[e] : v[e + 1], 1);
          const float gg = rbf(odd ? got : v[e]), uu = rbf(odd ? v[e + 1] : got);
          const float a = e == e4 ? (odd ? fa.y : fa.x) : (odd ? fa.w : fa.z);
          s16[(e + (odd ? 1 : 0)) * 16 + (lane >> 1)] = __half_as_ushort(__float2half_rn(rbf(tc_silu(gg) * uu) * a));
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NV; i++) {
      const int tok = t0 + i * (32 / LPT) + lane / LPT;
      const uint4 o = reinterpret_cast<const uint4*>(stage)[i * 32 + lane];
      if (tok < tend) *reinterpret_cast<uint4*>(at(P, wrow, tok, lane)) = o;
    }
    __syncwarp();
  }
};

// after a failure: the copies and MMAs in flight (see drain_phase); out of line, a healthy launch never comes here
template <int NRAW, int NS, int NB, int ND>
inline __device__ __noinline__ void tc_drain(uint64_t* bars, volatile int* s_issued) {
  uint64_t *raw_full = bars, *b_full = bars + 2 * NRAW + NS, *done = b_full + NB, *acc_full = done + ND;
  const uint32_t n = s_issued[1];
  drain_ring<NRAW>(raw_full, s_issued[0]);
  drain_ring<NB>(b_full, s_issued[2]);
  if (n) drain_phase(&done[(n - 1) % ND], ((n - 1) / ND) & 1);
  drain_ring<2>(acc_full, s_issued[3]);
  __syncwarp();
}

template <int EPI, bool HZ, int NT_>
__global__ void __launch_bounds__(kTcThreads, 1) v_gemm_tc(const __grid_constant__ VtcParams P) {
  using S = VtcSmem<HZ, NT_>;
  constexpr int NT = S::NT, NRAW = S::NRAW, NS = S::NS, NB = S::NB, ND = S::ND, REC = S::REC, HC = NT / 2;
  extern __shared__ __align__(1024) uint8_t tsm_raw[];
  // the swizzle pattern is a function of the absolute shared-memory address: tiles must start on 1024-byte boundaries
  uint8_t* tsm = tsm_raw + ((1024u - (smem_u32(tsm_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(tsm + S::BAR);
  uint64_t *raw_full = bars, *raw_empty = bars + NRAW, *a_full = bars + 2 * NRAW, *b_full = a_full + NS, *done = b_full + NB,
           *acc_full = done + ND, *acc_empty = acc_full + 2;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  volatile int* s_issued = s_abort + 1;                          // [4] copies or MMA groups that warps 0, 1, 2 have issued, whole items of warp 1
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < NRAW; i++) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 8); }
    for (int i = 0; i < NS; i++) mbar_init(&a_full[i], 8);
    for (int i = 0; i < NB; i++) mbar_init(&b_full[i], 1);
    for (int i = 0; i < ND; i++) mbar_init(&done[i], 1);
    for (int i = 0; i < 2; i++) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
    *s_abort = 0;
    mbar_fence_init();
  }
  constexpr int TCOLS = 512;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  WaitCtl wc{P.status, s_abort, P.spin_limit};
  pdl_trigger();
  const int quad = warp & 3, row = quad * 32 + lane;             // warps 4..19: row of the block = TMEM lane
  const int half = ((warp >> 2) & 1) ^ 1;                        // warps 4..11: half of a group's columns; 12..19: of the tokens
  bool ok = true;

  if (warp == 0) {
    // ---------------- producer: the groups' records (weights do not depend on the previous kernel)
    if (lane == 0) {
      uint32_t gi = 0;
      Ring<NRAW> r;
      for (TcWalk w(P); w.valid() && ok; w.next()) {
        const uint8_t* blk = P.w + (size_t)w.rb * tc_block_bytes(P.K, HZ);
        for (int g = 0; g < w.G; g++, gi++, r.next()) {
          ok = mbar_wait(&raw_empty[r.i], r.lap ^ 1u, wc, W_EMPTY, 2);
          if (!ok) break;
          mbar_expect_tx(&raw_full[r.i], REC);
          bulk_g2s(tsm + S::RAW + r.i * REC, blk + (size_t)g * REC, REC, &raw_full[r.i]);
        }
      }
      s_issued[0] = gi;
    }
  } else if (warp == 1) {
    // ---------------- MMA issue: the warp waits as one, an elected lane issues eight MMAs per group and one commit. (With the
    // whole loop under `lane == 0` every operand took a trip through the vector registers: 0.36 us per group on top of the MMAs.)
    const uint32_t idesc = (1u << 4) | ((uint32_t)(P.ntok >> 3) << 17) | ((128u >> 4) << 24);      // fp16 x fp16 -> fp32
    Ring<NS> rs;
    Ring<NB> rb;
    Ring<ND> rd;
    Ring<2> ra;
    uint32_t gi = 0, finished = 0;
    for (TcWalk w(P); w.valid() && ok; w.next(), ra.next()) {
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[ra.i], ra.lap ^ 1u, wc, W_EMPTY, 3));
      for (int g = 0; g < w.G && ok; g++, gi++, rs.next(), rb.next(), rd.next()) {
        // both are usually there already: test them side by side, a barrier test is a round trip of its own
        bool now = mbar_try(&a_full[rs.i], rs.lap);
        now = mbar_try(&b_full[rb.i], rb.lap) && now;
        if (!now) ok = mbar_wait(&a_full[rs.i], rs.lap, wc, W_FULL, 4) && mbar_wait(&b_full[rb.i], rb.lap, wc, W_FULL, 4);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t ta = tmem + S::T_A + rs.i * 64, tz = tmem + S::T_AZ + rs.i * 8, td = tmem + ra.i * NT;
          const uint64_t db0 = tc_desc(smem_u32(tsm + S::B + rb.i * S::BSTAGE));
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const uint64_t db = db0 + (uint64_t)(((k >> 2) * (NT * 128) + (k & 3) * 32) >> 4);
            tc_mma_ts(td, ta + k * 8, db, idesc, (g || k) ? 1u : 0u);
            if (HZ) tc_mma_ts(td, tz, db, idesc, 1u);
          }
          tc_commit(&done[rd.i]);
          if (g == w.G - 1) tc_commit(&acc_full[ra.i]);
        }
        __syncwarp();
      }
      if (ok) finished++;
    }
    if (lane == 0) { s_issued[1] = gi; s_issued[3] = finished; }
  } else if (warp == 2) {
    // ---------------- activations (the previous kernel's output): two tensor copies per group. Token rows past M are whatever
    // the buffer holds: they only feed accumulator columns that nobody reads.
    pdl_wait();
    if (lane == 0) {
      uint32_t gi = 0;
      Ring<NB> r;
      for (TcWalk w(P); w.valid() && ok; w.next()) {
        for (int g = 0; g < w.G; g++, gi++, r.next()) {
          // group gi - NB has retired
          ok = gi < NB || mbar_wait(&done[(gi - NB) % ND], ((gi - NB) / ND) & 1, wc, W_EMPTY, 8);
          if (!ok) break;
          mbar_expect_tx(&b_full[r.i], S::BSTAGE);
          uint8_t* dst = tsm + S::B + r.i * S::BSTAGE;
          tma_load_2d(dst, &P.xmap, g * 128, w.tt * P.ntok, &b_full[r.i]);
          tma_load_2d(dst + NT * 128, &P.xmap, g * 128 + 64, w.tt * P.ntok, &b_full[r.i]);
        }
      }
      s_issued[2] = gi;
    }
  } else if (warp >= 4 && warp < 12) {
    // ---------------- dequantise: thread = (row of the block = TMEM lane, half of the group's columns); 8 words -> 32 packed fp16
    // pairs per group. (Two warps sharing a group halve the time that a stage is busy; with each warp doing whole groups in turn
    // the stages did not cover the round trip to the MMA and back.)
    const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16) + half * 32;
    uint32_t gi = 0;
    Ring<NRAW> rr;
    Ring<NS> rs;
    for (TcWalk w(P); w.valid() && ok; w.next()) {
      const bool fast = !HZ && __ldg(reinterpret_cast<const int*>(P.w + (size_t)(w.rb + 1) * tc_block_bytes(P.K, HZ)) - 4) != 0;
      for (int g = 0; g < w.G; g++, gi++, rr.next(), rs.next()) {
        uint64_t* freed = &done[(gi - NS) % ND];                 // the stage's previous group has retired
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
        tc_st32(tl + S::T_A + rs.i * 64, v);
        if (HZ && half == 0) {
          // the group's zero point of this row as one k16 step: A_z = z for every column
          const uint16_t z = reinterpret_cast<const uint16_t*>(rec + 8448)[row];
          tc_st8(tl + S::T_AZ + rs.i * 8, (uint32_t)z | ((uint32_t)z << 16));
        }
        tc_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(&a_full[rs.i]); mbar_arrive(&raw_empty[rr.i]); }
      }
    }
  } else if (warp >= 12) {
    // ---------------- epilogue: thread = (row of the block, half of the tokens), 8 or 16 tokens at a time
    constexpr bool STAGED = EPI == EPI_RESID || EPI == EPI_SWIGLU;
    constexpr int CH = STAGED || EPI == EPI_LOGITS ? 16 : 8;
    const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16) + half * HC;
    uint8_t* area = tsm + S::EPI + (warp - 12) * kTcEpiBytes;
    TcFactorTable fac{reinterpret_cast<float*>(area), reinterpret_cast<float*>(area) + kTcTable};
    TcOperands<EPI, CH> pre;
    TcStaged<EPI> staged;
    Ring<2> ra;
    pdl_wait();
    for (TcWalk w(P); w.valid() && ok; w.next(), ra.next()) {
      const int tok0 = w.tt * P.ntok, tend = min(P.M, tok0 + P.ntok), srow = w.rb * 128 + row;
      // the row's factor and the first chunk's operands are fetched while the GEMM runs
      const float rf = __ldg(reinterpret_cast<const float*>(P.w + (size_t)(w.rb + 1) * tc_block_bytes(P.K, HZ)) - kTcTrailer / 4 + row);
      const int th0 = tok0 + half * HC, the = min(tend, th0 + HC);
      if constexpr (STAGED) staged.fetch(P, srow - lane, th0, the, lane);
      else pre.fetch(P, srow, th0, the);
      __syncwarp();
      TcFactors<EPI, HC / 32> mine;
      mine.fetch(P, th0, the, lane);
      fac.put<EPI, HC / 32>(mine, lane);
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[ra.i], ra.lap, wc, W_FULL, 10));
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int t0 = th0; t0 < the; t0 += CH) {
        uint32_t u[CH / 8][8];
#pragma unroll
        for (int c8 = 0; c8 < CH / 8; c8++) tc_ld8(tlane + ra.i * NT + (t0 - th0) + c8 * 8, u[c8]);
        TcOperands<EPI, CH> nxt;
        TcStaged<EPI> snxt;
        if constexpr (STAGED) snxt.fetch(P, srow - lane, t0 + CH, the, lane);
        else nxt.fetch(P, srow, t0 + CH, the);
        tc_ld_wait();
        float v[CH];
#pragma unroll
        for (int e = 0; e < CH; e++) v[e] = __uint_as_float(u[e >> 3][e & 7]);
        if constexpr (STAGED) {
          staged.run(P, area + 2 * kTcTable * 4, srow - lane, t0, the, v, rf, fac, t0 - th0, lane);
          staged = snxt;
        } else {
          vtc_epilogue<EPI, CH>(P, srow, t0, the, v, rf, fac, t0 - th0, pre, lane);
          pre = nxt;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[ra.i]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*s_abort) tc_drain<NRAW, NS, NB, ND>(bars, s_issued);
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS));
  }
}

}  // namespace fb
