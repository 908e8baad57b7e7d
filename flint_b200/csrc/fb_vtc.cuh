// int4 x bf16 GEMM of the M-token verify and prefill paths on the 5th-generation tensor cores (tcgen05): a weight row is
// read once and multiplied with a tile of up to NT tokens (NT = 16 / 32 / 64 for verify, 128 for prompts).
//
// D[128 weight rows][NT tokens] (fp32, in TENSOR MEMORY) = A[128][128] * B[NT][128]^T per group of 128 columns, issued by
// one thread as eight tcgen05.mma (K = 16 each). A is the group's weights dequantised to bf16 (nib - 8) / 64 -- exact -- by 128
// threads, thread = weight row = TMEM lane, and stored with tcgen05.st straight into tensor memory (a ring of four
// 64-column stages): routing A through shared memory would cost 8 bytes of shared-memory traffic per int4 byte and cap
// the kernel well below the HBM rate. B is the tokens' activations, fetched by tensor copies (box 64 columns x NT tokens)
// into the K-major 128-byte-swizzle layout the MMA reads. A group of 128 columns shares one bf16 scale per
// row, so every group accumulates into its own TMEM accumulator (a ring of them); eight warps read a finished group
// with tcgen05.ld and fold it into per-thread fp32 sums with the row's scale: the arithmetic is the
// reference's sum (nib - 8) * s * x with fp32 accumulation (reference: kernels/verify_mega.cu:18-75), only the order of
// summation differs. The asymmetric layout's zero points ride the same groups as a second MMA with A = z (exact in bf16)
// into an accumulator of their own.
//
// Weight layout ("TC layout", a library-owned copy made by tc_repack): per block of 128 rows, one record per group of 128
// columns: two 4 KB chunks [8 words][128 rows] -- word (w, r) holds columns 8w .. 8w+7 of row r with the nibbles ordered so
// that the four mask-and-fma conversions yield ADJACENT column pairs -- then the group's scales [128 rows] (and zeros).
// One 1-D bulk copy brings a record; the dequantising thread of row r reads its words without bank conflicts.
//
// Work item = (token tile, row block). Small matrices (QKV, O, down) are split along K over a CLUSTER of 2 or 4 CTAs: every
// CTA sends the sums of a quarter of the tokens to each CTA of its cluster through distributed shared memory, and each
// finishes its own tokens (sum in split order: deterministic), so the split costs one cluster barrier instead of a round
// trip through global memory and the epilogue is shared out as well. Every wait is bounded.
#pragma once
#include <cuda.h>

#include "fb_common.cuh"
#include "fb_verify.cuh"

namespace fb {

constexpr int kTcStages = 4;      // operand stages: A (dequantised group, 64 TMEM columns) and B (activations, shared memory)
constexpr int kTcThreads = 512;   // warps: 0 weights, 1 MMA issue, 2 activations, 4..7 dequantise, 8..15 sums and epilogue
constexpr int kTcRowBlock = 128;

__host__ __device__ constexpr int tc_rec_bytes(int has_zeros) { return 8192 + 256 * (has_zeros ? 2 : 1); }
__host__ __device__ constexpr size_t tc_block_bytes(int k, int has_zeros) { return (size_t)(k / 128) * tc_rec_bytes(has_zeros); }
__host__ __device__ constexpr size_t tc_matrix_bytes(int rows, int k, int has_zeros) {
  return (size_t)((rows + kTcRowBlock - 1) / kTcRowBlock) * tc_block_bytes(k, has_zeros);
}

// caller layout (word c of a row = columns 8c .. 8c+7, column 8c+m in bits [4m, 4m+4)) -> TC layout.
// grid (row blocks, layers), 256 threads.
__global__ void tc_repack(const uint32_t* q, const uint16_t* sc, const uint16_t* zr, int rows, int K, int order, int order_arg,
                          int order_rows, uint8_t* out) {
  const bool hz = zr != nullptr;
  const int rb = blockIdx.x, nrb = gridDim.x, G = K / 128, nw = K / 8, rec = tc_rec_bytes(hz);
  uint8_t* blk = out + ((size_t)blockIdx.y * nrb + rb) * tc_block_bytes(K, hz);
  __shared__ int src_row[128];
  if (threadIdx.x < 128) {
    const int j = rb * 128 + threadIdx.x;
    src_row[threadIdx.x] = j < rows ? (int)blockIdx.y * rows + perm_row(j, order, order_arg, order_rows) : -1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nw * 128; i += blockDim.x) {
    const int r = i & 127, wq = (i >> 7) & 15, g = i >> 11;      // word wq of the group's 16
    uint32_t d = 0x88888888u;                                  // padding rows: value 0
    if (src_row[r] >= 0) {
      const uint32_t s = __ldg(q + (size_t)src_row[r] * nw + g * 16 + wq);
      // column offset e goes to nibble slot [0, 4, 1, 5, 2, 6, 3, 7][e]: (w & 0x000F000F) is then columns (0, 1),
      // (w & 0x00F000F0) columns (2, 3), and the same two masks on w >> 8 columns (4, 5) and (6, 7)
      d = (s & 0xFu) | ((s >> 4 & 0xFu) << 16) | ((s >> 8 & 0xFu) << 4) | ((s >> 12 & 0xFu) << 20) | ((s >> 16 & 0xFu) << 8) |
          ((s >> 20 & 0xFu) << 24) | ((s >> 24 & 0xFu) << 12) | ((s >> 28 & 0xFu) << 28);
    }
    reinterpret_cast<uint32_t*>(blk + (size_t)g * rec)[wq * 128 + r] = d;
  }
  for (int i = threadIdx.x; i < G * 128; i += blockDim.x) {
    const int r = i & 127, g = i >> 7, row = src_row[r];
    uint16_t* meta = reinterpret_cast<uint16_t*>(blk + (size_t)g * rec + 8192);
    meta[r] = row >= 0 ? sc[(size_t)row * G + g] : 0;
    if (hz) meta[128 + r] = row >= 0 ? zr[(size_t)row * G + g] : 0;
  }
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
  CUtensorMap xmap;          // activations bf16 [rows >= M][K] as a 2-D tensor, box 64 columns x NT tokens, 128-byte swizzle
  const uint8_t* w;          // TC layout of this matrix
  int rows, K, M;
  int nsplit;                // CTAs of a cluster that share one item's K (1, 2 or 4)
  int ntok, ntile;           // tokens of one tile (a multiple of 16, <= NT; one tile unless this is a prompt) and tiles
  DevStatus* status;
  unsigned spin_limit;
  // epilogue operands
  uint16_t* h;               // RESID: bf16 [M][out_ld] in/out
  uint16_t* q;               // QKV: bf16 [M][n_head * HD]
  uint16_t *kc, *vc;         // QKV: layer base of the caches [max_seq][nkv][HD]
  uint16_t* act;             // SWIGLU: bf16 [M][out_ld]
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
// nibble pairs in bits (0..3, 16..19) / (4..7, 20..23) -> bf16 pair ((nib - 8) / 64, ...): the masked bits are the bf16
// subnormals nib * 2^-133 (16 nib * 2^-133); one bf16x2 fma with 2^127 (2^123) and -1/8
__device__ __forceinline__ uint32_t tc_cvt_lo(uint32_t w) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(w & 0x000F000Fu), "r"(0x7F007F00u), "r"(0xBE00BE00u));
  return d;
}
__device__ __forceinline__ uint32_t tc_cvt_hi(uint32_t w) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(w & 0x00F000F0u), "r"(0x7D007D00u), "r"(0xBE00BE00u));
  return d;
}
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

__device__ __forceinline__ void tc_st8(uint32_t taddr, uint32_t z) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
// cluster of the K splits: barrier over all threads of all its CTAs, and plain stores into a neighbour's shared memory
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// Shared-memory plan (bytes). The raw ring is what keeps HBM busy; a stage of activations is a group's two 64-column tiles.
template <int NT, bool HZ>
struct VtcSmem {
  static constexpr int REC = tc_rec_bytes(HZ);
  static constexpr int NS = NT > 64 ? 3 : kTcStages;                // operand stages
  static constexpr int NRAW = NT > 64 ? 6 : 10;                    // raw int4 groups in flight
  static constexpr int BSTAGE = NT * 256;                          // two [NT rows x 128 bytes] swizzled tiles
  static constexpr int B = 0;
  static constexpr int RAW = B + NS * BSTAGE;
  static constexpr int NSC = 8;                                    // ring of the groups' row scales (x 64), fp32 [128]
  static constexpr int SC = RAW + NRAW * REC;
  static constexpr int YS = SC + NSC * 512;                        // sums on their way to the epilogue, fp32 [tokens][128 rows]
  static constexpr int BAR = YS + NT * 512;
  static constexpr int TOTAL = BAR + 512 + 1024;                   // barriers + slack to align the base
  static_assert(TOTAL <= 227 * 1024, "verify GEMM shared memory");
  // tensor memory columns: group accumulators, zero-point accumulator, A stages (64 columns = 128 bf16 per row), A_z
  // (8 columns = one k16 step of the row's zero point, the same for every step of the group)
  static constexpr int NACC = (NT > 64 || (NT == 64 && HZ)) ? 2 : 4;
  static constexpr int T_ACCZ = NACC * NT, T_A = T_ACCZ + (HZ ? NT : 0), T_AZ = T_A + NS * 64;
  static_assert(T_AZ + (HZ ? NS * 8 : 0) <= 512, "tensor memory columns");
  // A scale slot of group g is rewritten for group g + NSC. The writer (dequantising group g + NSC) has seen the MMAs of group
  // g + NSC - NS retire, whose accumulator was free: the sums of group g + NSC - NS - NACC have been read. So:
  static_assert(NSC >= NS + NACC, "a scale slot must outlive its group's sums");
};

// work items of this CTA in order (token tile by token tile: the tile's activations stay in L2); every role walks the same
// sequence
struct TcWalk {
  int item, nitems, nrb, step, g0, g1, rb, tt;
  __device__ __forceinline__ TcWalk(const VtcParams& P) {
    const int ns = P.nsplit, G = P.K / 128, sp = (int)blockIdx.x % ns;
    nrb = (P.rows + kTcRowBlock - 1) / kTcRowBlock;
    nitems = nrb * P.ntile;
    item = (int)blockIdx.x / ns;
    step = (int)gridDim.x / ns;
    g0 = G * sp / ns;
    g1 = G * (sp + 1) / ns;
    set();
  }
  __device__ __forceinline__ bool valid() const { return item < nitems; }
  __device__ __forceinline__ void set() { tt = item / nrb; rb = item % nrb; }
  __device__ __forceinline__ void next() { item += step; set(); }
};

constexpr int kTcChunk = 8;       // tokens whose epilogue operands a thread loads before it uses the first

// What one chunk of the epilogue reads from global memory (issued early: it does not depend on the GEMM)
struct TcOperands {
  uint16_t h[kTcChunk];
  float2 cs[kTcChunk];
};
template <int EPI>
__device__ __forceinline__ void vtc_fetch(const VtcParams& P, int srow, int t0, int tend, TcOperands& o) {
  if (EPI == EPI_RESID) {
#pragma unroll
    for (int e = 0; e < kTcChunk; e++)
      o.h[e] = (srow < P.rows && t0 + e < tend) ? ld_cg_u16(P.h + (size_t)(t0 + e) * P.out_ld + srow) : (uint16_t)0;
  } else if (EPI == EPI_QKV) {
    const int HP = P.head_dim >> 1, head = srow / P.head_dim, i = (srow % P.head_dim) >> 1;
    const bool rot = head < P.n_head + P.nkv;
#pragma unroll
    for (int e = 0; e < kTcChunk; e++)
      o.cs[e] = (rot && t0 + e < tend) ? __ldg(P.rope + (size_t)(t0 + e) * HP + i) : make_float2(1.f, 0.f);
  }
}
// v[e] = the finished sum of (stream row srow, token t0 + e). The whole warp calls this together: lanes 2i, 2i + 1 hold the two
// rows of a RoPE or gate/up pair.
template <int EPI>
__device__ __forceinline__ void vtc_epilogue(const VtcParams& P, int srow, int t0, int tend, const float (&v)[kTcChunk],
                                             const TcOperands& o, int lane) {
  const bool live = srow < P.rows, odd = lane & 1;
  if (EPI == EPI_RESID) {
#pragma unroll
    for (int e = 0; e < kTcChunk; e++)
      if (live && t0 + e < tend) P.h[(size_t)(t0 + e) * P.out_ld + srow] = f2bf(bf2f(o.h[e]) + v[e] * P.resid);
  } else if (EPI == EPI_LOGITS) {
#pragma unroll
    for (int e = 0; e < kTcChunk; e++)
      if (live && t0 + e < tend) P.logits[(size_t)(t0 + e) * P.out_ld + srow] = v[e] / P.logits_scaling;
  } else if (EPI == EPI_SWIGLU) {
    // stream rows (2i, 2i+1) = (gate_i, up_i): the even lane takes the even tokens of the pair, the odd lane the odd ones
#pragma unroll
    for (int e = 0; e < kTcChunk; e += 2) {
      const float got = __shfl_xor_sync(0xffffffffu, odd ? v[e] : v[e + 1], 1);
      const float gg = rbf(odd ? got : v[e]), uu = rbf(odd ? v[e + 1] : got);
      const int t = t0 + e + (odd ? 1 : 0);
      if (live && t < tend) P.act[(size_t)t * P.out_ld + (srow >> 1)] = f2bf((gg / (1.0f + __expf(-gg))) * uu);
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
    for (int e = 0; e < kTcChunk; e++) {
      const float x = rbf(v[e]), y = __shfl_xor_sync(0xffffffffu, x, 1);
      const float r = odd ? x * o.cs[e].x + y * o.cs[e].y : x * o.cs[e].x - y * o.cs[e].y;
      if (live && t0 + e < tend) base[(size_t)(t0 + e) * ld] = f2bf(rot ? r : x);
    }
  }
}

template <int NT, int EPI, bool HZ>
__global__ void __launch_bounds__(kTcThreads, 1) v_gemm_tc(const __grid_constant__ VtcParams P) {
  using S = VtcSmem<NT, HZ>;
  constexpr int NRAW = S::NRAW, NS = S::NS, NACC = S::NACC, REC = S::REC, HC = NT / 2;
  extern __shared__ __align__(1024) uint8_t tsm_raw[];
  // the swizzle pattern is a function of the absolute shared-memory address: tiles must start on 1024-byte boundaries
  uint8_t* tsm = tsm_raw + ((1024u - (smem_u32(tsm_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(tsm + S::BAR);
  uint64_t *raw_full = bars, *raw_empty = bars + NRAW, *a_full = bars + 2 * NRAW, *b_full = a_full + NS, *s_empty = b_full + NS,
           *acc_full = s_empty + NS, *acc_empty = acc_full + NACC;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(acc_empty + NACC);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  float* scr = reinterpret_cast<float*>(tsm + S::SC);
  float* ys = reinterpret_cast<float*>(tsm + S::YS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < NRAW; i++) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4); }
    for (int i = 0; i < NS; i++) { mbar_init(&a_full[i], 4); mbar_init(&b_full[i], 1); mbar_init(&s_empty[i], 1); }
    for (int i = 0; i < NACC; i++) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
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
  const bool split = P.nsplit > 1;
  if (split) { cluster_arrive(); cluster_wait(); }               // the neighbours' shared memory exists from here on
  pdl_trigger();
  const int quad = warp & 3, row = quad * 32 + lane;             // warps 4..15: row of the block = TMEM lane
  const int half = (warp >> 2) & 1;                              // warps 8..15: which half of the token columns
  // splits: this CTA finishes tokens [rank * TPR, (rank + 1) * TPR) of the item
  const int TPR = NT / P.nsplit, lgT = 31 - __clz(TPR), rank = (int)blockIdx.x % P.nsplit;
  bool ok = true;
  TcOperands pre;
  int e_srow = 0, e_t0 = 0, e_tend = 0;                          // split items: the epilogue's row and first token

  if (warp == 0) {
    // ---------------- producer: the groups' records (weights do not depend on the previous kernel)
    if (lane == 0) {
      uint32_t gi = 0;
      for (TcWalk w(P); w.valid() && ok; w.next()) {
        const uint8_t* blk = P.w + (size_t)w.rb * tc_block_bytes(P.K, HZ);
        for (int g = w.g0; g < w.g1; g++, gi++) {
          const int s = gi % NRAW;
          ok = mbar_wait(&raw_empty[s], ((gi / NRAW) & 1) ^ 1, wc, W_EMPTY, 2);
          if (!ok) break;
          mbar_expect_tx(&raw_full[s], REC);
          bulk_g2s(tsm + S::RAW + s * REC, blk + (size_t)g * REC, REC, &raw_full[s]);
        }
      }
      // every copy issued must have landed before the CTA may exit: the consumers wait for all of them in a clean run;
      // after a failure, wait here (bounded)
      if (*s_abort) {
        for (int k = 0; k < NRAW && k < (int)gi; k++) {
          const uint32_t j = gi - 1 - k;
          for (unsigned i = 0; i < wc.limit; i++) {
            if (mbar_try(&raw_full[j % NRAW], (j / NRAW) & 1)) break;
            if ((i & 1023) == 1023) __nanosleep(64);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issue: one thread, eight MMAs per group, two commits
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(P.ntok >> 3) << 17) | ((128u >> 4) << 24);
      uint32_t gi = 0;
      for (TcWalk w(P); w.valid() && ok; w.next()) {
        for (int g = w.g0; g < w.g1 && ok; g++, gi++) {
          const int a = gi % NACC, s = gi % NS;
          ok = mbar_wait(&acc_empty[a], ((gi / NACC) & 1) ^ 1, wc, W_EMPTY, 3) && mbar_wait(&a_full[s], (gi / NS) & 1, wc, W_FULL, 4) &&
               mbar_wait(&b_full[s], (gi / NS) & 1, wc, W_FULL, 4);
          if (!ok) break;
          tc_fence_after();
          const uint32_t ta = tmem + S::T_A + s * 64, tz = tmem + S::T_AZ + s * 8;
          const uint32_t sb = smem_u32(tsm + S::B + s * S::BSTAGE);
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const uint64_t db = tc_desc(sb + (k >> 2) * (NT * 128) + (k & 3) * 32);
            tc_mma_ts(tmem + a * NT, ta + k * 8, db, idesc, k ? 1u : 0u);
            if (HZ) tc_mma_ts(tmem + S::T_ACCZ, tz, db, idesc, (g > w.g0 || k) ? 1u : 0u);
          }
          tc_commit(&s_empty[s]);
          tc_commit(&acc_full[a]);
        }
      }
    }
  } else if (warp == 2) {
    // ---------------- activations (the previous kernel's output): two tensor copies per group. Token rows past M are whatever
    // the buffer holds: they only feed accumulator columns that nobody reads.
    pdl_wait();
    if (lane == 0) {
      uint32_t gi = 0;
      for (TcWalk w(P); w.valid() && ok; w.next()) {
        for (int g = w.g0; g < w.g1; g++, gi++) {
          const int s = gi % NS;
          ok = mbar_wait(&s_empty[s], ((gi / NS) & 1) ^ 1, wc, W_EMPTY, 8);
          if (!ok) break;
          mbar_expect_tx(&b_full[s], S::BSTAGE);
          uint8_t* dst = tsm + S::B + s * S::BSTAGE;
          tma_load_2d(dst, &P.xmap, g * 128, w.tt * P.ntok, &b_full[s]);
          tma_load_2d(dst + NT * 128, &P.xmap, g * 128 + 64, w.tt * P.ntok, &b_full[s]);
        }
      }
      if (*s_abort) {
        for (int k = 0; k < NS && k < (int)gi; k++) {
          const uint32_t j = gi - 1 - k;
          for (unsigned i = 0; i < wc.limit; i++) {
            if (mbar_try(&b_full[j % NS], (j / NS) & 1)) break;
            if ((i & 1023) == 1023) __nanosleep(64);
          }
        }
      }
    }
  } else if (warp >= 4 && warp < 8) {
    // ---------------- dequantise: thread = row of the block = TMEM lane; 16 words -> 64 packed bf16 pairs per group
    const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16);
    uint32_t gi = 0;
    for (TcWalk w(P); w.valid() && ok; w.next()) {
      for (int g = w.g0; g < w.g1; g++, gi++) {
        const int sr = gi % NRAW, s = gi % NS;
        ok = mbar_wait(&raw_full[sr], (gi / NRAW) & 1, wc, W_FULL, 5) && mbar_wait(&s_empty[s], ((gi / NS) & 1) ^ 1, wc, W_EMPTY, 6);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint8_t* rec = tsm + S::RAW + sr * REC;
        const uint32_t raw = smem_u32(rec) + (uint32_t)row * 4;
        scr[(gi % S::NSC) * 128 + row] = bf2f(reinterpret_cast<const uint16_t*>(rec + 8192)[row]) * 64.0f;
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t v[32];
#pragma unroll
          for (int q8 = 0; q8 < 8; q8++) {
            const uint32_t wv = lds32(raw + c * 4096 + q8 * 512);
            v[4 * q8] = tc_cvt_lo(wv); v[4 * q8 + 1] = tc_cvt_hi(wv); v[4 * q8 + 2] = tc_cvt_lo(wv >> 8); v[4 * q8 + 3] = tc_cvt_hi(wv >> 8);
          }
          tc_st32(tl + S::T_A + s * 64 + c * 32, v);
        }
        if (HZ) {
          // the group's zero point of this row as one k16 step: A_z = z for every column
          const uint16_t z = reinterpret_cast<const uint16_t*>(rec + 8448)[row];
          tc_st8(tl + S::T_AZ + s * 8, (uint32_t)z | ((uint32_t)z << 16));
        }
        tc_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(&raw_empty[sr]); mbar_arrive(&a_full[s]); }
      }
    }
  } else if (warp >= 8) {
    // ---------------- sums: thread = (row of the block, half of the tokens), HC fp32 sums in registers
    const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16) + half * HC;
    uint32_t gi = 0;
    pdl_wait();
    for (TcWalk w(P); w.valid() && ok; w.next()) {
      float y[HC];
#pragma unroll
      for (int t = 0; t < HC; t++) y[t] = 0.f;
      const int tok0 = w.tt * P.ntok, tend = min(P.M, tok0 + P.ntok);
      if (split) {                                               // one item: fetch what its epilogue needs while the GEMM runs
        e_srow = w.rb * 128 + row; e_t0 = rank * TPR + half * (TPR / 2); e_tend = min(tend, e_t0 + TPR / 2);
        vtc_fetch<EPI>(P, e_srow, e_t0, e_tend, pre);
      }
      for (int g = w.g0; g < w.g1; g++, gi++) {
        const int a = gi % NACC;
        ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[a], (gi / NACC) & 1, wc, W_FULL, 10));
        if (!ok) break;
        tc_fence_after();
        const float s64 = scr[(gi % S::NSC) * 128 + row];
        constexpr int LB = HC > 32 ? 16 : HC;                    // columns per batch of loads: one wait per batch
#pragma unroll
        for (int h0 = 0; h0 < HC; h0 += LB) {
          uint32_t v[LB / 8][8];
#pragma unroll
          for (int c8 = 0; c8 < LB / 8; c8++) tc_ld8(tlane + a * NT + h0 + c8 * 8, v[c8]);
          tc_ld_wait();
#pragma unroll
          for (int c8 = 0; c8 < LB / 8; c8++)
#pragma unroll
            for (int e = 0; e < 8; e++) y[h0 + c8 * 8 + e] = fmaf(s64, __uint_as_float(v[c8][e]), y[h0 + c8 * 8 + e]);
        }
        if (HZ && g == w.g1 - 1) {                               // the item's zero-point sums: sum_g z_g * sum_k x_k
#pragma unroll
          for (int c8 = 0; c8 < HC / 8; c8++) {
            uint32_t v[8];
            tc_ld8(tlane + S::T_ACCZ + c8 * 8, v);
            tc_ld_wait();
#pragma unroll
            for (int e = 0; e < 8; e++) y[c8 * 8 + e] += __uint_as_float(v[e]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[a]);
      }
      if (!ok) break;
      if (split) {
        // token t of this half goes to the CTA that finishes it: its ys is [source rank][its tokens][128 rows]
        const uint32_t mine = smem_u32(ys) + (uint32_t)(rank * TPR * 128 + row) * 4;
#pragma unroll
        for (int t = 0; t < HC; t++) {
          const int tk = half * HC + t;
          st_cluster_f32(map_rank(mine + (uint32_t)(tk & (TPR - 1)) * 512, tk >> lgT), y[t]);
        }
      } else {
        // The sums go through shared memory ([token][row], a warp touches only its own rows and tokens) so that the per-token
        // work is a compact loop: unrolled over all tokens it is tens of KB of straight-line code that runs once per item, one
        // instruction-cache miss after the other.
        float* yw = ys + half * HC * 128 + row;
        __syncwarp();                                            // the previous item's readers are done
#pragma unroll
        for (int t = 0; t < HC; t++) yw[t * 128] = y[t];
        __syncwarp();
        const int srow = w.rb * 128 + row, th0 = tok0 + half * HC, the = min(tend, th0 + HC);
        for (int t0 = 0; th0 + t0 < the; t0 += kTcChunk) {
          vtc_fetch<EPI>(P, srow, th0 + t0, the, pre);
          float v[kTcChunk];
#pragma unroll
          for (int e = 0; e < kTcChunk; e++) v[e] = yw[(t0 + e) * 128];
          vtc_epilogue<EPI>(P, srow, th0 + t0, the, v, pre, lane);
        }
      }
    }
  }
  if (split) {
    __syncwarp();
    cluster_arrive();
    cluster_wait();                                              // every rank's sums are in
    if (warp >= 8 && __all_sync(0xffffffffu, ok && *s_abort == 0)) {
      const float* yw = ys + half * (TPR / 2) * 128 + row;
      for (int t0 = 0; e_t0 + t0 < e_tend; t0 += kTcChunk) {
        if (t0) vtc_fetch<EPI>(P, e_srow, e_t0 + t0, e_tend, pre);
        float v[kTcChunk];
#pragma unroll
        for (int e = 0; e < kTcChunk; e++) {
          v[e] = 0.f;
          if (t0 + e < TPR / 2)
            for (int r = 0; r < P.nsplit; r++) v[e] += yw[(r * TPR + t0 + e) * 128];
        }
        vtc_epilogue<EPI>(P, e_srow, e_t0 + t0, e_tend, v, pre, lane);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS));
}

}  // namespace fb
