// extern "C" boundary of libflintb200.so: context management, weight re-layout and the launches.
// No torch types, no CPU fallback: a failed CUDA call or an unsupported shape is an error code.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <new>

#include "../../include/flint_b200.h"
#include "fb_ctx.hpp"
#include "fb_decode.cuh"

using namespace fb;


namespace {

struct KernelEntry {
  int dim, ko, ffn, head_dim, rgqa, hz;
  const void* fn;          // the kernel of a single GPU; none where the attention output is not as wide as the model
  int nps;                 // K/V positions per ring stage (the box of the cache tensors)
  int copy, ring;          // bytes of a bulk copy of the matrices that read the model width, and of the whole ring
};

template <int KD, int KO, int KF, int HD, int R, bool HZ>
const void* single_gpu_kernel() {
  if constexpr (KO == KD) return (const void*)decode_mega2<KD, KO, KF, HD, R, HZ, false>;
  else return nullptr;
}
template <int KD, int KO, int KF, int HD, int R, bool HZ>
KernelEntry kernel_entry() {
  constexpr int stage = DecodePlan<KD, KO, KF>::STAGE;
  using C = TCfg<KD, stage>;
  return {KD, KO, KF, HD, R, HZ, single_gpu_kernel<KD, KO, KF, HD, R, HZ>(), AttnCfg<HD, stage>::NPS, C::CPS * C::chunk(HZ), kStages * stage};
}
#define FB_DECODE_ENTRY(KD, KO, KF, HD, R) kernel_entry<KD, KO, KF, HD, R, false>(), kernel_entry<KD, KO, KF, HD, R, true>()

const KernelEntry kDecodeKernels[] = {
#include "fb_decode_shapes.h"
};
constexpr int kNumDecodeKernels = sizeof(kDecodeKernels) / sizeof(kDecodeKernels[0]);

const void* kernel_of(int id, int tp_size) { return tp_size > 1 ? decode_tp_kernel(id) : kDecodeKernels[id].fn; }

int find_kernel(const fb_model_desc& d, int ko) {
  if (d.n_kv_head <= 0 || d.n_head % d.n_kv_head) return -1;
  for (int i = 0; i < kNumDecodeKernels; i++) {
    const KernelEntry& e = kDecodeKernels[i];
    if (e.dim == d.dim && e.ko == ko && e.ffn == d.ffn && e.head_dim == d.head_dim &&
        e.rgqa == d.n_head / d.n_kv_head && e.hz == (d.has_zeros ? 1 : 0))
      return i;
  }
  return -1;
}


int chunks_for(const fb_ctx* c, int T) {
  if (c->force_chunks > 0) return c->force_chunks < c->maxchunks ? c->force_chunks : c->maxchunks;
  // Two ring stages of positions per chunk (8 or 4 units of 16 positions for the 14 warps), until the CTAs run out: fewer, longer chunks
  // add passes of the warps, more of them a round trip of the merge and its poll traffic. Microseconds a token at 1 / 2 / 4 / 8 / 18
  // chunks: heads of 80, 200 cached positions 1038 / 1040 / 1048 / 1063 / 1111, 603 positions 1129 / 1102 / 1061 / 1067 / 1111; heads of
  // 128, 200 positions 1756 / 1741 / 1719 / 1733 / 1787, 1777 positions 2733 / 2235 / 1980 / 1849 / 1830.
  const int span = 2 * kDecodeKernels[c->kernel_id].nps, n = (T + span - 1) / span;
  return n < c->maxchunks ? n : c->maxchunks;
}

// Bulk copies a CTA keeps in flight while the layers run. A layer that brings each SM at most 1.8 rings of weights and K/V spends far
// longer on its hand-overs than on the copies, and the tagged words then wait behind less bulk traffic; more bytes, or copies of less than 20 KB (two of them
// are then too little to stream with), need the full rate. Measured are copies of 21.1 KB (width 2560) and 16.9 KB (2048; 4096 in layers of more than
// 1.8 rings); the line lies between the two, and widths of 512 and 640 make no difference. Microseconds a token at 1 / 2 / 3 / 4 copies (cached positions, rings a layer):
//   3B-class   20, 1.6: 739 / 730 / 734 / 733   200, 1.6: 804 / 794 / 799 / 798   2000, 1.8: 830 / 819 / 820 / 819   4000, 2.0: 900 / 883 / 877 / 875
//              8000, 2.3: 960 / 953 / 949 / 946   32700, 4.7: 1589 / 1473 / 1438 / 1431
//   40 heads   600, 1.7: 794 / 788 / 794 / 796   1500, 1.75: 810 / 802 / 809 / 809   3900, 1.9: 876 / 864 / 859 / 860
//   1B-class (copies of 17 KB)   22, 1.2: 289 / 284 / 281 / 280   3900, 1.6: 348 / 343 / 341 / 340        8B-class, 200: 1409 / 1326 / 1292 / 1287
// The LM head has no hand-over to disturb: always 4.
int fly_for(const fb_ctx* c, int T) {
  if (c->max_fly) return c->max_fly;
  const fb_model_desc& d = c->d;
  const KernelEntry& e = kDecodeKernels[c->kernel_id];
  const int HD = d.head_dim, hz = d.has_zeros ? 1 : 0;
  const int64_t bytes = (int64_t)(d.n_head + 2 * d.n_kv_head) * HD * rec_bytes_of(d.dim, hz) + (int64_t)d.dim * rec_bytes_of(c->ko, hz) +
                        (int64_t)2 * d.ffn * rec_bytes_of(d.dim, hz) + (int64_t)d.dim * rec_bytes_of(d.ffn, hz) +
                        (int64_t)T * d.n_kv_head * HD * 4;
  return bytes * 10 <= (int64_t)18 * e.ring * c->sm_count && e.copy >= 20000 ? 2 : 4;
}

// every K the stand-alone entry points (re-layout, dequantise, GEMV) are built for
#ifndef FB_EXTRA_K
#define FB_EXTRA_K(X)                             // widths of the build-time extra shapes that this list lacks
#endif
#define FB_FOR_EACH_K(X) X(256) X(384) X(512) X(640) X(768) X(1024) X(1280) X(1408) X(1536) X(1792) X(2048) X(2560) X(3584) X(4096) X(7168) X(8192) X(14336) FB_EXTRA_K(X)

template <int K>
int launch_gemv_k(bool hz, const GemvParams& p, int grid, cudaStream_t st) {
  cudaError_t e;
  if (hz) {
    e = cudaFuncSetAttribute(gemv_stream<K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    gemv_stream<K, true><<<grid, kThreads, kSmemBytes, st>>>(p);
  } else {
    e = cudaFuncSetAttribute(gemv_stream<K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    gemv_stream<K, false><<<grid, kThreads, kSmemBytes, st>>>(p);
  }
  return (int)cudaGetLastError();
}

bool supported_k(int k) {
  switch (k) {
#define X(K_) case K_:
    FB_FOR_EACH_K(X)
#undef X
    return true;
  }
  return false;
}

// caller layout -> tiles, for `layers` stacked matrices of `rows` rows each
cudaError_t launch_repack(const void* q, const void* s, const void* z, int layers, int rows, int k, int order, int arg,
                          int orows, uint8_t* out, cudaStream_t st) {
  const int tiles = (rows + tile_rt(k) - 1) / tile_rt(k);
  switch (k) {
#define X(K_)                                                                                                          \
  case K_:                                                                                                             \
    repack_tiles<K_><<<dim3(tiles, layers), 128, 0, st>>>((const uint32_t*)q, (const uint16_t*)s, (const uint16_t*)z, rows, \
                                                          order, arg, orows, out);                                     \
    break;
    FB_FOR_EACH_K(X)
#undef X
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// The caches as 4-D tensors for the decode kernel's producer: (column, column block of 64, kv head, n_layer * max_seq rows), box =
// one block x one head x one ring stage of positions; 128-byte blocks are swizzled (AttnCfg). Head dimensions that are no
// multiple of 64 are one unswizzled block. maps: K, V.
cudaError_t make_kv_maps(const fb_ctx* c, void* kc, void* vc, int max_seq, CUtensorMap (&maps)[2]) {
  EncodeFn fn = tensor_map_encoder();
  if (!fn) return cudaErrorNotSupported;
  const fb_model_desc& d = c->d;
  const int HD = d.head_dim, bcols = HD % 64 == 0 ? 64 : HD;
  const cuuint64_t row = (cuuint64_t)d.n_kv_head * HD * 2;
  const cuuint64_t dims[4] = {(cuuint64_t)bcols, (cuuint64_t)(HD / bcols), (cuuint64_t)d.n_kv_head, (cuuint64_t)d.n_layer * (cuuint64_t)max_seq};
  const cuuint64_t strides[3] = {(cuuint64_t)bcols * 2, (cuuint64_t)HD * 2, row};
  const cuuint32_t box[4] = {(cuuint32_t)bcols, 1u, 1u, (cuuint32_t)kDecodeKernels[c->kernel_id].nps};
  const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  void* bases[2] = {kc, vc};
  for (int i = 0; i < 2; i++)
    if (fn(&maps[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, bases[i], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           bcols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
  return cudaSuccess;
}

}  // namespace

extern "C" {

int fb_query(int device, fb_caps* out) {
  if (!out) return FB_ERR_ARG;
  cudaDeviceProp p;
  if (cudaGetDeviceProperties(&p, device) != cudaSuccess) return FB_ERR_CUDA;
  memset(out, 0, sizeof(*out));
  out->device = device;
  out->sm_count = p.multiProcessorCount;
  out->cc_major = p.major;
  out->cc_minor = p.minor;
  out->smem_per_block_optin = (int32_t)p.sharedMemPerBlockOptin;
  out->l2_bytes = p.l2CacheSize;
  out->cooperative_launch = p.cooperativeLaunch;
  out->total_mem_bytes = (int64_t)p.totalGlobalMem;
  cudaFuncAttributes fa;
  for (int i = 0; i < kNumDecodeKernels; i++)      /* registers of the 3B-class instantiation, the one the benchmark runs */
    if (kDecodeKernels[i].dim == 2560 && kDecodeKernels[i].head_dim == 80 && kDecodeKernels[i].ko == 2560 && !kDecodeKernels[i].hz) {
      if (cudaFuncGetAttributes(&fa, kDecodeKernels[i].fn) == cudaSuccess) out->regs_decode_kernel = fa.numRegs;
      break;
    }
  return FB_OK;
}

int fb_ctx_create(const fb_model_desc* desc, int device, fb_ctx** out) {
  return fb_ctx_create_tp(desc, device, 0, 1, 0, out);
}

int fb_ctx_create_tp(const fb_model_desc* desc, int device, int32_t tp_rank, int32_t tp_size, int32_t vocab_base,
                     fb_ctx** out) {
  if (!desc || !out) return FB_ERR_ARG;
  *out = nullptr;
  const fb_model_desc& d = *desc;
  if (tp_size < 1 || tp_size > 8 || tp_rank < 0 || tp_rank >= tp_size) return FB_ERR_ARG;
  if (d.n_layer <= 0 || d.vocab <= 0 || d.dim % 128 || d.ffn % 128 || d.n_head <= 0 || d.head_dim <= 0) return FB_ERR_SHAPE;
  if (tp_size == 1 && d.n_head * d.head_dim != d.dim) return FB_ERR_SHAPE;
  const OWindow win = o_window(d.n_head * d.head_dim, tp_rank);
  const int ko = win.ko, ao_off = win.off;
  if (tp_size == 1 && ao_off) return FB_ERR_SHAPE;
  const int kid = find_kernel(d, ko);
  if (kid < 0) return FB_ERR_SHAPE;
  DeviceGuard g(device);
  if (!g.ok) return FB_ERR_CUDA;
  cudaDeviceProp p;
  if (cudaGetDeviceProperties(&p, device) != cudaSuccess) return FB_ERR_CUDA;
  if (p.major < 10 || !p.cooperativeLaunch || (int)p.sharedMemPerBlockOptin < kSmemBytes) return FB_ERR_SHAPE;
  fb_ctx* c = new (std::nothrow) fb_ctx();
  if (!c) return FB_ERR_ARG;
  memset(c, 0, sizeof(*c));
  c->d = d;
  c->device = device;
  c->sm_count = p.multiProcessorCount;
  c->kernel_id = kid;
  c->rgqa = d.n_head / d.n_kv_head;
  c->spin_limit = 4000000u;
  c->tp_size = tp_size; c->tp_rank = tp_rank; c->vocab_base = vocab_base; c->ko = ko; c->ao_off = ao_off;
  c->tag_base = 8;
  c->maxchunks = c->sm_count / d.n_kv_head;
  if (c->maxchunks < 1) c->maxchunks = 1;
  if (c->maxchunks > 64) c->maxchunks = 64;
  {  // every chunk CTA merges its share of the attention output with one tagged load per thread:
     // chunks * (R + ceil(R * HD/2 / chunks)) loads must fit the consumer threads
    const int pairs = c->rgqa * d.head_dim / 2;
    const int cap = (kConsumerThreads - pairs) / (c->rgqa + 1);
    if (c->maxchunks > cap) c->maxchunks = cap;
    if (c->maxchunks < 1) c->maxchunks = 1;
  }
  cudaError_t e = cudaSuccess;
  auto A = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
  A(dmalloc(&c->invf, sizeof(float) * (d.head_dim / 2)));
  A(dmalloc(&c->status, sizeof(DevStatus)));
  {
    const size_t inbox_words = (size_t)2 * tp_size * d.dim + 2 * (size_t)tp_size + 16;
    A(dmalloc(&c->inbox, inbox_words * 8));
    if (e == cudaSuccess) A(cudaMemset(c->inbox, 0, inbox_words * 8));
    c->peer_inbox[tp_rank] = c->inbox;
  }
  const size_t hp = d.head_dim / 2;
  const size_t wpc = (size_t)c->rgqa * d.head_dim + 2 * c->rgqa;
  const size_t ll_words[8] = {(size_t)d.dim / 2, d.n_head * hp, d.n_kv_head * hp, d.n_kv_head * hp, (size_t)ko / 2,
                              (size_t)d.ffn / 2, 2 * (size_t)c->sm_count, (size_t)d.n_kv_head * c->maxchunks * wpc};
  uint64_t** ll_ptrs[8] = {&c->h_ll, &c->q_ll, &c->k_ll, &c->v_ll, &c->ao_ll, &c->act_ll, &c->cand_ll, &c->part_ll};
  for (int i = 0; i < 8; i++) {
    A(dmalloc(ll_ptrs[i], 8 * ll_words[i] + 16));
    if (e == cudaSuccess) A(cudaMemset(*ll_ptrs[i], 0, 8 * ll_words[i] + 16));
  }
  if (e == cudaSuccess) e = pass_alloc(c);
  if (c->sm_count > 256) e = cudaErrorInvalidValue;
  {  // rows of the residual stream one CTA owns (whole tiles of the O and the down matrix)
    const int uo = tile_rt(ko) > tile_rt(d.ffn) ? tile_rt(ko) : tile_rt(d.ffn);
    const int units = (d.dim + uo - 1) / uo;
    if ((units + c->sm_count - 1) / c->sm_count * uo > kMaxOwnRows || (2 * d.ffn) % 4) e = cudaErrorInvalidValue;
  }
  if (e == cudaSuccess) {
    float invf[128];
    for (int i = 0; i < d.head_dim / 2; i++) invf[i] = (float)pow((double)d.rope_base, -2.0 * i / d.head_dim);
    A(cudaMemcpy(c->invf, invf, sizeof(float) * (d.head_dim / 2), cudaMemcpyHostToDevice));
    A(cudaMemset(c->status, 0, sizeof(DevStatus)));
    A(cudaFuncSetAttribute(kernel_of(kid, tp_size), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
  }
  if (e != cudaSuccess) {
    fb_ctx_destroy(c);
    return FB_ERR_CUDA;
  }
  *out = c;
  return FB_OK;
}

int fb_ctx_destroy(fb_ctx* c) {
  if (!c) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  for (int p = 0; p < 8; p++)
    if (c->peers_open[p] && c->peer_inbox[p]) cudaIpcCloseMemHandle(c->peer_inbox[p]);
  void* ptrs[] = {c->w_qkv, c->w_o, c->w_gu, c->w_d, c->w_lm, c->invf,
                  c->status, c->h_ll, c->q_ll, c->k_ll, c->v_ll, c->ao_ll, c->act_ll, c->cand_ll,
                  c->part_ll, c->inbox};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  pass_free(c);
  delete c;
  return FB_OK;
}

int fb_set_option(fb_ctx* c, int32_t what, int64_t value) {
  if (!c) return FB_ERR_ARG;
  if (what == 0) { c->spin_limit = (unsigned)value; return FB_OK; }       // spin limit of every device-side wait
  if (what == 1) { c->force_chunks = (int)value; return FB_OK; }          // attention chunks per kv head (0 = auto)
  if (what == 5) return FB_OK;                                             // 5, 7, 8: accepted, without effect: one implementation
  if (what == 8) return value < 0 || value > 2 ? FB_ERR_ARG : FB_OK;
  if (what == 7) return value < 0 || value > 4 ? FB_ERR_ARG : FB_OK;
  if (what == 4) { if (value < 1 || value > kStages / 2) return FB_ERR_ARG; c->max_fly = (int)value; return FB_OK; }
  if (what == 2) { c->prof = (long long*)(uintptr_t)value; return FB_OK; } // device int64[sm_count * n_layer * 16] phase stamps (ns), 0 = off
  return FB_ERR_ARG;
}

int fb_last_status(fb_ctx* c, fb_status* out) {
  if (!c || !out) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  DevStatus s;
  cudaError_t e = cudaMemcpy(&s, c->status, sizeof(s), cudaMemcpyDeviceToHost);
  memset(out, 0, sizeof(*out));
  out->cuda_error = c->last_cuda_error;
  if (e != cudaSuccess) {
    out->code = FB_ERR_CUDA;
    out->cuda_error = (int)e;
    return FB_ERR_CUDA;
  }
  out->code = s.code;
  out->where = s.where;
  out->layer = s.layer;
  out->block = s.block;
  out->expected = s.expected;
  out->seen = s.seen;
  if (s.code != 0) {   // a launch gave up: clear the report so that the next launch starts clean
    cudaMemset(c->status, 0, sizeof(DevStatus));
  }
  return FB_OK;
}

size_t fb_stream_bytes(int32_t rows, int32_t k, int32_t has_zeros) {
  if (rows < 0 || !supported_k(k)) return 0;
  const int u = stream_row_unit(k);
  return (size_t)((rows + u - 1) / u * u) * rec_bytes_of(k, has_zeros);
}

int fb_repack(const void* d_q, const void* d_s, const void* d_z, int32_t rows, int32_t k, int32_t order, int32_t order_arg,
              int32_t order_rows, void* d_out, void* stream) {
  if (!d_q || !d_s || !d_out || rows <= 0 || k <= 0 || k % 128 || order < 0 || order > 2) return FB_ERR_ARG;
  if (order == 1 && (order_arg <= 0 || order_arg % 2 || order_rows % order_arg || order_rows > rows)) return FB_ERR_ARG;
  if (order == 2 && (order_arg * 2 != rows)) return FB_ERR_ARG;
  if (!supported_k(k)) return FB_ERR_SHAPE;
  const int full = rows / tile_rt(k) * tile_rt(k);
  cudaStream_t st = (cudaStream_t)stream;
  if (full && launch_repack(d_q, d_s, d_z, 1, full, k, order, order_arg, order_rows, (uint8_t*)d_out, st) != cudaSuccess) return FB_ERR_CUDA;
  if (rows > full)
    repack_plain<><<<rows - full, 128, 0, st>>>((const uint32_t*)d_q, (const uint16_t*)d_s, (const uint16_t*)d_z, full, k, order, order_arg, order_rows,
                                              (uint8_t*)d_out + (size_t)full * rec_bytes_of(k, d_z != nullptr));
  return cudaGetLastError() == cudaSuccess ? FB_OK : FB_ERR_CUDA;
}

int fb_dequant(const void* d_in, int32_t rows, int32_t k, int32_t has_zeros, int32_t order, int32_t order_arg,
               int32_t order_rows, float* d_out, void* stream) {
  if (!d_in || !d_out || rows <= 0 || k <= 0 || k % 128 || order < 0 || order > 2) return FB_ERR_ARG;
  const int full = rows / tile_rt(k) * tile_rt(k);
  cudaStream_t st = (cudaStream_t)stream;
  switch (k) {
#define X(K_)                                                                                                         \
  case K_:                                                                                                            \
    if (full) dequant_tiles<K_><<<full, 256, 0, st>>>((const uint8_t*)d_in, full, has_zeros, order, order_arg, \
                                                              order_rows, d_out);                                     \
    break;
    FB_FOR_EACH_K(X)
#undef X
    default: return FB_ERR_SHAPE;
  }
  if (rows > full)
    dequant_plain<><<<rows - full, 256, 0, st>>>((const uint8_t*)d_in + (size_t)full * rec_bytes_of(k, has_zeros), full, k, has_zeros, order, order_arg,
                                               order_rows, d_out);
  return cudaGetLastError() == cudaSuccess ? FB_OK : FB_ERR_CUDA;
}

int fb_gemv(const void* d_in, int32_t rows, int32_t k, int32_t has_zeros, int32_t order, int32_t order_arg,
            int32_t order_rows, const void* d_x, float* d_y, void* d_status, void* stream) {
  if (!d_in || !d_x || !d_y || !d_status || rows <= 0) return FB_ERR_ARG;
  if (((uintptr_t)d_in & 15) || ((uintptr_t)d_x & 15)) return FB_ERR_ARG;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return FB_ERR_CUDA;
  GemvParams p{(const uint8_t*)d_in, (const uint16_t*)d_x, d_y, (DevStatus*)d_status, rows, order, order_arg, order_rows,
               4000000u};
  const bool hz = has_zeros != 0;
  cudaStream_t st = (cudaStream_t)stream;
  int e;
  switch (k) {
#define X(K_) case K_: e = launch_gemv_k<K_>(hz, p, sms, st); break;
    FB_FOR_EACH_K(X)
#undef X
    default: return FB_ERR_SHAPE;
  }
  return e == 0 ? FB_OK : FB_ERR_CUDA;
}

// ---- GEMV for callers that must not allocate ----------------------------------------------------------------------
// The streaming-layout copy of the matrix is the scratch of this path. Here it lives in one fixed array inside the
// library image instead of a buffer from cudaMalloc: every GPU that loads the library carries these 9 MiB until the
// process exits. `g_static_scratch` in HOST code is only a stand-in for the symbol, not a device address: the address
// a kernel can use comes from cudaGetSymbolAddress, once per device, with that device current.
constexpr size_t kStaticScratchBytes = (size_t)9 << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
static void* g_static_scratch_addr[64];      // per device ordinal, filled by the first call on that device

int fb_gemv_static(const void* d_q, const void* d_s, const void* d_z, int32_t rows, int32_t k, const void* d_x, float* d_y,
                   void* d_status, void* stream) {
  if (!d_q || !d_s || !d_x || !d_y || !d_status || rows <= 0 || k <= 0 || k % 128) return FB_ERR_ARG;
  const int hz = d_z != nullptr;
  if (!supported_k(k)) return FB_ERR_SHAPE;
  const size_t need = fb_stream_bytes(rows, k, hz);
  if (need > kStaticScratchBytes) return FB_ERR_RANGE;       /* matrix larger than the built-in scratch: use fb_gemv */
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FB_ERR_CUDA;
  if (!g_static_scratch_addr[dev]) {                          /* set-up, once per device, with that device current */
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || !p) return FB_ERR_CUDA;
    g_static_scratch_addr[dev] = p;
  }
  void* scratch = g_static_scratch_addr[dev];
  cudaStream_t st = (cudaStream_t)stream;
  /* the caller's status words must start at zero; the scratch itself needs no clearing: every byte of the rows*record
     range that the GEMV reads is rewritten by the re-layout below (padding included) */
  if (cudaMemsetAsync(d_status, 0, 32, st) != cudaSuccess) return FB_ERR_CUDA;
  int rc = fb_repack(d_q, d_s, d_z, rows, k, 0, 0, 0, scratch, stream);
  if (rc != FB_OK) return rc;
  return fb_gemv(scratch, rows, k, hz, 0, 0, 0, d_x, d_y, d_status, stream);
}

int fb_bind_weights(fb_ctx* c, const fb_weight_ptrs* w, void* stream) {
  if (!c || !w) return FB_ERR_ARG;
  const fb_model_desc& d = c->d;
  const bool hz = d.has_zeros != 0;
  const void* need[] = {w->qkv_q, w->qkv_s, w->o_q, w->o_s, w->gu_q, w->gu_s, w->d_q, w->d_s, w->lm_q, w->lm_s,
                        w->n1, w->n2, w->nf};   /* embed may be NULL when every step supplies its own residual */
  for (const void* p : need)
    if (!p) return FB_ERR_ARG;
  if (hz && (!w->qkv_z || !w->o_z || !w->gu_z || !w->d_z || !w->lm_z)) return FB_ERR_ARG;
  if (((uintptr_t)w->n1 & 15) || ((uintptr_t)w->n2 & 15) || ((uintptr_t)w->nf & 15)) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int L = d.n_layer, D = d.dim, FF = d.ffn, HD = d.head_dim;
  const int QKV = (d.n_head + 2 * d.n_kv_head) * HD;
  struct M { uint8_t** dst; const void *q, *s, *z; int layers, rows, k, order, arg, orows; };
  M ms[] = {
      {&c->w_qkv, w->qkv_q, w->qkv_s, w->qkv_z, L, QKV, D, 1, HD, (d.n_head + d.n_kv_head) * HD},
      {&c->w_o, w->o_q, w->o_s, w->o_z, L, D, c->ko, 0, 0, 0},
      {&c->w_gu, w->gu_q, w->gu_s, w->gu_z, L, 2 * FF, D, 2, FF, 0},
      {&c->w_d, w->d_q, w->d_s, w->d_z, L, D, FF, 0, 0, 0},
      {&c->w_lm, w->lm_q, w->lm_s, w->lm_z, 1, d.vocab, D, 0, 0, 0},
  };
  for (M& m : ms) {
    const size_t bytes = (size_t)m.layers * pad_rows(m.rows, m.k) * rec_bytes_of(m.k, hz);
    if (*m.dst) { cudaFree(*m.dst); *m.dst = nullptr; }
    FB_CUDA(c, dmalloc(m.dst, bytes + 16));
    FB_CUDA(c, launch_repack(m.q, m.s, hz ? m.z : nullptr, m.layers, m.rows, m.k, m.order, m.arg, m.orows, *m.dst, st));
    FB_CUDA(c, pass_bind_matrix(c, (int)(&m - ms), m.q, m.s, hz ? m.z : nullptr, m.layers, m.rows, m.k, m.order, m.arg, m.orows, st));
  }
  c->n1 = w->n1; c->n2 = w->n2; c->nf = w->nf; c->embed = w->embed;
  c->weights_bound = true;
  return FB_OK;
}

int fb_bind_kv(fb_ctx* c, void* d_k, void* d_v, int32_t max_seq) {
  if (!c || !d_k || !d_v || max_seq <= 0) return FB_ERR_ARG;
  if (((uintptr_t)d_k & 15) || ((uintptr_t)d_v & 15)) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  CUtensorMap maps[2];
  FB_CUDA(c, make_kv_maps(c, d_k, d_v, max_seq, maps));        // refused: the context keeps the cache that it had, or none
  c->kc = d_k; c->vc = d_v; c->max_seq = max_seq; c->kmap = maps[0]; c->vmap = maps[1];
  return FB_OK;
}

int fb_decode(fb_ctx* c, int32_t token, const int32_t* d_token, void* d_h, int32_t pos, float* d_logits, int32_t* d_next,
              void* stream) {
  if (!c) return FB_ERR_ARG;
  if (!c->weights_bound || !c->kc) return FB_ERR_STATE;
  const fb_model_desc& d = c->d;
  if (pos < 0 || pos >= c->max_seq) return FB_ERR_RANGE;
  if (!d_token && !d_h && (token < 0 || (c->tp_size == 1 && token >= d.vocab))) return FB_ERR_RANGE;
  if (!d_h && !c->embed) return FB_ERR_STATE;
  if (d_h && ((uintptr_t)d_h & 1)) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  Decode2Params Q;
  memset(&Q, 0, sizeof(Q));
  Q.w_qkv = c->w_qkv; Q.w_o = c->w_o; Q.w_gu = c->w_gu; Q.w_d = c->w_d; Q.w_lm = c->w_lm;
  Q.n1 = (const uint16_t*)c->n1; Q.n2 = (const uint16_t*)c->n2; Q.nf = (const uint16_t*)c->nf;
  Q.embed = (const uint16_t*)c->embed; Q.invf = c->invf;
  Q.kc = (uint16_t*)c->kc; Q.vc = (uint16_t*)c->vc;
  Q.kmap = c->kmap; Q.vmap = c->vmap;
  Q.h_ll = c->h_ll; Q.q_ll = c->q_ll; Q.k_ll = c->k_ll; Q.v_ll = c->v_ll; Q.ao_ll = c->ao_ll; Q.act_ll = c->act_ll;
  Q.cand_ll = c->cand_ll; Q.part_ll = c->part_ll; Q.status = c->status;
  Q.d_token = d_token; Q.d_h = (uint16_t*)d_h; Q.d_logits = d_logits; Q.d_next = d_next;
  Q.token = token; Q.pos = pos; Q.max_seq = c->max_seq;
  Q.n_layer = d.n_layer; Q.dim = d.dim; Q.n_head = d.n_head; Q.n_kv = d.n_kv_head; Q.ffn = d.ffn; Q.vocab = d.vocab;
  Q.nchunks = chunks_for(c, pos + 1);
  Q.maxchunks = c->maxchunks;
  const unsigned span = (unsigned)(d.n_layer + 1) * 8u;
  if (c->tag_base > 0xffffffffu - 2 * span) c->tag_base = 8;      // tags never reach 0 (the value of fresh buffers)
  Q.tag_base = c->tag_base; Q.spin_limit = c->spin_limit;
  Q.eps = d.rms_eps; Q.attn_scale = d.attn_scale * 1.4426950408889634f; Q.resid = d.resid_mult; Q.emb_mult = d.emb_mult;
  Q.logits_scaling = d.logits_scaling; Q.prof = c->prof; Q.max_fly = (unsigned)fly_for(c, pos + 1); Q.lm_fly = c->max_fly ? Q.max_fly : 4u;
  Q.tp_size = c->tp_size; Q.tp_rank = c->tp_rank; Q.vocab_base = c->vocab_base; Q.inbox = c->inbox; Q.ao_off = c->ao_off;
  for (int p = 0; p < c->tp_size; p++) {
    if (!c->peer_inbox[p]) return FB_ERR_STATE;       /* fb_tp_connect has not been called */
    Q.peer_inbox[p] = c->peer_inbox[p];
  }
  void* args2[] = {&Q};
  FB_CUDA(c, cudaLaunchCooperativeKernel(kernel_of(c->kernel_id, c->tp_size), dim3(c->sm_count), dim3(kThreads), args2, (size_t)kSmemBytes,
                                         (cudaStream_t)stream));
  c->tag_base += span;
  return FB_OK;
}


int fb_tp_export(fb_ctx* c, void* handle_out64) {
  if (!c || !handle_out64) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  cudaIpcMemHandle_t h;
  FB_CUDA(c, cudaIpcGetMemHandle(&h, c->inbox));
  static_assert(sizeof(h) == 64, "IPC handle size");
  memcpy(handle_out64, &h, 64);
  return FB_OK;
}

int fb_tp_connect(fb_ctx* c, const void* handles, int32_t n) {
  if (!c || !handles || n != c->tp_size) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  for (int p = 0; p < n; p++) {
    if (p == c->tp_rank) continue;
    cudaIpcMemHandle_t h;
    memcpy(&h, (const char*)handles + 64 * p, 64);
    void* ptr = nullptr;
    FB_CUDA(c, cudaIpcOpenMemHandle(&ptr, h, cudaIpcMemLazyEnablePeerAccess));
    c->peer_inbox[p] = (uint64_t*)ptr;
    c->peers_open[p] = true;
  }
  return FB_OK;
}

int fb_tp_connect_local(fb_ctx* c, fb_ctx* const* ranks, int32_t n) {
  if (!c || !ranks || n != c->tp_size) return FB_ERR_ARG;
  DeviceGuard g(c->device);
  for (int p = 0; p < n; p++) {
    if (p == c->tp_rank) continue;
    fb_ctx* o = ranks[p];
    if (!o || o == c || o->tp_size != n || o->tp_rank != p || o->d.dim != c->d.dim) return FB_ERR_ARG;
    if (o->device != c->device) {
      int can = 0;
      FB_CUDA(c, cudaDeviceCanAccessPeer(&can, c->device, o->device));
      if (!can) return FB_ERR_STATE;
      cudaError_t e = cudaDeviceEnablePeerAccess(o->device, 0);
      if (e == cudaErrorPeerAccessAlreadyEnabled) cudaGetLastError();
      else if (e != cudaSuccess) return cuda_fail(c, e);
    }
    c->peer_inbox[p] = o->inbox;
    c->peers_open[p] = false;                          /* not an IPC mapping: the owner frees it */
  }
  return FB_OK;
}

int fb_kv_move(fb_ctx* c, const int32_t* src, const int32_t* dst, int32_t n, void* stream) {
  if (!c || !c->kc || (n > 0 && (!src || !dst))) return FB_ERR_ARG;
  const fb_model_desc& d = c->d;
  DeviceGuard g(c->device);
  const size_t row = (size_t)d.n_kv_head * d.head_dim * 2, layer = (size_t)c->max_seq * row;
  for (int i = 0; i < n; i++) {     /* sequential, like the reference loop (reference: spec_tree.py:126-128) */
    if (src[i] < 0 || dst[i] < 0 || src[i] >= c->max_seq || dst[i] >= c->max_seq) return FB_ERR_RANGE;
    if (src[i] == dst[i]) continue;
    for (void* base : {c->kc, c->vc})
      FB_CUDA(c, cudaMemcpy2DAsync((char*)base + dst[i] * row, layer, (char*)base + src[i] * row, layer, row, d.n_layer,
                                   cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
  }
  return FB_OK;
}

}  // extern "C"
