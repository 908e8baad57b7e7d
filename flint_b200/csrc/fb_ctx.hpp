// The context object behind the C ABI's opaque `fb_ctx`, shared by the translation units of the library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/flint_b200.h"

namespace fb { struct DevStatus; }
using fb::DevStatus;

struct fb_ctx {
  fb_model_desc d;
  int device, sm_count, kernel_id, rgqa;
  uint8_t *w_qkv, *w_o, *w_gu, *w_d, *w_lm;
  const void *n1, *n2, *nf, *embed;
  float* invf;
  DevStatus* status;
  void *kc, *vc;
  int max_seq, maxchunks;
  unsigned spin_limit;
  bool weights_bound;
  int last_cuda_error;
  int force_chunks;
  long long* prof;
  uint64_t *h_ll, *q_ll, *k_ll, *v_ll, *ao_ll, *act_ll, *cand_ll, *part_ll;   // tagged vectors of the data-flow kernel
  unsigned tag_base;
  int tp_size, tp_rank, vocab_base, ko, ao_off;                     // tensor parallelism (1 GPU: tp_size 1, ko = dim)
  uint64_t* inbox;                                                  // [2][tp][dim] partial words + [tp][2] candidates
  uint64_t* peer_inbox[8];
  bool peers_open[8];
  uint16_t *vh, *vxn, *vq, *vao, *vact;                             // verify / prompt activations, kPromptRows token rows each
  CUtensorMap m_xn[5], m_ao[5], m_act[5];                           // vxn, vao, vact as tensors: boxes of 16, 32, 64, 128, 192 token rows
  uint8_t *t_qkv, *t_o, *t_gu, *t_d, *t_lm;                          // verify: the matrices in the tensor-core (TC) layout
  float *vfx, *vfao, *vfa, *vfa_inv;                                // per token: inverse powers of two of xn / attention output, that of the SwiGLU output and its inverse
  unsigned* vamax;                                                  // per token: bound on the attention output (float bits)
  unsigned* gu_norms;                                               // [n_layer][2] largest squared row norms of gate and up (float bits)
  void* vrope;                                                      // verify: (cos, sin) per (token, rotation pair)
  int max_fly;                                                      // max_fly 0: chosen by the bytes of a layer (fly_for)
  CUtensorMap kmap, vmap;                                           // the caches as tensors (make_kv_maps)
};

inline int cuda_fail(fb_ctx* c, cudaError_t e) {
  if (c) c->last_cuda_error = (int)e;
  return FB_ERR_CUDA;
}

#define FB_CUDA(c, call)                                   \
  do {                                                     \
    cudaError_t e__ = (call);                              \
    if (e__ != cudaSuccess) return cuda_fail((c), e__);    \
  } while (0)

template <class T>
inline cudaError_t dmalloc(T** p, size_t n) { return cudaMalloc(reinterpret_cast<void**>(p), n); }

struct DeviceGuard {
  int prev;
  bool ok;
  explicit DeviceGuard(int dev) : prev(0), ok(false) {
    if (cudaGetDevice(&prev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) ok = true;
  }
  ~DeviceGuard() { if (ok) cudaSetDevice(prev); }
};

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeFn tensor_map_encoder() {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return nullptr;
  return (EncodeFn)fn;
}

// ---- the verify / prompt passes (fb_pass.cu)
constexpr int kPromptRows = 1024;  // token rows of the activation buffers: a prompt goes through the layers in chunks of at most this
cudaError_t pass_alloc(fb_ctx* c);
void pass_free(fb_ctx* c);
// one stacked weight matrix in the layouts the passes read (order / arg / orows as in fb_repack)
cudaError_t pass_bind_matrix(fb_ctx* c, int which, const void* q, const void* s, const void* z, int layers, int rows, int k, int order,
                             int arg, int orows, cudaStream_t st);

// ---- the decode kernels of tensor-parallel ranks (fb_decode_tp.cu), by index into fb_api.cu's table
const void* decode_tp_kernel(int id);
