// The M-token passes: tree verification and prompts. Launchers of their kernels, the activation buffers, fb_verify, fb_prefill.
#include <stdio.h>
#include <string.h>

#include "../../include/flint_b200.h"
#include "fb_ctx.hpp"
#include "fb_geometry.hpp"
#include "fb_verify.cuh"
#include "fb_vtc.cuh"
#include "fb_vtl.cuh"
#include "fb_vattn.cuh"

using namespace fb;

#define FB_TRY(call)                              \
  do {                                            \
    cudaError_t e__ = (call);                     \
    if (e__ != cudaSuccess) return e__;           \
  } while (0)

namespace {

template <int NT, int EPI, bool HZ>
cudaError_t launch_vtl_hz(const VtcParams& p, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    FB_TRY(cudaFuncSetAttribute(v_gemm_tl<NT, EPI, HZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, VtlSmem<NT, HZ>::TOTAL));
    configured[dev] = true;
  }
  if (p.K % 128 || p.ntok > NT || p.ntok % 16 || (NT < 128 && p.ntile > 1) || (NT == 128 && p.nsplit < 2) || (size_t)p.ntok * p.ntile < (size_t)p.M)
    return cudaErrorInvalidValue;
  const int items = (p.rows + kTcRowBlock - 1) / kTcRowBlock * p.ntile;
  return launch_pdl_cluster(v_gemm_tl<NT, EPI, HZ>, dim3(items * p.nsplit), dim3(kTlThreads), (size_t)VtlSmem<NT, HZ>::TOTAL, st,
                            (unsigned)p.nsplit, p);
}
template <int EPI, bool HZ, int NT>
cudaError_t launch_vtc_hz(const VtcParams& p, int sms, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    FB_TRY(cudaFuncSetAttribute(v_gemm_tc<EPI, HZ, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, VtcSmem<HZ, NT>::TOTAL));
    configured[dev] = true;
  }
  if (p.K % 128 || p.ntok % 16 || p.ntok > NT || (size_t)p.ntok * p.ntile < (size_t)p.M) return cudaErrorInvalidValue;
  const int items = ((p.rows + kTcRowBlock - 1) / kTcRowBlock) * p.ntile;
  return launch_pdl(v_gemm_tc<EPI, HZ, NT>, dim3(items < sms ? items : sms), dim3(kTcThreads), (size_t)VtcSmem<HZ, NT>::TOTAL, st, p);
}
// `maps`: the activation buffer as a tensor, one map per token tile height (16, 32, 64, 128, 192)
template <int EPI>
cudaError_t launch_vtc(VtcParams& p, const CUtensorMap* maps, bool hz, int sms, cudaStream_t st) {
  const GemmGeometry g = gemm_geometry(p.M, p.rows, p.K, hz, sms);
  p.ntok = g.ntok; p.ntile = g.ntile; p.nsplit = g.nsplit;
  p.xmap = maps[g.nt == 16 ? 0 : (g.nt == 32 ? 1 : (g.nt == 64 ? 2 : (g.nt == 128 ? 3 : 4)))];
  switch (g.nt) {
    case 16: return hz ? launch_vtl_hz<16, EPI, true>(p, st) : launch_vtl_hz<16, EPI, false>(p, st);
    case 32: return hz ? launch_vtl_hz<32, EPI, true>(p, st) : launch_vtl_hz<32, EPI, false>(p, st);
    case 64: return hz ? launch_vtl_hz<64, EPI, true>(p, st) : launch_vtl_hz<64, EPI, false>(p, st);
    case 128:
      if (g.nsplit > 1) return hz ? launch_vtl_hz<128, EPI, true>(p, st) : launch_vtl_hz<128, EPI, false>(p, st);
      return hz ? launch_vtc_hz<EPI, true, 128>(p, sms, st) : launch_vtc_hz<EPI, false, 128>(p, sms, st);
    case 192: return launch_vtc_hz<EPI, false, 192>(p, sms, st);
  }
  return cudaErrorInvalidValue;
}

// The activation buffers of the verify GEMMs as 2-D tensors [rows][K], box 64 columns x a token tile, in the swizzle the MMA reads
bool make_act_maps(fb_ctx* c) {
  EncodeFn enc = tensor_map_encoder();
  if (!enc) return false;
  const fb_model_desc& d = c->d;
  void* bases[3] = {c->vxn, c->vao, c->vact};
  const cuuint64_t widths[3] = {(cuuint64_t)d.dim, (cuuint64_t)d.n_head * d.head_dim, (cuuint64_t)d.ffn};
  CUtensorMap* maps[3] = {c->m_xn, c->m_ao, c->m_act};
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 5; j++) {
      const cuuint64_t dims[2] = {widths[i], (cuuint64_t)kPromptRows}, strides[1] = {widths[i] * 2};
      const cuuint32_t box[2] = {64u, j < 4 ? 16u << j : 192u}, estr[2] = {1u, 1u};
      if (enc(&maps[i][j], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, bases[i], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    }
  return true;
}

template <int HD, int R, int RT>
cudaError_t launch_vattn_rt(const VattnParams& a, dim3 grid, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  auto k = v_attn<HD, R, RT>;
  if (!configured[dev]) {
    FB_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, VaCfg<HD, RT>::TOTAL));
    configured[dev] = true;
  }
  return launch_pdl_cluster(k, grid, dim3(256), (size_t)VaCfg<HD, RT>::TOTAL, st, grid.x, a);
}
template <int HD, int R>
cudaError_t launch_vattn_hd(const VattnParams& a, int rt, dim3 grid, cudaStream_t st) {
  return rt == 1 ? launch_vattn_rt<HD, R, 1>(a, grid, st) : (rt == 2 ? launch_vattn_rt<HD, R, 2>(a, grid, st) : launch_vattn_rt<HD, R, 4>(a, grid, st));
}
cudaError_t launch_vattn_tc(const fb_ctx* c, const uint16_t* kc, const uint16_t* vc, const uint8_t* amask, int pos, int M, bool want_max,
                            cudaStream_t st) {
  const fb_model_desc& d = c->d;
  const AttnGeometry a = attn_geometry(M, pos, d.n_kv_head, c->rgqa, c->sm_count);
  const VattnParams p{c->vq, kc, vc, amask, c->vao, want_max ? c->vamax : nullptr, d.n_head, d.n_kv_head, pos, M, a.span,
                      d.attn_scale * 1.4426950408889634f, c->status, c->spin_limit};
  const dim3 grid(a.nspan, d.n_kv_head, a.groups);
  if (d.head_dim == 64 && c->rgqa == 4) return launch_vattn_hd<64, 4>(p, a.rt, grid, st);
  if (d.head_dim == 80 && c->rgqa == 4) return launch_vattn_hd<80, 4>(p, a.rt, grid, st);
  if (d.head_dim == 64 && c->rgqa == 5) return launch_vattn_hd<64, 5>(p, a.rt, grid, st);
  if (d.head_dim == 128 && c->rgqa == 4) return launch_vattn_hd<128, 4>(p, a.rt, grid, st);
  return cudaErrorInvalidValue;
}

// One pass of M tokens (1 .. kPromptRows) through the model on the tcgen05 GEMMs: natural-order activations, the matrices in the
// TC layout. depth / amask NULL: a causal chain (a chunk of a prompt).
int run_tc_pass(fb_ctx* c, const int32_t* d_tokens, const void* d_h, const int32_t* d_depth, const uint8_t* d_amask, int M,
                int pos, float* d_logits, void* d_feat, cudaStream_t st) {
  const fb_model_desc& d = c->d;
  const int D = d.dim, FF = d.ffn, HD = d.head_dim, QD = d.n_head * HD, QKV = (d.n_head + 2 * d.n_kv_head) * HD, sms = c->sm_count;
  const bool hz = d.has_zeros != 0;
  const bool tree = token_tile(M) <= 64;
  const size_t tQ = tc_matrix_bytes(QKV, D, hz), tO = tc_matrix_bytes(D, QD, hz), tG = tc_matrix_bytes(2 * FF, D, hz),
               tF = tc_matrix_bytes(D, FF, hz);
  FB_CUDA(c, launch_pdl(v_embed, dim3(M), dim3(256), 0, st, d_tokens, (const uint16_t*)c->embed, (const uint16_t*)d_h, c->vh,
                        D, d.vocab, d.emb_mult, &c->status->code));
  FB_CUDA(c, launch_pdl(v_rope_table, dim3(M), dim3(64), 0, st, d_depth, (const float*)c->invf, pos, HD / 2, (float2*)c->vrope));
  VtcParams t;
  memset(&t, 0, sizeof(t));
  t.M = M; t.status = c->status; t.spin_limit = c->spin_limit;
  t.rope = (const float2*)c->vrope; t.n_head = d.n_head; t.nkv = d.n_kv_head; t.pos = pos; t.head_dim = HD;
  t.resid = d.resid_mult; t.logits_scaling = d.logits_scaling; t.h = c->vh; t.q = c->vq; t.act = c->vact; t.fa = c->vfa;
  t.logits = d_logits;
  auto norm = [&](const void* w, uint16_t* feat, const unsigned* norms) {
    return D <= 8 * 256 ? launch_pdl(v_norm_f16<1>, dim3(M), dim3(256), 0, st, (const uint16_t*)c->vh, (const uint16_t*)w, c->vxn, feat,
                                     c->vfx, norms, c->vfa, c->vfa_inv, c->vamax, D, d.rms_eps)
                        : launch_pdl(v_norm_f16<2>, dim3(M), dim3(256), 0, st, (const uint16_t*)c->vh, (const uint16_t*)w, c->vxn, feat,
                                     c->vfx, norms, c->vfa, c->vfa_inv, c->vamax, D, d.rms_eps);
  };
  if (D > 8 * 256 * 2) return FB_ERR_SHAPE;
  for (int l = 0; l < d.n_layer; l++) {
    uint16_t* kcl = (uint16_t*)c->kc + (size_t)l * c->max_seq * d.n_kv_head * HD;
    uint16_t* vcl = (uint16_t*)c->vc + (size_t)l * c->max_seq * d.n_kv_head * HD;
    FB_CUDA(c, norm((const uint16_t*)c->n1 + (size_t)l * D, nullptr, nullptr));
    t.w = c->t_qkv + l * tQ; t.rows = QKV; t.K = D; t.kc = kcl; t.vc = vcl; t.fx = c->vfx;
    FB_CUDA(c, launch_vtc<EPI_QKV>(t, c->m_xn, hz, sms, st));
    // trees: the O GEMM converts the attention output to fp16 on its way in; prompts, whose activations come by tensor copies, have it
    // converted in place
    FB_CUDA(c, launch_vattn_tc(c, kcl, vcl, d_amask, pos, M, tree, st));
    if (!tree) FB_CUDA(c, launch_pdl(v_row_f16, dim3(M), dim3(256), 0, st, c->vao, c->vfao, QD));
    t.w = c->t_o + l * tO; t.rows = D; t.K = QD; t.out_ld = D; t.fx = c->vfao;
    t.xbf = tree ? c->vao : nullptr; t.amax = tree ? c->vamax : nullptr;
    FB_CUDA(c, launch_vtc<EPI_RESID>(t, c->m_ao, hz, sms, st));
    t.xbf = nullptr; t.amax = nullptr;
    FB_CUDA(c, norm((const uint16_t*)c->n2 + (size_t)l * D, nullptr, c->gu_norms + 2 * l));
    t.w = c->t_gu + l * tG; t.rows = 2 * FF; t.K = D; t.out_ld = FF; t.fx = c->vfx;
    FB_CUDA(c, launch_vtc<EPI_SWIGLU>(t, c->m_xn, hz, sms, st));
    t.w = c->t_d + l * tF; t.rows = D; t.K = FF; t.out_ld = D; t.fx = c->vfa_inv;
    FB_CUDA(c, launch_vtc<EPI_RESID>(t, c->m_act, hz, sms, st));
  }
  // the feature goes to the caller; the LM head reads the context's copy
  FB_CUDA(c, norm(c->nf, (uint16_t*)d_feat, nullptr));
  if (d_logits) {
    t.w = c->t_lm; t.rows = d.vocab; t.K = D; t.out_ld = d.vocab; t.fx = c->vfx;
    FB_CUDA(c, launch_vtc<EPI_LOGITS>(t, c->m_xn, hz, sms, st));
  }
  FB_CUDA(c, cudaGetLastError());
  return FB_OK;
}

}  // namespace

cudaError_t pass_alloc(fb_ctx* c) {
  const fb_model_desc& d = c->d;
  const int QD = d.n_head * d.head_dim;
  cudaError_t e = cudaSuccess;
  auto A = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
  {
    const size_t rowsz[5] = {(size_t)d.dim, (size_t)d.dim, (size_t)QD, (size_t)QD, (size_t)d.ffn};
    uint16_t** vp[5] = {&c->vh, &c->vxn, &c->vq, &c->vao, &c->vact};
    for (int i = 0; i < 5; i++) {
      A(dmalloc(vp[i], kPromptRows * rowsz[i] * 2));
      if (e == cudaSuccess) A(cudaMemset(*vp[i], 0, kPromptRows * rowsz[i] * 2));
    }
  }
  float** fp[4] = {&c->vfx, &c->vfao, &c->vfa, &c->vfa_inv};
  for (float** p : fp) A(dmalloc(p, kPromptRows * 4));
  A(dmalloc(&c->vamax, kPromptRows * 4));
  A(dmalloc(&c->gu_norms, (size_t)d.n_layer * 8));
  A(cudaMalloc(&c->vrope, (size_t)kPromptRows * (d.head_dim / 2) * 8));
  if (e == cudaSuccess && c->tp_size == 1 && !make_act_maps(c)) e = cudaErrorInvalidValue;
  return e;
}

void pass_free(fb_ctx* c) {
  void* ptrs[] = {c->vh, c->vxn, c->vq, c->vao, c->vact, c->t_qkv, c->t_o, c->t_gu, c->t_d, c->t_lm, c->vrope,
                  c->vfx, c->vfao, c->vfa, c->vfa_inv, c->vamax, c->gu_norms};
  for (void* p : ptrs)
    if (p) cudaFree(p);
}

cudaError_t pass_bind_matrix(fb_ctx* c, int which, const void* q, const void* s, const void* z, int layers, int rows, int k, int order,
                             int arg, int orows, cudaStream_t st) {
  uint8_t** dst[] = {&c->t_qkv, &c->t_o, &c->t_gu, &c->t_d, &c->t_lm};
  uint8_t*& t = *dst[which];
  if (t) { cudaFree(t); t = nullptr; }
  if (c->tp_size > 1) return cudaSuccess;          // a tensor-parallel rank decodes only
  FB_TRY(dmalloc(&t, (size_t)layers * tc_matrix_bytes(rows, k, z != nullptr) + 16));
  if (order == 2) FB_TRY(cudaMemsetAsync(c->gu_norms, 0, (size_t)layers * 8, st));
  tc_repack<<<dim3((rows + kTcRowBlock - 1) / kTcRowBlock, layers), 256, 0, st>>>((const uint32_t*)q, (const uint16_t*)s, (const uint16_t*)z, rows, k,
                                                                                  order, arg, orows, t, order == 2 ? c->gu_norms : nullptr);
  FB_TRY(cudaGetLastError());
  return cudaSuccess;
}

extern "C" {

int fb_prefill(fb_ctx* c, const int32_t* d_tokens, int32_t n, int32_t pos, float* d_logits, void* d_feat, void* stream) {
  if (!c || !d_tokens || n < 1 || ((uintptr_t)d_feat & 15)) return FB_ERR_ARG;       /* features are stored 16 bytes at a time */
  if (!c->weights_bound || !c->kc) return FB_ERR_STATE;
  if (c->tp_size > 1 || !c->embed) return FB_ERR_STATE;
  if (pos < 0 || n > c->max_seq - pos) return FB_ERR_RANGE;
  DeviceGuard g(c->device);
  const fb_model_desc& d = c->d;
  const int nchunk = (n + kPromptRows - 1) / kPromptRows;      // chunks of equal length: no short last one
  for (int i = 0; i < nchunk; i++) {
    const int t0 = (int)((int64_t)n * i / nchunk), t1 = (int)((int64_t)n * (i + 1) / nchunk);
    const int rc = run_tc_pass(c, d_tokens + t0, nullptr, nullptr, nullptr, t1 - t0, pos + t0,
                               d_logits ? d_logits + (size_t)t0 * d.vocab : nullptr,
                               d_feat ? (uint16_t*)d_feat + (size_t)t0 * d.dim : nullptr, (cudaStream_t)stream);
    if (rc != FB_OK) return rc;
  }
  return FB_OK;
}

int fb_verify(fb_ctx* c, const int32_t* d_tokens, const void* d_h, const int32_t* d_depth, const uint8_t* d_amask,
              int32_t M, int32_t pos, float* d_logits, void* d_feat, void* stream) {
  if (!c || !d_depth || !d_amask || (!d_tokens && !d_h) || ((uintptr_t)d_feat & 15)) return FB_ERR_ARG;
  if (!c->weights_bound || !c->kc) return FB_ERR_STATE;
  if (c->tp_size > 1) return FB_ERR_STATE;           /* a tensor-parallel rank holds slices only */
  if (!d_h && !c->embed) return FB_ERR_STATE;
  if (M < 1 || M > 64) return FB_ERR_RANGE;          /* never fall through to another M (reference: result.md:112-113) */
  if (pos < 0 || M > c->max_seq - pos) return FB_ERR_RANGE;
  DeviceGuard g(c->device);
  return run_tc_pass(c, d_tokens, d_h, d_depth, d_amask, M, pos, d_logits, d_feat, (cudaStream_t)stream);
}

}  // extern "C"
