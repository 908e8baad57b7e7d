// The M-token passes: tree verification and prompts. Launchers of their kernels, the activation buffers, fb_verify, fb_prefill.
#include <stdio.h>
#include <string.h>

#include "../../include/flint_b200.h"
#include "fb_ctx.hpp"
#include "fb_verify.cuh"
#include "fb_vsub.cuh"
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

template <int MT, int K, int EPI, int HD, int ROWS>
cudaError_t launch_vgemm_r(const VGemmParams& p, int sms, cudaStream_t st) {
  static bool configured[64] = {};        // the attribute belongs to a device's copy of the function: once per device
  using V = VG<MT, K, ROWS>;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(v_gemm<MT, K, EPI, HD, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, V::smem());
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int per_sm = (227 * 1024) / (V::smem() + 1024) >= 2 ? 2 : 1;      // persistent CTAs: as many as are resident
  const int nrb = (p.rows + V::ROWS - 1) / V::ROWS;
  const int grid = nrb < sms * per_sm ? nrb : sms * per_sm;
  return launch_pdl(v_gemm<MT, K, EPI, HD, ROWS>, dim3(grid), dim3(V::NTHR), V::smem(), st, p);
}
template <int MT, int K, int EPI, int HD>
cudaError_t launch_vgemm_k(const VGemmParams& p, int sms, cudaStream_t st) {
  // tall matrices (gate/up, LM head) with few tokens: 64-row blocks halve the per-chunk overhead per MMA and still
  // give every SM at least one block
  if constexpr (MT == 16 && (EPI == EPI_SWIGLU || EPI == EPI_LOGITS)) {
    if (p.rows >= 64 * sms) return launch_vgemm_r<MT, K, EPI, HD, 64>(p, sms, st);
  }
  return launch_vgemm_r<MT, K, EPI, HD, 32>(p, sms, st);
}
// the shapes the decode kernel table knows: K = model width for QKV / gate-up / LM head and O, FFN width for down
// whether the bf16 warp-level verify GEMM is instantiated for a model's widths (the other verify kernels take them at
// run time)
bool vgemm_known(int D, int QD, int FF, int HD) {
  const bool qkv = (D == 512 && HD == 64) || (D == 2560 && (HD == 80 || HD == 64)) || (D == 4096 && HD == 128);
  const bool kd = D == 512 || D == 2560 || D == 4096, kq = QD == 512 || QD == 2560 || QD == 4096;
  const bool kf = FF == 1408 || FF == 8192 || FF == 14336 || FF == 512 || FF == 2560 || FF == 4096;
  return qkv && kd && kq && kf;
}

template <int MT, int EPI>
cudaError_t launch_vgemm_shape(const VGemmParams& p, int k, int hd, int sms, cudaStream_t st) {
  if constexpr (EPI == EPI_QKV) {
    if (k == 512 && hd == 64) return launch_vgemm_k<MT, 512, EPI, 64>(p, sms, st);
    if (k == 2560 && hd == 80) return launch_vgemm_k<MT, 2560, EPI, 80>(p, sms, st);
    if (k == 2560 && hd == 64) return launch_vgemm_k<MT, 2560, EPI, 64>(p, sms, st);
    if (k == 4096 && hd == 128) return launch_vgemm_k<MT, 4096, EPI, 128>(p, sms, st);
    return cudaErrorInvalidValue;
  } else {
    switch (k) {
      case 512: return launch_vgemm_k<MT, 512, EPI, 64>(p, sms, st);
      case 2560: return launch_vgemm_k<MT, 2560, EPI, 64>(p, sms, st);
      case 4096: return launch_vgemm_k<MT, 4096, EPI, 64>(p, sms, st);
    }
    if constexpr (EPI == EPI_RESID) {
      switch (k) {
        case 1408: return launch_vgemm_k<MT, 1408, EPI_RESID, 64>(p, sms, st);
        case 8192: return launch_vgemm_k<MT, 8192, EPI_RESID, 64>(p, sms, st);
        case 14336: return launch_vgemm_k<MT, 14336, EPI_RESID, 64>(p, sms, st);
      }
    }
    return cudaErrorInvalidValue;
  }
}
template <int EPI>
cudaError_t launch_vgemm_mt(const VGemmParams& p, int mt, int k, int hd, int sms, cudaStream_t st) {
  switch (mt) {
    case 16: return launch_vgemm_shape<16, EPI>(p, k, hd, sms, st);
    case 32: return launch_vgemm_shape<32, EPI>(p, k, hd, sms, st);
    case 64: return launch_vgemm_shape<64, EPI>(p, k, hd, sms, st);
  }
  return cudaErrorInvalidValue;
}
constexpr size_t kVsplitFloats = (size_t)256 * 64 * 128;      // K-split partial sums of v_gemm_sub that the context can hold

template <int NT, int EPI>
cudaError_t launch_vsub_nt(const VsubParams& p, int sms, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(v_gemm_sub<NT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVsSmem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  return launch_pdl(v_gemm_sub<NT, EPI>, dim3(sms), dim3(kVsThreads), (size_t)p.plan.bar_off + 512, st, p);
}
template <int EPI>
cudaError_t launch_vsub(const VsubParams& p, int sms, cudaStream_t st) {
  switch ((p.M + 7) / 8) {
    case 1: return launch_vsub_nt<1, EPI>(p, sms, st);
    case 2: return launch_vsub_nt<2, EPI>(p, sms, st);
    case 3: return launch_vsub_nt<3, EPI>(p, sms, st);
    case 4: return launch_vsub_nt<4, EPI>(p, sms, st);
  }
  return cudaErrorInvalidValue;
}

// K splits (CTAs of a cluster) of one GEMM over a single token tile: two CTAs share an SM; matrices with few row blocks are cut while
// all CTAs are resident at once and each keeps two groups to multiply
int tl_splits(int items, int k, int nt, int sms) {
  const int G = k / 128;
  int ns = 1;
  while (ns < 8 && items * ns * 2 <= 2 * sms && G / (ns * 2) >= 2 && nt / (ns * 2) >= 2) ns *= 2;
  return ns;
}
template <int NT, int EPI, bool HZ>
cudaError_t launch_vtl_hz(VtcParams& p, int sms, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    FB_TRY(cudaFuncSetAttribute(v_gemm_tl<NT, EPI, HZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, VtlSmem<NT, HZ>::TOTAL));
    configured[dev] = true;
  }
  if (p.K % 128 || p.M > NT) return cudaErrorInvalidValue;
  const int items = (p.rows + kTcRowBlock - 1) / kTcRowBlock;
  p.nsplit = tl_splits(items, p.K, NT, sms);
  return launch_pdl_cluster(v_gemm_tl<NT, EPI, HZ>, dim3(items * p.nsplit), dim3(kTlThreads), (size_t)VtlSmem<NT, HZ>::TOTAL, st,
                            (unsigned)p.nsplit, p);
}
template <int EPI, bool HZ>
cudaError_t launch_vtc_hz(VtcParams& p, int sms, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    FB_TRY(cudaFuncSetAttribute(v_gemm_tc<EPI, HZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, VtcSmem<HZ>::TOTAL));
    configured[dev] = true;
  }
  if (p.K % 128 || p.ntok % 16 || p.ntok > kTcTokens || (size_t)p.ntok * p.ntile < (size_t)p.M) return cudaErrorInvalidValue;
  const int items = ((p.rows + kTcRowBlock - 1) / kTcRowBlock) * p.ntile;
  return launch_pdl(v_gemm_tc<EPI, HZ>, dim3(items < sms ? items : sms), dim3(kTcThreads), (size_t)VtcSmem<HZ>::TOTAL, st, p);
}
// `maps`: the activation buffer as a tensor, one map per token tile height (16, 32, 64, 128)
template <int EPI>
cudaError_t launch_vtc(VtcParams& p, const CUtensorMap* maps, int nt, bool hz, int sms, cudaStream_t st) {
  p.xmap = maps[nt == 16 ? 0 : (nt == 32 ? 1 : (nt == 64 ? 2 : 3))];
  switch (nt) {
    case 16: return hz ? launch_vtl_hz<16, EPI, true>(p, sms, st) : launch_vtl_hz<16, EPI, false>(p, sms, st);
    case 32: return hz ? launch_vtl_hz<32, EPI, true>(p, sms, st) : launch_vtl_hz<32, EPI, false>(p, sms, st);
    case 64: return hz ? launch_vtl_hz<64, EPI, true>(p, sms, st) : launch_vtl_hz<64, EPI, false>(p, sms, st);
    case 128: return hz ? launch_vtc_hz<EPI, true>(p, sms, st) : launch_vtc_hz<EPI, false>(p, sms, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_vnorm(const uint16_t* h, const uint16_t* w, uint16_t* xn_t, uint16_t* xn_nat, uint16_t* feat, int D, int M,
                         float eps, cudaStream_t st) {
  if (D % 16 || D > 8 * 256 * 2) return cudaErrorInvalidValue;
  if (D <= 8 * 256) return launch_pdl(v_rmsnorm<1>, dim3(M), dim3(256), 0, st, h, w, xn_t, xn_nat, feat, D, eps);
  return launch_pdl(v_rmsnorm<2>, dim3(M), dim3(256), 0, st, h, w, xn_t, xn_nat, feat, D, eps);
}
constexpr int kVSpans = 32;       // most spans of positions a kv head's attention is cut into

cudaError_t launch_vattn(const fb_ctx* c, const uint16_t* q, const uint16_t* kc, const uint16_t* vc, const uint8_t* amask,
                         uint16_t* ao, int pos, int M, cudaStream_t st) {
  const fb_model_desc& d = c->d;
  const int T = pos + M;
  // a CTA takes 64 query rows (four 16-row tiles); spans of positions are sized so that about two CTAs per SM exist
  const int mgroups = (M * c->rgqa + 63) / 64;
  int smax = (2 * c->sm_count) / (d.n_kv_head * mgroups);
  if (smax < 1) smax = 1;
  if (smax > kVSpans) smax = kVSpans;
  if (smax > kVSpans * 64 / M) smax = kVSpans * 64 / M > 0 ? kVSpans * 64 / M : 1;     // the partials' buffer
  int S = (T + 63) / 64;
  if (S > smax) S = smax;
  const int span = ((T + S - 1) / S + 63) / 64 * 64;
  S = (T + span - 1) / span;
#define FB_VATTN(HD_, R_)                                                                                               \
  if (d.head_dim == HD_ && c->rgqa == R_) {                                                                             \
    cudaError_t e = launch_pdl(v_attn_mma<HD_, R_>, dim3(d.n_kv_head, S, mgroups), dim3(128), 0, st, q, kc, vc, amask, c->vpart,  \
                               d.n_head, d.n_kv_head, pos, M, d.attn_scale, span);                                      \
    if (e != cudaSuccess) return e;                                                                                     \
    return launch_pdl(v_attn_merge<HD_, R_>, dim3(M, d.n_kv_head), dim3(256), 0, st, (const float*)c->vpart, ao, d.n_head, \
                      d.n_kv_head, M, S);                                                                      \
  }
  FB_VATTN(64, 4) FB_VATTN(80, 4) FB_VATTN(64, 5) FB_VATTN(128, 4)
#undef FB_VATTN
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
    for (int j = 0; j < 4; j++) {
      const cuuint64_t dims[2] = {widths[i], (cuuint64_t)kPromptRows}, strides[1] = {widths[i] * 2};
      const cuuint32_t box[2] = {64u, 16u << j}, estr[2] = {1u, 1u};
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
// Geometry. Few row tiles: one or two a CTA, its warps share the span's positions instead; four where that many CTAs would not fit the
// GPU with four spans each. Spans: a power of two up to 8 while there is a stage for each and all CTAs are resident at once (with one
// CTA per SM the GPU holds 15 clusters of 8 -- the 16th waited for a second wave, 22 us instead of 12 -- but 36 of 4).
cudaError_t launch_vattn_tc(const fb_ctx* c, const uint16_t* kc, const uint16_t* vc, const uint8_t* amask, int pos, int M, bool want_max,
                            cudaStream_t st) {
  const fb_model_desc& d = c->d;
  const int T = pos + M, tiles = (M * c->rgqa + 15) / 16, per4 = c->sm_count / (4 * d.n_kv_head);
  VattnParams a{c->vq, kc, vc, amask, c->vao, want_max ? c->vamax : nullptr, d.n_head, d.n_kv_head, pos, M, 0, d.attn_scale * 1.4426950408889634f};
  const int rt = tiles <= per4 ? 1 : (tiles <= 2 * per4 ? 2 : 4), mg = (tiles + rt - 1) / rt, groups = d.n_kv_head * mg;
  const int stages = (T + 63) / 64;
  int nspan = 1;
  while (nspan < 8 && nspan * 2 <= stages && groups * nspan * 2 <= (nspan == 4 ? c->sm_count * 2 / 3 : c->sm_count)) nspan *= 2;
  a.span = (stages + nspan - 1) / nspan * 64;
  const dim3 grid(nspan, d.n_kv_head, mg);
  if (d.head_dim == 64 && c->rgqa == 4) return launch_vattn_hd<64, 4>(a, rt, grid, st);
  if (d.head_dim == 80 && c->rgqa == 4) return launch_vattn_hd<80, 4>(a, rt, grid, st);
  if (d.head_dim == 64 && c->rgqa == 5) return launch_vattn_hd<64, 5>(a, rt, grid, st);
  if (d.head_dim == 128 && c->rgqa == 4) return launch_vattn_hd<128, 4>(a, rt, grid, st);
  return cudaErrorInvalidValue;
}

// One pass of M tokens (1 .. kPromptRows) through the model on the tcgen05 GEMMs: natural-order activations, the matrices in the
// TC layout. depth / amask NULL: a causal chain (a chunk of a prompt).
int run_tc_pass(fb_ctx* c, const int32_t* d_tokens, const void* d_h, const int32_t* d_depth, const uint8_t* d_amask, int M,
                int pos, float* d_logits, void* d_feat, cudaStream_t st) {
  const fb_model_desc& d = c->d;
  const int D = d.dim, FF = d.ffn, HD = d.head_dim, QD = d.n_head * HD, QKV = (d.n_head + 2 * d.n_kv_head) * HD, sms = c->sm_count;
  const bool hz = d.has_zeros != 0;
  // token tile: the smallest that holds the tokens; prompts go in tiles of up to 128, cut evenly
  const int nt = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
  const size_t tQ = tc_matrix_bytes(QKV, D, hz), tO = tc_matrix_bytes(D, QD, hz), tG = tc_matrix_bytes(2 * FF, D, hz),
               tF = tc_matrix_bytes(D, FF, hz);
  FB_CUDA(c, launch_pdl(v_embed, dim3(M), dim3(256), 0, st, d_tokens, (const uint16_t*)c->embed, (const uint16_t*)d_h, c->vh,
                        D, d.vocab, d.emb_mult, &c->status->code));
  FB_CUDA(c, launch_pdl(v_rope_table, dim3(M), dim3(64), 0, st, d_depth, (const float*)c->invf, pos, HD / 2, (float2*)c->vrope));
  VtcParams t;
  memset(&t, 0, sizeof(t));
  t.M = M; t.status = c->status; t.spin_limit = c->spin_limit;
  t.ntile = (M + nt - 1) / nt; t.ntok = ((M + t.ntile - 1) / t.ntile + 15) / 16 * 16;
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
    FB_CUDA(c, launch_vtc<EPI_QKV>(t, c->m_xn, nt, hz, sms, st));
    // trees: the O GEMM converts the attention output to fp16 on its way in; prompts, whose activations come by tensor copies, have it
    // converted in place
    FB_CUDA(c, launch_vattn_tc(c, kcl, vcl, d_amask, pos, M, nt <= 64, st));
    if (nt > 64) FB_CUDA(c, launch_pdl(v_row_f16, dim3(M), dim3(256), 0, st, c->vao, c->vfao, QD));
    t.w = c->t_o + l * tO; t.rows = D; t.K = QD; t.out_ld = D; t.fx = c->vfao;
    t.xbf = nt <= 64 ? c->vao : nullptr; t.amax = nt <= 64 ? c->vamax : nullptr;
    FB_CUDA(c, launch_vtc<EPI_RESID>(t, c->m_ao, nt, hz, sms, st));
    t.xbf = nullptr; t.amax = nullptr;
    FB_CUDA(c, norm((const uint16_t*)c->n2 + (size_t)l * D, nullptr, c->gu_norms + 2 * l));
    t.w = c->t_gu + l * tG; t.rows = 2 * FF; t.K = D; t.out_ld = FF; t.fx = c->vfx;
    FB_CUDA(c, launch_vtc<EPI_SWIGLU>(t, c->m_xn, nt, hz, sms, st));
    t.w = c->t_d + l * tF; t.rows = D; t.K = FF; t.out_ld = D; t.fx = c->vfa_inv;
    FB_CUDA(c, launch_vtc<EPI_RESID>(t, c->m_act, nt, hz, sms, st));
  }
  // the feature goes to the caller; the LM head reads the context's copy
  FB_CUDA(c, norm(c->nf, (uint16_t*)d_feat, nullptr));
  if (d_logits) {
    t.w = c->t_lm; t.rows = d.vocab; t.K = D; t.out_ld = d.vocab; t.fx = c->vfx;
    FB_CUDA(c, launch_vtc<EPI_LOGITS>(t, c->m_xn, nt, hz, sms, st));
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
  A(dmalloc(&c->vpart, (size_t)d.n_kv_head * 32 * 64 * c->rgqa * (d.head_dim + 2) * 4));
  A(dmalloc(&c->vsplit, kVsplitFloats * 4));
  A(dmalloc(&c->vcount, kVsCounters * 4));
  if (e == cudaSuccess) A(cudaMemset(c->vcount, 0, kVsCounters * 4));
  float** fp[4] = {&c->vfx, &c->vfao, &c->vfa, &c->vfa_inv};
  for (float** p : fp) A(dmalloc(p, kPromptRows * 4));
  A(dmalloc(&c->vamax, kPromptRows * 4));
  A(dmalloc(&c->gu_norms, (size_t)d.n_layer * 8));
  A(cudaMalloc(&c->vrope, (size_t)kPromptRows * (d.head_dim / 2) * 8));
  if (e == cudaSuccess && c->tp_size == 1 && !make_act_maps(c)) e = cudaErrorInvalidValue;
  return e;
}

void pass_free(fb_ctx* c) {
  void* ptrs[] = {c->vh, c->vxn, c->vq, c->vao, c->vact, c->vpart, c->t_qkv, c->t_o, c->t_gu, c->t_d, c->t_lm, c->s_qkv, c->s_o, c->s_gu,
                  c->s_d, c->s_lm, c->vsplit, c->vcount, c->vrope, c->vfx, c->vfao, c->vfa, c->vfa_inv, c->vamax, c->gu_norms};
  for (void* p : ptrs)
    if (p) cudaFree(p);
}

cudaError_t pass_bind_matrix(fb_ctx* c, int which, const void* q, const void* s, const void* z, int layers, int rows, int k, int order,
                             int arg, int orows, cudaStream_t st) {
  uint8_t** tdst[] = {&c->t_qkv, &c->t_o, &c->t_gu, &c->t_d, &c->t_lm};
  uint8_t** sdst[] = {&c->s_qkv, &c->s_o, &c->s_gu, &c->s_d, &c->s_lm};
  struct M { uint8_t **tdst, **sdst; const void *q, *s, *z; int layers, rows, k, order, arg, orows; } m =
      {tdst[which], sdst[which], q, s, z, layers, rows, k, order, arg, orows};
  const bool hz = z != nullptr;
    if (*m.tdst) { cudaFree(*m.tdst); *m.tdst = nullptr; }
    if (c->tp_size == 1) {     // the verify path's own copy, in the layout the tcgen05 GEMM streams
      const int nrb = (m.rows + kTcRowBlock - 1) / kTcRowBlock;
      FB_TRY(dmalloc(m.tdst, (size_t)m.layers * tc_matrix_bytes(m.rows, m.k, hz) + 16));
      if (m.order == 2) FB_TRY(cudaMemsetAsync(c->gu_norms, 0, (size_t)m.layers * 8, st));
      tc_repack<<<dim3(nrb, m.layers), 256, 0, st>>>((const uint32_t*)m.q, (const uint16_t*)m.s, (const uint16_t*)m.z,
                                                     m.rows, m.k, m.order, m.arg, m.orows, *m.tdst, m.order == 2 ? c->gu_norms : nullptr);
      FB_TRY(cudaGetLastError());
    }
    if (*m.sdst) { cudaFree(*m.sdst); *m.sdst = nullptr; }
    const int tiles32 = (m.rows + 31) / 32;
    const VsPlan vp = vs_plan(m.k, 1, tiles32);
    if (c->tp_size == 1 && !hz && vp.ok &&
        (size_t)tiles32 * vp.nkc * 8 * 512 <= kVsplitFloats * 4) {   // K-split partials fit the shared buffer
      // the small-tree verify GEMM's copy (symmetric layout only; other shapes keep the bf16 warp-level kernel)
      FB_TRY(dmalloc(m.sdst, (size_t)m.layers * vs_matrix_bytes(m.rows, m.k) + 16));
      vs_repack<<<dim3(tiles32, m.layers), 256, 0, st>>>((const uint32_t*)m.q, (const uint16_t*)m.s, m.rows, m.k, vp.ug, m.order,
                                                         m.arg, m.orows, *m.sdst);
      FB_TRY(cudaGetLastError());
    }
  return cudaSuccess;
}

extern "C" {

int fb_prefill(fb_ctx* c, const int32_t* d_tokens, int32_t n, int32_t pos, float* d_logits, void* d_feat, void* stream) {
  if (!c || !d_tokens || n < 1) return FB_ERR_ARG;
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
  if (!c || !d_depth || !d_amask || (!d_tokens && !d_h)) return FB_ERR_ARG;
  if (!c->weights_bound || !c->kc) return FB_ERR_STATE;
  if (c->tp_size > 1) return FB_ERR_STATE;           /* a tensor-parallel rank holds slices only */
  if (!d_h && !c->embed) return FB_ERR_STATE;
  if (M < 1 || M > 64) return FB_ERR_RANGE;          /* never fall through to another M (reference: result.md:112-113) */
  if (pos < 0 || pos + M > c->max_seq) return FB_ERR_RANGE;
  const fb_model_desc& d = c->d;
  DeviceGuard g(c->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int MT = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
  const int D = d.dim, FF = d.ffn, HD = d.head_dim, QD = d.n_head * HD, QKV = (d.n_head + 2 * d.n_kv_head) * HD;
  const bool hz = d.has_zeros != 0;
  if (c->verify_path == 2 || c->verify_path == 3 || (c->verify_path == 0 && (M > 8 || hz)) || !vgemm_known(D, QD, FF, HD))
    return run_tc_pass(c, d_tokens, d_h, d_depth, d_amask, M, pos, d_logits, d_feat, st);
  const size_t strQ = (size_t)pad_rows(QKV, D) * rec_bytes_of(D, hz), strO = (size_t)pad_rows(D, QD) * rec_bytes_of(QD, hz),
               strG = (size_t)pad_rows(2 * FF, D) * rec_bytes_of(D, hz), strF = (size_t)pad_rows(D, FF) * rec_bytes_of(FF, hz);
  FB_CUDA(c, launch_pdl(v_embed, dim3(M), dim3(256), 0, st, d_tokens, (const uint16_t*)c->embed, (const uint16_t*)d_h, c->vh,
                        D, d.vocab, d.emb_mult, &c->status->code));
  VGemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.has_zeros = hz; p.depth = d_depth; p.invf = c->invf; p.n_head = d.n_head; p.nkv = d.n_kv_head; p.pos = pos;
  p.resid = d.resid_mult; p.logits_scaling = d.logits_scaling;
  // small trees: every GEMM whose matrix has an R32 copy runs on the subnormal-operand kernel. It reads the same
  // activation buffers; the QKV and gate/up GEMMs read the residual rows and apply the RMSNorm themselves
  // by tree size: up to 8 tokens (one B tile) this kernel wins (2.07 vs 2.40 ms per pass of the 3B model); above, its
  // per-CTA conversion of the activations (linear in the tokens) costs more than the dequantisation it saves
  const bool use_sub = (c->verify_path == 4 || (c->verify_path == 0 && M <= 8)) && M <= kVsMaxTokens && !hz;
  VsubParams sp;
  memset(&sp, 0, sizeof(sp));
  sp.M = M; sp.part = c->vsplit; sp.counters = (int*)c->vcount; sp.status = c->status; sp.spin_limit = c->spin_limit;
  sp.rope = (const float2*)c->vrope; sp.n_head = d.n_head; sp.nkv = d.n_kv_head; sp.pos = pos; sp.head_dim = HD;
  sp.resid = d.resid_mult; sp.logits_scaling = d.logits_scaling; sp.eps = d.rms_eps;
  if (use_sub && c->s_qkv)
    FB_CUDA(c, launch_pdl(v_rope_table, dim3(M), dim3(64), 0, st, d_depth, (const float*)c->invf, (int)pos, HD / 2, (float2*)c->vrope));
  int nsub = 0;
  auto sub = [&](const uint8_t* sw, size_t layer, int rows, int K) -> bool {
    if (!use_sub || !sw) return false;
    sp.plan = vs_plan(K, M, (rows + 31) / 32);
    if (!sp.plan.ok) return false;
    sp.w = sw + layer * vs_matrix_bytes(rows, K); sp.rows = rows; sp.K = K; sp.norm_w = nullptr;
    sp.dbg = (c->prof && layer == 1) ? c->prof + 8 * (nsub++ & 7) : nullptr;   // stamps of the second layer's GEMMs
    return true;
  };
  for (int l = 0; l < d.n_layer; l++) {
    uint16_t* kcl = (uint16_t*)c->kc + (size_t)l * c->max_seq * d.n_kv_head * HD;
    uint16_t* vcl = (uint16_t*)c->vc + (size_t)l * c->max_seq * d.n_kv_head * HD;
    if (sub(c->s_qkv, l, QKV, D)) {
      if (sp.plan.nkc == 1) { sp.x = c->vh; sp.norm_w = (const uint16_t*)c->n1 + (size_t)l * D; }
      else {
        FB_CUDA(c, launch_vnorm(c->vh, (const uint16_t*)c->n1 + (size_t)l * D, c->vxn, nullptr, nullptr, D, M, d.rms_eps, st));
        sp.x = c->vxn;
      }
      sp.q = c->vq; sp.kc = kcl; sp.vc = vcl;
      FB_CUDA(c, launch_vsub<EPI_QKV>(sp, c->sm_count, st));
    } else {
      FB_CUDA(c, launch_vnorm(c->vh, (const uint16_t*)c->n1 + (size_t)l * D, c->vxn, nullptr, nullptr, D, M, d.rms_eps, st));
      p.w = c->w_qkv + l * strQ; p.x_t = c->vxn; p.rows = QKV;
      p.q = c->vq; p.kc = kcl; p.vc = vcl;
      FB_CUDA(c, launch_vgemm_mt<EPI_QKV>(p, MT, D, HD, c->sm_count, st));
    }
    FB_CUDA(c, launch_vattn(c, c->vq, kcl, vcl, d_amask, c->vao, pos, M, st));
    if (sub(c->s_o, l, D, QD)) {
      sp.x = c->vao; sp.h = c->vh; sp.out_ld = D;
      FB_CUDA(c, launch_vsub<EPI_RESID>(sp, c->sm_count, st));
    } else {
      p.w = c->w_o + l * strO; p.x_t = c->vao; p.rows = D; p.h = c->vh; p.out_ld = D;
      FB_CUDA(c, launch_vgemm_mt<EPI_RESID>(p, MT, QD, HD, c->sm_count, st));
    }
    if (sub(c->s_gu, l, 2 * FF, D)) {
      if (sp.plan.nkc == 1) { sp.x = c->vh; sp.norm_w = (const uint16_t*)c->n2 + (size_t)l * D; }
      else {
        FB_CUDA(c, launch_vnorm(c->vh, (const uint16_t*)c->n2 + (size_t)l * D, c->vxn, nullptr, nullptr, D, M, d.rms_eps, st));
        sp.x = c->vxn;
      }
      sp.act_t = c->vact; sp.out_ld = FF;
      FB_CUDA(c, launch_vsub<EPI_SWIGLU>(sp, c->sm_count, st));
    } else {
      FB_CUDA(c, launch_vnorm(c->vh, (const uint16_t*)c->n2 + (size_t)l * D, c->vxn, nullptr, nullptr, D, M, d.rms_eps, st));
      p.w = c->w_gu + l * strG; p.x_t = c->vxn; p.rows = 2 * FF; p.act_t = c->vact;
      p.out_ld = FF;
      FB_CUDA(c, launch_vgemm_mt<EPI_SWIGLU>(p, MT, D, HD, c->sm_count, st));
    }
    if (sub(c->s_d, l, D, FF)) {
      sp.x = c->vact; sp.h = c->vh; sp.out_ld = D;
      FB_CUDA(c, launch_vsub<EPI_RESID>(sp, c->sm_count, st));
    } else {
      p.w = c->w_d + l * strF; p.x_t = c->vact; p.rows = D; p.h = c->vh; p.out_ld = D;
      FB_CUDA(c, launch_vgemm_mt<EPI_RESID>(p, MT, FF, HD, c->sm_count, st));
    }
  }
  FB_CUDA(c, launch_vnorm(c->vh, (const uint16_t*)c->nf, c->vxn, nullptr, (uint16_t*)d_feat, D, M, d.rms_eps, st));
  if (d_logits) {
    if (sub(c->s_lm, 0, d.vocab, D)) {
      sp.x = c->vxn; sp.logits = d_logits; sp.out_ld = d.vocab;
      FB_CUDA(c, launch_vsub<EPI_LOGITS>(sp, c->sm_count, st));
    } else {
      p.w = c->w_lm; p.x_t = c->vxn; p.rows = d.vocab; p.logits = d_logits; p.out_ld = d.vocab;
      FB_CUDA(c, launch_vgemm_mt<EPI_LOGITS>(p, MT, D, HD, c->sm_count, st));
    }
  }
  FB_CUDA(c, cudaGetLastError());
  return FB_OK;
}

}  // extern "C"
