// extern "C" entry points of the speculative-decoding side: sampling, acceptance, KV compaction, the EAGLE draft head.
// No torch types, no CPU fallback: a failed CUDA call or an unsupported shape is an error code.
#include <string.h>

#include <new>

#include "../../include/flint_b200.h"
#include "fb_ctx.hpp"
#include "fb_geometry.hpp"
#include "fb_spec.cuh"

using namespace fb;

struct fb_draft {
  fb_draft_desc d;
  int device;
  fb_draft_weights w;
  bool bound;
  uint16_t *x, *h, *q, *k, *v, *att, *x2, *act, *hh, *fn;     // [max_tokens] rows of activations
  uint16_t *kc, *vc;                                           // [max_roll, n_kv, hd]
  float* logits;                                               // [max_heads rows, vocab]
  int last_cuda_error, sm_count;
};

namespace {

constexpr int kMaxHeadRows = 16;
constexpr int kAttnSmem = 200 * 1024;            // d_attn's scores of every cache slot and the query (more than the 48 KB that need no asking) ...
constexpr int kAttnSmemNew = 8 * 1024;           // ... and the new k and v of a single token (d_attn_one)

template <int NT, int MT, int MODE>
cudaError_t launch_linear_nt(DLin p, int t0, int sms, cudaStream_t st) {
  int blocks = 0;
  for (int i = 0; i < (MODE == DL_STORE ? 3 : 1) && p.W[i]; i++) blocks += (p.N[i] + 16 * MT - 1) / (16 * MT);
  p.ks = MODE == DL_LOGITS ? 1 : draft_splits(blocks, (p.k0 + p.k1 + 31) / 32, NT, sms);
  const dim3 grid(blocks * p.ks), block(kDraftWarps * 32);
  constexpr bool FOLDS = NT == 1 && (MODE == DL_STORE || MODE == DL_SWIGLU);
  if (MODE == DL_STORE && p.x1) return launch_pdl_cluster(d_gemm<NT, MT, MODE, MODE == DL_STORE, false>, grid, block, 0, st, (unsigned)p.ks, p, t0);
  if (FOLDS && p.norm_w) return launch_pdl_cluster(d_gemm<NT, MT, MODE, false, FOLDS>, grid, block, 0, st, (unsigned)p.ks, p, t0);
  return launch_pdl_cluster(d_gemm<NT, MT, MODE, false, false>, grid, block, 0, st, (unsigned)p.ks, p, t0);
}
// All T tokens, up to 32 per pass over the weights. Up to 8 tokens: 16 rows per CTA and three CTAs per SM. More tokens: 32 rows per CTA (one
// matrix) or 16 of each of two, so that a CTA reads about as many bytes of activations from L2 as of weights, and two CTAs per SM.
template <int MODE>
cudaError_t launch_linear(const DLin& p, int sms, cudaStream_t st) {
  if ((p.k0 + p.k1) % 8 || p.k0 % 8 || p.N[0] <= 0 || p.T <= 0) return cudaErrorInvalidValue;
  constexpr int MW = MODE == DL_SWIGLU ? 1 : 2;
  cudaError_t e = cudaSuccess;
  for (int t0 = 0; t0 < p.T && e == cudaSuccess; t0 += 32) {
    const int left = p.T - t0;
    if (left <= 8) e = launch_linear_nt<1, 1, MODE>(p, t0, sms, st);
    else if (left <= 16) e = launch_linear_nt<2, MW, MODE>(p, t0, sms, st);
    else e = launch_linear_nt<4, MW, MODE>(p, t0, sms, st);
  }
  return e;
}
// RMSNorm of n rows, `first`: the first kernel of a call, which nothing hides: in registers (one row, step and token head 118.5 -> 117.2 us at 3B, 136.6 -> 135.4 at 1B;
// inside the block no faster at 3B and 1 us slower at 1B)
cudaError_t launch_norm(const uint16_t* x, int ldx, const void* w, uint16_t* y, int n, int D, float eps, bool first, cudaStream_t st) {
  return launch_pdl(first && D <= kNormRegs * 256 ? d_rmsnorm_regs : d_rmsnorm, dim3(n), dim3(256), 0, st, x, ldx, (const uint16_t*)w, y, D, D, eps, first);
}
// CTAs per row of the token choice: slices of at least 4096 values, at most 8 CTAs (the portable cluster)
int row_ctas(int vocab) {
  int c = 1;
  while (c < 8 && vocab >= 4096 * 2 * c) c *= 2;
  return c;
}

int dfail(fb_draft* d, cudaError_t e) {
  if (d) d->last_cuda_error = (int)e;
  return FB_ERR_CUDA;
}
#define FB_DCUDA(d, call)                                 \
  do {                                                    \
    cudaError_t e__ = (call);                             \
    if (e__ != cudaSuccess) return dfail((d), e__);       \
  } while (0)

}  // namespace

extern "C" {

int fb_sample(const float* d_logits, int32_t vocab, int32_t rows, int64_t row_stride, float temperature, int32_t top_k,
              uint64_t seed, uint64_t counter, int32_t* d_out, void* stream) {
  if (!d_logits || !d_out || vocab <= 0 || rows <= 0 || row_stride < 0) return FB_ERR_ARG;
  const int c = row_ctas(vocab);
  const bool reg = (vocab + c - 1) / c <= kSampleRegs * 1024;
  const bool select = temperature > 0.f && top_k > 0 && top_k < vocab;
  const auto kern = select ? (reg ? sample_rows<true, true> : sample_rows<false, true>) : (reg ? sample_rows<true, false> : sample_rows<false, false>);
  const int64_t most = 0x7fffffff / c;              // rows of one launch: grid.x holds every CTA of every row
  for (int64_t r0 = 0; r0 < rows; r0 += most) {
    const int64_t n = rows - r0 < most ? rows - r0 : most;
    const SampleParams p{d_logits + r0 * row_stride, (long long)row_stride, vocab, top_k, temperature, (unsigned long long)seed,
                         (unsigned long long)counter + (unsigned long long)r0, d_out + r0, c};
    const cudaError_t e = launch_pdl_cluster(kern, dim3((unsigned)(n * c)), dim3(1024), 0, (cudaStream_t)stream, c, p);
    if (e != cudaSuccess) return FB_ERR_CUDA;
  }
  return FB_OK;
}

int fb_accept_chain(const int32_t* d_target, const int32_t* d_draft, int32_t k, int32_t* d_out, void* stream) {
  if (!d_target || !d_out || k < 0 || (k > 0 && !d_draft)) return FB_ERR_ARG;
  accept_chain<<<1, 32, 0, (cudaStream_t)stream>>>(d_target, d_draft, k, d_out);
  return cudaGetLastError() == cudaSuccess ? FB_OK : FB_ERR_CUDA;
}

int fb_accept_tree(const int32_t* d_cand, const int32_t* d_parent, const int32_t* d_target, int32_t m, int32_t* d_out,
                   void* stream) {
  if (!d_cand || !d_parent || !d_target || !d_out || m < 1 || m > 64) return FB_ERR_ARG;
  accept_tree<<<1, 32, 0, (cudaStream_t)stream>>>(d_cand, d_parent, d_target, m, d_out);
  return cudaGetLastError() == cudaSuccess ? FB_OK : FB_ERR_CUDA;
}

int fb_kv_compact(fb_ctx* c, const int32_t* d_accept, int32_t pos, void* stream) {
  if (!c || !c->kc || !d_accept) return FB_ERR_ARG;
  if (pos < 0 || pos >= c->max_seq) return FB_ERR_RANGE;
  const fb_model_desc& d = c->d;
  DeviceGuard g(c->device);
  const int row = d.n_kv_head * d.head_dim;
  if (row % 8) return FB_ERR_SHAPE;
  kv_compact<<<dim3(d.n_layer, 2), 128, 0, (cudaStream_t)stream>>>((uint16_t*)c->kc, (uint16_t*)c->vc, d_accept, pos,
                                                                  (size_t)c->max_seq * row, row, c->max_seq);
  return cudaGetLastError() == cudaSuccess ? FB_OK : FB_ERR_CUDA;
}

int fb_draft_create(const fb_draft_desc* desc, int device, fb_draft** out) {
  if (!desc || !out) return FB_ERR_ARG;
  *out = nullptr;
  const fb_draft_desc& d = *desc;
  if (d.dim <= 0 || d.n_head <= 0 || d.n_kv_head <= 0 || d.dim % d.n_head || d.n_head % d.n_kv_head || d.inter <= 0 ||
      d.fuse < 1 || d.vocab <= 0 || d.max_roll < 1 || d.max_tokens < 1)
    return FB_ERR_SHAPE;
  const int hd = d.dim / d.n_head;
  if (d.dim % 8 || d.inter % 8 || hd % 2 || (d.n_kv_head * hd) % 8) return FB_ERR_SHAPE;
  DeviceGuard g(device);
  if (!g.ok) return FB_ERR_CUDA;
  fb_draft* r = new (std::nothrow) fb_draft();
  if (!r) return FB_ERR_ARG;
  memset(r, 0, sizeof(*r));
  r->d = d;
  r->device = device;
  const size_t T = d.max_tokens, D = d.dim, kvd = (size_t)d.n_kv_head * hd, F = (size_t)d.fuse * d.dim;
  cudaError_t e = cudaSuccess;
  auto A = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
  A(cudaDeviceGetAttribute(&r->sm_count, cudaDevAttrMultiProcessorCount, device));
  A(cudaFuncSetAttribute(d_attn, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmem));
  A(cudaFuncSetAttribute(d_attn_one, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmem + kAttnSmemNew));
  A(dmalloc(&r->x, T * D * 2)); A(dmalloc(&r->h, T * D * 2)); A(dmalloc(&r->q, T * D * 2));
  A(dmalloc(&r->k, T * kvd * 2)); A(dmalloc(&r->v, T * kvd * 2)); A(dmalloc(&r->att, T * D * 2));
  A(dmalloc(&r->x2, T * D * 2)); A(dmalloc(&r->act, T * (size_t)d.inter * 2)); A(dmalloc(&r->hh, T * D * 2));
  A(dmalloc(&r->fn, (size_t)kMaxHeadRows * D * 2));
  A(dmalloc(&r->kc, (size_t)d.max_roll * kvd * 2)); A(dmalloc(&r->vc, (size_t)d.max_roll * kvd * 2));
  A(dmalloc(&r->logits, (size_t)kMaxHeadRows * d.vocab * 4));
  if (e == cudaSuccess) A(cudaMemset(r->kc, 0, (size_t)d.max_roll * kvd * 2));
  if (e == cudaSuccess) A(cudaMemset(r->vc, 0, (size_t)d.max_roll * kvd * 2));
  (void)F;
  if (e != cudaSuccess) { fb_draft_destroy(r); return FB_ERR_CUDA; }
  *out = r;
  return FB_OK;
}

int fb_draft_destroy(fb_draft* r) {
  if (!r) return FB_ERR_ARG;
  DeviceGuard g(r->device);
  void* ptrs[] = {r->x, r->h, r->q, r->k, r->v, r->att, r->x2, r->act, r->hh, r->fn, r->kc, r->vc, r->logits};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  delete r;
  return FB_OK;
}

int fb_draft_bind(fb_draft* r, const fb_draft_weights* w) {
  if (!r || !w) return FB_ERR_ARG;
  const void* need[] = {w->merge, w->n1, w->n2, w->q, w->k, w->v, w->o, w->gate, w->up, w->down, w->fout, w->nf, w->embed};
  for (const void* p : need)
    if (!p || ((uintptr_t)p & 15)) return FB_ERR_ARG;
  r->w = *w;
  r->bound = true;
  return FB_OK;
}

int fb_draft_forward(fb_draft* r, const void* d_feat, const void* d_emb, const int32_t* d_tokens, const int32_t* d_positions,
                     const int32_t* d_slots, int32_t T, void* d_out, void* stream) {
  if (!r || !d_feat || !d_positions || !d_out || (!d_emb && !d_tokens)) return FB_ERR_ARG;
  if (!r->bound) return FB_ERR_STATE;
  const fb_draft_desc& d = r->d;
  if (T < 1 || T > d.max_tokens || (!d_slots && T > d.max_roll)) return FB_ERR_RANGE;
  if (((uintptr_t)d_feat & 15) || ((uintptr_t)d_emb & 15) || ((uintptr_t)d_out & 1)) return FB_ERR_ARG;
  DeviceGuard g(r->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int D = d.dim, F = d.fuse * d.dim, hd = D / d.n_head, kvd = d.n_kv_head * hd;
  DLin p;
  // x = merge(cat(feat, emb))
  memset(&p, 0, sizeof(p));
  p.W[0] = (const uint16_t*)r->w.merge; p.x0 = (const uint16_t*)d_feat; p.ldx0 = F; p.k0 = F;
  if (d_emb) { p.x1 = (const uint16_t*)d_emb; p.ldx1 = D; }
  else { p.x1 = (const uint16_t*)r->w.embed; p.ldx1 = D; p.x1_tokens = d_tokens; p.x1_rows = d.vocab; }
  p.k1 = D; p.N[0] = D; p.T = T; p.y[0] = r->x; p.ldy[0] = D; p.first = true;
  FB_DCUDA(r, launch_linear<DL_STORE>(p, r->sm_count, st));
  const bool fold = draft_folds_norm(T, D);
  if (!fold) FB_DCUDA(r, launch_norm(r->x, D, r->w.n1, r->h, T, D, d.rms_eps, false, st));
  // q, k, v in one launch
  memset(&p, 0, sizeof(p));
  const void* qkvw[3] = {r->w.q, r->w.k, r->w.v};
  uint16_t* qkvo[3] = {r->q, r->k, r->v};
  const int qkvn[3] = {D, kvd, kvd};
  for (int i = 0; i < 3; i++) { p.W[i] = (const uint16_t*)qkvw[i]; p.N[i] = qkvn[i]; p.y[i] = qkvo[i]; p.ldy[i] = qkvn[i]; }
  p.x0 = fold ? r->x : r->h; p.ldx0 = D; p.k0 = D; p.T = T; p.norm_w = fold ? (const uint16_t*)r->w.n1 : nullptr; p.norm_eps = d.rms_eps;
  FB_DCUDA(r, launch_linear<DL_STORE>(p, r->sm_count, st));
  const size_t asmem = (size_t)(d.max_roll + hd) * 4, news = (size_t)hd * 8;
  if (T == 1 && news <= kAttnSmemNew && asmem <= kAttnSmem) {
    FB_DCUDA(r, launch_pdl(d_attn_one, dim3(d.n_head), dim3(128), asmem + news, st, (const uint16_t*)r->q, (const uint16_t*)r->k, (const uint16_t*)r->v,
                           d_positions, d_slots, r->kc, r->vc, r->att, d.n_head, d.n_kv_head, hd, d.rope_base, d.max_roll));
  } else {
    FB_DCUDA(r, launch_pdl(d_rope_store, dim3(T, d.n_head + d.n_kv_head), dim3(64), 0, st, r->q, (const uint16_t*)r->k, (const uint16_t*)r->v, d_positions,
                           d_slots, r->kc, r->vc, d.n_head, d.n_kv_head, hd, d.rope_base, d.max_roll));
    FB_DCUDA(r, launch_pdl(d_attn, dim3(T, d.n_head), dim3(128), asmem, st, (const uint16_t*)r->q, d_slots, (const uint16_t*)r->kc,
                           (const uint16_t*)r->vc, r->att, d.n_head, d.n_kv_head, hd, d.max_roll));
  }
  // x2 = x + o(att)
  memset(&p, 0, sizeof(p));
  p.W[0] = (const uint16_t*)r->w.o; p.x0 = r->att; p.ldx0 = D; p.k0 = D; p.N[0] = D; p.T = T; p.y[0] = r->x2; p.ldy[0] = D;
  p.resid = r->x; p.ldr = D;
  FB_DCUDA(r, launch_linear<DL_RESID>(p, r->sm_count, st));
  if (!fold) FB_DCUDA(r, launch_norm(r->x2, D, r->w.n2, r->h, T, D, d.rms_eps, false, st));
  // act = silu(gate h) * up h
  memset(&p, 0, sizeof(p));
  p.W[0] = (const uint16_t*)r->w.gate; p.W2 = (const uint16_t*)r->w.up; p.x0 = fold ? r->x2 : r->h; p.ldx0 = D;
  p.norm_w = fold ? (const uint16_t*)r->w.n2 : nullptr; p.norm_eps = d.rms_eps; p.k0 = D; p.N[0] = d.inter; p.T = T;
  p.y[0] = r->act; p.ldy[0] = d.inter;
  FB_DCUDA(r, launch_linear<DL_SWIGLU>(p, r->sm_count, st));
  // hh = x2 + down(act)
  memset(&p, 0, sizeof(p));
  p.W[0] = (const uint16_t*)r->w.down; p.x0 = r->act; p.ldx0 = d.inter; p.k0 = d.inter; p.N[0] = D; p.T = T; p.y[0] = r->hh; p.ldy[0] = D;
  p.resid = r->x2; p.ldr = D;
  FB_DCUDA(r, launch_linear<DL_RESID>(p, r->sm_count, st));
  // out = fout(hh)
  memset(&p, 0, sizeof(p));
  p.W[0] = (const uint16_t*)r->w.fout; p.x0 = r->hh; p.ldx0 = D; p.k0 = D; p.N[0] = F; p.T = T; p.y[0] = (uint16_t*)d_out; p.ldy[0] = F;
  FB_DCUDA(r, launch_linear<DL_STORE>(p, r->sm_count, st));
  FB_DCUDA(r, cudaGetLastError());
  return FB_OK;
}

int fb_draft_head(fb_draft* r, const void* d_feat_rows, int32_t n, int32_t top_b, int32_t* d_tokens, float* d_scores,
                  void* stream) {
  if (!r || !d_feat_rows || !d_tokens) return FB_ERR_ARG;
  if (!r->bound) return FB_ERR_STATE;
  const fb_draft_desc& d = r->d;
  if (n < 1 || n > kMaxHeadRows || top_b < 1 || top_b > 16 || top_b > d.vocab) return FB_ERR_RANGE;
  DeviceGuard g(r->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int D = d.dim, F = d.fuse * d.dim;
  // the token head reads the HIGH slice (last dim elements) of the fused feature (reference: spec_mega.py:43-44)
  const uint16_t* rows = (const uint16_t*)d_feat_rows + (F - D);
  FB_DCUDA(r, launch_norm(rows, F, r->w.nf, r->fn, n, D, d.rms_eps, true, st));
  DLin p;
  memset(&p, 0, sizeof(p));
  p.W[0] = (const uint16_t*)r->w.embed; p.x0 = r->fn; p.ldx0 = D; p.k0 = D; p.N[0] = d.vocab; p.T = n; p.yf = r->logits; p.ldy[0] = d.vocab;
  p.scale = d.logits_scaling;
  FB_DCUDA(r, launch_linear<DL_LOGITS>(p, r->sm_count, st));
  const int nc = row_ctas(d.vocab);
  const bool reg = (d.vocab + nc - 1) / nc <= kSampleRegs * 1024;
  FB_DCUDA(r, launch_pdl_cluster(reg ? topb_rows<true> : topb_rows<false>, dim3(nc, n), dim3(1024), 0, st, nc, (const float*)r->logits,
                                 (long long)d.vocab, d.vocab, top_b, d_tokens, d_scores));
  FB_DCUDA(r, cudaGetLastError());
  return FB_OK;
}

}  // extern "C"
