// M-token passes: tree verification (EAGLE) and prompts. Every weight row is read once and applied to all M tokens; a short sequence
// of kernels per layer on one stream, graph-capturable. This file: what the kernels share (GEMMs: fb_vtc.cuh, fb_vtl.cuh; attention:
// fb_vattn.cuh).
#pragma once
#include "fb_common.cuh"

namespace fb {

enum { EPI_QKV = 0, EPI_RESID = 1, EPI_SWIGLU = 2, EPI_LOGITS = 3 };

// the power of two that brings a bound `a` on some magnitudes into [2^14, 2^15), and its inverse (both finite for every a >= 0)
__device__ __forceinline__ float2 pow2_for(float a) {
  uint32_t mf = 268u - ((__float_as_uint(a) >> 23) & 255u);
  mf = mf > 253u ? 253u : (mf < 24u ? 24u : mf);
  return make_float2(__uint_as_float(mf << 23), __uint_as_float((254u - mf) << 23));
}

// h[m] = bf16(float(embed[token[m]]) * mult), or a copy of the caller's residual rows
__global__ void v_embed(const int32_t* tokens, const uint16_t* embed, const uint16_t* h_in, uint16_t* h, int D, int vocab,
                        float mult, int* status_code) {
  const int m = blockIdx.x;
  pdl_begin(true);
  int tok = 0;
  if (!h_in) {
    tok = tokens[m];
    if ((unsigned)tok >= (unsigned)vocab) { tok = 0; if (threadIdx.x == 0) atomicCAS(status_code, 0, 6); }
  }
  for (int i = threadIdx.x; i < D; i += blockDim.x)
    h[(size_t)m * D + i] = h_in ? h_in[(size_t)m * D + i] : f2bf(bf2f(embed[(size_t)tok * D + i]) * mult);
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

}  // namespace fb
