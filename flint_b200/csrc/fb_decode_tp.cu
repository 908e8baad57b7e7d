// The decode kernels of tensor-parallel ranks, apart from those of a single GPU: a translation unit of its own, so that both compile side by side.
#include "fb_ctx.hpp"
#include "fb_decode.cuh"

using namespace fb;

namespace {
#define FB_DECODE_ENTRY(KD, KO, KF, HD, R) \
  (const void*)decode_mega2<KD, KO, KF, HD, R, false, true>, (const void*)decode_mega2<KD, KO, KF, HD, R, true, true>
const void* const kTpKernels[] = {
#include "fb_decode_shapes.h"
};
}  // namespace

const void* decode_tp_kernel(int id) { return kTpKernels[id]; }
