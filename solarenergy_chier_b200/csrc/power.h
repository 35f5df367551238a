// Compensated, fixed-order per-heliostat FP64 power of a trace launch
// (power.cu): adds the per-chunk partials the tracer wrote to
// TraceParams::chunk_power into TraceParams::power.
#pragma once

#include <cuda_runtime.h>

#include "device_scene.h"

namespace qm {
// Images deposited through copies (DevReceiver::copy_mask): each copy's pixels
// are added to the image and left zero.
struct CopiedImage {
  float* image;
  float* copies;  // `copies_n` of them, `stride` floats apart
  int pixels, copies_n, stride;
};
constexpr int kMaxCopiedImages = 4;
struct CopiedImages {
  int n = 0;
  CopiedImage at[kMaxCopiedImages];
};
// The end of a trace launch: the power sums, and the copied images' merge.
cudaError_t launch_trace_end(const TraceParams& p, const CopiedImages& images, cudaStream_t stream);
}  // namespace qm
