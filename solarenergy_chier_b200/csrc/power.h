// Compensated, fixed-order per-heliostat FP64 power of a trace launch
// (power.cu): adds the per-chunk partials the tracer wrote to
// TraceParams::chunk_power into TraceParams::power.
#pragma once

#include <cuda_runtime.h>

#include "device_scene.h"

namespace qm {
// An image deposited through a spread one, where pixel i is at i * step and
// which holds zeros between launches.
struct SpreadImage {
  float* image = nullptr;
  float* spread = nullptr;
  int pixels = 0, step = 0;
};
constexpr int kMaxSpreadImages = 4;
struct SpreadImages {
  int n = 0;
  SpreadImage at[kMaxSpreadImages];
};
// The end of a trace launch: the power sums, and the spread images added to
// theirs.
cudaError_t launch_trace_end(const TraceParams& p, const SpreadImages& images, cudaStream_t stream);
}  // namespace qm
