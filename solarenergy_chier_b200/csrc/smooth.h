#pragma once

#include <cuda_runtime.h>

namespace qm {

// Floats per heap per thread: int((2r+1)^2 * ratio) + 1, the reference's
// heap_size (Tool/Smoother/ImageSmoother.cu:103).
int smooth_heap_stride(int radius, float ratio);

// Trimmed mean of an image in place, without scratch memory.
// cudaErrorNotSupported (nothing launched): a window trims more than 15 values
// at each end, or the image does not fit the SMs' shared memory; then
// launch_trimmed_mean does it from a copy.
cudaError_t launch_trimmed_mean_in_place(float* image, int width, int height, int radius, float ratio,
                                         cudaStream_t stream);

// Trimmed mean of `src`, a copy of the image, into `dst`.
cudaError_t launch_trimmed_mean(const float* src, float* dst, int width, int height, int radius, float ratio,
                                cudaStream_t stream);

}  // namespace qm
