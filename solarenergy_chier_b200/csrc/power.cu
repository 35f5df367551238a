// Per-heliostat FP64 power of a trace launch, summed with compensation and
// in a fixed order.
//
// The tracer's warps write one FP64 partial per warp chunk (the sum of its
// rays' energies: per-lane sums of at most 64 float energies, exact in
// double for the magnitudes of one heliostat, then a warp shuffle tree) to
// TraceParams::chunk_power.  This kernel adds each task's partials, one warp
// or one block of 8 or 32 warps per task: every lane runs a Neumaier-compensated
// sum over a strided subset, the 32 (sum, compensation) pairs of a warp merge
// by error-free two-sums down a fixed shuffle tree, the warps' pairs likewise
// in warp order, and lane 0 adds the rounded result to the task's power slot.
// The order depends on the launch's chunks alone, never on scheduling, so a
// launch's per-heliostat powers are the same on every run, and the total
// error stays at the last bit of the double result instead of growing with
// the number of chunks, as one double atomic per chunk let it.
#include "device_scene.h"
#include "power.h"

namespace qm {
namespace {

__device__ __forceinline__ void neumaier(double& s, double& c, double x) {
  const double t = s + x;
  c += fabs(s) >= fabs(x) ? (s - t) + x : (x - t) + s;
  s = t;
}

// (s, c) += (s2, c2): s + s2 = sum + err exactly (two-sum).
__device__ __forceinline__ void merge(double& s, double& c, double s2, double c2) {
  const double sum = s + s2;
  const double bb = sum - s;
  c += c2 + ((s - (sum - bb)) + (s2 - bb));
  s = sum;
}

// Adds pixel i of the spread images to its image, where a caller's other
// streams may read or deposit at the same time.  A spread image belongs to
// launches of one stream at a time (see spread_images in capi.cpp).
__device__ __forceinline__ void add_spread(const SpreadImages& images, long long i) {
  for (int r = 0; r < images.n; ++r) {
    const SpreadImage& m = images.at[r];
    if (i >= m.pixels) {
      i -= m.pixels;
      continue;
    }
    float* wide = m.spread + i * m.step;
    const float v = __ldcg(wide);
    if (v != 0.0f) {
      *wide = 0.0f;
      atomicAdd(m.image + i, v);
    }
    return;
  }
}

long long pixels_of(const SpreadImages& images) {
  long long pixels = 0;
  for (int r = 0; r < images.n; ++r) pixels += images.at[r].pixels;
  return pixels;
}

// A task's partials are a chain of loads and dependent adds per lane, so the
// kernel's time is its longest chain: 8 or 32 warps shorten it for tasks of
// many chunks, where a warp alone would take hundreds of steps.  Blocks from
// power_blocks on add the spread images, in the same launch.
template <int kWarps>
__global__ void __launch_bounds__(kWarps > 4 ? 32 * kWarps : 128)
    power_reduce_kernel(TraceParams p, SpreadImages images, int power_blocks) {
  __shared__ double part[kWarps][2];
  wait_previous();
  begin_next();
  if ((int)blockIdx.x >= power_blocks) {
    add_spread(images, (long long)(blockIdx.x - power_blocks) * blockDim.x + threadIdx.x);
    return;
  }
  const int lane = threadIdx.x & 31, warp = kWarps > 1 ? threadIdx.x >> 5 : 0;
  const long long t = kWarps > 1 ? blockIdx.x : ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= p.num_tasks) return;
  const long long c0 = max(__ldg(p.facet_prefix + t), p.chunk_begin);
  const long long c1 = min(__ldg(p.facet_prefix + t + 1), p.total_facets);
  if (c1 <= c0) return;  // the same for all of the task's warps
  // Written by the launch that wait_previous waits for: not __restrict__, which
  // would let the compiler read it as data that no kernel changes, ahead of the wait.
  const double* in = p.chunk_power - p.chunk_begin;
  constexpr int kStride = 32 * kWarps;
  double s = 0.0, c = 0.0;
  long long k = c0 + (kWarps > 1 ? (int)threadIdx.x : lane);
  for (; k + 3 * kStride < c1; k += 4 * kStride) {
    const double x0 = in[k], x1 = in[k + kStride], x2 = in[k + 2 * kStride], x3 = in[k + 3 * kStride];
    neumaier(s, c, x0);
    neumaier(s, c, x1);
    neumaier(s, c, x2);
    neumaier(s, c, x3);
  }
  for (; k < c1; k += kStride) neumaier(s, c, in[k]);
  for (int off = 16; off > 0; off >>= 1)
    merge(s, c, __shfl_down_sync(0xffffffffu, s, off), __shfl_down_sync(0xffffffffu, c, off));
  if (kWarps > 1) {
    if (lane == 0) {
      part[warp][0] = s;
      part[warp][1] = c;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int w = 1; w < kWarps; ++w) merge(s, c, part[w][0], part[w][1]);
  }
  if (lane == 0) {
    const double v = s + c;
    if (v != 0.0) atomicAdd(p.power + p.tasks[t].power_slot, v);
  }
}

}  // namespace

cudaError_t launch_trace_end(const TraceParams& p, const SpreadImages& images, cudaStream_t stream) {
  const bool power = p.chunk_power && p.num_tasks > 0;
  const long long pixels = pixels_of(images);
  if (!power && pixels == 0) return cudaSuccess;
  // 8 warps per task from 256 chunks a task on (one step per lane), 32 from
  // 1,024: a lone heliostat of 6,400 chunks takes 7 steps of 32 warps, where 8
  // took 25 and a warp alone 200.
  const long long per_task = power ? (p.total_facets - p.chunk_begin) / p.num_tasks : 0;
  const int warps = per_task >= 1024 ? 32 : (per_task >= 256 ? 8 : 1);
  const int threads = warps > 1 ? 32 * warps : 128;
  const int power_blocks = !power ? 0 : (int)(warps > 1 ? p.num_tasks : ((long long)p.num_tasks * 32 + 127) / 128);
  const long long blocks = power_blocks + (pixels + threads - 1) / threads;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  switch (warps) {
    case 32: return launch_overlapped(power_reduce_kernel<32>, (unsigned)blocks, threads, stream, p, images, power_blocks);
    case 8: return launch_overlapped(power_reduce_kernel<8>, (unsigned)blocks, threads, stream, p, images, power_blocks);
    default: return launch_overlapped(power_reduce_kernel<1>, (unsigned)blocks, threads, stream, p, images, power_blocks);
  }
}

}  // namespace qm
