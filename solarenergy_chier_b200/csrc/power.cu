// Per-heliostat FP64 power of a trace launch, summed with compensation and
// in a fixed order.
//
// The tracer's warps write one FP64 partial per warp chunk (the sum of its
// rays' energies: per-lane sums of at most 64 float energies, exact in
// double for the magnitudes of one heliostat, then a warp shuffle tree) to
// TraceParams::chunk_power.  This kernel adds each task's partials, one warp
// or one block of 8 warps per task: every lane runs a Neumaier-compensated
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

// A task's partials are a chain of loads and dependent adds per lane, so the
// kernel's time is its longest chain: kWarps = 8 shortens it for tasks of
// many chunks, where a warp alone would take hundreds of steps.
template <int kWarps>
__global__ void __launch_bounds__(128 * (kWarps > 4 ? kWarps / 4 : 1)) power_reduce_kernel(TraceParams p) {
  __shared__ double part[kWarps][2];
  const int lane = threadIdx.x & 31, warp = kWarps > 1 ? threadIdx.x >> 5 : 0;
  const long long t = kWarps > 1 ? blockIdx.x : ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= p.num_tasks) return;
  const long long c0 = max(__ldg(p.facet_prefix + t), p.chunk_begin);
  const long long c1 = min(__ldg(p.facet_prefix + t + 1), p.total_facets);
  if (c1 <= c0) return;  // the same for all of the task's warps
  const double* __restrict__ in = p.chunk_power - p.chunk_begin;
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

cudaError_t launch_power_reduce(const TraceParams& p, cudaStream_t stream) {
  if (!p.chunk_power || p.num_tasks <= 0) return cudaSuccess;
  // 8 warps per task from 256 chunks a task on: one step per lane (a lone
  // heliostat of 1,600 chunks: 50 steps of a warp or 7 of 8 warps).
  if ((p.total_facets - p.chunk_begin) / p.num_tasks >= 256) {
    power_reduce_kernel<8><<<(unsigned)p.num_tasks, 256, 0, stream>>>(p);
  } else {
    const int threads = 128;
    const long long blocks = ((long long)p.num_tasks * 32 + threads - 1) / threads;
    power_reduce_kernel<1><<<(unsigned)blocks, threads, 0, stream>>>(p);
  }
  return cudaGetLastError();
}

}  // namespace qm
