// Sample pools and per-facet pool offsets, generated on the device.
//
// The reference draws both pools from cuRAND XORWOW seeded with time(NULL)
// (Scene/SceneProcessor.cu:147-271, Tool/RandomNumberGenerator/).  Here they
// come from the scrambled Sobol streams of sampling.h, so a seed reproduces
// a pool exactly; the mapping from uniforms to directions follows the
// reference.
#include "pools.h"
#include "device_scene.h"
#include "sampling.h"
#include "vecmath.h"

namespace qm {
namespace {

// samplelights::max_less_index (Scene/SceneProcessor.cu:46-59).
__device__ __forceinline__ int max_less_index(const float2* cdf, float value, int n) {
  int left = 0, right = n;
  while (left <= right) {
    int mid = (left + right) >> 1;
    float y = cdf[mid].y;
    if (value > y)
      left = mid + 1;
    else if (value < y)
      right = mid - 1;
    else
      return mid;
  }
  return right;
}

// samplelights::linear_interpolation (Scene/SceneProcessor.cu:61-81): the
// reference's Buie inverse CDF, including its arctangent warp of the core
// and its tail formula that lands at >= 9.3 mrad.
__device__ __forceinline__ float buie_theta(float uniform, const BuieTable& b) {
  float u = uniform * b.A;
  if (u < b.less_465) {
    int id = max_less_index(b.cdf, u, b.n);
    u = (u - b.cdf[id].y) * b.k[id] + b.cdf[id].x;
    u = atanf(sqrtf(u / 4.65f) * 0.5016916f);
  } else {
    u = powf((u - b.less_465) * b.B + b.C, 1 / (b.gamma + 1));
    float ri2 = 0.5016916f * 0.5016916f;
    float ro2 = 1.340874f * 1.340874f;
    u = atanf(sqrtf(ro2 + (u - 4.65f) / 4.65f * (ro2 - ri2)));
  }
  return u / 100.0f;
}

__global__ void pool_kernel(PoolParams p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.pool_size) return;
  uint32_t a, b;
  sobol2_owen((uint32_t)i, p.seed_sun, a, b);
  float3 s;
  if (p.sunshape == kSunshapePillbox) {
    // Uniform over the disc of half-angle h: cos(theta) uniform in [cos h, 1].
    double th = 2.0 * asin(sqrt(unit_open(a)) * sin(0.5 * (double)p.half_angle));
    double ph = 2.0 * M_PI * unit_open(b);
    s = make_float3((float)(sin(th) * cos(ph)), (float)cos(th), (float)(sin(th) * sin(ph)));
  } else {
    // samplelights::map_angle2xyz (Scene/SceneProcessor.cu:95-103) with the
    // reference's float constants.
    float theta = buie_theta(unit_float(a), p.buie);
    float phi = unit_float(b) * 2 * 3.141592654f;
    s = make_float3(sinf(theta) * cosf(phi), cosf(theta), sinf(theta) * sinf(phi));
  }
  p.samples[i] = make_float4(s.x, s.y, s.z, 0.0f);

  // Slope error: samplelights::map_permuation (Scene/SceneProcessor.cu:83-93),
  // normalize(N(0, sigma), 1, N(0, sigma)), Gaussians by Box-Muller.
  sobol2_owen((uint32_t)i, p.seed_slope, a, b);
  double r = sqrt(-2.0 * log(unit_open(a)));
  double w = 2.0 * M_PI * unit_open(b);
  float3 d = make_float3((float)((double)p.sigma * r * cos(w)), 1.0f, (float)((double)p.sigma * r * sin(w)));
  d = normalize(d);
  p.perturbations[i] = make_float4(d.x, d.y, d.z, 0.0f);
}

// Facet offsets of every heliostat in one launch: element i of the buffer
// belongs to heliostat h with seg[h] <= i < seg[h + 1].
__global__ void offsets_all_kernel(int* out, const long long* seg, int heliostats, uint32_t seed, int pool) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= seg[heliostats]) return;
  int lo = 0, hi = heliostats - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (seg[mid] <= i) lo = mid; else hi = mid - 1;
  }
  out[i] = facet_offset(seed, (uint32_t)lo, (uint32_t)(i - seg[lo]), (uint32_t)pool);
}

// The pools as the tracer reads them: n_out = P + L entries, entry i holding
// pool entry i % P, so that offset + light index never wraps; sun-shape
// samples turned into world space by the sun frame, exactly as the reference
// turns each one per ray (local2world_rotate of the sample about
// -sun_direction, RectangleReceiverRectangleGridRayTracing.cu:16).
__global__ void trace_pools_kernel(const float4* in, const float4* pert, int n, int n_out, SunFrame sun, float4* out,
                                   float4* pert_out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_out) return;
  const int k = i % n;
  pert_out[i] = pert[k];
  float3 d = make_float3(in[k].x, in[k].y, in[k].z);
  if (!sun.identity) {
    Frame f;
    f.u = sun.u;
    f.n = sun.n;
    f.v = sun.v;
    f.identity = false;
    d = qs::to_world(f, d);
  }
  out[i] = make_float4(d.x, d.y, d.z, 0.0f);
}

// Both pools' checks and bounds in one pass: vectors whose squared length
// lies outside [0.25, 4] or is NaN, and the largest tan(angle from +y) of each
// pool as float bits (non-negative floats order like their bit patterns); +inf
// when some direction has y <= 0.
// Reduced per block: an atomic per warp made two words' 16,384 maxima the
// kernel's time (12 us for 262,144 vectors, 3 so).
__global__ void __launch_bounds__(256) pool_stats_kernel(const float* dirs, const float* perts, int stride, int n,
                                                         PoolStats* out) {
  __shared__ unsigned found[3];  // bad, tan bits
  if (threadIdx.x < 3) found[threadIdx.x] = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned bad = 0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    float t = 0.0f;
    if (i < n) {
      const float* v = (k ? perts : dirs) + (size_t)stride * i;
      const float x = v[0], y = v[1], z = v[2];
      const float s = x * x + y * y + z * z;
      bad += !(s >= 0.25f && s <= 4.0f);
      t = y > 0.0f ? sqrtf(x * x + z * z) / y : __int_as_float(0x7f800000);
    }
    const unsigned most = __reduce_max_sync(0xffffffffu, __float_as_uint(t));
    if ((threadIdx.x & 31) == 0) atomicMax(found + 1 + k, most);
  }
  bad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(found, bad);
  __syncthreads();
  if (threadIdx.x == 0 && found[0]) atomicAdd(&out->bad, found[0]);
  if (threadIdx.x < 2) atomicMax(out->tan_bits + threadIdx.x, found[1 + threadIdx.x]);
}

__global__ void xyz_to_float4_kernel(const float* xyz, float4* out, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 0.0f);
}

}  // namespace

cudaError_t launch_pool(const PoolParams& p, cudaStream_t stream) {
  if (p.pool_size <= 0) return cudaSuccess;
  pool_kernel<<<(p.pool_size + 255) / 256, 256, 0, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_offsets_all(int* out, const long long* seg, int heliostats, long long total, uint32_t seed, int pool,
                               cudaStream_t stream) {
  if (total <= 0 || heliostats <= 0) return cudaSuccess;
  offsets_all_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(out, seg, heliostats, seed, pool);
  return cudaGetLastError();
}

cudaError_t launch_trace_pools(const float4* samples, const float4* perturbations, int n, int n_out,
                               const SunFrame& sun, float4* out, float4* pert_out, cudaStream_t stream) {
  if (n <= 0 || n_out <= 0) return cudaSuccess;
  trace_pools_kernel<<<(n_out + 255) / 256, 256, 0, stream>>>(samples, perturbations, n, n_out, sun, out, pert_out);
  return cudaGetLastError();
}

cudaError_t launch_pool_stats(const float* dirs, const float* perts, int stride, int n, PoolStats* out,
                              cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  pool_stats_kernel<<<(n + 255) / 256, 256, 0, stream>>>(dirs, perts, stride, n, out);
  return cudaGetLastError();
}

cudaError_t launch_xyz_to_float4(const float* xyz, float4* out, int n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  xyz_to_float4_kernel<<<(n + 255) / 256, 256, 0, stream>>>(xyz, out, n);
  return cudaGetLastError();
}

}  // namespace qm
