// Trimmed-mean smoother (Tool/Smoother/ImageSmoother.cu:13-113, heaps in
// Tool/Smoother/heap.cuh:16-225).
//
// Each output pixel is the mean of its (2r+1)^2 window clipped to the image,
// after dropping k = int(count * ratio) values at each end, where the k
// smallest and k largest are tracked by the reference's streaming max- and
// min-heaps in the reference's visiting order (row by row).  The heap
// updates and the summation order are kept, so the float result matches the
// reference's kernel, including the cases where its streaming selection
// differs from a sorted trim (k >= 2 with some value orders).
//
// The reference reads a texture copy of the image and writes in place.  Here
// windows that trim at most 15 values at each end are smoothed in place
// from tiles held in shared memory while the image fits there; otherwise the
// kernel reads an explicit copy (`src`) and writes `dst`.
#include "smooth.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <type_traits>

namespace qm {
namespace {

// heap.cuh's array heap, 1-based, comparator `larger` (max-heap) or
// `smaller` (min-heap).
template <bool kMax>
struct ArrayHeap {
  float* e;
  int num;  // next free slot (1 when empty)
  int cap;  // size + 1
  __device__ __forceinline__ static bool cmp(float a, float b) { return kMax ? a > b : a < b; }
  __device__ __forceinline__ bool full() const { return num == cap; }
  __device__ __forceinline__ bool empty() const { return num == 1; }
  __device__ __forceinline__ float top() const { return empty() ? 0.0f : e[1]; }
  __device__ __forceinline__ void insert(float x) {
    if (full()) return;
    int i = num++;
    for (; i != 1 && cmp(x, e[i / 2]); i /= 2) e[i] = e[i / 2];
    e[i] = x;
  }
  __device__ __forceinline__ void replace_top(float x) {
    if (empty()) return;
    int i = 1;
    while (2 * i < num) {
      int c = (2 * i + 1 >= num || cmp(e[2 * i], e[2 * i + 1])) ? 2 * i : 2 * i + 1;
      if (cmp(e[c], x)) {
        e[i] = e[c];
        i = c;
      } else {
        break;
      }
    }
    e[i] = x;
  }
  __device__ __forceinline__ float sum() const {
    float s = 0.0f;
    for (int i = 1; i < num; ++i) s += e[i];
    return s;
  }
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// The same two heaps with every element in a register (K >= k elements, known
// when compiled).  `sgn` folds both kinds into one: the min-heap holds negated
// values, so element order, comparisons and moves mirror the max-heap's.
// Slots above k hold -inf: they lose every comparison against a real child
// and never change, so a thread at the image's border keeps its smaller heap.
template <int K>
struct RegisterHeap {
  float e[K + 1];  // e[1..K]
  __device__ __forceinline__ RegisterHeap() {
#pragma unroll
    for (int i = 0; i <= K; ++i) e[i] = -INFINITY;
  }
  __device__ __forceinline__ float top() const { return e[1]; }
  // Sift-up of x appended as element J (ArrayHeap::insert).
  template <int J>
  __device__ __forceinline__ void insert_at(float x) {
    if constexpr (J == 1) {
      e[1] = x;
    } else if (x > e[J / 2]) {
      e[J] = e[J / 2];
      insert_at<J / 2>(x);
    } else {
      e[J] = x;
    }
  }
  template <int J = 1>
  __device__ __forceinline__ void insert(float x, int j) {
    if constexpr (J <= K) {
      if (j == J) insert_at<J>(x);
      else insert<J + 1>(x, j);
    }
  }
  // ArrayHeap::replace_top without a branch, for any x (x >= top changes
  // nothing): below a node on x's path, where x < e[I], the node takes the
  // larger of its larger child and x, and x goes on into that child -- also
  // when it stops here, since then it is not below that child and every
  // min() further down leaves its element.
  template <int I = 1>
  __device__ __forceinline__ void replace_top(float x, bool on = true) {
    if constexpr (2 * I + 1 <= K) {
      const bool left = e[2 * I] > e[2 * I + 1];
      const float m = max3(e[2 * I], e[2 * I + 1], x);
      if (on) e[I] = fminf(e[I], m);
      replace_top<2 * I>(x, on && left);
      replace_top<2 * I + 1>(x, on && !left);
    } else if constexpr (2 * I <= K) {
      if (on) e[I] = fminf(e[I], fmaxf(e[2 * I], x));
      if (on) e[2 * I] = fminf(e[2 * I], x);
    } else if constexpr (I <= K) {
      if (on) e[I] = fminf(e[I], x);
    }
  }
  // The first k elements, in ArrayHeap::sum's order; sgn -1 for the min-heap.
  __device__ __forceinline__ float sum(int k, float sgn) const {
    float s = 0.0f;
#pragma unroll
    for (int i = 1; i <= K; ++i) s += i <= k ? sgn * e[i] : 0.0f;
    return s;
  }
};

constexpr int kTileX = 32, kTileY = 8;  // a warp is one row of 32 pixels

// Trimmed mean with both heaps in registers, for at most K trimmed values at
// each end.  Bound by the min/max and compare rate (64 lanes a cycle per SM,
// half the FMA rate): about 2.3 operations per heap element per window value.
// The heaps are updated without branches, as on lit pixels some lane of a
// warp replaces a value at almost every tap (heaps in shared memory, walked
// with dynamic indexes, spent their time on that divergence); where no lane
// does (dark or constant regions), a vote skips both.  A 1257 x 600 flux map
// with an 11 x 11 window and 6 values trimmed at each end: 300 -> 165 us (its
// min/max, compares and selects alone take about 135 us at that rate).
//
// Block b computes tiles b, b + gridDim.x, ...  In place (src == dst, a
// cooperative launch), every block first loads all its tiles with their
// halos and the grid waits for that once, so the image needs no copy and no
// scratch memory; otherwise src is a copy and the grid has a block per tile.
template <int K, bool kInPlace>
__global__ void __launch_bounds__(kTileX* kTileY, K <= 7 ? 6 : 4)
    trimmed_mean_register_kernel(const float* src, float* dst, int radius, float ratio, int width, int height,
                                 int tiles_x, int tiles) {
  extern __shared__ float held_tiles[];  // each (kTileY + 2 radius) rows of kTileX + 2 radius values
  const int tw = kTileX + 2 * radius, th = kTileY + 2 * radius;
  float* tile = held_tiles;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x, tile += tw * th) {
    const int bx = t % tiles_x * kTileX - radius, by = t / tiles_x * kTileY - radius;
    for (int i = threadIdx.y * kTileX + threadIdx.x; i < tw * th; i += kTileX * kTileY) {
      const int c = bx + i % tw, r = by + i / tw;
      const bool in = (unsigned)c < (unsigned)width && (unsigned)r < (unsigned)height;
      tile[i] = in ? src[(size_t)r * width + c] : 0.0f;
    }
  }
  if constexpr (kInPlace) cooperative_groups::this_grid().sync();
  else __syncthreads();
  tile = held_tiles;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x, tile += tw * th) {
    const int x = t % tiles_x * kTileX + threadIdx.x, y = t / tiles_x * kTileY + threadIdx.y;
    if (y >= height) continue;  // a whole warp
    const bool inside = x < width;
    // Columns of the window inside the image, as offsets from the window's
    // left end; none for a lane beyond the image.
    const int c0 = max(radius - x, 0);
    const int span = inside ? min(x + radius, width - 1) - max(x - radius, 0) + 1 : 0;
    const int r0 = max(y - radius, 0), r1 = min(y + radius, height - 1);
    const int cnt = span * (r1 - r0 + 1);
    const int k = cnt * ratio;
    RegisterHeap<K> lo, hi;  // the k smallest, the k largest (negated)
    float value = 0.0f;
    int held = 0;          // values in each heap, while they fill
    bool filling = K > 0;  // warp-uniform
    auto taps = [&](auto whole) {  // whole: every lane's window lies inside the image's columns
      for (int r = r0; r <= r1; ++r) {
        const float* row = tile + (r - (y - (int)threadIdx.y) + radius) * tw + threadIdx.x;
        for (int c = 0; c <= 2 * radius; ++c) {
          const bool ok = decltype(whole)::value || (unsigned)(c - c0) < (unsigned)span;
          const float cur = row[c];
          value += ok ? cur : 0.0f;
          if constexpr (K > 0) {
            const bool low = cur < lo.top();
            if (filling) {
              if (ok && held < k) {
                ++held;
                lo.insert(cur, held);
                hi.insert(-cur, held);
              } else if (ok) {
                lo.replace_top(cur);
                hi.replace_top(low ? INFINITY : -cur);
              }
              filling = __any_sync(0xffffffffu, held < k);
              continue;
            }
            if (!__any_sync(0xffffffffu, ok && (low || -cur < hi.top()))) continue;
            lo.replace_top(ok ? cur : INFINITY);
            hi.replace_top(ok && !low ? -cur : INFINITY);
          }
        }
      }
    };
    if (__all_sync(0xffffffffu, span == 2 * radius + 1)) taps(std::true_type{});
    else taps(std::false_type{});
    if (inside) dst[(size_t)y * width + x] = (value - lo.sum(k, 1.0f) - hi.sum(k, -1.0f)) / float(cnt - 2 * k);
  }
}

__global__ void trimmed_mean_kernel(const float* __restrict__ src, float* __restrict__ dst, int radius, float ratio,
                                    int width, int height, int heap_stride) {
  extern __shared__ float heaps[];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x > width - 1 || y > height - 1) return;
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int x0 = (x - radius >= 0) ? x - radius : 0;
  const int y0 = (y - radius >= 0) ? y - radius : 0;
  const int x1 = (x + radius < width) ? x + radius : width - 1;
  const int y1 = (y + radius < height) ? y + radius : height - 1;
  const int cnt = (x1 - x0 + 1) * (y1 - y0 + 1);
  const int k = cnt * ratio;
  ArrayHeap<true> lo{heaps + (size_t)(2 * tid) * heap_stride, 1, k + 1};
  ArrayHeap<false> hi{heaps + (size_t)(2 * tid + 1) * heap_stride, 1, k + 1};
  float value = 0.0f;
  for (int r = y0; r <= y1; ++r) {
    for (int c = x0; c <= x1; ++c) {
      const float cur = __ldg(src + (size_t)r * width + c);
      value += cur;
      if (!lo.full()) {
        lo.insert(cur);
        hi.insert(cur);
      } else if (cur < lo.top()) {
        lo.replace_top(cur);
      } else if (cur > hi.top()) {
        hi.replace_top(cur);
      }
    }
  }
  dst[(size_t)y * width + x] = (value - lo.sum() - hi.sum()) / float(cnt - 2 * k);
}

}  // namespace

int smooth_heap_stride(int radius, float ratio) {
  return (2 * radius + 1) * (2 * radius + 1) * ratio + 1;
}

namespace {

// Largest trim that keeps both heaps in registers.
constexpr int kMaxRegisterTrim = 15;

constexpr size_t kMaxShared = 227 * 1024;  // of a block, and of an SM's blocks together

// Lets a kernel's launches use `smem` bytes of shared memory.  The limit is the
// kernel's, for all host threads: always the largest one, so that no thread
// lowers it between another's call here and its launch.
cudaError_t allow_shared(const void* kernel, size_t smem) {
  return smem <= 48 * 1024 ? cudaSuccess
                           : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxShared);
}

struct RegisterLaunch {
  float* image;      // in place when src is NULL
  const float* src;  // else a copy of the image
  int width, height, radius;
  float ratio;
  cudaStream_t stream;
};

template <int K, bool kInPlace>
cudaError_t start_register(RegisterLaunch a, int blocks, size_t smem, int tiles_x, int tiles) {
  auto kernel = trimmed_mean_register_kernel<K, kInPlace>;
  if constexpr (!kInPlace) {
    kernel<<<blocks, dim3(kTileX, kTileY), smem, a.stream>>>(a.src, a.image, a.radius, a.ratio, a.width, a.height,
                                                            tiles_x, tiles);
    return cudaGetLastError();
  } else {
    const float* src = a.image;
    void* args[] = {&src, &a.image, &a.radius, &a.ratio, &a.width, &a.height, &tiles_x, &tiles};
    return cudaLaunchCooperativeKernel((const void*)kernel, dim3(blocks), dim3(kTileX, kTileY), args, smem, a.stream);
  }
}

// cudaErrorNotSupported: the image's tiles do not fit the SMs' shared memory
// (or the device has no cooperative launch) and the caller must pass a copy.
template <int K, bool kInPlace>
cudaError_t launch_register(int trim, const RegisterLaunch& a) {
  if constexpr (K < kMaxRegisterTrim) {
    if (trim > K) return launch_register<K + 1, kInPlace>(trim, a);
  }
  const size_t tile_bytes = sizeof(float) * (kTileX + 2 * a.radius) * (kTileY + 2 * a.radius);
  const int tiles_x = (a.width + kTileX - 1) / kTileX;
  const long long tiles = (long long)tiles_x * ((a.height + kTileY - 1) / kTileY);
  if (tiles > INT_MAX) return cudaErrorNotSupported;
  const void* kernel = (const void*)trimmed_mean_register_kernel<K, kInPlace>;
  if constexpr (!kInPlace) {
    const cudaError_t e = allow_shared(kernel, tile_bytes);
    return e != cudaSuccess ? e : start_register<K, false>(a, (int)tiles, tile_bytes, tiles_x, (int)tiles);
  } else {
    int dev = 0, sms = 0, coop = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (e != cudaSuccess) return e;
    if (!coop || sms <= 0) return cudaErrorNotSupported;
    // The most resident blocks per SM whose share of the tiles fits beside
    // each other: the same number on every SM, so the tiles, dealt round,
    // differ by at most one per block.
    for (int want = 2048 / (kTileX * kTileY); want >= 1; --want) {
      const long long share = (tiles + (long long)sms * want - 1) / ((long long)sms * want);
      const size_t smem = tile_bytes * share;
      if (smem * want > kMaxShared) continue;
      e = allow_shared(kernel, smem);
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTileX * kTileY, smem);
      if (e != cudaSuccess) return e;
      if (per_sm < want) continue;
      return start_register<K, true>(a, (int)std::min<long long>(tiles, (long long)sms * want), smem, tiles_x,
                                     (int)tiles);
    }
    return cudaErrorNotSupported;
  }
}

}  // namespace

cudaError_t launch_trimmed_mean_in_place(float* image, int width, int height, int radius, float ratio,
                                         cudaStream_t stream) {
  const int trim = smooth_heap_stride(radius, ratio) - 1;  // at least every window's k
  if (trim > kMaxRegisterTrim) return cudaErrorNotSupported;
  const cudaError_t e = launch_register<0, true>(trim, RegisterLaunch{image, nullptr, width, height, radius, ratio, stream});
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();  // fewer SMs than the device reports are ours: smooth from a copy
    return cudaErrorNotSupported;
  }
  return e;
}

cudaError_t launch_trimmed_mean(const float* src, float* dst, int width, int height, int radius, float ratio,
                                cudaStream_t stream) {
  const int trim = smooth_heap_stride(radius, ratio) - 1;  // at least every window's k
  if (trim <= kMaxRegisterTrim) {
    const cudaError_t e =
        launch_register<0, false>(trim, RegisterLaunch{dst, src, width, height, radius, ratio, stream});
    if (e != cudaErrorNotSupported) return e;
  }
  const dim3 block(16, 16);
  const dim3 grid((width + block.x - 1) / block.x, (height + block.y - 1) / block.y);
  const int stride = smooth_heap_stride(radius, ratio);
  const size_t smem = sizeof(float) * (size_t)stride * 2 * block.x * block.y;
  if (smem > kMaxShared) return cudaErrorInvalidValue;
  const cudaError_t e = allow_shared((const void*)trimmed_mean_kernel, smem);
  if (e != cudaSuccess) return e;
  trimmed_mean_kernel<<<grid, block, smem, stream>>>(src, dst, radius, ratio, width, height, stride);
  return cudaGetLastError();
}

}  // namespace qm
