// Per-sun scene preparation on the device: for every (sun, heliostat) of a
// batch, the sun-dependent half of SceneProcessor::processScene
// (Scene/SceneProcessor.cpp:22-39): the heliostat normal
// (Heliostat::CSetNormal, Heliostat.cu:15-20), its corner / sub-heliostat
// parallelograms (Heliostat::CSetWorldVertex, Heliostat.cu:22-40;
// FocusFlatRectangleHelio::CGetSubHeliostatVertexes, FocusFlatRectangleHelio.cu:123-227),
// the traversal record and the tracer's facet frame; and the world-space
// sun-shape pool of every sun.
//
// The arithmetic is helio_geom.h's, shared with the host scene code; this
// unit is compiled with -fmad=false, so a heliostat prepared here equals the
// host's bit for bit.
#include "prep.h"

#include "helio_geom.h"
#include "ray_geom.h"
#include "shadow.h"

namespace qm {
namespace {

// A thread per heliostat, in blocks of one warp so that a few hundred
// heliostats still spread over the SMs: a chain of dependent double
// arithmetic per sub-heliostat, 16 us for 648 heliostats of 4, 86 us for 1,872
// of 28.  Moving a plain scene's sun here from the host (with its uploads)
// took a sun of 648 heliostats from 1.6 to 0.5 ms, its trace included.
__global__ void prep_kernel(PrepInputs p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  const PrepItem it = p.items[i];
  DevTask& T = p.tasks[it.task];
  const float4 offset = p.params ? p.params[it.param] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float3 aim = it.focus;
  if (offset.x != 0.0f || offset.y != 0.0f)
    aim = qs::add(qs::add(aim, qs::mul(it.aim_u, offset.x)), qs::mul(it.aim_v, offset.y));
  float3 normal = helio_normal(T.pos, aim, p.suns[it.sun].dir);
  if (offset.z != 0.0f || offset.w != 0.0f) {
    const Frame f0 = qs::make_frame(normal, false);
    normal = qs::normalize(qs::add(qs::add(normal, qs::mul(f0.u, offset.z)), qs::mul(f0.v, offset.w)));
  }
  T.normal = normal;
  const Frame hf = qs::make_frame(normal, T.type == 1);
  T.fu = hf.u;
  T.fn = hf.n;
  T.fv = hf.v;
  T.frame_identity = hf.identity ? 1 : 0;
  float3* v = it.verts;
  if (T.type == 0) {
    float3 c[4];
    flat_vertices(T.size, normal, T.pos, c);
    v[0] = c[0];
    v[1] = c[1];
    v[2] = c[2];
  } else {
    const float2 len = sub_lengths(T.size, T.gap, T.row_col);
    for (int s = 0; s < it.num_sub; ++s)
      focus_flat_sub_vertices(len, T.local_centers[s], T.local_normals[s], normal, T.pos, v + 3 * s);
  }
  for (int s = 0; s < it.num_sub; ++s) {
    const float3 B = v[3 * s], A = v[3 * s + 1], C = v[3 * s + 2];
    const float3 ab = qs::sub(B, A), ac = qs::sub(C, A);
    it.subv[3 * s] = make_float4(A.x, A.y, A.z, ab.x);
    it.subv[3 * s + 1] = make_float4(ab.y, ab.z, ac.x, ac.y);
    it.subv[3 * s + 2] = make_float4(ac.z, 0.f, 0.f, 0.f);
  }
  int2 rc;
  heliostat_record(v, it.num_sub, T.row_col, T.pos, normal, it.bound, &rc);
  *it.hsub = make_int4(it.sub_first, it.num_sub, rc.x, rc.y);
  // A box without a finite top (a heliostat whose aim lies exactly along the
  // sun's direction has no normal) must not lower the height at which the walks
  // of the others end: the NaN's key is the largest of all.
  const float4 *c = it.bound;
  const float top = c[0].y + fabsf(c[1].y) * c[1].w + fabsf(c[2].y) * c[2].w + fabsf(c[3].y) * c[3].w;
  atomicMax(it.top_key, height_key(isfinite(top) ? __float_as_int(top) : 0x7f800000));
}

// DevGrid::sub_free code of a warp_candidates result: 1 nothing to hit,
// k + 1 for k listed candidates, 0 walk (too many, or not enumerable).
__device__ __forceinline__ int candidate_code(int k) {
  return k == 0 ? 1 : (k > 0 && k <= kMaxCandidates ? k + 1 : 0);
}

// Code and candidate list of one cone (state: make_cone's result), by a whole
// warp; `cand` holds kMaxCandidates entries.
__device__ __forceinline__ int warp_code(const ShadowGrid& view, int own, int state, const Cone& cone, int* cand) {
  if (state < 0) return 0;
  if (state == 0) return 1;
  int found;
  const int k = warp_candidates(view, own, cone, kMaxCandidates, found);
  if (k <= kMaxCandidates && (int)(threadIdx.x & 31) < k) cand[threadIdx.x & 31] = found;
  return candidate_code(k);
}

__device__ __forceinline__ float3 sub_normal(const DevTask& T, int s) {
  Frame hf;
  hf.u = T.fu;
  hf.n = T.fn;
  hf.v = T.fv;
  hf.identity = T.frame_identity != 0;
  return T.type == 1 ? qs::to_world(hf, T.local_normals[s]) : T.normal;
}

// Walk codes of the prepared tasks: warp j handles task j / (1 + max_sub),
// slot j % (1 + max_sub): slot 0 its shadow walks, slot 1 + s the block
// walks of its sub-heliostat s (each a capsule enumeration of its own).
__global__ void shadow_kernel(PrepInputs p, int max_sub, const DevGrid* grids) {
  const long long j = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int i = (int)(j / (1 + max_sub)), slot = (int)(j % (1 + max_sub));
  if (i >= p.n) return;
  const PrepItem& it = p.items[i];
  const SunParams& sun = p.suns[it.sun];
  DevTask& T = p.tasks[it.task];
  const DevGrid& G = grids[T.grid];
  const ShadowGrid view{G.pos,       G.interval, G.cells, G.bound, G.cell_range, G.entries,
                        __int_as_float(height_key(G.top_key))};
  Cone cone;
  if (slot == 0) {
    const int state = sun.shadow_tan >= 0.0f ? shadow_cone(view, T.own, sun.shadow_axis, sun.shadow_tan, cone) : -1;
    const int code = warp_code(view, T.own, state, cone, T.shadow_cand);
    if (lane == 0) T.shadow_free = code;
    return;
  }
  const int s = slot - 1;
  if (s >= it.num_sub) return;
  if (lane == 0) sub_frames(T, s, it.sub_frames + 6 * s);
  const int state = sun.block_theta >= 0.0f
                        ? block_cone(view, it.verts + 3 * s, sun.dir, sub_normal(T, s), sun.block_theta, cone)
                        : -1;
  const int code = warp_code(view, T.own, state, cone, it.sub_cand + kMaxCandidates * s);
  if (lane == 0) it.sub_free[s] = code;
}

__global__ void gather_tasks_kernel(const DevTask* tasks, const int* ids, int n, DevTask* out) {
  constexpr int kWords = sizeof(DevTask) / 4;
  static_assert(sizeof(DevTask) % 4 == 0, "copied by words");
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(j / kWords), w = (int)(j % kWords);
  if (i < n) reinterpret_cast<int*>(out + i)[w] = reinterpret_cast<const int*>(tasks + ids[i])[w];
}

// Pool of instance blockIdx.y turned by that instance's sun frame.
__global__ void rotate_pools_kernel(const PoolRotation* jobs) {
  const PoolRotation J = jobs[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= J.n_out) return;
  const int k = i % J.n;
  float3 d = make_float3(J.in[k].x, J.in[k].y, J.in[k].z);
  if (!J.sun.identity) {
    Frame f;
    f.u = J.sun.u;
    f.n = J.sun.n;
    f.v = J.sun.v;
    f.identity = false;
    d = qs::to_world(f, d);
  }
  J.out[i] = make_float4(d.x, d.y, d.z, 0.0f);
}

}  // namespace

cudaError_t launch_prep(const PrepInputs& p, DevGrid* grids, int num_grids, cudaStream_t stream) {
  if (p.n <= 0) return cudaSuccess;
  static_assert(kNoHeight == (int)0x80808080, "set by bytes");
  const cudaError_t e = cudaMemset2DAsync(&grids->top_key, sizeof(DevGrid), 0x80, sizeof(int), num_grids, stream);
  if (e != cudaSuccess) return e;
  prep_kernel<<<(p.n + 31) / 32, 32, 0, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_shadow_flags(const PrepInputs& p, int max_sub, const DevGrid* grids, cudaStream_t stream) {
  if (p.n <= 0) return cudaSuccess;
  if (max_sub < 0) return cudaErrorInvalidValue;
  const long long warps = (long long)p.n * (1 + max_sub);
  const long long blocks = (warps + 3) / 4;  // four warps a block, a warp per cone
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  shadow_kernel<<<(unsigned)blocks, 128, 0, stream>>>(p, max_sub, grids);
  return cudaGetLastError();
}

cudaError_t launch_gather_tasks(const DevTask* tasks, const int* ids, int n, DevTask* out, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const long long words = (long long)n * (sizeof(DevTask) / 4);
  gather_tasks_kernel<<<(unsigned)((words + 255) / 256), 256, 0, stream>>>(tasks, ids, n, out);
  return cudaGetLastError();
}

cudaError_t launch_rotate_pools(const PoolRotation* jobs, int n_jobs, int max_out, cudaStream_t stream) {
  if (n_jobs <= 0 || max_out <= 0) return cudaSuccess;
  if (n_jobs > 65535) return cudaErrorInvalidValue;
  rotate_pools_kernel<<<dim3((max_out + 255) / 256, n_jobs), 256, 0, stream>>>(jobs);
  return cudaGetLastError();
}

}  // namespace qm
