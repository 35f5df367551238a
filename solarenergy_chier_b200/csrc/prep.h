// Device-side per-sun preparation (prep.cu).
#pragma once

#include <cuda_runtime.h>

#include "device_scene.h"

namespace qm {

// One sun of a preparation: its direction of travel, and what the walk-free
// tests need (csrc/shadow.h): the axis toward the sun with the world-space
// tangent of the largest sun-shape angle (< 0: unbounded, no test), and
// theta_sun + 2 theta_slope (< 0: no test).
struct SunParams {
  float3 dir;
  float3 shadow_axis;
  float shadow_tan;
  float block_theta;
};

// One (sun, heliostat) to prepare, the same for every sun direction: uploaded
// once, so that a new sun costs its SunParams alone.  The task already holds
// the heliostat's sun-independent fields; the kernels fill its normal, facet
// frame and walk code and write the heliostat's sub-heliostat parallelograms
// and traversal record into the sun's grid arrays.
struct PrepItem {
  int task;         // index into the task array
  int sun;          // index into the SunParams
  int param;        // index into the differentiable parameters
  int num_sub;      // sub-heliostats of the heliostat
  int sub_first;    // grid-local id of its first sub-heliostat
  float3 focus;     // aim point (sun-independent)
  float3 aim_u, aim_v;  // aim axes of the differentiable parameters
  int* sub_free;
  int* sub_cand;  // kMaxCandidates per sub-heliostat
  float4* sub_frames;  // 6 per sub-heliostat (DevGrid::sub_frames)
  float3* verts;    // out: 3 float3 (B, A, C) per sub-heliostat
  float4* subv;     // out: 3 float4 per sub-heliostat (A, B - A, C - A)
  float4* bound;    // out: 5 float4 traversal record
  int4* hsub;       // out: (first, count, lattice rows, lattice columns)
  int* top_key;     // out: raised to the box's highest point (DevGrid::top_key)
};

// Inputs of the preparation kernels.  params (NULL: none): per heliostat
// (aim x, aim y, normal x, normal y): the aim point moves by x aim_u + y
// aim_v; the normal then turns by (x, y) radians about the u and v axes of its
// own frame.
struct PrepInputs {
  const PrepItem* items;
  int n;
  DevTask* tasks;
  const SunParams* suns;
  const float4* params;
};

struct PoolRotation {
  const float4* in;  // local sun-shape pool, n entries
  float4* out;       // world-space tracer copy, n_out = n + L entries (entry i = pool entry i % n)
  int n, n_out;
  SunFrame sun;
};

// grids, num_grids: the grids that the items' records belong to.
cudaError_t launch_prep(const PrepInputs& p, DevGrid* grids, int num_grids, cudaStream_t stream);
// Walk codes and sub-heliostat frames of the prepared tasks; grids: the
// tasks' grids with their prepared traversal records.  Run after launch_prep.
// max_sub: the most sub-heliostats of any item (one warp per heliostat and
// per sub-heliostat).
cudaError_t launch_shadow_flags(const PrepInputs& p, int max_sub, const DevGrid* grids, cudaStream_t stream);
// out[i] = tasks[ids[i]].
cudaError_t launch_gather_tasks(const DevTask* tasks, const int* ids, int n, DevTask* out, cudaStream_t stream);
// max_out: the largest n_out of the jobs.
cudaError_t launch_rotate_pools(const PoolRotation* jobs, int n_jobs, int max_out, cudaStream_t stream);

}  // namespace qm
