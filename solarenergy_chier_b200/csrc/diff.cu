// Differentiable forward and hand-written adjoint of the tracer.
//
// Forward (diff.cpp drives it): the heliostats are prepared with their
// parameters -- aim point moved by (du, dv) along the receiver's aim axes,
// normal then turned by (a, b) radians about its frame's u and v axes --
// every ray is traced as in the plain path, each receiver hit deposits its
// energy bilinearly at its continuous pixel position (trace kernel output
// mode 2, which also records one hit bit per ray), the deposit D is smoothed
// by a separable Gaussian G (flux F = G * D) and L = sum (F - T)^2.
//
// Adjoint: with R = dL/dF = 2 (F - T) and P = G * R (G is symmetric, so
// dL/dD = P), a ray depositing energy e at pixel position (X, Y) contributes
//   dL/dtheta = e (dPb/dX dX/dtheta + dPb/dY dY/dtheta) + Pb de/dtheta,
// Pb the bilinear interpolation of P at (X, Y) -- the exact derivative of
// the discretised forward.  The chain from the heliostat's normal and frame
// over the facet position and normal, the slope-error normal, the reflection,
// the receiver intersection (implicitly: the hit point stays on the receiver
// surface) and the energy (cosine and atmospheric attenuation) is run
// backwards per ray, down to the heliostat's frame axes, whose derivatives
// with respect to its four parameters (forward-mode, once per heliostat) are
// applied to a warp chunk's sums.
// Shadowing and blocking are treated as constants (indicators detached):
// only rays whose hit bit the forward set contribute, and no grid walk is
// repeated.  The receiver's own edges (a cylinder's silhouette, the image's
// first and last rows and a rectangle's columns) are handled by band
// estimates of their boundary terms.  The bias left is the change of loss
// from rays that cross a blocker's edge.
#include "diff.h"

#include "ray_geom.h"

namespace qm {
namespace {

constexpr int K = kDiffParams;
// Smallest |cos(incidence)| on the receiver of a ray whose interior
// derivative is used (about 84 degrees from the surface normal); grazing rays
// on a cylinder estimate its silhouette's boundary term instead.
constexpr float kGrazing = 0.1f;
// Width in pixels of the bands along the image edges whose rays estimate
// the edges' boundary terms.
constexpr float kEdgeBand = 1.0f;
constexpr float kTwoPi = 6.28318530717959f;

// ---- value + tangent arithmetic ----------------------------------------------
template <int N>
__device__ __forceinline__ DualT<N> dc(float v) {
  DualT<N> r;
  r.v = v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = 0.0;
  return r;
}
template <int N>
__device__ __forceinline__ DualT<N> dvar(float v, int k) {
  DualT<N> r = dc<N>(v);
  r.d[k] = 1.0;
  return r;
}
template <int N>
__device__ __forceinline__ DualT<N> operator+(DualT<N> a, DualT<N> b) {
  DualT<N> r;
  r.v = a.v + b.v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] + b.d[k];
  return r;
}
template <int N>
__device__ __forceinline__ DualT<N> operator-(DualT<N> a, DualT<N> b) {
  DualT<N> r;
  r.v = a.v - b.v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] - b.d[k];
  return r;
}
template <int N>
__device__ __forceinline__ DualT<N> operator-(DualT<N> a) {
  DualT<N> r;
  r.v = -a.v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = -a.d[k];
  return r;
}
template <int N>
__device__ __forceinline__ DualT<N> operator*(DualT<N> a, DualT<N> b) {
  DualT<N> r;
  r.v = a.v * b.v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] * b.v + a.v * b.d[k];
  return r;
}
template <int N>
__device__ __forceinline__ DualT<N> operator*(DualT<N> a, float s) {
  DualT<N> r;
  r.v = a.v * s;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] * s;
  return r;
}
// 1 / sqrt(a)
template <int N>
__device__ __forceinline__ DualT<N> drsqrt(DualT<N> a) {
  const float r = rsqrtf(a.v);
  DualT<N> o;
  o.v = r;
  if constexpr (N > 0) {
    const double dr = -0.5 / ((double)a.v * sqrt((double)a.v));
#pragma unroll
    for (int k = 0; k < N; ++k) o.d[k] = dr * a.d[k];
  }
  return o;
}

template <int N>
__device__ __forceinline__ Dual3T<N> d3(float3 c) {
  return Dual3T<N>{dc<N>(c.x), dc<N>(c.y), dc<N>(c.z)};
}
template <int N>
__device__ __forceinline__ float3 val(const Dual3T<N>& a) {
  return make_float3(a.x.v, a.y.v, a.z.v);
}
template <int N>
__device__ __forceinline__ Dual3T<N> operator+(const Dual3T<N>& a, const Dual3T<N>& b) {
  return Dual3T<N>{a.x + b.x, a.y + b.y, a.z + b.z};
}
template <int N>
__device__ __forceinline__ Dual3T<N> operator-(const Dual3T<N>& a, const Dual3T<N>& b) {
  return Dual3T<N>{a.x - b.x, a.y - b.y, a.z - b.z};
}
template <int N>
__device__ __forceinline__ Dual3T<N> operator-(const Dual3T<N>& a) {
  return Dual3T<N>{-a.x, -a.y, -a.z};
}
template <int N>
__device__ __forceinline__ Dual3T<N> operator*(const Dual3T<N>& a, DualT<N> s) {
  return Dual3T<N>{a.x * s, a.y * s, a.z * s};
}
template <int N>
__device__ __forceinline__ Dual3T<N> operator*(const Dual3T<N>& a, float s) {
  return Dual3T<N>{a.x * s, a.y * s, a.z * s};
}
template <int N>
__device__ __forceinline__ DualT<N> dot(const Dual3T<N>& a, const Dual3T<N>& b) {
  return a.x * b.x + a.y * b.y + a.z * b.z;
}
template <int N>
__device__ __forceinline__ Dual3T<N> cross(const Dual3T<N>& a, const Dual3T<N>& b) {
  return Dual3T<N>{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <int N>
__device__ __forceinline__ Dual3T<N> normalize(const Dual3T<N>& a) {
  return a * drsqrt(dot(a, a));
}

// Frame (u, n, v) of a normal, as qm::make_frame (Util/global_function.cuh:19-36
// and the flipped focus-flat variant), with tangents.
template <int N>
struct DFrameT {
  Dual3T<N> u, n, v;
  bool identity;
};
template <int N>
__device__ __forceinline__ DFrameT<N> make_dframe(const Dual3T<N>& n, bool flip) {
  DFrameT<N> f;
  f.n = n;
  f.identity = qm_below_eps(fabsf(n.x.v)) && qm_below_eps(fabsf(n.z.v));
  if (f.identity) {
    f.u = d3<N>(make_float3(1.f, 0.f, 0.f));
    f.v = d3<N>(make_float3(0.f, 0.f, 1.f));
    return f;
  }
  f.u = normalize(cross(d3<N>(make_float3(0.f, 1.f, 0.f)), n));
  f.v = normalize(cross(f.u, n));
  if (flip && n.z.v < 0) {
    f.u = -f.u;
    f.v = -f.v;
  }
  return f;
}
template <int N>
__device__ __forceinline__ Dual3T<N> to_world(const DFrameT<N>& f, float3 d) {
  if (f.identity) return d3<N>(d);
  return f.u * d.x + f.n * d.y + f.v * d.z;
}

// ---- preparation: normal and frame of every heliostat with tangents --------
__global__ void diff_prep_kernel(PrepInputs p, DiffTask* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  const PrepItem it = p.items[i];
  const DevTask& T = p.tasks[it.task];
  const float3 sun_dir = p.suns[it.sun].dir;
  const float4 offset = p.params[it.param];
  // aim point a = focus + du aim_u + dv aim_v
  Dual3T<K> a = d3<K>(make_float3(it.focus.x + it.aim_u.x * offset.x + it.aim_v.x * offset.y,
                                  it.focus.y + it.aim_u.y * offset.x + it.aim_v.y * offset.y,
                                  it.focus.z + it.aim_u.z * offset.x + it.aim_v.z * offset.y));
  a.x.d[0] = it.aim_u.x;
  a.y.d[0] = it.aim_u.y;
  a.z.d[0] = it.aim_u.z;
  a.x.d[1] = it.aim_v.x;
  a.y.d[1] = it.aim_v.y;
  a.z.d[1] = it.aim_v.z;
  const Dual3T<K> r = normalize(a - d3<K>(T.pos));
  const Dual3T<K> n0 = normalize(r - d3<K>(sun_dir));
  const DFrameT<K> f0 = make_dframe(n0, false);
  const Dual3T<K> nrm =
      normalize(n0 + f0.u * dvar<K>(offset.z, 2) + f0.v * dvar<K>(offset.w, 3));
  const DFrameT<K> hf = make_dframe(nrm, T.type == 1);
  DiffTask o;
  o.n = nrm;
  o.u = hf.u;
  o.fn = hf.n;
  o.v = hf.v;
  o.identity = hf.identity ? 1 : 0;
  out[it.task] = o;
}

// ---- adjoint ------------------------------------------------------------------
// P at the four pixels around pixel position (xs + 0.5, ys + 0.5), with the
// forward deposit's wrap / zero conventions.
struct Quad {
  float p00, p10, p01, p11;  // p<column><row>
  float fx, fy;
};
__device__ __forceinline__ Quad sample_quad(const DevReceiver& R, float xs, float ys) {
  const float x0 = floorf(xs), y0 = floorf(ys);
  Quad q;
  q.fx = xs - x0;
  q.fy = ys - y0;
  const int w = R.resolution.x, h = R.resolution.y;
  int c0 = (int)x0, c1 = c0 + 1;
  const int r0 = (int)y0, r1 = r0 + 1;
  if (R.type == 1) {
    c0 = c0 < 0 ? c0 + w : (c0 >= w ? c0 - w : c0);
    c1 = c1 < 0 ? c1 + w : (c1 >= w ? c1 - w : c1);
  }
  const bool in0 = (unsigned)c0 < (unsigned)w, in1 = (unsigned)c1 < (unsigned)w;
  const bool up = (unsigned)r0 < (unsigned)h, down = (unsigned)r1 < (unsigned)h;
  const float* row = R.image + (long long)r0 * w;
  q.p00 = up && in0 ? __ldg(row + c0) : 0.0f;
  q.p10 = up && in1 ? __ldg(row + c1) : 0.0f;
  q.p01 = down && in0 ? __ldg(row + w + c0) : 0.0f;
  q.p11 = down && in1 ? __ldg(row + w + c1) : 0.0f;
  return q;
}
__device__ __forceinline__ float bilinear(const Quad& q) {
  return (1 - q.fx) * (1 - q.fy) * q.p00 + q.fx * (1 - q.fy) * q.p10 + (1 - q.fx) * q.fy * q.p01 + q.fx * q.fy * q.p11;
}

// Bilinear interpolation of P at continuous pixel position (X, Y).
__device__ __noinline__ float bilinear_p(const DevReceiver& R, float X, float Y) {
  return bilinear(sample_quad(R, X - 0.5f, Y - 0.5f));
}

// What the rays of one facet share: its origin and the frame of its normal
// (the slope-error perturbation's frame), its point and its sub-heliostat's
// normal in the heliostat's local frame, and its two pool offsets.
struct Facet {
  float3 origin, u, n, v, local, local_normal;
  bool identity;
  int g0, g1;
};

// The values follow the dual arithmetic of the preparation (value parts).  Not
// inlined: once per 32 facets, beside a sweep whose code the one-warp blocks
// of an SM, each at another place in it, must hold in one instruction cache.
__device__ __noinline__ Facet make_facet(const DevTask& T, const DiffTask& DT, int f) {
  Facet fd;
  const bool focus_flat = facet_local(T, f, fd.local, fd.local_normal);
  DFrameT<0> hf;
  hf.u = d3<0>(val(DT.u));
  hf.n = d3<0>(val(DT.fn));
  hf.v = d3<0>(val(DT.v));
  hf.identity = DT.identity != 0;
  fd.origin = val(to_world(hf, fd.local) + d3<0>(T.pos));
  const Dual3T<0> normal = focus_flat ? to_world(hf, fd.local_normal) : d3<0>(val(DT.n));
  const DFrameT<0> fr = make_dframe(normal, false);
  fd.u = val(fr.u);
  fd.n = val(fr.n);
  fd.v = val(fr.v);
  fd.identity = fr.identity;
  fd.g0 = __ldg(T.offsets + f);
  fd.g1 = __ldg(T.offsets + (f + 1) % T.pool_size);
  return fd;
}

// Adjoint of the heliostat's facet frame, one lane's sum: row j is d/d(axis j).
struct FrameSum {
  float3 u, n, v;
};
__device__ __forceinline__ void add_outer(FrameSum& s, float3 a, float3 l) {
  s.u.x += a.x * l.x; s.u.y += a.y * l.x; s.u.z += a.z * l.x;
  s.n.x += a.x * l.y; s.n.y += a.y * l.y; s.n.z += a.z * l.y;
  s.v.x += a.x * l.z; s.v.y += a.y * l.z; s.v.z += a.z * l.z;
}
// abar . da/d(parameter k)
__device__ __forceinline__ double along(float3 abar, const Dual3T<K>& a, int k) {
  return abar.x * a.x.d[k] + abar.y * a.y.d[k] + abar.z * a.z.d[k];
}
__device__ __forceinline__ float3 axpy(float s, float3 x, float3 y) {
  return make_float3(s * x.x + y.x, s * x.y + y.y, s * x.z + y.z);
}

// What a chunk's rays share, in shared memory: read per ray, and a read from
// the task and receiver tables would wait on the L1.
struct ChunkConstants {
  DevReceiver R;
  const float4* samples;
  const float4* perturbations;
  float factor;
  float sx, sy;  // cylinder: pixels per radian, per metre of height
};

// Adds the contribution of one ray (facet fd, light lab) that hit the
// receiver in the forward to `sum`.
__device__ __forceinline__ void ray_adjoint(const ChunkConstants& T, const Facet& fd, int lab, FrameSum& sum) {
  const DevReceiver& R = T.R;
  const float3 o = fd.origin;
  const float3 din = xyz(__ldg(T.samples + fd.g0 + lab));
  const float3 pert = xyz(__ldg(T.perturbations + fd.g1 + lab));
  DFrameT<0> fr;
  fr.u = d3<0>(fd.u);
  fr.n = d3<0>(fd.n);
  fr.v = d3<0>(fd.v);
  fr.identity = fd.identity;
  const Dual3T<0> slope = to_world(fr, pert);
  const Dual3T<0> dnp = normalize(slope);
  const Dual3T<0> din3 = d3<0>(make_float3(-din.x, -din.y, -din.z));
  const DualT<0> c0 = dot(dnp, din3);
  const Dual3T<0> refl = din3 - dnp * (c0 * 2.0f);
  const DualT<0> inv_len = drsqrt(dot(refl, refl));
  const Dual3T<0> drd = refl * inv_len;  // normalize(refl)
  const float3 d = val(drd), np = val(dnp), in = val(din3);
  float t, u, v;
  // The receiver test with its decisions rounded as the forward's and the
  // hit point, (u, v) and distance in approximate arithmetic: the direction
  // here is a contracted value, not the forward's, so the exact position
  // arithmetic would buy nothing.  A ray the rounding moves off the receiver
  // edge adds nothing.
  if (!receiver_hit_rx(R, o, d, t, u, v)) return;
  // energy |rd . np| eta(t) factor (receiverIntersectionUtil.cuh:17-34)
  const float c = dot(drd, dnp).v;
  const float sgn = c >= 0.0f ? 1.0f : -1.0f;
  float eta, deta;
  if (t <= 1000.0f) {
    eta = 0.99331f - 0.0001176f * t + 1.97e-8f * t * t;
    deta = -0.0001176f + 2.0f * 1.97e-8f * t;
  } else {
    eta = expf(-0.0001106f * t);
    deta = -0.0001106f * eta;
  }
  const float e = fabsf(c) * eta * T.factor;
  // The adjoints of the hit point's path: of the origin, of the reflected
  // direction and of c = rd . np.
  float3 obar, rdbar;
  float cbar = 0.0f;
  bool band = false;
  float x = 0.0f, z = 0.0f, den = 0.0f, rr = 0.0f, dxz2 = 0.0f;
  if (R.type == 1) {
    const float3 p = make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
    x = p.x - R.pos.x;
    z = p.z - R.pos.z;
    den = x * d.x + z * d.z;
    rr = x * x + z * z;
    dxz2 = d.x * d.x + d.z * d.z;
    if (!(rr > 0.0f) || !(dxz2 > 0.0f)) return;
    band = !(fabsf(den) > kGrazing * sqrtf(rr * dxz2));  // rounded thus: one ray on the other side shows
  }
  if (band) {
    // Silhouette band: rays whose impact parameter b (distance of the
    // ray's horizontal line from the axis) lies within w of the radius
    // (|cos incidence| < kGrazing).  Their interior derivative grows as
    // 1/cos(incidence) and is not summed; across the band it integrates
    // to rho e v (P(silhouette) - P(inner band edge)), and the boundary
    // term of rays crossing the silhouette is -rho e v P(silhouette), so
    // together the band contributes -rho e v P(inner band edge), with
    // v = d|b|/dtheta and rho ~ (rays in the band) / w.  P is taken where
    // this ray's line would meet the cylinder with impact parameter R - w.
    const float radius = R.size.x;
    const float w = radius * (1.0f - sqrtf(1.0f - kGrazing * kGrazing));
    const float inv_dxz = rsqrtf(dxz2);
    const float ox = o.x - R.pos.x, oz = o.z - R.pos.z;
    const float b = (ox * d.z - oz * d.x) * inv_dxz;
    const float out = b >= 0.0f ? 1.0f : -1.0f;
    const float hx = d.x * inv_dxz, hz = d.z * inv_dxz;  // horizontal unit direction
    const float tca = -(ox * d.x + oz * d.z) / dxz2;
    const float cx = o.x + tca * d.x - R.pos.x, cz = o.z + tca * d.z - R.pos.z;  // closest approach
    const float cl = sqrtf(cx * cx + cz * cz);
    const float ux = cl > 0.0f ? cx / cl : -hz, uz = cl > 0.0f ? cz / cl : hx;
    const float back = radius * kGrazing;  // sqrt(R^2 - (R - w)^2)
    const float ex = (radius - w) * ux - back * hx, ez = (radius - w) * uz - back * hz;
    float phi = atan2f(ez, ex);
    if (phi < 0.0f) phi += kTwoPi;
    const float Xs = phi * (float)R.resolution.x / kTwoPi;
    const float ys = o.y + (tca - back * inv_dxz) * d.y;
    const float Ys = ((ys - R.pos.y) / R.size.y + 0.5f) * (float)R.resolution.y;
    const float pe = bilinear_p(R, Xs, Ys);
    // b = (ox d.z - oz d.x) / |d_xz|
    const float bbar = -e * pe * out / w;
    const float bl = bbar * inv_dxz;
    obar = make_float3(bl * d.z, 0.0f, -bl * d.x);
    rdbar = make_float3(-bl * (oz + b * hx), 0.0f, bl * (ox - b * hz));
  } else {
    // bilinear P at the deposit position (as the forward's splat)
    const float X = v * (float)R.resolution.x, Y = u * (float)R.resolution.y;
    const float xs = X - 0.5f, ys = Y - 0.5f;
    const Quad q = sample_quad(R, xs, ys);
    const float pb = bilinear(q);
    float xbar = e * ((1 - q.fy) * (q.p10 - q.p00) + q.fy * (q.p11 - q.p01));
    float ybar = e * ((1 - q.fx) * (q.p01 - q.p00) + q.fx * (q.p11 - q.p10));
    // Image edges (rows of both receivers, columns of a rectangle): rays
    // within kEdgeBand pixels of an edge estimate the boundary term -rho e P
    // (outward pixel velocity) of rays leaving or entering across it, with P
    // taken on the edge itself (half of an edge deposit falls outside).
    const float by = kEdgeBand;
    const float H = (float)R.resolution.y, W = (float)R.resolution.x;
    if (Y < by) ybar += e * bilinear_p(R, X, 0.0f) / by;
    if (H - Y < by) ybar -= e * bilinear_p(R, X, H) / by;
    if (R.type == 0) {
      if (X < by) xbar += e * bilinear_p(R, 0.0f, Y) / by;
      if (W - X < by) xbar -= e * bilinear_p(R, W, Y) / by;
    }
    // e = |c| eta(t) factor
    const float pf = pb * T.factor;
    cbar = pf * sgn * eta;
    float tbar = pf * fabsf(c) * deta;
    // The hit point q = o + t rd, kept on the surface by dt = -(m . (do + t drd)) / (m . rd), m its normal.
    float3 qbar, m;
    float md;
    if (R.type == 1) {
      const float a = __fdividef(xbar * T.sx, rr);
      qbar = make_float3(-a * z, ybar * T.sy, a * x);
      m = make_float3(x, 0.0f, z);
      md = den;
    } else {
      const float3 N = qm::cross(R.ab, R.ac);
      const float nd = qm::dot(N, d), nn = qm::dot(N, N);
      if (!(fabsf(nd) > kGrazing * sqrtf(nn))) return;  // grazing on a plane: no boundary, detached
      const float3 abs_ = qm::mul(qm::cross(R.ac, N), 1.0f / nn), acs = qm::mul(qm::cross(N, R.ab), 1.0f / nn);
      qbar = axpy(ybar * H, abs_, qm::mul(acs, xbar * W));
      m = N;
      md = nd;
    }
    tbar += qm::dot(qbar, d);
    obar = axpy(-__fdividef(tbar, md), m, qbar);
    rdbar = make_float3(t * obar.x, t * obar.y, t * obar.z);
  }
  add_outer(sum, obar, fd.local);
  if (fd.identity) return;  // the slope-error frame does not turn
  // rd = (in - 2 (np . in) np) / |in| and c = -(np . in) / |in| (np is a unit
  // vector, so the reflection keeps in's length, which no parameter moves but
  // which is not always 1: pools and suns need not be of unit length), then
  // np = slope / |slope|.
  const float rn = qm::dot(rdbar, np);
  const float3 npbar = qm::mul(axpy(-2.0f * rn - cbar, in, qm::mul(rdbar, -2.0f * c0.v)), inv_len.v);
  const float il = rsqrtf(dot(slope, slope).v);
  const float3 wbar = qm::mul(axpy(-qm::dot(npbar, np), np, npbar), il);
  // slope = pert.x u + pert.y n + pert.z v with, for n = (s sin psi, n.y,
  // s cos psi), u = (cos psi, 0, -sin psi) and v = (n.y sin psi, -s, n.y cos psi).
  const float sn = -fd.u.z, cs = fd.u.x, s = -fd.v.y;
  const float along = wbar.x * sn + wbar.z * cs, across = wbar.x * cs - wbar.z * sn;
  const float psibar = __fdividef(pert.z * fd.n.y * across - pert.x * along, s), sbar = -pert.z * wbar.y;
  const float3 nbar = make_float3(pert.y * wbar.x + psibar * cs + sbar * sn, pert.y * wbar.y + pert.z * along,
                                  pert.y * wbar.z - psibar * sn + sbar * cs);
  add_outer(sum, nbar, fd.local_normal);
}

// Facet window of the adjoint, per warp (as the trace kernel's): 32
// consecutive facets, one per lane, stored component-major so that lanes
// reading different slots touch different banks; and the queue of recorded
// hits (window slot, light) waiting for a full warp.
#ifndef QM_BWD_THREADS
#define QM_BWD_THREADS 32
#endif
#ifndef QM_BWD_MIN_BLOCKS
#define QM_BWD_MIN_BLOCKS 24
#endif
constexpr int kBwdThreads = QM_BWD_THREADS;
constexpr int kFacetFloats = 18;
struct AdjointWindow {
  float value[kFacetFloats][kBwdThreads];
  int g0[kBwdThreads], g1[kBwdThreads], identity[kBwdThreads];
  int slot[2 * kBwdThreads], light[2 * kBwdThreads];
  ChunkConstants shared[kBwdThreads / 32];
};

__device__ __forceinline__ void put3(AdjointWindow& w, int first, int slot, float3 a) {
  w.value[first][slot] = a.x;
  w.value[first + 1][slot] = a.y;
  w.value[first + 2][slot] = a.z;
}
__device__ __forceinline__ float3 get3(const AdjointWindow& w, int first, int slot) {
  return make_float3(w.value[first][slot], w.value[first + 1][slot], w.value[first + 2][slot]);
}

// Bound by instruction issue.  Run backwards a ray costs its value chain, one
// sweep of vector adjoints and 18 multiply-adds into the frame sums, against
// four tangents through every operation; the queue gives every sweep 32 hits
// where a chunk's iterations hold 22 on the benchmark field.  The call on 462 M
// rays, 32 lights per facet: 17.9 -> 7.7 ms; on 256 M rays, 4 lights: 11.9 -> 5.8.
// Distance (2-norm) from 64-bit tangents of the same rays, over four fields x 16
// seeds: 3.3e-8 to 4.6e-8, where the forward-mode kernel's was 3.6e-8 to 8.1e-8:
// what counts is the factors that a heliostat's rays share (its tangents, the
// pixels per radian), hence in double; the sweep's three approximate divisions
// round each ray on its own, and IEEE ones (0.3 ms more) leave the distance at
// 3.4e-8 to 4.4e-8.
// 20 / 24 / 28 blocks per SM: 8.2 / 7.9 / 8.3 ms with the facets still inlined.
__global__ void __launch_bounds__(kBwdThreads, QM_BWD_MIN_BLOCKS) diff_backward_kernel(BackwardParams p) {
  __shared__ AdjointWindow win;
  const int lane = threadIdx.x & 31;
  const int wbase = threadIdx.x & ~31;
  const long long warp = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long chunk = p.chunk_begin + warp;
  if (chunk >= p.total_chunks) return;
  const int nl = p.light_end - p.light_begin;
  const int t = find_task(p.chunk_prefix, p.num_tasks, chunk);
  const int r0 = (int)(chunk - __ldg(p.chunk_prefix + t)) * kChunk;
  const DevTask& T = p.tasks[t];
  const DiffTask& DT = p.dtasks[t];
  if (lane == 0) {
    ChunkConstants& c = win.shared[threadIdx.x >> 5];
    c.R = p.receivers[T.receiver];
    c.samples = T.samples;
    c.perturbations = T.perturbations;
    c.factor = T.factor;
    c.sx = (float)(c.R.resolution.x / 6.283185307179586);
    c.sy = (float)c.R.resolution.y / c.R.size.y;
  }
  const int r_end = T.num_facets * nl;
  const int iters = min(kChunkIters, (r_end - r0 + 31) >> 5);
  int f = (r0 + lane) / nl;
  int l = (r0 + lane) - f * nl;
  FrameSum sum{};
  int base = 0;
  bool filled = false;  // warp-uniform
  int queued = 0;       // warp-uniform, at most 63
  int* q_slot = win.slot + 2 * wbase;
  int* q_light = win.light + 2 * wbase;
  unsigned words = 0;  // lane i: hit bits of iteration 32 (it / 32) + i
  for (int it = 0;; ++it) {
    const bool more = it < iters;  // a last step runs what still waits
    if ((it & 31) == 0) words = it + lane < iters ? __ldg(p.hit_bits + warp * kChunkIters + it + lane) : 0u;
    const unsigned bits = __shfl_sync(0xffffffffu, words, it & 31);
    const bool hit = more && r0 + it * 32 + lane < r_end && ((bits >> lane) & 1u);
    // The facets of an iteration lie within 32 of lane 0's (see the trace
    // kernel); refill the window when a lane with a hit needs one past it,
    // after the hits that are waiting with the present one.
    const int f0 = __shfl_sync(0xffffffffu, f, 0);
    const bool fill = __any_sync(0xffffffffu, hit && (!filled || f - base >= 32));
    // Runs the last queued hits, one per lane, at this one place in the code.
    while (fill || !more ? queued > 0 : queued >= 32) {
      const int n = min(queued, 32);
      __syncwarp();
      if (lane < n) {
        const int slot = q_slot[queued - n + lane], light = q_light[queued - n + lane];
        Facet fd;
        fd.origin = get3(win, 0, slot);
        fd.u = get3(win, 3, slot);
        fd.n = get3(win, 6, slot);
        fd.v = get3(win, 9, slot);
        fd.local = get3(win, 12, slot);
        fd.local_normal = get3(win, 15, slot);
        fd.identity = win.identity[slot] != 0;
        fd.g0 = win.g0[slot];
        fd.g1 = win.g1[slot];
        ray_adjoint(win.shared[threadIdx.x >> 5], fd, light, sum);
      }
      queued -= n;
      __syncwarp();
    }
    if (!more) break;
    if (fill) {
      __syncwarp();
      base = f0;
      filled = true;
      const int fw = base + lane;
      if (fw < T.num_facets) {
        const Facet fd = make_facet(T, DT, fw);
        const int slot = wbase + lane;
        put3(win, 0, slot, fd.origin);
        put3(win, 3, slot, fd.u);
        put3(win, 6, slot, fd.n);
        put3(win, 9, slot, fd.v);
        put3(win, 12, slot, fd.local);
        put3(win, 15, slot, fd.local_normal);
        win.g0[slot] = fd.g0;
        win.g1[slot] = fd.g1;
        win.identity[slot] = fd.identity ? 1 : 0;
      }
    }
    const unsigned hits = __ballot_sync(0xffffffffu, hit);
    if (hit) {
      const int k = queued + __popc(hits & ((1u << lane) - 1u));
      q_slot[k] = wbase + (f - base);
      q_light[k] = p.light_begin + l;
    }
    queued += __popc(hits);
    f += p.lights_q32;
    l += p.lights_r32;
    if (l >= nl) {
      l -= nl;
      ++f;
    }
  }
  // d(axes)/d(parameters) of the heliostat's facet frame; constant axes when
  // the frame is the identity.
  if (DT.identity) return;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double s = along(sum.u, DT.u, k) + along(sum.n, DT.fn, k) + along(sum.v, DT.v, k);
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0 && s != 0.0) atomicAdd(p.grad + (size_t)T.power_slot * K + k, s);
  }
}

// ---- smoothing and loss ---------------------------------------------------------
__global__ void gauss_rows_kernel(const float* in, float* out, int w, int h, const float* wt, int radius, bool wrap) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= w || y >= h) return;
  float s = 0.0f;
  for (int k = -radius; k <= radius; ++k) {
    int c = x + k;
    if (wrap) c = ((c % w) + w) % w;
    if (c < 0 || c >= w) continue;
    s += wt[k < 0 ? -k : k] * in[(size_t)y * w + c];
  }
  out[(size_t)y * w + x] = s;
}

__global__ void gauss_cols_kernel(const float* in, float* out, int w, int h, const float* wt, int radius) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= w || y >= h) return;
  float s = 0.0f;
  for (int k = -radius; k <= radius; ++k) {
    const int r = y + k;
    if (r < 0 || r >= h) continue;
    s += wt[k < 0 ? -k : k] * in[(size_t)r * w + x];
  }
  out[(size_t)y * w + x] = s;
}

__global__ void round_kernel(const double* in, float* out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)in[i];
}

__global__ void loss_kernel(const float* flux, const float* target, float* resid, long long n, double* loss) {
  __shared__ double part[8];
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double s = 0.0;
  if (i < n) {
    const float diff = flux[i] - target[i];
    resid[i] = 2.0f * diff;
    s = (double)diff * diff;
  }
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) b += part[k];
    if (b != 0.0) atomicAdd(loss, b);
  }
}

}  // namespace

cudaError_t launch_diff_prep(const PrepInputs& p, DiffTask* out, cudaStream_t stream) {
  if (p.n <= 0) return cudaSuccess;
  if (!p.params) return cudaErrorInvalidValue;
  diff_prep_kernel<<<(p.n + 31) / 32, 32, 0, stream>>>(p, out);
  return cudaGetLastError();
}

cudaError_t launch_diff_backward(const BackwardParams& params, cudaStream_t stream) {
  const long long nl = params.light_end - params.light_begin;
  if (params.chunk_begin < 0) return cudaErrorInvalidValue;
  if (nl <= 0 || params.total_chunks <= params.chunk_begin) return cudaSuccess;
  BackwardParams p = params;
  p.lights_q32 = (int)(32 / nl);
  p.lights_r32 = (int)(32 % nl);
  const long long warps_per_block = kBwdThreads / 32;
  const long long blocks = (p.total_chunks - p.chunk_begin + warps_per_block - 1) / warps_per_block;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  diff_backward_kernel<<<(unsigned)blocks, kBwdThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_gauss(const float* in, float* tmp, float* out, int width, int height, const float* weights,
                         int radius, bool wrap_cols, cudaStream_t stream) {
  if (width <= 0 || height <= 0) return cudaSuccess;
  const dim3 grid((width + 127) / 128, height);
  gauss_rows_kernel<<<grid, 128, 0, stream>>>(in, tmp, width, height, weights, radius, wrap_cols);
  gauss_cols_kernel<<<grid, 128, 0, stream>>>(tmp, out, width, height, weights, radius);
  return cudaGetLastError();
}

cudaError_t launch_round_deposit(const double* in, float* out, long long n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  round_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(in, out, n);
  return cudaGetLastError();
}

cudaError_t launch_loss(const float* flux, const float* target, float* resid, long long n, double* loss,
                        cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  loss_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(flux, target, resid, n, loss);
  return cudaGetLastError();
}

}  // namespace qm
