// Single-axis projections (the beam has no y component: every ray stays in
// one y plane): the launch's steps and orientation, and the pixel layout of
// its kernels. Shared by the forward projector (esb_projector_fast.cu) and
// the gradients (esb_adjoint.cu).
#pragma once

#include <math.h>

#include "esb_ray_core.cuh"

namespace esb {
namespace raycore {

__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }

// Ceilings of two sample parameters in [0, 2^22] (additions that round up;
// no conversion-unit instruction).
__device__ __forceinline__ float2 ceil2(float a, float b) {
  return __fadd2_rn(__fadd2_ru(make_float2(a, b), splat(8388608.0f)), splat(-8388608.0f));
}

// Steps of the walk, the same for every ray of a launch whose samples lie in
// one binade of the ray parameter (axis_step on the host; a ray with another
// step takes ray_sum).
struct AxisStep {
  float step;          // of the ray parameter
  float dM, dN;        // |step| of the major and minor coordinate, dM >= dN
  float isM, isN;      // 1 / dM, and 1 / dN (0 for dN = 0)
  float hM, hN;        // dM / 2, dN / 2
  float g;             // dN dM / 12
};

// Beam directions whose rays all stay in one y plane take the axis kernels.
inline bool axis_projection(const KConst& c) { return fabsf(c.n.y) <= 1e-6f; }

// Instance of the axis kernels for the launch's beam direction (major axis z
// when |dq.z| >= |dq.x|, step signs) and its steps: the step of the ray
// parameter is the one of the binade that holds the volume's centre.
inline AxisStep axis_step(const KConst& c, bool& zmaj, int& sm, int& sn) {
  const float h = c.vs.x * 0.15f;
  double t = 0.0;
  const double n[3] = {c.n.x, c.n.y, c.n.z}, d[3] = {c.det.x, c.det.y, c.det.z};
  const double lo[3] = {c.bbMin.x, c.bbMin.y, c.bbMin.z}, hi[3] = {c.bbMax.x, c.bbMax.y, c.bbMax.z};
  for (int j = 0; j < 3; ++j) t += n[j] * (0.5 * (lo[j] + hi[j]) - d[j]);
  int e = 0;
  frexp(t, &e);
  volatile float t0 = (float)ldexp(0.5, e), t1 = t0 + h;  // single roundings, as the kernel's
  AxisStep A;
  A.step = t > 0.0 ? t1 - t0 : 0.0f;  // 0: no ray takes the walk
  volatile float qx = A.step * c.n.x, qz = A.step * c.n.z;
  qx = qx * c.bbRcp.x;
  qz = qz * c.bbRcp.z;
  qx = qx * c.dim.x;
  qz = qz * c.dim.z;
  zmaj = fabsf(qz) >= fabsf(qx);
  const float m = zmaj ? qz : qx, nn = zmaj ? qx : qz;
  sm = m < 0.f ? -1 : 1;
  sn = nn < 0.f ? -1 : 1;
  A.dM = fabsf(m);
  A.dN = fabsf(nn);
  if (!(A.dM > 0.f)) A.step = 0.0f;
  A.isM = 1.0f / A.dM;
  A.isN = A.dN > 0.f ? 1.0f / A.dN : 0.f;
  A.hM = 0.5f * A.dM;
  A.hN = 0.5f * A.dN;
  A.g = A.dN * A.dM * (1.0f / 12.0f);
  return A;
}

// Whether the warps of the axis kernels span detector columns (u) instead of
// rows: when a pixel step along u moves the ray less across the volume's y
// planes than one along v. 1024 x 1024 x 64 at 84 degrees, where rows cross
// 8 planes a warp and lose half the lanes: 1905 us with rows, 844 with columns
// and the walk's other changes (worth 20 % where rows stay in one plane).
inline int axis_swap(const KConst& c) {
  const float uy = c.aniso[0] * c.u.y + c.aniso[3] * c.v.y, vy = c.aniso[1] * c.u.y + c.aniso[4] * c.v.y;
  return fabsf(uy) < fabsf(vy) ? 1 : 0;
}

inline dim3 axis_grid(int swap, int nw, int w, int h) {
  const int along = swap ? w : h, across = swap ? h : w;
  return dim3((across + nw - 1) / nw, (along + 7) / 8);
}

}  // namespace raycore
}  // namespace esb
