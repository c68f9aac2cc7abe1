// The HLLC flux of the plain FP64 kernels.  Include it only where products and
// sums are not contracted (--fmad=false).
#pragma once

#include "euler_device.cuh"

namespace wasl_b200 {

// The HLLC flux of hllc() (euler_device.cuh; cpp/include/wasl/flux/hllc.hpp:40-74)
// with the side whose state the flux is built on chosen before its physical
// flux and star state are evaluated, not after both sides' are: the same
// expressions on the chosen side, so the same doubles, one evaluation of each
// for every branch, and no divergence between the branches of a warp.
__device__ __forceinline__ void hllc_selected(double gamma, const double (&l)[4],
                                              const double (&r)[4], double nx, double ny,
                                              double (&f)[4]) {
  const Prim<double> lv = primitive(gamma, l);
  const Prim<double> rv = primitive(gamma, r);
  const double lu = lv.vx * nx + lv.vy * ny;
  const double ru = rv.vx * nx + rv.vy * ny;
  const double lc = sound_speed(gamma, lv);
  const double rc = sound_speed(gamma, rv);
  const double sl = smin(lu - lc, ru - rc);
  const double sr = smax(lu + lc, ru + rc);
  const double contact = (rv.p - lv.p + l[0] * lu * (sl - lu) - r[0] * ru * (sr - ru)) /
                         (l[0] * (sl - lu) - r[0] * (sr - ru));
  // The reference's tests in its order (NaN speeds fall through to the right
  // star state, as there).
  const bool left_flow = sl >= 0.0, right_flow = sr <= 0.0;
  const bool left = left_flow || (!right_flow && contact >= 0.0);
  double s[4];
#pragma unroll
  for (int v = 0; v < 4; ++v)
    s[v] = left ? l[v] : r[v];
  const double vx = left ? lv.vx : rv.vx, vy = left ? lv.vy : rv.vy, p = left ? lv.p : rv.p;
  const double un = left ? lu : ru, wave = left ? sl : sr;
  const double energy = s[3] + p;
  f[0] = nx * s[1] + ny * s[2];
  f[1] = nx * (s[1] * vx + p) + ny * (s[1] * vy);
  f[2] = nx * (s[2] * vx) + ny * (s[2] * vy + p);
  f[3] = nx * (energy * vx) + ny * (energy * vy);
  if (!left_flow && !right_flow) {
    const double rho_star = s[0] * (wave - un) / (wave - contact);
    const double shift = contact - un;
    const double e_star = s[3] / s[0] + shift * (contact + p / (s[0] * (wave - un)));
    f[0] = f[0] + wave * (rho_star - s[0]);
    f[1] = f[1] + wave * (rho_star * (vx + shift * nx) - s[1]);
    f[2] = f[2] + wave * (rho_star * (vy + shift * ny) - s[2]);
    f[3] = f[3] + wave * (rho_star * e_star - s[3]);
  }
}

} // namespace wasl_b200
