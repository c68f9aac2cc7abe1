// Whether an element provably keeps density and pressure at or above the
// positivity limiter's check-point floors, from bounds on its point values:
// |sum_{m>=1} c_m phi_m| <= sum_{m>=1} |c_m| max|phi_m| (max over the check
// points), then the pressure's lower bound from the bounds on density, momentum
// and energy.  Where it holds the limiter would scale by exactly 1, so skipping
// it gives the same bits.  Small margins cover the rounding of the point sums
// and of these bounds themselves (with or without contraction).
#pragma once

#include "euler_device.cuh"
#include "kernels.hpp"

namespace wasl_b200 {

// mode0[v]: the mean modes; reach[v] = sum_{m>=1} |c_m| bound[m].
__device__ __forceinline__ bool positivity_clear(double gamma, const PositivityFloors &floors,
                                                 const double (&mode0)[4],
                                                 const double (&reach)[4]) {
  const double inv_root2 = 1.0 / sqrt(2.0);
  const double avg[4] = {mode0[0] * inv_root2, mode0[1] * inv_root2, mode0[2] * inv_root2,
                         mode0[3] * inv_root2};
  if (!(avg[0] > floors.density && primitive(gamma, avg).p > floors.pressure))
    return false; // the limiter reports it
  const double rf =
      floors.relative > 0.0 ? fmax(floors.density, floors.relative * avg[0]) : floors.density;
  const double pf =
      floors.relative > 0.0 ? fmax(floors.pressure, floors.relative * avg[3]) : floors.pressure;
  const double rho_lo = avg[0] - reach[0] - 1e-12 * (avg[0] + reach[0]);
  if (!(rho_lo >= rf))
    return false;
  const double mx = fabs(avg[1]) + reach[1], my = fabs(avg[2]) + reach[2];
  const double energy_lo = avg[3] - reach[3];
  const double kinetic = 0.5 * (mx * mx + my * my) / rho_lo;
  const double p_lo = (gamma - 1.0) * (energy_lo - kinetic) -
                      1e-12 * (gamma - 1.0) * (fabs(avg[3]) + reach[3] + kinetic);
  return p_lo >= pf;
}

// The active lanes' elements with `listed` set appended to a list, one atomic
// per warp.
__device__ __forceinline__ void append_listed(bool listed, std::int64_t e, std::int32_t *list,
                                              std::int32_t *count) {
  const unsigned mask = __activemask();
  const unsigned ballot = __ballot_sync(mask, listed);
  if (!ballot)
    return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(ballot) - 1;
  int base = 0;
  if (lane == leader)
    base = atomicAdd(count, __popc(ballot));
  base = __shfl_sync(mask, base, leader);
  if (listed)
    list[base + __popc(ballot & ((1u << lane) - 1u))] = static_cast<std::int32_t>(e);
}

} // namespace wasl_b200
