// Plain FP64 kernels of the 1D SSP-RK3 stage on line meshes, bit-consistent
// with the reference CPU solver:
//   compressible Euler  cpp/include/wasl/dg/euler/line_residual.hpp:24-86
//   scalar advection    cpp/include/wasl/dg/scalar_advection/line_residual.hpp:48-111
// with the boundary exteriors evaluated inline:
//   Euler ends          cpp/src/boundaries/line_euler_exterior.cpp:13-43
//   scalar ends         cpp/include/wasl/boundaries/line_boundary_conditions.hpp:36-57
//
// Compiled with --fmad=false.  One thread owns one element; the reference's
// face loop runs in ascending face index and element e owns faces e (left)
// and e+1 (right), so the thread adds the volume term, then its left face,
// then its right face.  An Euler face's flux is computed once, by the thread of
// its right element, and passed to the left one (which computes it again only
// between two blocks); an advection flux is one product, which both elements
// form from the same trace.  Either way both use the same double.  Then
// rhs *= 1/J and the Shu-Osher combination (time/ssp_rk3.hpp:44-60).
#include <algorithm>
#include <stdexcept>
#include <string>

#include "basis.hpp"
#include "euler_device.cuh"
#include "hllc_selected.cuh"
#include "kernels.hpp"

namespace wasl_b200 {
namespace {

// Trace of a thread-local element at an endpoint (modes summed from 0.0).
template <int V, int M>
__device__ __forceinline__ void trace_local(const double (&c)[V][M], const double *b, double *s) {
#pragma unroll
  for (int v = 0; v < V; ++v) {
    double acc = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m)
      acc += c[v][m] * b[m];
    s[v] = acc;
  }
}

template <int V, int M>
__device__ __forceinline__ void trace_global(const double *u, std::int64_t ne,
                                             std::int64_t e, const double *b, double *s) {
#pragma unroll
  for (int v = 0; v < V; ++v) {
    double acc = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m)
      acc += u[(static_cast<std::int64_t>(v) * M + m) * ne + e] * b[m];
    s[v] = acc;
  }
}

// scalar_advection.hpp:36-42
__device__ __forceinline__ double upwind(double a, double l, double r) {
  return a >= 0.0 ? a * l : a * r;
}

// One element's stage: residual of `in`, scaled by 1/J, and the Shu-Osher
// combination into `out`; rho receives the new density (or scalar) modes.
// The pointers carry no __restrict__: the whole-run kernel reads buffers that
// other threads of its block wrote earlier in the same launch.
template <int V, int P>
__device__ __forceinline__ void line_element_stage(const LineStageArgs &a, std::int64_t e,
                                                   const double *in, const double *u0,
                                                   double *out, int stage, double dt,
                                                   double (&rho)[P + 1]) {
  constexpr int M = P + 1;
  constexpr int NQ = V == 4 ? P + 1 : (P > 0 ? P : 1);
  const std::int64_t ne = a.ne;
  const LineTable &T = a.table;
  const double *lb = T.lb, *rb = T.rb;

  double c[V][M], r[V][M];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      c[v][m] = in[(static_cast<std::int64_t>(v) * M + m) * ne + e];
      r[v][m] = 0.0;
    }
  if constexpr (V == 4) {
    const double gamma = a.gamma;
    // Volume term: sum_q w_q F(u_q) dphi/dxi (line_residual.hpp:34-45).
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double s[4], fx[4], fy[4];
      trace_local<4, M>(c, T.phi[q], s);
      flux_xy(gamma, s, fx, fy);
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int m = 0; m < M; ++m)
          r[v][m] += T.w[q] * fx[v] * T.dphi[q][m];
    }
    // Left face (face e): the flux runs from the left state to this element's
    // left trace; at the left end the exterior is the periodic image (the last
    // element's right trace) or this element's own trace (outflow).
    {
      double own[4], other[4], f[4];
      trace_local<4, M>(c, lb, own);
      if (e > 0)
        trace_global<4, M>(in, ne, e - 1, rb, other);
      else if (a.left_kind == 0)
        trace_global<4, M>(in, ne, ne - 1, rb, other);
      else
        trace_local<4, M>(c, lb, other);
      hllc(gamma, other, own, 1.0, 0.0, f);
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int m = 0; m < M; ++m)
          r[v][m] += lb[m] * f[v];
    }
    // Right face (face e+1).
    {
      double own[4], other[4], f[4];
      trace_local<4, M>(c, rb, own);
      if (e + 1 < ne)
        trace_global<4, M>(in, ne, e + 1, lb, other);
      else if (a.right_kind == 0)
        trace_global<4, M>(in, ne, 0, lb, other);
      else
        trace_local<4, M>(c, rb, other);
      hllc(gamma, own, other, 1.0, 0.0, f);
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int m = 0; m < M; ++m)
          r[v][m] += -rb[m] * f[v];
    }
  } else {
    const double speed = a.speed;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double s;
      trace_local<1, M>(c, T.phi[q], &s);
      const double flux = speed * s;
#pragma unroll
      for (int m = 0; m < M; ++m)
        r[0][m] += T.w[q] * flux * T.dphi[q][m];
    }
    {
      double own, other;
      trace_local<1, M>(c, lb, &own);
      double flux;
      if (e > 0) {
        trace_global<1, M>(in, ne, e - 1, rb, &other);
        flux = upwind(speed, other, own);
      } else {
        if (a.left_kind == 1)
          other = a.left_value;
        else if (a.left_kind == 2)
          trace_local<1, M>(c, lb, &other);
        else
          trace_global<1, M>(in, ne, ne - 1, rb, &other);
        flux = upwind(speed, other, own);
      }
#pragma unroll
      for (int m = 0; m < M; ++m)
        r[0][m] += lb[m] * flux;
    }
    {
      double own, other;
      trace_local<1, M>(c, rb, &own);
      if (e + 1 < ne)
        trace_global<1, M>(in, ne, e + 1, lb, &other);
      else if (a.right_kind == 1)
        other = a.right_value;
      else if (a.right_kind == 2)
        trace_local<1, M>(c, rb, &other);
      else
        trace_global<1, M>(in, ne, 0, lb, &other);
      const double flux = upwind(speed, own, other);
#pragma unroll
      for (int m = 0; m < M; ++m)
        r[0][m] -= rb[m] * flux;
    }
  }

  const double inv = a.inv_jacobian[e];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const std::int64_t idx = (static_cast<std::int64_t>(v) * M + m) * ne + e;
      const double rr = r[v][m] * inv;
      double o;
      if (stage == 0)
        o = c[v][m] + dt * rr;
      else if (stage == 1)
        o = 0.75 * u0[idx] + 0.25 * (c[v][m] + dt * rr);
      else
        o = (1.0 / 3.0) * u0[idx] + (2.0 / 3.0) * (c[v][m] + dt * rr);
      out[idx] = o;
      if (v == 0)
        rho[m] = o;
    }
}

// Modal-decay sensor on the density modes (modal_decay.hpp:23-33).
template <int M>
__device__ __forceinline__ void line_sensor(const LineStageArgs &a, std::int64_t e,
                                            const double (&rho)[M]) {
  if (!a.sense)
    return;
  double total = 0.0, high = 0.0;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    total += rho[m] * rho[m];
    if (m >= a.highest_degree_begin)
      high += rho[m] * rho[m];
  }
  const bool troubled = !(total == 0.0 || high / total <= a.threshold);
  a.flags[e] = troubled ? 1 : 0;
  const unsigned active = __activemask();
  const unsigned ballot = __ballot_sync(active, troubled);
  if (ballot) {
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(ballot) - 1;
    int base = 0;
    if (lane == leader)
      base = atomicAdd(a.troubled_count, __popc(ballot));
    base = __shfl_sync(active, base, leader);
    if (troubled)
      a.troubled[base + __popc(ballot & ((1u << lane) - 1u))] = static_cast<std::int32_t>(e);
  }
}

// Trace of a thread's element at an endpoint, the modes summed from the first
// product (a zero's sign apart, which no flux keeps, the sum from 0.0).
template <int M> __device__ __forceinline__ double trace_of(const double (&c)[M], const double *b) {
  double s = c[0] * b[0];
#pragma unroll
  for (int m = 1; m < M; ++m)
    s += c[m] * b[m];
  return s;
}

// Volume term of the Euler residual into r: sum_q w_q F(u_q) dphi/dxi
// (cpp/include/wasl/dg/euler/line_residual.hpp:34-45).  Mode 0's derivative is
// zero: its term is zero, or NaN where a flux is not finite (which mode 1's sum
// then is not either).
template <int M>
__device__ __forceinline__ void euler_volume(const LineTable &T, double gamma,
                                             const double (&c)[4][M], double (&r)[4][M]) {
#pragma unroll
  for (int v = 0; v < 4; ++v)
#pragma unroll
    for (int m = 0; m < M; ++m)
      r[v][m] = 0.0;
  if constexpr (M > 1) {
#pragma unroll
    for (int q = 0; q < M; ++q) {
      double s[4], fx[4], fy[4];
#pragma unroll
      for (int v = 0; v < 4; ++v)
        s[v] = trace_of(c[v], T.phi[q]);
      flux_xy(gamma, s, fx, fy);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const double wf = T.w[q] * fx[v];
#pragma unroll
        for (int m = 1; m < M; ++m)
          r[v][m] += wf * T.dphi[q][m];
      }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
      r[v][0] = 0.0 + 0.0 * r[v][1];
  } else {
    // (P0: the same rule, for the NaN of a flux that is not finite.)
    double s[4], fx[4], fy[4];
#pragma unroll
    for (int v = 0; v < 4; ++v)
      s[v] = trace_of(c[v], T.phi[0]);
    flux_xy(gamma, s, fx, fy);
#pragma unroll
    for (int v = 0; v < 4; ++v)
      r[v][0] += T.w[0] * fx[v] * T.dphi[0][0];
  }
}

// The Shu-Osher combination of one coefficient (time/ssp_rk3.hpp:44-60).
__device__ __forceinline__ double combine(int stage, double u0, double c, double dt, double rr) {
  if (stage == 0)
    return c + dt * rr;
  if (stage == 1)
    return 0.75 * u0 + 0.25 * (c + dt * rr);
  return (1.0 / 3.0) * u0 + (2.0 / 3.0) * (c + dt * rr);
}

// One Euler stage with each face's flux evaluated once: a block of 128 threads
// computes the 128 faces first .. first + 127 (thread t: face first + t, the
// left face of element first + t) and updates the 127 elements between them;
// right traces and fluxes pass between neighbouring threads through shared
// memory.  Bound by the FP64 pipe (two HLLC fluxes of 190 operations per
// element were more than half of its work) and by the 96 M bytes per element
// that stages 2 and 3 move.  Four steps at 1,000,003 cells, P2: 1978 -> 843 us
// (with one thread per element evaluating both its faces: 150 us a stage).
constexpr int kLineBlock = 128;

// Resident blocks per SM the registers are sized for; at P0 to P3 the bound spills
// (36, 72, 88 and 188 bytes of stores) and pays all the same.  Measured, four
// steps: P0 (1,000,003 cells) 438 us (7: 444, 9: 431, 10: 494, no bound: 482; at
// 300,000 cells 174, 177, 179, 197, 186); P1 (700,001) 486 us (7: 510, 9: 505, no
// bound: 595); P2 (1,000,003) 843 us (6: 883, 8: 888, no bound: 977); P3 (700,001)
// 868 us (5: 885, 7: 1002); from P4 on it costs (100,001 cells: 272 us without,
// 312 at 6).
template <int P> constexpr int kLineBlocks = P <= 1 ? 8 : P == 2 ? 7 : P == 3 ? 6 : 1;

template <int P>
__global__ void __launch_bounds__(kLineBlock, kLineBlocks<P>) line_euler_stage_f64(const LineStageArgs a) {
  constexpr int M = P + 1;
  __shared__ double right[4][kLineBlock], flux[4][kLineBlock];
  const int t = threadIdx.x;
  const std::int64_t ne = a.ne;
  const std::int64_t e = static_cast<std::int64_t>(blockIdx.x) * (kLineBlock - 1) + t;
  const bool present = e < ne;
  const LineTable &T = a.table;
  const double *lb = T.lb, *rb = T.rb;
  double c[4][M];
  if (present) {
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
      for (int m = 0; m < M; ++m)
        c[v][m] = a.in[(static_cast<std::int64_t>(v) * M + m) * ne + e];
#pragma unroll
    for (int v = 0; v < 4; ++v)
      right[v][t] = trace_of(c[v], rb);
  }
  const bool updates = present && t < kLineBlock - 1;
  if (a.stage > 0 && updates) {
    // u^n (read by the combination) into L1 meanwhile.
#pragma unroll
    for (int row = 0; row < 4 * M; ++row)
      asm volatile("prefetch.global.L1 [%0];\n" ::"l"(a.u0 + static_cast<std::int64_t>(row) * ne + e));
  }
  __syncthreads();
  double f[4] = {0.0, 0.0, 0.0, 0.0};
  if (e <= ne) {
    // Left and right states of face e: the ends take the periodic image or the
    // end element's own trace (outflow).
    double ls[4], rs[4];
    if (e > 0 && t > 0) {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        ls[v] = right[v][t - 1];
    } else if (e > 0 || a.left_kind == 0) {
      trace_global<4, M>(a.in, ne, e > 0 ? e - 1 : ne - 1, rb, ls);
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        ls[v] = trace_of(c[v], lb);
    }
    if (present) {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        rs[v] = trace_of(c[v], lb);
    } else if (a.right_kind == 0) {
      trace_global<4, M>(a.in, ne, 0, lb, rs);
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        rs[v] = ls[v];
    }
    hllc_selected(a.gamma, ls, rs, 1.0, 0.0, f);
#pragma unroll
    for (int v = 0; v < 4; ++v)
      flux[v][t] = f[v];
  }
  __syncthreads();
  if (!updates)
    return;
  double r[4][M], rho[M], mean[4];
  euler_volume(T, a.gamma, c, r);
  const double inv = a.inv_jacobian[e];
  const double dt = a.dt ? *a.dt : a.dt_value;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const double after = flux[v][t + 1];
#pragma unroll
    for (int m = 0; m < M; ++m) {
      r[v][m] += lb[m] * f[v];
      r[v][m] += -rb[m] * after;
      const std::int64_t idx = (static_cast<std::int64_t>(v) * M + m) * ne + e;
      const double o = combine(a.stage, a.stage > 0 ? a.u0[idx] : 0.0, c[v][m], dt, r[v][m] * inv);
      a.out[idx] = o;
      if (v == 0)
        rho[m] = o;
      if (m == 0)
        mean[v] = o;
    }
  }
  if (a.speed_max) {
    // The next step's CFL speed from this stage's cell averages (the CFL
    // kernels' formula), the warp's largest to the word.
    const double scale = 1.0 / sqrt(2.0);
    const double sa[4] = {scale * mean[0], scale * mean[1], scale * mean[2], scale * mean[3]};
    bool physical = true;
    const double speed = cfl_speed(a.gamma, sa, 1, physical);
    unsigned long long best = 0;
    if (physical)
      best = __double_as_longlong(speed);
    else
      raise_error(a.error, kNonPhysicalAverage, e);
    const unsigned mask = __activemask();
    const unsigned hi = __reduce_max_sync(mask, static_cast<unsigned>(best >> 32));
    const unsigned lo = __reduce_max_sync(
        mask, static_cast<unsigned>(best >> 32) == hi ? static_cast<unsigned>(best) : 0u);
    if ((t & 31) == __ffs(mask) - 1)
      atomicMax(a.speed_max, (static_cast<unsigned long long>(hi) << 32) | lo);
  }
  line_sensor<M>(a, e, rho);
}

// One scalar advection stage, one thread per element (bound by the state's
// bytes: 90% of the HBM rate).
template <int P>
__global__ void __launch_bounds__(128) line_scalar_stage_f64(const LineStageArgs a) {
  constexpr int M = P + 1;
  const std::int64_t e = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= a.ne)
    return;
  double rho[M];
  line_element_stage<1, P>(a, e, a.in, a.u0, a.out, a.stage, a.dt ? *a.dt : a.dt_value, rho);
}

// A whole run in one launch of one CTA (meshes whose three state buffers fit
// in its shared memory): the serial run loop of cpp/src/case/serial_case_runner.cpp:107-142
// (dt clipped to land on end_time; "timestep cannot advance time" ends the
// run) around the SSP-RK3 stages of the stage kernels, with a block barrier
// between stages instead of a kernel boundary.  The CFL step is fixed
// (fixed_dt > 0: scalar advection, cfl_timestep.cpp:55-60) or taken from the
// state each step (Euler: the largest |u| + c of the cell averages,
// cfl_timestep.cpp:33-47 and 70-76, the arithmetic of the CFL kernels).
template <int V, int P> __global__ void __launch_bounds__(512) line_run_f64(LineRunArgs r) {
  constexpr int M = P + 1;
  extern __shared__ double buffers[]; // u, stage 1, stage 2: V M ne each
  const std::int64_t ne = r.stage.ne, n = static_cast<std::int64_t>(V) * M * ne;
  double *u = buffers, *s1 = buffers + n, *s2 = buffers + 2 * n;
  for (std::int64_t i = threadIdx.x; i < n; i += blockDim.x)
    u[i] = r.state[i];
  __shared__ unsigned long long speed_bits[32];
  __shared__ int status;
  if (threadIdx.x == 0)
    status = 0;
  __syncthreads();
  double time = r.start_time;
  unsigned long long steps = 0;
  while (time < r.end_time && steps < r.max_steps) {
    double stable = r.fixed_dt;
    if (V == 4) {
      // Largest cell-average speed, with the CFL kernels' physical-state check.
      unsigned long long best = 0;
      for (std::int64_t e = threadIdx.x; e < ne; e += blockDim.x) {
        const double scale = 1.0 / sqrt(2.0);
        const double sa[4] = {scale * u[e], scale * u[M * ne + e], scale * u[2 * M * ne + e],
                              scale * u[3 * M * ne + e]};
        bool physical = true;
        const double speed = cfl_speed(r.stage.gamma, sa, 1, physical);
        if (!physical) {
          raise_error(r.error, kNonPhysicalAverage, e);
          status = 2;
        } else {
          const unsigned long long bits = __double_as_longlong(speed);
          best = bits > best ? bits : best;
        }
      }
      for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, best, off);
        best = o > best ? o : best;
      }
      if ((threadIdx.x & 31) == 0)
        speed_bits[threadIdx.x >> 5] = best;
      __syncthreads();
      best = 0;
      for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w)
        best = speed_bits[w] > best ? speed_bits[w] : best;
      __syncthreads();
      if (status)
        break;
      const double speed = __longlong_as_double(static_cast<long long>(best));
      stable = speed > 0.0 ? r.cfl * r.length / (speed * (2 * P + 1)) : 0.0;
    }
    const double remaining = r.end_time - time;
    const double dt = stable > 0.0 ? (remaining < stable ? remaining : stable) : remaining;
    if (dt <= 0.0 || time + dt == time) {
      status = 1; // every thread finds the same dt: the same value, one break
      break;
    }
    double *ins[3] = {u, s1, s2}, *outs[3] = {s1, s2, u};
    for (int k = 0; k < 3; ++k) {
      double rho[M];
      for (std::int64_t e = threadIdx.x; e < ne; e += blockDim.x)
        line_element_stage<V, P>(r.stage, e, ins[k], u, outs[k], k, dt, rho);
      __syncthreads();
    }
    time += dt;
    ++steps;
  }
  __syncthreads();
  for (std::int64_t i = threadIdx.x; i < n; i += blockDim.x)
    r.state[i] = u[i];
  if (threadIdx.x == 0) {
    r.result[0] = steps;
    r.result[1] = static_cast<unsigned long long>(__double_as_longlong(time));
    r.result[2] = static_cast<unsigned long long>(status);
  }
}

// The same run with one element per thread, for meshes of fewer than
// kRunThreads elements: the stage's coefficients stay in registers over the whole
// run (and u^n too, for scalar advection; in the thread's column of shared memory
// for Euler), and only what a neighbour needs passes through shared memory: the
// one trace an upwind flux reads, or Euler's right traces and face fluxes.
// Against the kernel above, which keeps the three state buffers in shared memory,
// evaluates every trace twice and reads each coefficient it needs, 300 Euler
// cells at P2 take 7.7 instead of 12.8 ms a run.  Bound by the FP64 pipe of one
// SM and the barriers (one per advection stage, two per Euler stage).
//
// Advection from kRunClusterFrom cells on runs on a cluster (launch_run), whose
// blocks have up to kRunClusterThreads threads; Euler from P4 on does not fit
// the registers.
constexpr int kRunClusterFrom = 96;
template <int V, int P> constexpr int kRunThreads = V == 1 ? kRunClusterFrom : P <= 3 ? 512 : 0;
template <int P> constexpr int kRunClusterThreads = P <= 2 ? 1024 : 512;

template <int V, int P>
__global__ void __launch_bounds__(kRunThreads<V, P>) line_run_registers_f64(LineRunArgs r) {
  constexpr int M = P + 1;
  extern __shared__ double run_smem[];
  const int n = static_cast<int>(r.stage.ne), e = threadIdx.x, T = blockDim.x;
  const bool active = e < n;
  const LineTable &table = r.stage.table;
  const double *lb = table.lb, *rb = table.rb;
  __shared__ unsigned long long speed_bits[32];
  __shared__ double first_left[4]; // element 0's left trace (Euler)
  __shared__ int status;
  if (e == 0)
    status = 0;
  double c[V][M];
  double un[V == 1 ? M : 1]; // u^n (scalar)
  double *held = run_smem;   // u^n (Euler): [V M][T]
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int m = 0; m < M; ++m)
      c[v][m] = active ? r.state[(v * M + m) * n + e] : 0.0;
  const double inv = active ? r.stage.inv_jacobian[e] : 0.0;
  __syncthreads();
  double time = r.start_time;
  unsigned long long steps = 0;
  int buffer = 0;
  while (time < r.end_time && steps < r.max_steps) {
    double stable = r.fixed_dt;
    if constexpr (V == 4) {
      // Largest cell-average speed, with the CFL kernels' physical-state check.
      unsigned long long best = 0;
      if (active) {
        const double scale = 1.0 / sqrt(2.0);
        const double sa[4] = {scale * c[0][0], scale * c[1][0], scale * c[2][0], scale * c[3][0]};
        bool physical = true;
        const double speed = cfl_speed(r.stage.gamma, sa, 1, physical);
        if (!physical) {
          raise_error(r.error, kNonPhysicalAverage, e);
          status = 2;
        } else {
          best = __double_as_longlong(speed);
        }
      }
      for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, best, off);
        best = o > best ? o : best;
      }
      if ((e & 31) == 0)
        speed_bits[e >> 5] = best;
      __syncthreads();
      best = 0;
      for (int w = 0; w < (T >> 5); ++w)
        best = speed_bits[w] > best ? speed_bits[w] : best;
      __syncthreads();
      if (status)
        break;
      const double speed = __longlong_as_double(static_cast<long long>(best));
      stable = speed > 0.0 ? r.cfl * r.length / (speed * (2 * P + 1)) : 0.0;
    }
    const double remaining = r.end_time - time;
    const double dt = stable > 0.0 ? (remaining < stable ? remaining : stable) : remaining;
    if (dt <= 0.0 || time + dt == time) {
      status = 1; // every thread finds the same dt: the same value, one break
      break;
    }
    if constexpr (V == 1) {
#pragma unroll
      for (int m = 0; m < M; ++m)
        un[m] = c[0][m];
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int m = 0; m < M; ++m)
          held[(v * M + m) * T + e] = c[v][m];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if constexpr (V == 1) {
        // The upwind flux reads the left state's trace for a speed >= 0 and
        // the right state's otherwise (scalar_advection.hpp:36-42); two
        // buffers, so one barrier per stage keeps readers and writers apart.
        const double speed = r.stage.speed;
        const bool forward = speed >= 0.0;
        double *traces = run_smem + buffer * T;
        buffer ^= 1;
        const double own = trace_of(c[0], forward ? rb : lb);
        traces[e] = own;
        double rhs[M];
#pragma unroll
        for (int m = 0; m < M; ++m)
          rhs[m] = 0.0;
        if constexpr (P > 0) {
#pragma unroll
          for (int q = 0; q < P; ++q) {
            const double wf = table.w[q] * (speed * trace_of(c[0], table.phi[q]));
#pragma unroll
            for (int m = 1; m < M; ++m)
              rhs[m] += wf * table.dphi[q][m];
          }
          rhs[0] = 0.0 + 0.0 * rhs[1]; // (mode 0's derivative is zero)
        } else {
          rhs[0] += table.w[0] * (speed * trace_of(c[0], table.phi[0])) * table.dphi[0][0];
        }
        __syncthreads();
        double before, after;
        if (forward) {
          double left;
          if (e > 0)
            left = traces[e - 1];
          else if (r.stage.left_kind == 1)
            left = r.stage.left_value;
          else if (r.stage.left_kind == 2)
            left = trace_of(c[0], lb);
          else
            left = traces[n - 1];
          before = speed * left;
          after = speed * own;
        } else {
          double right;
          if (e + 1 < n)
            right = traces[e + 1];
          else if (r.stage.right_kind == 1)
            right = r.stage.right_value;
          else if (r.stage.right_kind == 2)
            right = trace_of(c[0], rb);
          else
            right = traces[0];
          before = speed * own;
          after = speed * right;
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
          rhs[m] += lb[m] * before;
          rhs[m] -= rb[m] * after;
          c[0][m] = combine(k, un[m], c[0][m], dt, rhs[m] * inv);
        }
      } else {
        double(*right)[kRunThreads<V, P>] = reinterpret_cast<
            double(*)[kRunThreads<V, P>]>(run_smem + V * M * T);
        double(*flux)[kRunThreads<V, P>] = right + 4;
        double own[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          right[v][e] = trace_of(c[v], rb);
          own[v] = trace_of(c[v], lb);
          if (e == 0)
            first_left[v] = own[v];
        }
        __syncthreads();
        double f[4] = {0.0, 0.0, 0.0, 0.0};
        if (e <= n) {
          // Face e, between element e - 1 and this thread's.
          double ls[4];
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            ls[v] = e > 0 ? right[v][e - 1] : r.stage.left_kind == 0 ? right[v][n - 1] : own[v];
            if (e == n)
              own[v] = r.stage.right_kind == 0 ? first_left[v] : ls[v];
          }
          hllc_selected(r.stage.gamma, ls, own, 1.0, 0.0, f);
#pragma unroll
          for (int v = 0; v < 4; ++v)
            flux[v][e] = f[v];
        }
        double rhs[4][M];
        euler_volume(table, r.stage.gamma, c, rhs);
        __syncthreads();
        if (active) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const double after = flux[v][e + 1];
#pragma unroll
            for (int m = 0; m < M; ++m) {
              rhs[v][m] += lb[m] * f[v];
              rhs[v][m] += -rb[m] * after;
              c[v][m] = combine(k, held[(v * M + m) * T + e], c[v][m], dt, rhs[v][m] * inv);
            }
          }
        }
      }
    }
    time += dt;
    ++steps;
  }
  __syncthreads();
  if (active) {
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int m = 0; m < M; ++m)
        r.state[(v * M + m) * n + e] = c[v][m];
  }
  if (e == 0) {
    r.result[0] = steps;
    r.result[1] = static_cast<unsigned long long>(__double_as_longlong(time));
    r.result[2] = static_cast<unsigned long long>(status);
  }
}

// The advection run spread over a cluster of four blocks.  An upwind stage reads
// one element upstream only, so a block that also holds the kRunHalo elements
// upstream of its chunk can take kRunHalo / 3 steps on its own, the halo's
// outermost element going stale with each stage; then the blocks exchange their
// downstream ends through distributed shared memory, behind one cluster barrier
// (which costs more than a stage, so every stage would not pay: measured twice
// as slow).  Per stage a block has a quarter of the warps: at 400 cells one per
// sub-core instead of three or four, and the stage is its chain of dependent
// FP64 operations and a barrier of four warps instead of the pipe's 464 cycles.
// (The block count is a template argument: read from the grid it cost 8%.)
// The elements' arithmetic is the one-block kernel's.  400 cells at P2: 0.34 ->
// 0.18 us per stage (0.67 us when every block exchanged every stage).
constexpr int kRunHalo = 24;

template <int P, int BLOCKS>
__global__ void __launch_bounds__(kRunClusterThreads<P>) line_run_cluster_f64(LineRunArgs r) {
  constexpr int M = P + 1;
  extern __shared__ double cluster_smem[]; // traces [2][T], then edges [2][M][kRunHalo]
  const int n = static_cast<int>(r.stage.ne), t = threadIdx.x, T = blockDim.x;
  const LineTable &table = r.stage.table;
  const double *lb = table.lb, *rb = table.rb;
  const double speed = r.stage.speed;
  const bool forward = speed >= 0.0;
  const int inflow_kind = forward ? r.stage.left_kind : r.stage.right_kind;
  const double inflow_value = forward ? r.stage.left_value : r.stage.right_value;
  unsigned rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  // Positions along the flow: element s is the s-th from the inflow end; this
  // block's chunk is [begin, end), its threads hold [begin - kRunHalo, end).
  const int begin = static_cast<int>(rank) * n / BLOCKS;
  const int end = (static_cast<int>(rank) + 1) * n / BLOCKS;
  const int s = begin - kRunHalo + t;
  const bool wraps = inflow_kind == 0;
  const bool holds = s < end && (s >= 0 || wraps);
  const int along = s < 0 ? s + n : s;
  const int e = forward ? along : n - 1 - along;
  double *edges = cluster_smem + 2 * T;
  double c[M], un[M];
#pragma unroll
  for (int m = 0; m < M; ++m)
    c[m] = holds ? r.state[m * n + e] : 0.0;
  const double inv = holds ? r.stage.inv_jacobian[e] : 0.0;
  const bool at_inflow = s == 0 && !wraps;
  // The upstream block's edges (the last block's for the first, across the period).
  unsigned upstream_edges;
  {
    const unsigned local = static_cast<unsigned>(__cvta_generic_to_shared(edges));
    const unsigned from = (rank + BLOCKS - 1) % BLOCKS;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(upstream_edges) : "r"(local), "r"(from));
  }
  double time = r.start_time;
  unsigned long long steps = 0;
  unsigned long long status = 0;
  int buffer = 0, edge_buffer = 0, fresh = kRunHalo / 3;
  while (time < r.end_time && steps < r.max_steps) {
    const double remaining = r.end_time - time;
    const double dt =
        r.fixed_dt > 0.0 ? (remaining < r.fixed_dt ? remaining : r.fixed_dt) : remaining;
    if (dt <= 0.0 || time + dt == time) {
      status = 1; // every thread of the cluster finds the same dt
      break;
    }
    if (fresh == 0) {
      // The halo is stale: the downstream end of every chunk to its edges, and
      // after the barrier the upstream block's into the halo.  Two buffers:
      // a block rewrites one only after the next barrier, behind every read.
      double *mine = edges + edge_buffer * M * kRunHalo;
      const int at = s - (end - kRunHalo);
      if (at >= 0 && s < end) {
#pragma unroll
        for (int m = 0; m < M; ++m)
          mine[m * kRunHalo + at] = c[m];
      }
      asm volatile("barrier.cluster.arrive.release.aligned;\n"
                   "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
      if (t < kRunHalo && holds) {
#pragma unroll
        for (int m = 0; m < M; ++m)
          asm volatile("ld.shared::cluster.f64 %0, [%1];"
                       : "=d"(c[m])
                       : "r"(upstream_edges +
                             8u * static_cast<unsigned>((edge_buffer * M + m) * kRunHalo + t))
                       : "memory");
      }
      edge_buffer ^= 1;
      fresh = kRunHalo / 3;
    }
    --fresh;
#pragma unroll
    for (int m = 0; m < M; ++m)
      un[m] = c[m];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double *traces = cluster_smem + buffer * T;
      buffer ^= 1;
      const double own = trace_of(c, forward ? rb : lb);
      traces[t] = own;
      double rhs[M];
#pragma unroll
      for (int m = 0; m < M; ++m)
        rhs[m] = 0.0;
      if constexpr (P > 0) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const double wf = table.w[q] * (speed * trace_of(c, table.phi[q]));
#pragma unroll
          for (int m = 1; m < M; ++m)
            rhs[m] += wf * table.dphi[q][m];
        }
        rhs[0] = 0.0 + 0.0 * rhs[1]; // (mode 0's derivative is zero)
      } else {
        rhs[0] += table.w[0] * (speed * trace_of(c, table.phi[0])) * table.dphi[0][0];
      }
      __syncthreads();
      double upstream = t > 0 ? traces[t - 1] : 0.0; // (t = 0 is halo: stale)
      if (at_inflow)
        upstream = inflow_kind == 1 ? inflow_value : trace_of(c, forward ? lb : rb);
      const double in = speed * upstream, out = speed * own;
      const double before = forward ? in : out, after = forward ? out : in;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        rhs[m] += lb[m] * before;
        rhs[m] -= rb[m] * after;
        c[m] = combine(k, un[m], c[m], dt, rhs[m] * inv);
      }
    }
    time += dt;
    ++steps;
  }
  // The chunks go back to r.state only when every block has loaded its halo from
  // there (a run of up to kRunHalo / 3 steps passes no barrier above), and no
  // block leaves while another may still read its edges.
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  if (holds && s >= begin) {
#pragma unroll
    for (int m = 0; m < M; ++m)
      r.state[m * n + e] = c[m];
  }
  if (rank == 0 && t == 0) {
    r.result[0] = steps;
    r.result[1] = static_cast<unsigned long long>(__double_as_longlong(time));
    r.result[2] = status;
  }
}

template <int V, int P> void launch(const LineStageArgs &a, cudaStream_t s) {
  if constexpr (V == 4) {
    constexpr int E = kLineBlock - 1;
    // (ne + 1 faces; the last one may fall on a block's last thread)
    line_euler_stage_f64<P><<<static_cast<unsigned>((a.ne + E - 1) / E), kLineBlock, 0, s>>>(a);
  } else {
    line_scalar_stage_f64<P><<<static_cast<unsigned>((a.ne + 127) / 128), 128, 0, s>>>(a);
  }
}

template <int V> void launch_order(int p, const LineStageArgs &a, cudaStream_t s) {
  switch (p) {
  case 0: launch<V, 0>(a, s); break;
  case 1: launch<V, 1>(a, s); break;
  case 2: launch<V, 2>(a, s); break;
  case 3: launch<V, 3>(a, s); break;
  case 4: launch<V, 4>(a, s); break;
  case 5: launch<V, 5>(a, s); break;
  case 6: launch<V, 6>(a, s); break;
  default: throw std::invalid_argument("line polynomial order must be 0..6");
  }
}

// Shared memory above the default needs the opt-in attribute, once per device.
template <typename Kernel> void run_opt_in(Kernel kernel, std::size_t bytes, bool (&opted_in)[64]) {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64)
    throw std::runtime_error("resident run: no usable CUDA device");
  if (opted_in[device])
    return;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(bytes)) != cudaSuccess)
    throw std::runtime_error("resident run: shared memory opt-in failed");
  opted_in[device] = true;
}

// Advection from 96 cells on (four chunks of a halo's length): the cluster, of
// four blocks while a chunk and its halo fit in four warps, of eight above.  P2,
// us per stage, one block and the cluster: 0.220 and 0.179 at 96 cells, 0.244 and
// 0.179 at 128, 0.285 and 0.181 at 300; at 480 cells 0.346, 0.219 with four
// blocks and 0.181 with eight; P1 at 2000: 1.45, 0.30 and 0.22.  Else one element
// (and, for Euler, one face) per thread where the block has the threads and the
// registers for it; else the elements of a thread in turn.
constexpr int kRunCluster4To = 416;

template <int P, int BLOCKS> void launch_run_cluster(const LineRunArgs &r, cudaStream_t s) {
  const auto threads =
      static_cast<unsigned>(((r.stage.ne + BLOCKS - 1) / BLOCKS + kRunHalo + 31) / 32 * 32);
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(BLOCKS);
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = sizeof(double) * (2 * threads + 2 * (P + 1) * kRunHalo);
  config.stream = s;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = BLOCKS;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  if (cudaLaunchKernelEx(&config, line_run_cluster_f64<P, BLOCKS>, r) != cudaSuccess)
    throw std::runtime_error("resident run: cluster launch failed");
}

template <int V, int P> void launch_run(const LineRunArgs &r, cudaStream_t s) {
  if constexpr (V == 1) {
    if (r.stage.ne >= kRunClusterFrom && r.stage.ne <= kRunCluster4To) {
      launch_run_cluster<P, 4>(r, s);
      return;
    }
    if (r.stage.ne > kRunCluster4To && (r.stage.ne + 7) / 8 + kRunHalo <= kRunClusterThreads<P>) {
      launch_run_cluster<P, 8>(r, s);
      return;
    }
  }
  constexpr int limit = kRunThreads<V, P>;
  if constexpr (limit > 0) {
    if (r.stage.ne < limit) {
      static bool opted_in[64] = {};
      constexpr std::size_t most = sizeof(double) * limit * (V == 1 ? 2 : V * (P + 1) + 8);
      run_opt_in(line_run_registers_f64<V, P>, most, opted_in);
      const unsigned threads = static_cast<unsigned>((r.stage.ne + 1 + 31) / 32 * 32);
      const std::size_t bytes =
          sizeof(double) * (V == 1 ? 2 * threads : V * (P + 1) * threads + 8 * limit);
      line_run_registers_f64<V, P><<<1, threads, bytes, s>>>(r);
      return;
    }
  }
  // Advection from P1 on never comes here: a state of at most kLineRunMaxBytes
  // has no more cells than the cluster of eight takes.
  constexpr std::int64_t most_cells = kLineRunMaxBytes / (3 * sizeof(double) * V * (P + 1));
  if constexpr (V == 4 || (most_cells + 7) / 8 + kRunHalo > kRunClusterThreads<P>) {
    const std::size_t bytes = line_run_bytes(V, P, r.stage.ne);
    static bool opted_in[64] = {};
    run_opt_in(line_run_f64<V, P>, kLineRunMaxBytes, opted_in);
    const std::int64_t threads = std::min<std::int64_t>(512, (r.stage.ne + 31) / 32 * 32);
    line_run_f64<V, P><<<1, static_cast<unsigned>(threads), bytes, s>>>(r);
  }
}

template <int V> void launch_run_order(int p, const LineRunArgs &r, cudaStream_t s) {
  switch (p) {
  case 0: launch_run<V, 0>(r, s); break;
  case 1: launch_run<V, 1>(r, s); break;
  case 2: launch_run<V, 2>(r, s); break;
  case 3: launch_run<V, 3>(r, s); break;
  case 4: launch_run<V, 4>(r, s); break;
  case 5: launch_run<V, 5>(r, s); break;
  case 6: launch_run<V, 6>(r, s); break;
  default: throw std::invalid_argument("line polynomial order must be 0..6");
  }
}

} // namespace

std::size_t line_run_bytes(int variables, int p, std::int64_t ne) {
  return 3 * sizeof(double) * static_cast<std::size_t>(variables) * (p + 1) *
         static_cast<std::size_t>(ne);
}

void launch_line_run_f64(int variables, int p, const LineRunArgs &r, cudaStream_t s) {
  if (line_run_bytes(variables, p, r.stage.ne) > kLineRunMaxBytes || r.stage.ne < 1)
    throw std::invalid_argument("resident run: the state does not fit in one CTA's shared memory");
  if (variables == 4)
    launch_run_order<4>(p, r, s);
  else if (variables == 1)
    launch_run_order<1>(p, r, s);
  else
    throw std::invalid_argument("resident run: 1 or 4 variables");
}

bool line_order_supported(int p) { return p >= 0 && p <= 6; }

void fill_line_table(int p, int points, LineTable &t) {
  if (!line_order_supported(p) || points < 1 || points > 7)
    throw std::invalid_argument("line table: unsupported order or point count");
  t = LineTable{};
  const Rule1D rule = gauss_legendre(points);
  for (int q = 0; q < points; ++q) {
    const auto b = legendre(rule.x[q], p);
    const auto g = legendre_gradient(rule.x[q], p);
    for (int m = 0; m <= p; ++m) {
      t.phi[q][m] = b[m];
      t.dphi[q][m] = g[m];
    }
    t.w[q] = rule.w[q];
  }
  const auto l = legendre(-1.0, p), r = legendre(1.0, p);
  for (int m = 0; m <= p; ++m) {
    t.lb[m] = l[m];
    t.rb[m] = r[m];
  }
}

void launch_line_stage_f64(int variables, int p, const LineStageArgs &a, cudaStream_t s) {
  if (variables == 4)
    launch_order<4>(p, a, s);
  else if (variables == 1)
    launch_order<1>(p, a, s);
  else
    throw std::invalid_argument("line stage: 1 or 4 variables");
}

} // namespace wasl_b200
