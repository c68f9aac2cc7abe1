// The mixed form's dispatch by polynomial order and volume rule (its kernels:
// euler_tri_mixed_kernels.cu), and the per-case CFL speed of a batch.
#include <stdexcept>

#include "euler_device.cuh"
#include "euler_tri_mixed.hpp"
#include "kernels.hpp"

namespace wasl_b200 {

// Per-case CFL speed over a tile work list: the largest cell-average wave
// speed |u| + c of each case (the CFL kernels' formula), max-reduced as FP64
// bits into speed[case]; a non-physical average sets the error word.
__global__ void batch_speed(const double *state, std::int64_t ne, int M, double gamma,
                            const TileWork *work, unsigned long long *speed,
                            unsigned long long *error, int *status) {
  const TileWork w = work[blockIdx.x];
  const int lane = threadIdx.x & 31;
  unsigned long long best = 0;
  for (int i = threadIdx.x; i < w.count; i += blockDim.x) {
    const std::int64_t e = w.first + i;
    const double scale = 1.0 / sqrt(2.0);
    const std::int64_t plane = static_cast<std::int64_t>(M) * ne;
    const double s[4] = {__dmul_rn(scale, state[e]), __dmul_rn(scale, state[plane + e]),
                         __dmul_rn(scale, state[2 * plane + e]),
                         __dmul_rn(scale, state[3 * plane + e])};
    bool physical = true;
    const double speed = cfl_speed(gamma, s, 2, physical);
    if (physical) {
      const unsigned long long bits = __double_as_longlong(speed);
      best = bits > best ? bits : best;
    } else if (status) {
      atomicCAS(status + w.case_id, 0, static_cast<int>(kNonPhysicalAverage));
    } else {
      raise_error(error, kNonPhysicalAverage, e);
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_down_sync(0xffffffffu, best, off);
    best = o > best ? o : best;
  }
  if (lane == 0 && best)
    atomicMax(speed + w.case_id, best);
}

namespace {

// Op<P, R>::run(args...) for a supported (p, rule order) pair.
template <int P, int R> struct UploadMixed {
  static void run() { MixedForm<P, R>::upload(); }
};
template <int P, int R> struct StageMixed {
  static void run(const StageArgs &a, cudaStream_t s) { MixedForm<P, R>::stage(a, s); }
};
template <int P, int R> struct StageTile {
  static void run(int shape, const StageArgs &a, cudaStream_t s) {
    MixedForm<P, R>::stage_tile(shape, a, s);
  }
};
template <int P, int R> struct PrepareTile {
  static void run() { MixedForm<P, R>::prepare_tile(); }
};

template <template <int, int> class Op, typename... A> void dispatch_mixed(int p, int rule, A &&...args) {
  if (rule == 0)
    rule = p + 2;
  else if (rule == kSymmetricVolumeRule)
    rule = 0; // the template's code for the symmetric rule
  switch (p * 10 + rule) {
  case 11: Op<1, 1>::run(args...); break;
  case 12: Op<1, 2>::run(args...); break;
  case 13: Op<1, 3>::run(args...); break;
  case 22: Op<2, 2>::run(args...); break;
  case 23: Op<2, 3>::run(args...); break;
  case 24: Op<2, 4>::run(args...); break;
  case 33: Op<3, 3>::run(args...); break;
  case 34: Op<3, 4>::run(args...); break;
  case 35: Op<3, 5>::run(args...); break;
  case 10: Op<1, 0>::run(args...); break;
  case 20: Op<2, 0>::run(args...); break;
  case 30: Op<3, 0>::run(args...); break;
  default:
    throw std::invalid_argument("mixed form: polynomial order must be 1..3 and the volume rule"
                                " order p..p+2");
  }
}

} // namespace

bool euler_tri_mixed_supported(int p, int rule) {
  if (rule == 0)
    rule = p + 2;
  return p >= 1 && p <= 3 && (rule == kSymmetricVolumeRule || (rule >= p && rule <= p + 2));
}

std::size_t euler_tri_mixed_face_record_bytes(int p) {
  switch (p) {
  case 1: return MixedForm<1, 0>::face_record_bytes();
  case 2: return MixedForm<2, 0>::face_record_bytes();
  case 3: return MixedForm<3, 0>::face_record_bytes();
  default: throw std::invalid_argument("mixed form: polynomial order must be 1..3");
  }
}

void upload_euler_tri_tables_mixed(int p, int rule) {
  dispatch_mixed<UploadMixed>(p, rule);
}

int euler_tri_tile_shapes() { return kTileShapes; }

int euler_tri_tile_elements(int shape) {
  return shape >= 0 && shape < kTileShapes ? kTileElements[shape] : 0;
}

bool euler_tri_tile_is_patch(int shape) { return shape >= kFirstPatchShape && shape < kPatchShapeEnd; }

bool euler_tri_tile_limits(int shape) { return shape != 12 && shape != 13; }



void prepare_euler_tri_stage_tile(int p, int rule) { dispatch_mixed<PrepareTile>(p, rule); }

void launch_euler_tri_stage_tile(int p, int rule, int shape, const StageArgs &a, cudaStream_t s) {
  dispatch_mixed<StageTile>(p, rule, shape, a, s);
}

void launch_batch_speed(const double *state, std::int64_t ne, int M, double gamma,
                        const TileWork *work, std::int64_t work_count, unsigned long long *speed,
                        unsigned long long *error, int *status, cudaStream_t s) {
  if (work_count > 0)
    batch_speed<<<static_cast<unsigned>(work_count), 128, 0, s>>>(state, ne, M, gamma, work, speed,
                                                                  error, status);
}

void launch_euler_tri_stage_mixed(int p, int rule, const StageArgs &a, cudaStream_t s) {
  dispatch_mixed<StageMixed>(p, rule, a, s);
}

} // namespace wasl_b200
