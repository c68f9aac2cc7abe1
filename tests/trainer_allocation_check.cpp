// The indicator trainer's host code (mlp_trainer.cpp) on a CUDA runtime whose
// device memory is the heap and whose allocations fail on request: whatever the
// launches are given must be allocated and large enough, also in calls that follow
// a failed one.  Run by tests/test_host_trainer_allocation.py.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "mlp.hpp"

namespace {
std::map<const void *, std::size_t> live;
int until_failure = -1; // allocations that still succeed; -1: all
int bad = 0;

void need(const void *p, std::size_t bytes, const char *what) {
  const auto it = live.find(p);
  if (!p || it == live.end() || it->second < bytes) {
    std::printf("%s: %zu bytes of %s\n", what, bytes, p ? "a smaller allocation" : "nothing");
    ++bad;
  }
}
} // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, std::size_t n) {
  if (until_failure == 0)
    return cudaErrorMemoryAllocation;
  if (until_failure > 0)
    --until_failure;
  *p = std::malloc(n);
  live[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  live.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, std::size_t n, cudaMemcpyKind kind, cudaStream_t) {
  const int before = bad;
  need(kind == cudaMemcpyHostToDevice ? d : s, n, "copy");
  if (bad == before)
    std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, std::size_t n, cudaStream_t) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "out of memory"; }
}

namespace wasl_b200 {
void cuda_check(cudaError_t rc, const char *what) {
  if (rc != cudaSuccess)
    throw SolverError(WASL_ERR_CUDA, what);
}
MlpShape mlp_shape(int features) {
  MlpShape s;
  s.features = features;
  s.count = kMlpHidden * kMlpHidden + 1; // (the offsets all 0)
  return s;
}
int mlp_train_rows(std::int64_t samples) { return static_cast<int>(samples / kMlpBatch); }
std::size_t mlp_packed_floats(const MlpShape &s) { return s.count; }
void launch_mlp_pack(const MlpShape &, const float *, const MlpWorkspace &, cudaStream_t) {}
void launch_mlp_train(const MlpShape &s, const float *features, const std::uint8_t *labels,
                      std::int64_t n, std::int64_t, std::int64_t samples, float,
                      const MlpWorkspace &w, cudaStream_t) {
  const std::size_t rows = mlp_train_rows(samples);
  need(features, sizeof(float) * n * s.features, "features");
  need(labels, n, "labels");
  need(w.rows, sizeof(float) * rows * s.count, "gradient rows");
  need(w.losses, sizeof(double) * rows, "losses");
}
void launch_mlp_gradient(const MlpShape &, std::int64_t, const MlpWorkspace &, float *, double *,
                         cudaStream_t) {}
void launch_mlp_adam(const MlpShape &, std::int64_t, const MlpWorkspace &, double *loss, float *,
                     float *, float *, float, float, float, float, std::int64_t, cudaStream_t) {
  *loss = 0.0;
}
void launch_mlp_predict(const MlpShape &, const float *, const float *, std::int64_t, float *,
                        cudaStream_t) {}
} // namespace wasl_b200

int main() {
  using namespace wasl_b200;
  const std::vector<float> x(512 * 16, 0.5f);
  const std::vector<std::uint8_t> y(512, 1);
  for (const int first : {0, 64, 256})   // samples of a training before the failure
    for (const int fail : {0, 1}) {      // the allocation that fails
      MlpTrainer t(16, 1, 0);
      t.set_data(x.data(), y.data(), 256);
      if (first)
        t.train(1, first, 1e-3, 1.0);
      int thrown = 0;
      const auto failing = [&](auto &&call) {
        until_failure = fail;
        try {
          call();
        } catch (const SolverError &) {
          ++thrown;
        }
        until_failure = -1;
      };
      failing([&] { t.train(1, 512, 1e-3, 1.0); }); // the scratch grows
      for (const int batch : {64, 256, 512})
        t.train(1, batch, 1e-3, 1.0);
      failing([&] { t.set_data(x.data(), y.data(), 512); });
      try { // without data: refused, or trained on what there is
        t.train(1, 64, 1e-3, 1.0);
      } catch (const SolverError &) {
        ++thrown;
      }
      t.set_data(x.data(), y.data(), 512);
      t.train(1, 512, 1e-3, 1.0);
      if (thrown != 3) {
        std::printf("%d errors instead of 3 (first %d, failing %d)\n", thrown, first, fail);
        ++bad;
      }
    }
  std::printf("%d failures\n", bad);
  return bad != 0;
}
