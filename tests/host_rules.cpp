// The rules of dtq_host.h as plain functions for ctypes, with a stand-in for the runtime's error state: no GPU, no CUDA library.
#include "dtq_host.h"

namespace {
cudaError_t pending = cudaSuccess;
std::atomic<int> known[1];
int asked = 0;
}  // namespace

extern "C" {
cudaError_t cudaGetLastError() {
  const cudaError_t e = pending;
  pending = cudaSuccess;
  return e;
}

int rule_tensorwise(long long bytes, int aligned, int clusters, int cooperative) {
  return static_cast<int>(dtq::tensorwise_path(bytes, aligned != 0, clusters != 0, cooperative != 0));
}
int rule_asks_ahead(int kernel, long long bytes) { return dtq::asks_ahead(static_cast<dtq::Asks>(kernel), bytes); }
int rule_amax_asks(long long bytes, int f32, int grid, int tile_chunks) { return dtq::amax_ask_chunks(bytes, f32 != 0, grid, tile_chunks); }
int rule_turned_down(int error) { return dtq::turned_down_for_room(static_cast<cudaError_t>(error)); }

// One question about clusters: the runtime answers `n`, or fails with `error` as its runtime would.
int rule_clusters(int forget, int error, int n, int pending_before, int *pending_after, int *questions) {
  if (forget) {
    known[0] = 0;
    asked = 0;
  }
  pending = static_cast<cudaError_t>(pending_before);
  const int fit = dtq::clusters_that_fit(known[0], [&](int *out) {
    ++asked;
    *out = n;
    if (error) pending = static_cast<cudaError_t>(error);
    return static_cast<cudaError_t>(error);
  });
  *pending_after = pending;
  *questions = asked;
  return fit;
}
}
