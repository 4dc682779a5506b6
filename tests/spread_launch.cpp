// launch_spread of dtq_host.h against a stand-in for the runtime's rule on shared memory: a kernel may have 48 KB, static and dynamic
// together, until it has been allowed more on that device, at most 227 KB.  No GPU, no CUDA library.
#include <cuda.h>
#include <map>
#include <utility>

#include "dtq_host.h"

namespace {
constexpr size_t kDefault = 48 * 1024, kMost = 227 * 1024;
std::map<std::pair<const void *, int>, size_t> allowed;  // static and dynamic bytes, by kernel and device
int device = 0;
size_t static_bytes = 0;  // of the kernel being launched
bool grants = true;
cudaError_t pending = cudaSuccess;
int launches = 0;
bool in_green_context = false;
size_t launched_with = 0;

cudaError_t answer(cudaError_t e) {
  if (e != cudaSuccess) pending = e;
  return e;
}
template <int I>
void kernel(int, dtq::LaunchPad<4>) {}
template <size_t... I>
cudaError_t launch(std::index_sequence<I...>, int which, unsigned grid, int most, const dtq::DeviceInfo &dev) {
  using Kernel = void (*)(int, dtq::LaunchPad<4>);
  static const Kernel kernels[] = {kernel<I>...};
  return dtq::launch_spread(kernels[which], grid, 256, static_bytes, most, dev, nullptr, 0, dtq::LaunchPad<4>{});
}
}  // namespace

extern "C" {
cudaError_t cudaGetLastError() { return std::exchange(pending, cudaSuccess); }
cudaError_t cudaFuncSetAttribute(const void *kernel, cudaFuncAttribute, int dynamic) {
  if (!grants || static_bytes + dynamic > kMost) return answer(cudaErrorInvalidValue);
  allowed[{kernel, device}] = static_bytes + dynamic;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *kernel, void **) {
  const auto it = allowed.find({kernel, device});
  if (static_bytes + cfg->dynamicSmemBytes > (it == allowed.end() ? kDefault : it->second)) return answer(cudaErrorInvalidValue);
  ++launches;
  launched_with = cfg->dynamicSmemBytes;
  return cudaSuccess;
}

CUresult stand_in_for_the_query(CUstream, CUgreenCtx *ctx) {
  *ctx = reinterpret_cast<CUgreenCtx>(in_green_context ? &in_green_context : nullptr);
  return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPoint(const char *, void **f, unsigned long long, cudaDriverEntryPointQueryResult *found) {
  *f = reinterpret_cast<void *>(stand_in_for_the_query);
  *found = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

// The launch of kernel `which` (0 to 63) on device `dev` of 148 SMs.  Returns the runtime's error; *bytes: what it was launched with.
int spread_launch(int which, int dev, unsigned grid, long long statically, int most, int granted, long long *bytes, int *times, int *error_left) {
  device = dev;
  static_bytes = static_cast<size_t>(statically);
  grants = granted != 0;
  launches = 0;
  pending = cudaSuccess;
  dtq::DeviceInfo info;
  info.id = dev;
  info.sm_count = 148;
  const cudaError_t e = launch(std::make_index_sequence<64>{}, which, grid, most, info);
  *bytes = static_cast<long long>(launched_with);
  *times = launches;
  *error_left = pending;
  return e;
}
void move_to_green_context(int green) { in_green_context = green != 0; }
void forget_what_was_allowed() { allowed.clear(); }  // as a device reset does
}
