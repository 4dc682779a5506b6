// Host-side helpers shared by the launchers: status mapping, per-device facts, the workspace
// layout that kernels and launchers agree on.
#pragma once

#include <atomic>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/dtq_b200.h"

namespace dtq {

constexpr int kMaxGridBlocks = 4096;  // upper bound on any persistent grid (148 SMs x 16 CTAs fits)
constexpr int kMaxShares = 1024;      // upper bound on the grid of the fused kernel

// Scratch shared by the single-launch reductions.  Zero-filled once by dtq_workspace_init;
// every kernel leaves `arrivals` at zero again and only ever advances `generation`.
struct alignas(256) Workspace {
  unsigned int arrivals;    // blocks that have published their partial in the current launch
  unsigned int generation;  // bumped by the last-arriving block; waiters spin on it (bounded)
  int status;               // sticky: DTQ_ERR_TIMEOUT if a bounded wait ever gave up
  float amax;               // the reduced value of the current launch, valid after the bump
  // The grid barrier of the fused kernel that exchanges with other GPUs: arrival count and running maximum (as float bits), one
  // pair per parity of `generation`; a launch uses the pair of its parity and clears the other.
  unsigned int bar_count[2];
  unsigned int bar_max[2];
  // Running maxima of kernels whose blocks fold their value into a few words (atomicMax, block b
  // into word b % 32) instead of publishing partials; a one-warp finishing launch takes them and
  // leaves zeros behind.
  unsigned int slot_max[32];
  // Limit of a wait in the GEMMs and in the fused kernel, in microseconds; 0, as initialised, is a second or two.  Tests shorten it
  // to see one run out.
  unsigned int wait_limit_us;
  // The fused kernel on one GPU (see dtq_grid.cuh): the shares that are in and their maximum (as float bits), one pair per parity of
  // the launch; a launch clears the other.
  unsigned int shares_in[2];
  unsigned int shares_max[2];
  unsigned int pad[19];
  // Its shares of the input, one word each: twice the launches so far, between launches the same in all.
  unsigned int shares[kMaxShares];
  float partials[kMaxGridBlocks];
};

struct DeviceInfo {
  int id = 0;
  int sm_count = 0;
  int cooperative = 0;
};

// Facts about the current device, queried once per device and cached (thread-safe).
int current_device_info(DeviceInfo *info);

inline int cuda_status(cudaError_t e) { return e == cudaSuccess ? DTQ_OK : DTQ_ERR_CUDA_BASE + static_cast<int>(e); }

#define DTQ_CUDA_TRY(expr)                             \
  do {                                                 \
    cudaError_t _e = (expr);                           \
    if (_e != cudaSuccess) return dtq::cuda_status(_e); \
  } while (0)

// ---- bytes of parameters ----------------------------------------------------------------------------------------------
// What a launch costs the host depends on how many bytes of parameters the kernel has: on a B200 with driver 580, launched as
// a programmatic dependent, 1.70 to 1.77 us where they end in the second quarter of a 64-byte line (17 to 32, 81 to 96, ... of
// them) and 2.05 to 2.15 us otherwise, from 0 to 768 bytes; clusters the same, cooperative launches 1.95 against 2.4 and only where they
// end on its last byte.  On another host 2.0 against 2.4.  So every kernel that small calls reach has as many as end there: its last
// parameter is padding.
constexpr size_t kLaunchLine = 64, kLaunchEnd = 32;
template <size_t BEFORE>  // bytes of parameters in front of it
struct LaunchPad {
  unsigned char unused[(kLaunchLine + kLaunchEnd - 1 - BEFORE % kLaunchLine) % kLaunchLine + 1];
};
template <typename... KArgs>
constexpr size_t parameter_bytes() {
  size_t at = 0;
  ((at = (at + alignof(KArgs) - 1) / alignof(KArgs) * alignof(KArgs) + sizeof(KArgs)), ...);
  return at;
}
template <typename... KArgs>
constexpr bool quick_to_launch = parameter_bytes<KArgs...>() % kLaunchLine == kLaunchEnd;

// cudaLaunchKernelEx for kernels that small calls reach.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_quickly(const cudaLaunchConfig_t &cfg, void (*kernel)(KArgs...), Args... args) {
  static_assert(quick_to_launch<KArgs...>, "see LaunchPad");
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Launches `kernel` so that it may start while the kernel queued before it on `st` is still
// draining (programmatic dependent launch).  The kernel must call pdl_wait() before its first
// access to memory that its predecessor on the stream may read or write.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_after_dependency(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem_bytes,
                                           cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  static_assert(quick_to_launch<KArgs...>, "see LaunchPad");
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// ---- blocks of a small grid, spread over the device --------------------------------------------------------------------
// A programmatic dependent becomes resident while the kernel before it drains.  Where that leaves some SMs free and others full (a
// product with one CTA of 225 KB on each of 105 of the 148 SMs), the blocks of a small grid that follows all settle on the free
// ones, as many as fit each, and stay there when the others come free.  So a grid of less than a full wave asks for as much shared
// memory as keeps more than its even share of blocks off an SM (sixteen blocks or fewer: more than two).  `most` is what fits without.
// Not for more: all that leaves room for the share kept the blocks off every SM on which another kernel has any; us on a stream beside
// other work, with all -> with the least: 1024 x 4096 beside a row-wise quantization 270 -> 234, beside an amax 64 -> 18, beside an elementwise
// two-orientation cast 378 -> 339.
// Measured, us per pass, without -> with, the two-orientation MX casts in MXFP8 training steps: 864 x 1920 x 1920 45.1 -> 36.9, 768 x 800 x
// 4576 53.3 -> 40.8, 2048^3 56.8 -> 48.5, 4096 x 1024 x 4096 82.2 -> 79.6.
// Only for kernels whose own shared memory keeps them off an SM that a product holds anyway, like these.  The MX and row-wise casts have
// none, and run beside a product on another stream: spread, they waited for it (64 x 8192 beside MXFP8 8192^3 15 -> 364 us, 1024 x 4096 beside 4096^3 15 ->
// 64), which is more than their layers lose (row-wise 1024 x 2048 x 2048 12.1 -> 13.0, MXFP4 1024 x 4096 x 4096 13.5 -> 14.8, MXFP8 64 x 8192 x 4096 12.6 -> 12.7,
// 1024 x 1024 x 4096 9.1 -> 10.6).
// The amax and the elementwise two-orientation cast, whose kernels follow one another, release their dependents late instead: with an amax
// in front of it spread, 5003 x 4096 took 25.7 instead of 22.0.  (So do the products gain for the casts, but a product behind a product
// loses: MXFP8 300 x 2048 x 1024 5.8 -> 6.4, 1024 x 1024 x 4096 7.0 -> 7.2.)
constexpr size_t kSmemPerSm = 228 * 1024, kSmemReserved = 1024, kSmemUnit = 128;  // of an SM; taken by each block besides its own
constexpr size_t least_for_share(int64_t per_sm) { return (kSmemPerSm / kSmemUnit / (per_sm + 1) + 1) * kSmemUnit - kSmemReserved; }
inline size_t spread_bytes(int64_t grid, int sm_count, size_t static_smem, int most) {
  const int64_t per_sm = grid <= 16 ? 2 : (grid + sm_count - 1) / sm_count;
  if (per_sm >= most) return 0;
  return least_for_share(per_sm) > static_smem ? least_for_share(per_sm) - static_smem : 0;
}
// Lets `kernel` have that much on the current device: asked of the runtime once per kernel and device (again, harmlessly, should the
// table ever be full).  Until then a launch may have 48 KB, static and dynamic together, so any spread launch asks.
inline cudaError_t allow_spread(const void *kernel, int dev_id, size_t static_smem) {
  constexpr unsigned kSlots = 1024;
  static std::atomic<uintptr_t> seen[kSlots];
  const uintptr_t key = reinterpret_cast<uintptr_t>(kernel) * 64 + static_cast<uintptr_t>(dev_id & 63) + 1;
  unsigned slot = static_cast<unsigned>((key * 0x9E3779B97F4A7C15ull) >> 54);
  for (unsigned i = 0; i < kSlots; ++i, slot = (slot + 1) % kSlots) {
    const uintptr_t there = seen[slot].load(std::memory_order_acquire);
    if (there == key) return cudaSuccess;
    if (there) continue;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(least_for_share(1) - static_smem));
    uintptr_t empty = 0;
    if (e == cudaSuccess) seen[slot].compare_exchange_strong(empty, key, std::memory_order_acq_rel);
    return e;
  }
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(least_for_share(1) - static_smem));
}
// Whether work on `st` has the whole device, as against the SMs of a green context.  What the driver cannot tell is a yes.
inline bool has_whole_device(cudaStream_t st) {
  using GreenCtxOf = CUresult (*)(CUstream, CUgreenCtx *);
  static const GreenCtxOf green_ctx_of = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuStreamGetGreenCtx", &f, cudaEnableDefault, &found) != cudaSuccess) (void)cudaGetLastError();
    return reinterpret_cast<GreenCtxOf>(f);
  }();
  CUgreenCtx green = nullptr;
  return !green_ctx_of || green_ctx_of(st, &green) != CUDA_SUCCESS || !green;
}
// launch_after_dependency with the blocks spread, on a stream that has the whole device: the even share of fewer SMs is larger, and blocks that
// keep one another off them take turns (1024 x 2048 on 32 SMs 6.5 -> 9.2 us).  Where the runtime does not grant the memory (the answer above was another context's,
// say, or one from before the device was reset), the kernel is launched without: it runs as well.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_spread(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t static_smem, int most, const DeviceInfo &dev,
                                 cudaStream_t st, Args... args) {
  size_t bytes = spread_bytes(grid, dev.sm_count, static_smem, most);
  if (bytes && !has_whole_device(st)) bytes = 0;
  if (bytes && allow_spread(reinterpret_cast<const void *>(kernel), dev.id, static_smem) == cudaSuccess) {
    const cudaError_t e = launch_after_dependency(kernel, dim3(grid), dim3(block), bytes, st, args...);
    if (e != cudaErrorInvalidValue && e != cudaErrorLaunchOutOfResources) return e;
  }
  if (bytes) (void)cudaGetLastError();  // the question's own, or the refused launch's
  return launch_after_dependency(kernel, dim3(grid), dim3(block), 0, st, args...);
}

// ---- thread-block clusters: whether the device can place them ------------------------------------------------------
// The runtime's word that there is no such thing on this device, as against a failure of the moment (no memory to load the
// kernel, say).
inline bool means_no_such_clusters(cudaError_t e) {
  return e == cudaErrorNotSupported || e == cudaErrorInvalidClusterSize || e == cudaErrorInvalidConfiguration ||
         e == cudaErrorInvalidDeviceFunction || e == cudaErrorInvalidValue;
}
// How many clusters of a kernel the device holds at once, 0 where it cannot place them.  `ask(&n)` puts the question, and
// `known` (0: no answer yet, else the answer + 1) keeps the answer for the process.  A failure of the moment is 0 for this
// call and is not kept.  An error that was pending before stays pending: it is the caller's.  Asking twice is harmless.
template <typename Ask>
int clusters_that_fit(std::atomic<int> &known, Ask ask) {
  const int answer = known.load(std::memory_order_acquire);
  if (answer) return answer - 1;
  int n = 0;
  const cudaError_t e = ask(&n);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();  // the question's own
    n = 0;
  }
  if (e == cudaSuccess || means_no_such_clusters(e)) known.store(n + 1, std::memory_order_release);
  return n;
}
// Whether a launch was turned down for what a cluster needs: the answer above is the device's, and the context may have
// fewer SMs (a green context, a partition).
inline bool turned_down_for_room(cudaError_t e) {
  return e == cudaErrorLaunchOutOfResources || e == cudaErrorInvalidClusterSize || e == cudaErrorInvalidConfiguration ||
         e == cudaErrorNotSupported;
}

// ---- tensor-wise quantization: which kernels -------------------------------------------------------------------------
enum class Tensorwise { kCluster, kGrid, kTwoLaunches, kScalar };
constexpr int64_t kClusterMaxBytes = int64_t(1) << 20;  // of input; figures at dsq_cluster_kernel
// Inputs above this many bytes are quantised as amax kernel + cast kernel instead of the single
// fused launch: what the chip can keep between the two looks (about 140 MB) no longer matters at
// that size, and the two stream kernels run at higher occupancy than the persistent fused one
// (measured, bf16, fused / two launches: 128 MiB 44.8 / 49.5 us, 256 MiB 94.3 / 100.8, 320 MiB 118.3 / 120.2; fp32 320 MiB
// 105.7 / 104.9).
constexpr int64_t kFusedMaxBytes = int64_t(320) << 20;
// `aligned`: input and output allow 16-byte loads and whole stores.
inline Tensorwise tensorwise_path(int64_t input_bytes, bool aligned, bool clusters, bool cooperative) {
  if (!aligned) return Tensorwise::kScalar;
  if (input_bytes > kFusedMaxBytes) return Tensorwise::kTwoLaunches;
  if (input_bytes <= kClusterMaxBytes && clusters) return Tensorwise::kCluster;
  return cooperative ? Tensorwise::kGrid : Tensorwise::kScalar;
}

inline bool aligned_to(const void *p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// Which stream kernels call prefetch_first_tile, by bytes of input (dtq_device.cuh has the figures).  They have an instantiation
// for either answer: with the question at run time the compiler orders the rest of them differently, and those that do not
// ask ahead lost up to 2 %.
enum class Asks { kCastBf16, kCastF32, kMx, kMxBlocked, kMxFormats, kRowwise };
constexpr int64_t kAskSmallBytes = int64_t(2) << 20;  // the tokens of a decode step: 128 of K = 8192
inline bool asks_ahead(Asks kernel, int64_t input_bytes) {
  if (input_bytes <= kAskSmallBytes) return true;
  const auto mebibytes = [=](int64_t from, int64_t to) { return input_bytes >= from << 20 && input_bytes <= to << 20; };
  switch (kernel) {
    case Asks::kCastBf16: return mebibytes(16, 48) || mebibytes(80, 128);
    case Asks::kCastF32: return mebibytes(28, 128);
    case Asks::kMx: return input_bytes >= int64_t(16) << 20;
    case Asks::kMxBlocked: return mebibytes(16, 128);
    case Asks::kRowwise: return mebibytes(16, 128);
    default: return false;
  }
}

// How much of its first tile, in 16-byte chunks, every block of the amax asks for ahead of its dependency; 0: nothing (figures in
// amax.cu).
inline int amax_ask_chunks(int64_t input_bytes, bool f32, int grid, int tile_chunks) {
  if (input_bytes > int64_t(f32 ? 40 : 20) << 20) return 0;
  const int64_t in_all = int64_t(f32 && input_bytes > int64_t(22) << 20 ? 16 : 4) << 20;
  const int64_t share = in_all / 16 / grid;
  return static_cast<int>(share < tile_chunks ? share : tile_chunks);
}

inline int64_t ceil_div64(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Grid for a persistent kernel that walks `tiles` tiles grid-stride: at most `max_grid` blocks,
// and when every block needs several tiles, as few blocks as keep the number of rounds, so that
// all blocks run the same number of tiles (no straggler round with most of the GPU idle).
inline int balanced_grid(int64_t tiles, int64_t max_grid) {
  if (tiles < 1) return 1;
  if (tiles <= max_grid) return static_cast<int>(tiles);
  const int64_t rounds = ceil_div64(tiles, max_grid);
  return static_cast<int>(ceil_div64(tiles, rounds));
}

}  // namespace dtq
