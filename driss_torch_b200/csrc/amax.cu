// amax: out[0] = max |in[i]| as fp32, finished grid-wide in a single launch.
//
// Replaces src/amax.cu:50-80 (+ the -inf fill launch at :115): a persistent grid streams the
// input with several 128-bit loads in flight per thread, reduces with packed bf16 max, one
// integer warp-max instruction per warp, and a last-block finish instead of one same-address
// atomic per block on a pre-filled output.  The value is order independent, so the result is
// bit-identical; NaNs are dropped and an empty input gives -inf, as in the reference.
#include <atomic>
#include <cmath>
#include <mutex>

#include "dtq_device.cuh"
#include "dtq_grid.cuh"
#include "dtq_host.h"

namespace dtq {

constexpr int kAmaxUnroll = 8;       // 128-bit loads in flight per thread
constexpr int kAmaxBlocksPerSm = 4;  // persistent grid: blocks per SM
constexpr int kAmaxThreads = 512;

template <int IN>
struct AbsMax;

template <>
struct AbsMax<DTQ_BF16> {
  static constexpr int kElemBytes = 2;
  __nv_bfloat162 a, b;
  __device__ explicit AbsMax(float identity) { a = b = __float2bfloat162_rn(identity); }
  __device__ void chunk(uint4 v) {
    a = absmax_bf162(a, v.x);
    b = absmax_bf162(b, v.y);
    a = absmax_bf162(a, v.z);
    b = absmax_bf162(b, v.w);
  }
  __device__ void one(const void *p, int64_t i) {
    const uint32_t h = static_cast<const uint16_t *>(p)[i];
    a = absmax_bf162(a, h | (h << 16));
  }
  __device__ float result() const { return bf162_hmax_to_float(__hmax2(a, b)); }
};

template <>
struct AbsMax<DTQ_F32> {
  static constexpr int kElemBytes = 4;
  float a, b;
  __device__ explicit AbsMax(float identity) { a = b = identity; }
  __device__ void chunk(uint4 v) {
    a = fmaxf(a, fabsf(__uint_as_float(v.x)));
    b = fmaxf(b, fabsf(__uint_as_float(v.y)));
    a = fmaxf(a, fabsf(__uint_as_float(v.z)));
    b = fmaxf(b, fabsf(__uint_as_float(v.w)));
  }
  __device__ void one(const void *p, int64_t i) { a = fmaxf(a, fabsf(static_cast<const float *>(p)[i])); }
  __device__ float result() const { return fmaxf(a, b); }
};

// Streams chunks [0, nchunks) of `body` grid-stride in tiles of blockDim.x * UNROLL chunks.
template <int IN, int UNROLL>
__device__ __forceinline__ void absmax_stream(AbsMax<IN> &acc, const uint4 *__restrict__ body, int64_t nchunks) {
  const int64_t tile_chunks = int64_t(blockDim.x) * UNROLL;
  for (int64_t tile = blockIdx.x; tile * tile_chunks < nchunks; tile += gridDim.x) {
    const int64_t first = tile * tile_chunks + threadIdx.x;
    uint4 v[UNROLL];
    if ((tile + 1) * tile_chunks <= nchunks) {
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) v[u] = ldg_stream(body + first + int64_t(u) * blockDim.x);
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) acc.chunk(v[u]);
    } else {
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int64_t c = first + int64_t(u) * blockDim.x;
        if (c < nchunks) acc.chunk(ldg_stream(body + c));
      }
    }
  }
}

// `in` may have any element alignment: up to `head` leading and `tail` trailing elements are
// read one by one by block 0, the 16-byte aligned middle is streamed.
// PREFETCH: every block asks for the first `ask_chunks` chunks of its first tile ahead of the dependency.
template <int IN, int UNROLL, bool PREFETCH>
__global__ void __launch_bounds__(kAmaxThreads)
amax_kernel(const void *__restrict__ in, float *__restrict__ out, int64_t numel, int64_t head, Workspace *ws, int ask_chunks,
            LaunchPad<44>) {
  __shared__ float smem32[32];
  __shared__ int flag;
  constexpr int kElems = 16 / AbsMax<IN>::kElemBytes;
  // What is queued behind this kernel becomes resident when its blocks end, not earlier: the blocks that settled beside these, or
  // another amax's, settled unevenly (and a cast's first tiles are asked for in vain).  Amax alone, us, released at the start -> at the end:
  // 6 MiB 5.0 -> 3.7, 39 MiB 10.9 -> 9.5; with both casts see cast_transposed_kernel.
  const char *base = static_cast<const char *>(in);
  const uint4 *body = reinterpret_cast<const uint4 *>(base + head * AbsMax<IN>::kElemBytes);
  const int64_t nchunks = (numel - head) / kElems;
  // This launch itself may have started under the tail of its predecessor: part of the block's first tile is asked into L2
  // meanwhile, harmless whatever the predecessor still writes (see l2_prefetch_bulk).  What it hides is the start of the stream.
  // 4 MiB in all of inputs of up to 20 MiB of bf16 and 22 MiB of fp32, 16 MiB of up to 40 MiB of fp32 (amax_ask_chunks).  Measured in a
  // graph, outputs that stay, us with nothing asked, and the change in percent with 4 / 8 / 16 / 32 MiB; inputs from memory (400 MB of them in
  // turn), the last column three inputs in turn:
  //                 amax                          amax, static cast             amax, both casts              amax, both casts, three
  //   bf16   8 MiB   4.6  -8.4 -11.7 -11.5 -11.5   7.1  -3.5  -6.4  -6.8  -6.1   8.2  +5.1  +6.8  +6.7  +6.8   7.5 +4.5  +7.4  +8.0  +7.6
  //         16 MiB   5.5  -6.5  -8.2  -1.8  -1.6  10.3  -7.0 -10.1  -8.0  -7.8  11.8  +3.6  +5.5  +6.4  +6.7  11.2 +4.5  +5.2  +6.4  +7.1
  //         20 MiB   6.1  -5.1  -8.4  -2.8  -3.0  11.7  -4.4  -7.9  -8.1  -5.9  12.9 +11.1 +10.6 +15.1 +17.5  13.0 +8.1  +7.5  +9.8 +11.8
  //         24 MiB   6.6  -5.3  -8.3  -2.3  +0.3  13.2  -3.8  -6.0  -8.8  -6.8  14.5 +11.9 +13.3 +15.3 +20.4  14.4 +8.6 +10.0  +9.8 +13.0
  //         40 MiB   8.9  -3.7  -6.3  -6.2  -5.0  19.1  -2.4  -3.9  -4.0  -2.9  21.0 +13.2 +13.0 +15.3 +17.0  21.3 +9.1  +9.7 +10.5 +11.4
  //         20 MiB, rows no multiple of 16                                      16.4  -1.3  -4.3  -3.5  -2.2  16.4 -1.9  -5.1  -5.3  -3.9
  //   fp32   8 MiB   4.5  -7.9 -12.1 -12.1 -12.3   7.0  +0.1  -1.0  -1.0  -1.0   7.3  -1.2  +1.8  +1.5  +1.5   6.2 -3.9  -3.1  -3.2  -2.8
  //         16 MiB   5.5  -5.6  -7.1  -2.0  -0.9   9.2  -2.0  -3.7  -0.7  -0.7   9.7  -0.2  +2.1  +1.8  +2.2   8.7 +1.8  +4.8  +4.9  +3.7
  //         24 MiB   6.6  -4.4  -7.3  -2.0  +1.4  11.5  +0.3  +0.6  +1.4  +4.5  12.3  +3.6  +1.1  +1.1  +4.6  12.1 +3.6  -0.7  -1.5  -1.6
  //         32 MiB   7.7  -3.1  -5.7  -6.6  +0.4  14.9  -3.0  -3.1  -5.0  -2.6  15.1  +4.9  +2.5  -0.6  +5.8  15.0 +2.4  +0.8  -4.9  -3.2
  //         40 MiB   8.8  -3.5  -5.3  -5.8  -1.7  17.5  -2.5  -3.4  -2.5  -1.5  17.7  +5.2  +3.4  +5.2  +7.7  17.7 +3.2  +1.9  +2.0  +2.7
  // An amax alone or with a static cast gains; with both casts aligned rows of bf16 lose, and more beyond 20 MiB, where it stops.  Which will follow
  // the amax cannot see.
  constexpr int64_t kTile = int64_t(kAmaxThreads) * UNROLL;
  if constexpr (PREFETCH) {
    if (threadIdx.x == 0) prefetch_first_tile(body, blockIdx.x * kTile, ask_chunks, nchunks);
  }
  pdl_wait();
  const float identity = -INFINITY;
  AbsMax<IN> acc(identity);
  absmax_stream<IN, UNROLL>(acc, body, nchunks);
  if (blockIdx.x == 0) {
    const int64_t tail0 = head + nchunks * kElems;
    if (threadIdx.x < head) acc.one(in, threadIdx.x);
    if (tail0 + threadIdx.x < numel) acc.one(in, tail0 + threadIdx.x);
  }

  const float block_value = block_max_nonneg(acc.result(), smem32, identity);
  if (publish_and_ticket(ws, block_value, &flag)) {
    const float total = reduce_partials(ws, smem32, identity);
    if (threadIdx.x == 0) {
      out[0] = total;
      ws->arrivals = 0;
    }
  }
}

int amax_grid(int64_t numel, int elem_bytes, const DeviceInfo &dev) {
  const int64_t tiles = ceil_div64(numel * elem_bytes / 16, int64_t(kAmaxThreads) * kAmaxUnroll);
  const int64_t max_grid = int64_t(dev.sm_count) * kAmaxBlocksPerSm;
  return balanced_grid(tiles, max_grid);
}

int64_t head_elems(const void *p, int elem_bytes, int64_t numel) {
  const int64_t h = static_cast<int64_t>((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / elem_bytes;
  return h < numel ? h : numel;
}

// Arguments already validated; `out` may be any device float (the fused op points it into its
// workspace when it splits a very large tensor into amax + cast).
int launch_amax(const void *in, float *out, int64_t numel, int in_dtype, Workspace *ws, const DeviceInfo &dev,
                cudaStream_t st) {
  const int eb = in_dtype == DTQ_BF16 ? 2 : 4;
  const int grid = amax_grid(numel, eb, dev);
  const int64_t head = head_elems(in, eb, numel);
  const int ask_chunks = amax_ask_chunks(numel * eb, in_dtype == DTQ_F32, grid, kAmaxThreads * kAmaxUnroll);
  const bool ask = ask_chunks > 0;
  auto kernel = in_dtype == DTQ_BF16 ? (ask ? amax_kernel<DTQ_BF16, kAmaxUnroll, true> : amax_kernel<DTQ_BF16, kAmaxUnroll, false>)
                                     : (ask ? amax_kernel<DTQ_F32, kAmaxUnroll, true> : amax_kernel<DTQ_F32, kAmaxUnroll, false>);
  return cuda_status(launch_after_dependency(kernel, dim3(grid), dim3(kAmaxThreads), 0, st, in, out, numel, head, ws, ask_chunks,
                                             LaunchPad<44>{}));
}

}  // namespace dtq

extern "C" int dtq_amax(const void *in, float *out, int64_t numel, int in_dtype, void *workspace,
                        size_t workspace_bytes, void *stream) {
  using namespace dtq;
  if (numel < 0 || !out || (numel > 0 && !in)) return DTQ_ERR_INVALID_ARGUMENT;
  if (in_dtype != DTQ_BF16 && in_dtype != DTQ_F32) return DTQ_ERR_UNSUPPORTED_DTYPE;
  if (!workspace || workspace_bytes < sizeof(Workspace) || !aligned_to(workspace, 256)) return DTQ_ERR_WORKSPACE;
  if (numel > 0 && !aligned_to(in, in_dtype == DTQ_BF16 ? 2 : 4)) return DTQ_ERR_INVALID_ARGUMENT;
  DeviceInfo dev;
  if (int e = current_device_info(&dev)) return e;
  return launch_amax(in, out, numel, in_dtype, static_cast<Workspace *>(workspace), dev, static_cast<cudaStream_t>(stream));
}

// ---- amax without any caller- or library-allocated scratch -------------------------------------------------
//
// Some hosts may not allocate device memory at the point where they need an amax: a runtime that
// hands the whole device heap to its own pool and forbids cudaMalloc in plugins, or a
// latency-critical section that cannot afford the device-wide synchronisation cudaMalloc and
// cudaFree imply.  For them the scratch of the reduction lives in this library's image: one
// Workspace in a file-scope __device__ array, present on every GPU that loads the library until
// the process exits.
//
// In host code the array's NAME is only a host-side handle, not a device address, so the address
// is looked up once per device with cudaGetSymbolAddress (with that device current) and cached.
// One block per tile is launched, so the array's kMaxGridBlocks partial slots bound the input:
// kMaxGridBlocks tiles of kAmaxThreads * kAmaxUnroll 16-byte chunks = DTQ_AMAX_STATIC_MAX_BYTES.
namespace dtq {
namespace {

static __device__ __align__(256) unsigned char g_static_scratch[sizeof(Workspace)];

constexpr int kStaticMaxDevices = 64;
void *g_static_scratch_ptr[kStaticMaxDevices];
std::atomic<int> g_static_scratch_ready[kStaticMaxDevices];
std::mutex g_static_scratch_mutex;

// Device address of the scratch array on the current device (looked up on first use).
int static_scratch_address(Workspace **ws) {
  int dev = 0;
  DTQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kStaticMaxDevices) return DTQ_ERR_INVALID_ARGUMENT;
  if (!g_static_scratch_ready[dev].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (!g_static_scratch_ready[dev].load(std::memory_order_relaxed)) {
      void *ptr = nullptr;
      DTQ_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_static_scratch));
      g_static_scratch_ptr[dev] = ptr;
      g_static_scratch_ready[dev].store(1, std::memory_order_release);
    }
  }
  *ws = static_cast<Workspace *>(g_static_scratch_ptr[dev]);
  return DTQ_OK;
}

}  // namespace
}  // namespace dtq

extern "C" int dtq_amax_static_scratch(const void *in, float *out, int64_t numel, int in_dtype, void *stream) {
  using namespace dtq;
  static_assert(int64_t(kMaxGridBlocks) * kAmaxThreads * kAmaxUnroll * 16 == DTQ_AMAX_STATIC_MAX_BYTES,
                "the documented limit must match the scratch array");
  if (numel < 0 || !out || (numel > 0 && !in)) return DTQ_ERR_INVALID_ARGUMENT;
  if (in_dtype != DTQ_BF16 && in_dtype != DTQ_F32) return DTQ_ERR_UNSUPPORTED_DTYPE;
  const int eb = in_dtype == DTQ_BF16 ? 2 : 4;
  if (numel > DTQ_AMAX_STATIC_MAX_BYTES / eb) return DTQ_ERR_TOO_LARGE;  // needs more partial slots than the array has
  if (numel > 0 && !aligned_to(in, eb)) return DTQ_ERR_INVALID_ARGUMENT;
  Workspace *ws = nullptr;
  if (int e = static_scratch_address(&ws)) return e;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // The array keeps whatever the previous call left: start the arrival counter from zero.
  DTQ_CUDA_TRY(cudaMemsetAsync(&ws->arrivals, 0, sizeof(ws->arrivals), st));
  const int64_t tiles = ceil_div64(numel * eb / 16, int64_t(kAmaxThreads) * kAmaxUnroll);
  const int grid = static_cast<int>(tiles < 1 ? 1 : tiles);  // <= kMaxGridBlocks by the size check
  const int64_t head = head_elems(in, eb, numel);
  if (in_dtype == DTQ_BF16)
    amax_kernel<DTQ_BF16, kAmaxUnroll, false><<<grid, kAmaxThreads, 0, st>>>(in, out, numel, head, ws, 0, {});
  else
    amax_kernel<DTQ_F32, kAmaxUnroll, false><<<grid, kAmaxThreads, 0, st>>>(in, out, numel, head, ws, 0, {});
  return cuda_status(cudaGetLastError());
}
