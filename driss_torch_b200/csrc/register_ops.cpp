// PyTorch operator boundary: TORCH_LIBRARY(DrissTorch) over the torch-free C ABI.
//
// This translation unit and direct_calls.cpp are the only ones that see torch headers.  It keeps the reference's
// operator names and schema strings for the quantization path (src/register_ops.cpp:20-30,
// :40-41), its argument checks and error behaviour (src/saturated_cast.cu:227-252,
// src/amax.cu:106-119, src/dynamic_scaled_quant.cu:157-176, src/mx_cast.cu:168-246), CUDA-only
// dispatch (no CPU kernel, no autograd formula), and adds three ops the reference lacks.  Unlike
// the reference it launches on the current stream of the input's device.
//
// Each op: check -> allocate outputs with the caching allocator -> one C-ABI call.  Nothing
// here computes.
#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <c10/core/DispatchKey.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/library.h>

#include <cstdint>
#include <mutex>
#include <optional>
#include <tuple>
#include <unordered_map>

#include "dtq_b200.h"

namespace {

void check_status(int status, const char *what) {
  TORCH_CHECK(status == DTQ_OK, what, " failed: ", dtq_status_string(status), " (status ", status, ")");
}

int in_code(at::ScalarType t) { return t == at::kBFloat16 ? DTQ_BF16 : DTQ_F32; }
int out_code(at::ScalarType t) { return t == at::kFloat8_e4m3fn ? DTQ_E4M3 : DTQ_E5M2; }

// The device of an operator's input, current from here on, and the current stream there.  Comes before the outputs: they are
// allocated on the current device.
struct OnDeviceOf {
  c10::cuda::OptionalCUDAGuard guard;  // set only where another device was current
  c10::cuda::CUDAStream stream;
  explicit OnDeviceOf(const at::Tensor &t) : stream(c10::cuda::getCurrentCUDAStream(t.device().index())) {
    if (C10_UNLIKELY(c10::cuda::current_device() != t.device().index())) guard.set_index(t.device().index());
  }
};

// Outputs straight from the CUDA allocator: what at::empty / at::empty_like end in.  The smallest calls are bound by the host, and
// each at::empty was 0.4 us of their 5 to 9; at::detail::empty_cuda, which makes the device current once more for each output, 0.51,
// this 0.38 (0.29 of it the allocator's).
// at::empty also fills what it returns under torch.use_deterministic_algorithms (unless told not to), so then it is asked.
at::Tensor new_here(const OnDeviceOf &, const at::Tensor &like, at::IntArrayRef sizes, at::ScalarType dtype) {
  if (C10_UNLIKELY(at::globalContext().deterministicAlgorithms())) return at::empty(sizes, like.options().dtype(dtype));
  return at::Tensor(at::detail::empty_generic(sizes, c10::cuda::CUDACachingAllocator::get(), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                              dtype, std::nullopt));
}
at::Tensor new_same_layout(const OnDeviceOf &, const at::Tensor &like, at::ScalarType dtype) {  // `like` is dense: its strides are kept as they are
  if (C10_UNLIKELY(at::globalContext().deterministicAlgorithms()))
    return at::empty_strided(like.sizes(), like.strides(), like.options().dtype(dtype));
  return at::Tensor(at::detail::empty_strided_generic(like.sizes(), like.strides(), c10::cuda::CUDACachingAllocator::get(),
                                                      c10::DispatchKeySet(c10::DispatchKey::CUDA), dtype));
}

void check_fp8(at::ScalarType dtype) {
  TORCH_CHECK(dtype == at::kFloat8_e4m3fn || dtype == at::kFloat8_e5m2,
              "Output tensor must be of type Float8_e4m3fn or Float8_e5m2");
}
void check_input(const at::Tensor &input) {
  TORCH_CHECK(input.is_cuda(), "Input tensor must be a CUDA tensor");
  TORCH_CHECK(input.scalar_type() == at::kBFloat16 || input.scalar_type() == at::kFloat,
              "Input tensor must be of type BFloat16 or Float, but got ", input.dtype());
  TORCH_CHECK(input.dim() == 2, "Input tensor must be 2D, but got ", input.dim());
}

// One zero-initialised workspace per (device, stream): launches on one stream are ordered, so
// they can share it; launches on different streams may overlap and must not.
struct WorkspaceCache {
  std::mutex mutex;
  std::unordered_map<uint64_t, at::Tensor> map;
  void *get(const c10::cuda::CUDAStream &stream) {
    const uint64_t key = (static_cast<uint64_t>(stream.device_index()) << 48) ^ static_cast<uint64_t>(stream.id());
    std::lock_guard<std::mutex> lock(mutex);
    auto it = map.find(key);
    if (it == map.end()) {
      at::Tensor t = at::zeros({static_cast<int64_t>(dtq_workspace_bytes())},
                               at::TensorOptions().dtype(at::kByte).device(at::kCUDA, stream.device_index()));
      it = map.emplace(key, std::move(t)).first;
    }
    return it->second.data_ptr();
  }
  // Synchronises; raises if any workspace recorded a device-side timeout.
  void check_all() {
    std::lock_guard<std::mutex> lock(mutex);
    for (auto &kv : map) {
      c10::cuda::CUDAGuard guard(kv.second.device());
      int status = 0;
      check_status(dtq_workspace_status(kv.second.data_ptr(), &status, nullptr), "dtq_workspace_status");
      TORCH_CHECK(status == DTQ_OK, "a quantization kernel reported: ", dtq_status_string(status));
    }
  }
};
WorkspaceCache &workspaces() {
  static WorkspaceCache *cache = new WorkspaceCache();  // leaked on purpose: outlives CUDA teardown
  return *cache;
}

// ---- reference ops --------------------------------------------------------------------------------

std::tuple<at::Tensor, at::Tensor> cast_transposed(const at::Tensor &input, const at::Tensor &scale,
                                                   at::ScalarType dtype, bool both, const char *what);

at::Tensor saturated_cast(const at::Tensor &input, const at::Tensor &scale, at::ScalarType dtype, bool transpose) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(scale.scalar_type() == at::kFloat, "Scale tensor must be of type Float, but got ", scale.dtype());
  TORCH_CHECK(scale.numel() == 1, "Scale tensor must be a scalar, but got ", scale.numel());
  TORCH_CHECK(scale.is_cuda() && scale.device() == input.device(), "Scale tensor must live on the input's device");
  // transpose: the cast of input.t() as a contiguous [cols, rows] tensor, in one pass.  (The reference declares
  // the flag, asserts it off in its Python wrapper and only uses it to choose a kernel; this package's wrapper
  // keeps that assert, the operator itself honours the flag.)
  if (transpose) return std::get<1>(cast_transposed(input, scale, dtype, false, "saturated_cast"));
  // The op is elementwise over storage: row-major or exactly transposed inputs at storage offset
  // zero are processed in place and the output keeps their strides; anything else is made
  // contiguous first (same rule as the reference).
  const auto strides = input.strides();
  const bool transposed = strides[0] == 1 && strides[1] == input.size(0);
  const bool as_is = (input.is_contiguous() || transposed) && input.storage_offset() == 0;
  const at::Tensor x = as_is ? input : input.contiguous();
  const OnDeviceOf here(x);
  at::Tensor out = new_same_layout(here, x, dtype);
  check_status(dtq_saturated_cast(x.data_ptr(), out.data_ptr(), scale.data_ptr<float>(), x.numel(),
                                  in_code(x.scalar_type()), out_code(dtype), here.stream.stream()),
               "saturated_cast");
  return out;
}

// The cast of input.t() as a contiguous [cols, rows] tensor and, with `both`, also the cast of input.
std::tuple<at::Tensor, at::Tensor> cast_transposed(const at::Tensor &input, const at::Tensor &scale,
                                                   at::ScalarType dtype, bool both, const char *what) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(scale.scalar_type() == at::kFloat, "Scale tensor must be of type Float, but got ", scale.dtype());
  TORCH_CHECK(scale.numel() == 1, "Scale tensor must be a scalar, but got ", scale.numel());
  TORCH_CHECK(scale.is_cuda() && scale.device() == input.device(), "Scale tensor must live on the input's device");
  const at::Tensor x = input.contiguous();
  const int64_t rows = x.size(0), cols = x.size(1);
  const OnDeviceOf here(x);
  at::Tensor out_t = new_here(here, x, {cols, rows}, dtype);
  at::Tensor out = both ? new_here(here, x, {rows, cols}, dtype) : at::Tensor();
  check_status(dtq_saturated_cast_transposed(x.data_ptr(), both ? out.data_ptr() : nullptr, out_t.data_ptr(),
                                             scale.data_ptr<float>(), rows, cols, in_code(x.scalar_type()),
                                             out_code(dtype), here.stream.stream()),
               what);
  return {out, out_t};
}

at::Tensor saturated_cast_transposed(const at::Tensor &input, const at::Tensor &scale, at::ScalarType dtype) {
  return std::get<1>(cast_transposed(input, scale, dtype, false, "saturated_cast_transposed"));
}

std::tuple<at::Tensor, at::Tensor> saturated_cast_dual(const at::Tensor &input, const at::Tensor &scale,
                                                       at::ScalarType dtype) {
  return cast_transposed(input, scale, dtype, true, "saturated_cast_dual");
}

// Both orientations of the dynamic cast for a device-resident amax: (payload, payload_t, scale).
std::tuple<at::Tensor, at::Tensor, at::Tensor> cast_with_amax_dual(const at::Tensor &input, const at::Tensor &amax_value,
                                                                   at::ScalarType dtype) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  TORCH_CHECK(amax_value.scalar_type() == at::kFloat && amax_value.numel() == 1 && amax_value.is_cuda() &&
                  amax_value.device() == input.device(),
              "amax must be a one-element fp32 tensor on the input's device");
  const int64_t rows = input.size(0), cols = input.size(1);
  const OnDeviceOf here(input);
  at::Tensor out = new_here(here, input, {rows, cols}, dtype);
  at::Tensor out_t = new_here(here, input, {cols, rows}, dtype);
  at::Tensor scale = new_here(here, input, {1}, at::kFloat);
  if (input.numel() == 0) {  // nothing is launched: derive the scale like the cast kernels do
    scale.copy_((dtype == at::kFloat8_e4m3fn ? 448.0 : 57344.0) / (amax_value.clamp_min(0).to(at::kDouble) + 1e-12));
    return {out, out_t, scale};
  }
  check_status(dtq_cast_with_amax_transposed(input.data_ptr(), out.data_ptr(), out_t.data_ptr(),
                                             amax_value.data_ptr<float>(), scale.data_ptr<float>(), rows, cols,
                                             in_code(input.scalar_type()), out_code(dtype), here.stream.stream()),
               "cast_with_amax_dual");
  return {out, out_t, scale};
}

// amax, then both orientations of the cast: (payload, payload_t, amax, scale); one C-ABI call that queues the
// amax kernel and, overlapping its tail, the kernel that casts into both orientations.
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> dynamic_scaled_quant_dual(const at::Tensor &input,
                                                                                      at::ScalarType dtype) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  const int64_t rows = input.size(0), cols = input.size(1);
  const OnDeviceOf here(input);
  at::Tensor out = new_here(here, input, {rows, cols}, dtype);
  at::Tensor out_t = new_here(here, input, {cols, rows}, dtype);
  if (input.numel() == 0) {  // nothing is launched: the fused op's maximum starts at 0
    at::Tensor amax_value = at::zeros({1}, input.options().dtype(at::kFloat));
    at::Tensor scale = at::full({1}, (dtype == at::kFloat8_e4m3fn ? 448.0 : 57344.0) / 1e-12, input.options().dtype(at::kFloat));
    return {out, out_t, amax_value, scale};
  }
  at::Tensor amax_value = new_here(here, input, {1}, at::kFloat);
  at::Tensor scale = new_here(here, input, {1}, at::kFloat);
  check_status(dtq_dynamic_scaled_quant_dual(input.data_ptr(), out.data_ptr(), out_t.data_ptr(), amax_value.data_ptr<float>(),
                                             scale.data_ptr<float>(), rows, cols, in_code(input.scalar_type()),
                                             out_code(dtype), workspaces().get(here.stream), dtq_workspace_bytes(),
                                             here.stream.stream()),
               "dynamic_scaled_quant_dual");
  return {out, out_t, amax_value, scale};
}

at::Tensor amax(const at::Tensor &input) {
  check_input(input);
  // max is order independent, so any dense layout can be reduced over its storage.
  const at::Tensor x = input.is_non_overlapping_and_dense() ? input : input.contiguous();
  const OnDeviceOf here(x);
  at::Tensor out = new_here(here, x, {1}, at::kFloat);
  check_status(dtq_amax(x.data_ptr(), out.data_ptr<float>(), x.numel(), in_code(x.scalar_type()),
                        workspaces().get(here.stream), dtq_workspace_bytes(), here.stream.stream()),
               "amax");
  return out;
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> dynamic_scaled_quant_with_scale(const at::Tensor &input,
                                                                                at::ScalarType dtype) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  const OnDeviceOf here(input);
  at::Tensor out = new_same_layout(here, input, dtype);
  at::Tensor amax_value = new_here(here, input, {1}, at::kFloat);
  at::Tensor scale = new_here(here, input, {1}, at::kFloat);
  check_status(dtq_dynamic_scaled_quant(input.data_ptr(), out.data_ptr(), amax_value.data_ptr<float>(),
                                        scale.data_ptr<float>(), input.numel(),
                                        in_code(input.scalar_type()), out_code(dtype), workspaces().get(here.stream),
                                        dtq_workspace_bytes(), here.stream.stream()),
               "dynamic_scaled_quant");
  return {out, amax_value, scale};
}

at::Tensor dynamic_scaled_quant(const at::Tensor &input, at::ScalarType dtype) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  const OnDeviceOf here(input);
  at::Tensor out = new_same_layout(here, input, dtype);
  check_status(dtq_dynamic_scaled_quant(input.data_ptr(), out.data_ptr(), nullptr, nullptr, input.numel(),
                                        in_code(input.scalar_type()), out_code(dtype), workspaces().get(here.stream),
                                        dtq_workspace_bytes(), here.stream.stream()),
               "dynamic_scaled_quant");
  return out;
}

int mx_in_code(at::ScalarType t) { return t == at::kBFloat16 ? DTQ_BF16 : (t == at::kHalf ? DTQ_F16 : DTQ_F32); }

std::tuple<at::Tensor, at::Tensor> mx_fp8_quantize(at::Tensor input, int64_t block_size, int64_t axis, bool transpose,
                                                   c10::ScalarType fp8_type) {
  TORCH_CHECK(input.is_cuda(), "Input tensor must be a CUDA tensor");
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  TORCH_CHECK(input.dim() == 2, "Input tensor must be 2D");
  // The reference accepts fp16 / fp32 inputs and fp8_type = e5m2 and then computes bf16 -> e4m3 on the
  // bytes it was given; here they are computed with the same scale rule for the asked format.  What
  // the reference ignores and no kernel here implements is rejected instead of mis-computed.
  const auto in_type = input.scalar_type();
  TORCH_CHECK(in_type == at::kBFloat16 || in_type == at::kHalf || in_type == at::kFloat,
              "Input tensor must be bfloat16, float16 or float32, but got ", input.dtype());
  TORCH_CHECK(block_size == 32, "Block size must be 32, but got ", block_size);
  const bool along_rows = axis == 0 || axis == -2;
  TORCH_CHECK(along_rows || axis == 1 || axis == -1, "axis must be 0 or 1, but got ", axis);
  TORCH_CHECK(fp8_type == at::kFloat8_e4m3fn || fp8_type == at::kFloat8_e5m2,
              "FP8 type must be Float8_e4m3fn or Float8_e5m2");
  const int64_t m = input.size(0), n = input.size(1);
  // axis / transpose (the reference declares both and ignores them).  `transpose`: the result is that of
  // the op on input.t(); axis = 0: blocks of 32 run down the columns instead of along the rows.  One of the
  // two alone means blocks along the input's dimension 0, produced by the transposing kernel in one read
  // (payload_t [n, m] contiguous, one scale per 32 rows of a column): `transpose` returns payload_t itself,
  // axis = 0 returns it viewed as [m, n].  Both together cancel: the ordinary blocks, payload viewed as [n, m].
  const OnDeviceOf here(input);
  if (along_rows != transpose) {
    TORCH_CHECK(in_type == at::kBFloat16 && fp8_type == at::kFloat8_e4m3fn,
                "axis=0 / transpose=True need a bfloat16 input and an e4m3 payload");
    TORCH_CHECK(m % 32 == 0 && n % 32 == 0, "Both dimensions must be multiples of the block size 32, but got ", m, " x ", n);
    at::Tensor out_t = new_here(here, input, {n, m}, fp8_type);
    at::Tensor scale_t = new_here(here, input, {n * (m / 32)}, at::kFloat8_e8m0fnu);
    check_status(dtq_mx_fp8_quantize_dual(input.data_ptr(), nullptr, nullptr, out_t.data_ptr(), scale_t.data_ptr(), m, n,
                                          here.stream.stream()),
                 "mx_fp8_quantize");
    return {transpose ? out_t : out_t.t(), scale_t};
  }
  TORCH_CHECK(n % 32 == 0, "The last dimension must be a multiple of the block size 32, but got ", n);
  at::Tensor out = new_same_layout(here, input, fp8_type);
  at::Tensor scale = new_here(here, input, {m * (n / 32)}, at::kFloat8_e8m0fnu);
  if (in_type == at::kBFloat16 && fp8_type == at::kFloat8_e4m3fn) {
    check_status(dtq_mx_fp8_quantize(input.data_ptr(), out.data_ptr(), scale.data_ptr(), m, n, here.stream.stream()),
                 "mx_fp8_quantize");
  } else {
    check_status(dtq_mx_quantize(input.data_ptr(), out.data_ptr(), scale.data_ptr(), m, n, mx_in_code(in_type),
                                 out_code(fp8_type), here.stream.stream()),
                 "mx_fp8_quantize");
  }
  return {transpose ? out.t() : out, scale};
}

// ---- additions ---------------------------------------------------------------------------------------

// MX cast + the tensor's amax (>= 0) from one read of the input: the first half of a step that also
// quantises the tensor tensor-wise (follow with cast_with_amax).
std::tuple<at::Tensor, at::Tensor, at::Tensor> mx_fp8_quantize_with_amax(at::Tensor input) {
  TORCH_CHECK(input.is_cuda(), "Input tensor must be a CUDA tensor");
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  TORCH_CHECK(input.dim() == 2, "Input tensor must be 2D");
  TORCH_CHECK(input.scalar_type() == at::kBFloat16, "Input tensor must be bfloat16, but got ", input.dtype());
  const int64_t m = input.size(0), n = input.size(1);
  TORCH_CHECK(n % 32 == 0, "The last dimension must be a multiple of the block size 32, but got ", n);
  const OnDeviceOf here(input);
  at::Tensor out = new_same_layout(here, input, at::kFloat8_e4m3fn);
  at::Tensor scale = new_here(here, input, {m * (n / 32)}, at::kFloat8_e8m0fnu);
  at::Tensor amax = new_here(here, input, {1}, at::kFloat);
  check_status(dtq_mx_fp8_quantize_amax(input.data_ptr(), out.data_ptr(), scale.data_ptr(), amax.data_ptr<float>(), m, n,
                                        workspaces().get(here.stream), dtq_workspace_bytes(), here.stream.stream()),
               "mx_fp8_quantize_with_amax");
  return {out, scale, amax};
}

// MXFP4: e2m1 payload packed two per byte ([M, N/2] uint8, lower index in the low nibble: the operand
// layout of the reference's mx_fp4_bf16, which reads K as a.size(1) * 2) + E8M0 scales.
std::tuple<at::Tensor, at::Tensor> mx_fp4_quantize(at::Tensor input, bool blocked) {
  TORCH_CHECK(input.is_cuda(), "Input tensor must be a CUDA tensor");
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  TORCH_CHECK(input.dim() == 2, "Input tensor must be 2D");
  const auto in_type = input.scalar_type();
  TORCH_CHECK(in_type == at::kBFloat16 || in_type == at::kHalf || in_type == at::kFloat,
              "Input tensor must be bfloat16, float16 or float32, but got ", input.dtype());
  const int64_t m = input.size(0), n = input.size(1);
  TORCH_CHECK(n % 32 == 0, "The last dimension must be a multiple of the block size 32, but got ", n);
  const OnDeviceOf here(input);
  at::Tensor out = new_here(here, input, {m, n / 2}, at::kByte);
  if (blocked) {  // scales in the layout mx_fp4_bf16 takes, zero in the padding
    at::Tensor scale = new_here(here, input, {static_cast<int64_t>(dtq_mx_blocked_scale_bytes(m, n))}, at::kFloat8_e8m0fnu);
    check_status(dtq_mx_quantize_blocked(input.data_ptr(), out.data_ptr(), scale.data_ptr(), m, n, mx_in_code(in_type),
                                         DTQ_E2M1, here.stream.stream()),
                 "mx_fp4_quantize");
    return {out, scale};
  }
  at::Tensor scale = new_here(here, input, {m * (n / 32)}, at::kFloat8_e8m0fnu);
  check_status(dtq_mx_quantize(input.data_ptr(), out.data_ptr(), scale.data_ptr(), m, n, mx_in_code(in_type), DTQ_E2M1,
                               here.stream.stream()),
               "mx_fp4_quantize");
  return {out, scale};
}

// MX cast of the input and of its transpose from one read of the input; `blocked`: both scale tensors in the
// blocked layout of the MX GEMM (zero in the padding).
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> mx_fp8_quantize_dual(at::Tensor input, bool blocked) {
  TORCH_CHECK(input.is_cuda(), "Input tensor must be a CUDA tensor");
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  TORCH_CHECK(input.dim() == 2, "Input tensor must be 2D");
  TORCH_CHECK(input.scalar_type() == at::kBFloat16, "Input tensor must be bfloat16, but got ", input.dtype());
  const int64_t m = input.size(0), n = input.size(1);
  TORCH_CHECK(m % 32 == 0 && n % 32 == 0, "Both dimensions must be multiples of the block size 32, but got ", m, " x ", n);
  const OnDeviceOf here(input);
  at::Tensor out = new_here(here, input, {m, n}, at::kFloat8_e4m3fn), out_t = new_here(here, input, {n, m}, at::kFloat8_e4m3fn);
  at::Tensor scale, scale_t;
  if (blocked) {
    scale = new_here(here, input, {static_cast<int64_t>(dtq_mx_blocked_scale_bytes(m, n))}, at::kFloat8_e8m0fnu);
    scale_t = new_here(here, input, {static_cast<int64_t>(dtq_mx_blocked_scale_bytes(n, m))}, at::kFloat8_e8m0fnu);
  } else {
    scale = new_here(here, input, {m * (n / 32)}, at::kFloat8_e8m0fnu);
    scale_t = new_here(here, input, {n * (m / 32)}, at::kFloat8_e8m0fnu);
  }
  auto fn = blocked ? dtq_mx_fp8_quantize_dual_blocked : dtq_mx_fp8_quantize_dual;
  check_status(fn(input.data_ptr(), out.data_ptr(), scale.data_ptr(), out_t.data_ptr(), scale_t.data_ptr(), m, n,
                  here.stream.stream()),
               "mx_fp8_quantize_dual");
  return {out, scale, out_t, scale_t};
}

// MX cast whose scales come out in the blocked layout of the MX GEMM (1-D e8m0 tensor of
// 512 * ceil(M/128) * ceil(N/128) bytes, zero in the padding).
std::tuple<at::Tensor, at::Tensor> mx_fp8_quantize_blocked(at::Tensor input) {
  TORCH_CHECK(input.is_cuda(), "Input tensor must be a CUDA tensor");
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  TORCH_CHECK(input.dim() == 2, "Input tensor must be 2D");
  TORCH_CHECK(input.scalar_type() == at::kBFloat16, "Input tensor must be bfloat16, but got ", input.dtype());
  const int64_t m = input.size(0), n = input.size(1);
  TORCH_CHECK(n % 32 == 0, "The last dimension must be a multiple of the block size 32, but got ", n);
  const OnDeviceOf here(input);
  at::Tensor out = new_same_layout(here, input, at::kFloat8_e4m3fn);
  at::Tensor scale = new_here(here, input, {static_cast<int64_t>(dtq_mx_blocked_scale_bytes(m, n))}, at::kFloat8_e8m0fnu);
  check_status(dtq_mx_fp8_quantize_blocked(input.data_ptr(), out.data_ptr(), scale.data_ptr(), m, n, here.stream.stream()),
               "mx_fp8_quantize_blocked");
  return {out, scale};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> dynamic_scaled_quant_rowwise(const at::Tensor &input,
                                                                             at::ScalarType dtype) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  const int64_t m = input.size(0), n = input.size(1);
  TORCH_CHECK(m == 0 || n > 0, "Rows must not be empty");
  const OnDeviceOf here(input);
  at::Tensor out = new_same_layout(here, input, dtype);
  at::Tensor amax_rows = new_here(here, input, {m, 1}, at::kFloat);
  at::Tensor scale_rows = new_here(here, input, {m, 1}, at::kFloat);
  check_status(dtq_dynamic_scaled_quant_rowwise(input.data_ptr(), out.data_ptr(), amax_rows.data_ptr<float>(),
                                                scale_rows.data_ptr<float>(), m, n, in_code(input.scalar_type()),
                                                out_code(dtype), here.stream.stream()),
               "dynamic_scaled_quant_rowwise");
  return {out, amax_rows, scale_rows};
}

std::tuple<at::Tensor, at::Tensor> cast_with_amax(const at::Tensor &input, const at::Tensor &amax_value,
                                                  at::ScalarType dtype) {
  check_fp8(dtype);
  check_input(input);
  TORCH_CHECK(input.is_contiguous(), "Input tensor must be contiguous");
  TORCH_CHECK(amax_value.scalar_type() == at::kFloat && amax_value.numel() == 1 && amax_value.is_cuda() &&
                  amax_value.device() == input.device(),
              "amax must be one fp32 value on the input's device");
  const OnDeviceOf here(input);
  at::Tensor out = new_same_layout(here, input, dtype);
  at::Tensor scale = new_here(here, input, {1}, at::kFloat);
  check_status(dtq_cast_with_amax(input.data_ptr(), out.data_ptr(), amax_value.data_ptr<float>(),
                                  scale.data_ptr<float>(), input.numel(), in_code(input.scalar_type()),
                                  out_code(dtype), here.stream.stream()),
               "cast_with_amax");
  return {out, scale};
}

// The MX block-scaled GEMM; checks and messages follow the reference's validate() (src/mx_fp8_bf16.cu:168-215).
at::Tensor mx_fp8_bf16(at::Tensor a, at::Tensor b, at::Tensor a_scale, at::Tensor b_scale) {
  TORCH_CHECK(a.is_cuda(), "a must be CUDA tensor");
  TORCH_CHECK(b.is_cuda(), "b must be CUDA tensor");
  TORCH_CHECK(a_scale.is_cuda(), "a_scale must be CUDA tensor");
  TORCH_CHECK(b_scale.is_cuda(), "b_scale must be CUDA tensor");
  TORCH_CHECK(a.dim() == 2, "a must be a matrix");
  TORCH_CHECK(b.dim() == 2, "b must be a matrix");
  TORCH_CHECK(a.scalar_type() == at::kFloat8_e4m3fn && b.scalar_type() == at::kFloat8_e4m3fn,
              "a and b must be float8_e4m3fn, but got ", a.dtype(), " and ", b.dtype());
  const int64_t M = a.size(0), K = a.size(1), N = b.size(1);
  TORCH_CHECK(b.size(0) == K, "Incompatible matrix dimensions: a is ", M, "x", K, " but b is ", b.size(0), "x", N);
  TORCH_CHECK(N % 8 == 0, "N must be a multiple of 16 but got, ", N);
  TORCH_CHECK(K % 32 == 0, "K must be a multiple of the block size 32, but got ", K);
  TORCH_CHECK(reinterpret_cast<std::uintptr_t>(a.data_ptr()) % 16 == 0, "Input tensor 'a' must be 16-byte aligned");
  TORCH_CHECK(reinterpret_cast<std::uintptr_t>(b.data_ptr()) % 16 == 0, "Input tensor 'b' must be 16-byte aligned");
  const int64_t expected_a = static_cast<int64_t>(dtq_mx_gemm_scale_bytes(M, K));
  const int64_t expected_b = static_cast<int64_t>(dtq_mx_gemm_scale_bytes(N, K));
  // the reference checks 128 * ceil(rows / 128) * ceil(K / 32) and its kernel reads whole 4-block atoms; the two
  // agree whenever K is a multiple of 128, and the blocked casts of this library always produce whole atoms
  TORCH_CHECK(a_scale.numel() == expected_a || (K % 128 == 0 && a_scale.numel() == 128 * ((M + 127) / 128) * (K / 32)),
              "Expected a_scale_size to be ", expected_a, " but got ", a_scale.numel());
  TORCH_CHECK(b_scale.numel() == expected_b || (K % 128 == 0 && b_scale.numel() == 128 * ((N + 127) / 128) * (K / 32)),
              "Expected b_scale_size to be ", expected_b, " but got ", b_scale.numel());
  TORCH_CHECK(a_scale.element_size() == 1 && b_scale.element_size() == 1, "scales must be one byte per block (float8_e8m0fnu)");
  TORCH_CHECK(a_scale.is_contiguous() && b_scale.is_contiguous(), "scale tensors must be contiguous");
  TORCH_CHECK(a.stride(1) == 1 && a.stride(0) == K, "Input tensor 'a' must be contiguous in the K dimension (row-major)");
  TORCH_CHECK(b.stride(0) == 1 && b.stride(1) == K, "Input tensor 'b' must be contiguous in the K dimension (column-major)");
  const OnDeviceOf here(a);
  at::Tensor out = new_here(here, a, {M, N}, at::kBFloat16);
  check_status(dtq_mx_fp8_bf16(a.data_ptr(), b.data_ptr(), a_scale.data_ptr(), b_scale.data_ptr(), out.data_ptr(), M, N, K,
                               workspaces().get(here.stream), dtq_workspace_bytes(), here.stream.stream()),
               "mx_fp8_bf16");
  return out;
}

// The MXFP4 GEMM (src/mx_fp8_bf16.cu:243-271): e2m1 operands packed two per byte, K = 2 * a.size(1).  The reference
// runs no checks of its own here; the ones below are mx_fp8_bf16's applied to the packed shapes.
at::Tensor mx_fp4_bf16(at::Tensor a, at::Tensor b, at::Tensor a_scale, at::Tensor b_scale) {
  TORCH_CHECK(a.is_cuda(), "a must be CUDA tensor");
  TORCH_CHECK(b.is_cuda(), "b must be CUDA tensor");
  TORCH_CHECK(a_scale.is_cuda(), "a_scale must be CUDA tensor");
  TORCH_CHECK(b_scale.is_cuda(), "b_scale must be CUDA tensor");
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2, "a and b must be matrices");
  TORCH_CHECK(a.element_size() == 1 && b.element_size() == 1, "a and b must hold two e2m1 values per byte (uint8 or float4_e2m1fn_x2)");
  const int64_t M = a.size(0), Kb = a.size(1), K = Kb * 2, N = b.size(1);
  TORCH_CHECK(b.size(0) == Kb, "Incompatible matrix dimensions: a is ", M, "x", Kb, " but b is ", b.size(0), "x", N, " (packed bytes)");
  TORCH_CHECK(N % 8 == 0, "N must be a multiple of 16 but got, ", N);
  TORCH_CHECK(K % 32 == 0, "K must be a multiple of the block size 32, but got ", K);
  TORCH_CHECK(reinterpret_cast<std::uintptr_t>(a.data_ptr()) % 16 == 0, "Input tensor 'a' must be 16-byte aligned");
  TORCH_CHECK(reinterpret_cast<std::uintptr_t>(b.data_ptr()) % 16 == 0, "Input tensor 'b' must be 16-byte aligned");
  TORCH_CHECK(a_scale.numel() == static_cast<int64_t>(dtq_mx_gemm_scale_bytes(M, K)), "Expected a_scale_size to be ",
              dtq_mx_gemm_scale_bytes(M, K), " but got ", a_scale.numel());
  TORCH_CHECK(b_scale.numel() == static_cast<int64_t>(dtq_mx_gemm_scale_bytes(N, K)), "Expected b_scale_size to be ",
              dtq_mx_gemm_scale_bytes(N, K), " but got ", b_scale.numel());
  TORCH_CHECK(a_scale.element_size() == 1 && b_scale.element_size() == 1, "scales must be one byte per block (float8_e8m0fnu)");
  TORCH_CHECK(a_scale.is_contiguous() && b_scale.is_contiguous(), "scale tensors must be contiguous");
  TORCH_CHECK(a.stride(1) == 1 && a.stride(0) == Kb, "Input tensor 'a' must be contiguous in the K dimension (row-major)");
  TORCH_CHECK(b.stride(0) == 1 && b.stride(1) == Kb, "Input tensor 'b' must be contiguous in the K dimension (column-major)");
  const OnDeviceOf here(a);
  at::Tensor out = new_here(here, a, {M, N}, at::kBFloat16);
  check_status(dtq_mx_fp4_bf16(a.data_ptr(), b.data_ptr(), a_scale.data_ptr(), b_scale.data_ptr(), out.data_ptr(), M, N, K,
                               workspaces().get(here.stream), dtq_workspace_bytes(), here.stream.stream()),
               "mx_fp4_bf16");
  return out;
}

// The row-wise scaled fp8 GEMM under the reference's name and schema; checks as src/sweep_mm.cu:11-58.
at::Tensor sweep_mm(at::Tensor XQ, at::Tensor WQ, at::Tensor x_scale, at::Tensor w_scale, std::optional<at::Tensor> bias,
                    at::ScalarType out_dtype, bool use_fast_accum, int64_t cluster_shape_x, int64_t cluster_shape_y,
                    int64_t cluster_shape_z, bool transposed, int64_t swizzle) {
  // tuning arguments of the reference's CUTLASS kernels (no effect on the result): accepted, not used
  (void)use_fast_accum, (void)cluster_shape_x, (void)cluster_shape_y, (void)cluster_shape_z, (void)transposed, (void)swizzle;
  TORCH_CHECK(XQ.is_cuda());
  TORCH_CHECK(XQ.device() == WQ.device() && x_scale.device() == XQ.device() && w_scale.device() == WQ.device());
  TORCH_CHECK(XQ.scalar_type() == at::kFloat8_e4m3fn || XQ.scalar_type() == at::kFloat8_e5m2);
  TORCH_CHECK(WQ.scalar_type() == at::kFloat8_e4m3fn);
  TORCH_CHECK(x_scale.scalar_type() == at::kFloat && w_scale.scalar_type() == at::kFloat);
  TORCH_CHECK(out_dtype == at::kBFloat16, "out_dtype must be bfloat16");
  TORCH_CHECK(XQ.dim() == 2 && WQ.dim() == 2 && XQ.size(1) == WQ.size(0));
  const int64_t M = XQ.size(0), K = XQ.size(1), N = WQ.size(1);
  TORCH_CHECK(x_scale.dim() == 2 && w_scale.dim() == 2);
  TORCH_CHECK(x_scale.size(0) == M && x_scale.size(1) == 1);
  TORCH_CHECK(w_scale.size(0) == 1 && w_scale.size(1) == N);
  TORCH_CHECK(XQ.stride(1) == 1 && XQ.stride(0) == K, "x must be row-major and dense");
  TORCH_CHECK(WQ.stride(0) == 1 && WQ.stride(1) == K, "w must be column-major and dense");
  TORCH_CHECK(x_scale.stride(0) == 1 && w_scale.stride(1) == 1);
  TORCH_CHECK(N % 8 == 0 && K % 16 == 0, "N must be a multiple of 8 and K of 16");
  const void *bias_ptr = nullptr;
  int bias_code = DTQ_F32;
  if (bias.has_value()) {
    TORCH_CHECK(bias->device() == WQ.device());
    TORCH_CHECK(bias->scalar_type() == at::kFloat || bias->scalar_type() == at::kBFloat16);
    TORCH_CHECK(bias->dim() == 1 && bias->size(0) == N && bias->stride(0) == 1);
    bias_ptr = bias->data_ptr();
    bias_code = bias->scalar_type() == at::kBFloat16 ? DTQ_BF16 : DTQ_F32;
  }
  const OnDeviceOf here(XQ);
  at::Tensor out = new_here(here, XQ, {M, N}, out_dtype);
  check_status(dtq_rowwise_fp8_bf16(XQ.data_ptr(), WQ.data_ptr(), x_scale.data_ptr<float>(), w_scale.data_ptr<float>(), bias_ptr,
                                    bias_code, out.data_ptr(), M, N, K, out_code(XQ.scalar_type()), DTQ_GEMM_AUTO,
                                    workspaces().get(here.stream), dtq_workspace_bytes(), here.stream.stream()),
               "sweep_mm");
  return out;
}

void check_device_status() { workspaces().check_all(); }

}  // namespace

TORCH_LIBRARY(DrissTorch, m) {
  m.set_python_module("driss_torch_b200.abstract_impls");
  // the reference's schemas, verbatim
  m.def("saturated_cast(Tensor input, Tensor scale, ScalarType dtype, bool transpose) -> Tensor");
  m.impl("saturated_cast", c10::DispatchKey::CUDA, TORCH_FN(saturated_cast));
  m.def("amax(Tensor input) -> Tensor");
  m.impl("amax", c10::DispatchKey::CUDA, TORCH_FN(amax));
  m.def("dynamic_scaled_quant(Tensor input, ScalarType dtype) -> Tensor");
  m.impl("dynamic_scaled_quant", c10::DispatchKey::CUDA, TORCH_FN(dynamic_scaled_quant));
  m.def("mx_fp8_quantize(Tensor input, int block_size, int axis, bool transpose, ScalarType fp8_type) -> (Tensor, Tensor)");
  m.impl("mx_fp8_quantize", c10::DispatchKey::CUDA, TORCH_FN(mx_fp8_quantize));
  // additions: the fused op's amax and scale as outputs, the row-wise variant, the cast phase alone
  m.def("dynamic_scaled_quant_with_scale(Tensor input, ScalarType dtype) -> (Tensor, Tensor, Tensor)");
  m.impl("dynamic_scaled_quant_with_scale", c10::DispatchKey::CUDA, TORCH_FN(dynamic_scaled_quant_with_scale));
  m.def("dynamic_scaled_quant_rowwise(Tensor input, ScalarType dtype) -> (Tensor, Tensor, Tensor)");
  m.impl("dynamic_scaled_quant_rowwise", c10::DispatchKey::CUDA, TORCH_FN(dynamic_scaled_quant_rowwise));
  m.def("cast_with_amax(Tensor input, Tensor amax, ScalarType dtype) -> (Tensor, Tensor)");
  m.impl("cast_with_amax", c10::DispatchKey::CUDA, TORCH_FN(cast_with_amax));
  m.def("cast_with_amax_dual(Tensor input, Tensor amax, ScalarType dtype) -> (Tensor, Tensor, Tensor)");
  m.impl("cast_with_amax_dual", c10::DispatchKey::CUDA, TORCH_FN(cast_with_amax_dual));
  m.def("dynamic_scaled_quant_dual(Tensor input, ScalarType dtype) -> (Tensor, Tensor, Tensor, Tensor)");
  m.impl("dynamic_scaled_quant_dual", c10::DispatchKey::CUDA, TORCH_FN(dynamic_scaled_quant_dual));
  m.def("saturated_cast_transposed(Tensor input, Tensor scale, ScalarType dtype) -> Tensor");
  m.impl("saturated_cast_transposed", c10::DispatchKey::CUDA, TORCH_FN(saturated_cast_transposed));
  m.def("saturated_cast_dual(Tensor input, Tensor scale, ScalarType dtype) -> (Tensor, Tensor)");
  m.impl("saturated_cast_dual", c10::DispatchKey::CUDA, TORCH_FN(saturated_cast_dual));
  m.def("mx_fp8_quantize_with_amax(Tensor input) -> (Tensor, Tensor, Tensor)");
  m.impl("mx_fp8_quantize_with_amax", c10::DispatchKey::CUDA, TORCH_FN(mx_fp8_quantize_with_amax));
  m.def("mx_fp4_quantize(Tensor input, bool blocked=False) -> (Tensor, Tensor)");
  m.impl("mx_fp4_quantize", c10::DispatchKey::CUDA, TORCH_FN(mx_fp4_quantize));
  m.def("mx_fp8_quantize_dual(Tensor input, bool blocked=False) -> (Tensor, Tensor, Tensor, Tensor)");
  m.impl("mx_fp8_quantize_dual", c10::DispatchKey::CUDA, TORCH_FN(mx_fp8_quantize_dual));
  m.def("mx_fp8_quantize_blocked(Tensor input) -> (Tensor, Tensor)");
  m.impl("mx_fp8_quantize_blocked", c10::DispatchKey::CUDA, TORCH_FN(mx_fp8_quantize_blocked));
  // the consumer GEMM, the reference's schema verbatim (src/register_ops.cpp:35-36)
  m.def("mx_fp8_bf16(Tensor a, Tensor b, Tensor a_scale, Tensor b_scale) -> Tensor");
  m.impl("mx_fp8_bf16", c10::DispatchKey::CUDA, TORCH_FN(mx_fp8_bf16));
  m.def("mx_fp4_bf16(Tensor a, Tensor b, Tensor a_scale, Tensor b_scale) -> Tensor");  // src/register_ops.cpp:37-38
  m.impl("mx_fp4_bf16", c10::DispatchKey::CUDA, TORCH_FN(mx_fp4_bf16));
  // src/register_ops.cpp:32-33
  m.def("sweep_mm(Tensor x, Tensor w, Tensor x_scale, Tensor w_scale, Tensor? bias , ScalarType out_dtype, bool use_fast_accum, int cluster_shape_x, int cluster_shape_y, int cluster_shape_z, bool transposed, int swizzle) -> Tensor");
  m.impl("sweep_mm", c10::DispatchKey::CUDA, TORCH_FN(sweep_mm));
  m.def("check_device_status() -> ()");
  m.impl("check_device_status", c10::DispatchKey::CompositeExplicitAutograd, TORCH_FN(check_device_status));
}
