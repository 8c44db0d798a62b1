// Compiled torch binding over the C ABI of libfa8_b200.so.
//
// Provides what the reference extension provides: a pybind11 module named
// attention_cutlass_fp8 (setup.py:45, csrc/attention_api.cpp:6-10) whose one function
//   flash_attention_v2_cutlass(q, k, v, is_causal = false, softmax_scale = 1) -> [O]
// takes torch tensors (include/attention_api.h:10-11).  The body stands where the reference
// has csrc/flash_attention.cu:639-668: input checks, output allocation with torch's allocator,
// parameter packing, dispatch - here one call of fa8_fwd on torch's current stream.  Nothing
// in this file touches the GPU except through that call.
//
// Differences from the reference, as everywhere in this library: O is fp16, the call does not
// synchronise the device, and every failure is a C++ exception (RuntimeError in Python) instead
// of exit().  Two keyword arguments are added after the reference's five: v_layout
// ("transposed", the reference's [batch, heads, head_dim, seqlen], or "natural") and o_scale.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>
#include <optional>
#include <string>
#include <vector>

#include "fa8_b200.h"

namespace {

// CHECK_INPUT of include/attention_api.cuh:12-18
void check_input(const torch::Tensor& x, const char* name) {
  TORCH_CHECK(x.device().is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(x.is_contiguous(), name, " must be contiguous");
}

std::vector<torch::Tensor> flash_attention_v2_cutlass(torch::Tensor q, torch::Tensor k, torch::Tensor v,
                                                      bool is_causal, float softmax_scale,
                                                      const std::string& v_layout, float o_scale) {
  check_input(q, "q");
  check_input(k, "k");
  check_input(v, "v");
  const auto dtype = q.scalar_type();
  TORCH_CHECK(dtype == at::kFloat8_e4m3fn || dtype == at::kFloat8_e5m2,
              "q must be float8_e4m3fn (or float8_e5m2), got ", q.dtype());
  TORCH_CHECK(k.scalar_type() == dtype && v.scalar_type() == dtype, "k and v must have q's dtype");
  TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && v.dim() == 4,
              "q, k and v must have 4 dimensions [batch, heads, seqlen, head_dim]");
  TORCH_CHECK(k.device() == q.device() && v.device() == q.device(), "q, k and v must be on the same device");
  const int64_t B = q.size(0), H = q.size(1), S = q.size(2), D = q.size(3);
  const int64_t Hk = k.size(1), Sk = k.size(2);
  TORCH_CHECK(k.size(0) == B && k.size(3) == D && Hk >= 1 && H % Hk == 0,
              "k must be [batch, heads_kv, seqlen_k, head_dim] with heads_kv dividing q's heads");
  int32_t layout;
  if (v_layout == "transposed") {
    layout = FA8_V_TRANSPOSED;
    TORCH_CHECK(v.size(0) == B && v.size(1) == Hk && v.size(2) == D && v.size(3) == Sk,
                "v must be [batch, heads_kv, head_dim, seqlen_k] for v_layout='transposed'");
  } else if (v_layout == "natural") {
    layout = FA8_V_NATURAL;
    TORCH_CHECK(v.size(0) == B && v.size(1) == Hk && v.size(2) == Sk && v.size(3) == D,
                "v must be [batch, heads_kv, seqlen_k, head_dim] for v_layout='natural'");
  } else {
    TORCH_CHECK(false, "v_layout must be 'transposed' or 'natural'");
  }
  TORCH_CHECK(B <= INT32_MAX && H <= INT32_MAX && S <= INT32_MAX && Sk <= INT32_MAX && D <= INT32_MAX,
              "tensor extents must fit 32 bits");

  const c10::cuda::CUDAGuard guard(q.device());
  // The reference allocates with torch's allocator as well (csrc/flash_attention.cu:656), in e4m3.
  torch::Tensor out = torch::empty({B, H, S, D}, q.options().dtype(torch::kFloat16));

  fa8_fwd_params p{};
  p.q = q.data_ptr();
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  p.o = out.data_ptr();
  p.batch = static_cast<int32_t>(B);
  p.heads = static_cast<int32_t>(H);
  p.seqlen = static_cast<int32_t>(S);
  p.head_dim = static_cast<int32_t>(D);
  p.softmax_scale = softmax_scale;
  p.is_causal = is_causal ? 1 : 0;
  p.v_layout = layout;
  p.o_scale = o_scale;
  p.status_word = nullptr;   // the library's own word; a failed launch surfaces at the next call
  p.heads_kv = static_cast<int32_t>(Hk);
  p.fp8_format = (dtype == at::kFloat8_e5m2) ? FA8_FP8_E5M2 : FA8_FP8_E4M3;
  p.seqlen_k = static_cast<int32_t>(Sk);
  const int rc = fa8_fwd(&p, c10::cuda::getCurrentCUDAStream(q.device().index()).stream());
  TORCH_CHECK(rc == FA8_OK, "fa8 error ", rc, ": ", fa8_error_string(rc), " [", fa8_last_error_detail(), "]");
  return {out};
}

// Synchronises torch's current stream on `device_index` (-1 = current device) and raises if a
// launch of this library reported an expired wait; stands where the reference has
// cudaDeviceSynchronize + CUDA_ERROR_CHECK (csrc/flash_attention.cu:663-665).
void check_status(int64_t device_index) {
  const c10::DeviceIndex idx =
      device_index < 0 ? c10::cuda::current_device() : static_cast<c10::DeviceIndex>(device_index);
  const c10::cuda::CUDAGuard guard(idx);
  int32_t code = 0;
  const int rc = fa8_check_status(nullptr, c10::cuda::getCurrentCUDAStream(idx).stream(), &code);
  TORCH_CHECK(rc == FA8_OK, "fa8 error ", rc, ": ", fa8_error_string(rc), " (device code ", code, ") [",
              fa8_last_error_detail(), "]");
}

// ---- the package's operators (api.py) -----------------------------------------------------
// What api.py does around a call - checks, outputs, parameter block - in native code: through
// Python and ctypes it took 15 us of host time a call, twice what the smallest launch takes on the
// GPU.  These take only calls that nothing is wrong with; for any other they return None, and
// api.py's own checks then say what it is.  An error code of the library is returned as an integer.

// Status word of the package per device, registered by api.py (0 = not yet).
constexpr int kMaxDevices = 64;
std::atomic<int64_t> g_status_words[kMaxDevices];

void set_status_word(int64_t device_index, int64_t address) {
  if (device_index >= 0 && device_index < kMaxDevices) g_status_words[device_index].store(address);
}

bool plain(const torch::Tensor& x, const c10::Device& dev) { return x.device() == dev && x.is_contiguous(); }

py::object forward(const torch::Tensor& q, const torch::Tensor& k, const torch::Tensor& v, bool is_causal,
                   double softmax_scale, bool v_natural, double o_scale, const std::optional<torch::Tensor>& out_given,
                   bool return_lse, const std::optional<torch::Tensor>& descale_q,
                   const std::optional<torch::Tensor>& descale_k, const std::optional<torch::Tensor>& descale_v,
                   const std::optional<torch::Tensor>& status) {
  const auto dev = q.device();
  const auto dtype = q.scalar_type();
  if (!dev.is_cuda() || !plain(q, dev) || !plain(k, dev) || !plain(v, dev)) return py::none();
  if (dtype != at::kFloat8_e4m3fn && dtype != at::kFloat8_e5m2) return py::none();
  if (k.scalar_type() != dtype || v.scalar_type() != dtype) return py::none();
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return py::none();
  const int64_t B = q.size(0), H = q.size(1), S = q.size(2), D = q.size(3), Hk = k.size(1), Sk = k.size(2);
  if (k.size(0) != B || k.size(3) != D || Hk < 1 || H % Hk != 0) return py::none();
  if (v.size(0) != B || v.size(1) != Hk || v.size(2) != (v_natural ? Sk : D) || v.size(3) != (v_natural ? D : Sk)) return py::none();
  if (B > INT32_MAX || H > INT32_MAX || S > INT32_MAX || Sk > INT32_MAX || D > INT32_MAX) return py::none();
  torch::Tensor out;
  if (out_given) {
    out = *out_given;
    if (!plain(out, dev) || out.scalar_type() != at::kHalf || out.sizes() != q.sizes()) return py::none();
  }
  const std::optional<torch::Tensor>* descales[3] = {&descale_q, &descale_k, &descale_v};
  const int64_t full[3] = {B * H, B * Hk, B * Hk};
  bool per_head = false;
  for (const auto* d : descales) per_head = per_head || (*d && (*d)->numel() > 1);
  const float* dp[3] = {nullptr, nullptr, nullptr};
  for (int i = 0; i < 3; ++i) {
    if (!*descales[i]) continue;
    const torch::Tensor& d = **descales[i];
    if (!plain(d, dev) || d.scalar_type() != at::kFloat || d.numel() != (per_head ? full[i] : 1)) return py::none();
    dp[i] = static_cast<const float*>(d.data_ptr());
  }
  int64_t word = 0;
  if (status) {
    if (!status->device().is_cuda()) return py::none();
    word = reinterpret_cast<int64_t>(status->data_ptr());
  } else if (dev.index() >= 0 && dev.index() < kMaxDevices) {
    word = g_status_words[dev.index()].load();
  }
  if (word == 0) return py::none();

  const c10::cuda::OptionalCUDAGuard guard(dev);
  if (!out_given) out = at::empty({B, H, S, D}, q.options().dtype(at::kHalf));
  torch::Tensor lse;
  if (return_lse) lse = at::empty({B, H, S}, q.options().dtype(at::kFloat));
  fa8_fwd_params p{};
  p.q = q.data_ptr();
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  p.o = out.data_ptr();
  p.batch = static_cast<int32_t>(B);
  p.heads = static_cast<int32_t>(H);
  p.seqlen = static_cast<int32_t>(S);
  p.head_dim = static_cast<int32_t>(D);
  p.softmax_scale = static_cast<float>(softmax_scale);
  p.is_causal = is_causal ? 1 : 0;
  p.v_layout = v_natural ? FA8_V_NATURAL : FA8_V_TRANSPOSED;
  p.o_scale = static_cast<float>(o_scale);
  p.status_word = reinterpret_cast<int32_t*>(word);
  p.softmax_lse = return_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
  p.heads_kv = static_cast<int32_t>(Hk);
  p.descale_q = dp[0];
  p.descale_k = dp[1];
  p.descale_v = dp[2];
  p.fp8_format = dtype == at::kFloat8_e5m2 ? FA8_FP8_E5M2 : FA8_FP8_E4M3;
  p.seqlen_k = static_cast<int32_t>(Sk);
  p.descale_per_head = per_head ? 1 : 0;
  int rc;
  {
    const py::gil_scoped_release nogil;
    rc = fa8_fwd(&p, c10::cuda::getCurrentCUDAStream(dev.index()).stream());
  }
  if (rc != FA8_OK) return py::int_(rc);
  py::list result;
  result.append(out);
  if (return_lse) result.append(lse);
  return std::move(result);
}

py::object quantize(const torch::Tensor& x, bool per_head) {
  const auto dev = x.device();
  if (!dev.is_cuda() || !x.is_contiguous() || (x.scalar_type() != at::kHalf && x.scalar_type() != at::kBFloat16)) return py::none();
  if (per_head && x.dim() < 3) return py::none();
  const int64_t n_seg = per_head ? x.size(0) * x.size(1) : 1;
  if (x.numel() <= 0 || n_seg > INT32_MAX) return py::none();
  const c10::cuda::OptionalCUDAGuard guard(dev);
  torch::Tensor x8 = at::empty(x.sizes(), x.options().dtype(at::kFloat8_e4m3fn));
  torch::Tensor scal = at::empty({2 * n_seg}, x.options().dtype(at::kFloat));       // [amax..., descale...]
  float* const amax = static_cast<float*>(scal.data_ptr());
  const int32_t dt = x.scalar_type() == at::kBFloat16 ? FA8_DTYPE_BF16 : FA8_DTYPE_FP16;
  int rc;
  {
    const py::gil_scoped_release nogil;
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    rc = per_head ? fa8_quantize_e4m3_segments(x.data_ptr(), dt, x8.data_ptr(), x.numel() / n_seg,
                                               static_cast<int32_t>(n_seg), amax, amax + n_seg, stream)
                  : fa8_quantize_e4m3(x.data_ptr(), dt, x8.data_ptr(), x.numel(), amax, amax + 1, stream);
  }
  if (rc != FA8_OK) return py::int_(rc);
  return py::make_tuple(x8, scal.slice(0, n_seg));
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("flash_attention_v2_cutlass", &flash_attention_v2_cutlass,
        "FP8 flash-attention forward on sm_100a: e4m3 (or e5m2) q, k [batch, heads, seqlen, head_dim] and "
        "v -> [fp16 O]",
        py::arg("q"), py::arg("k"), py::arg("v"), py::arg("is_causal") = false, py::arg("softmax_scale") = 1.0f,
        py::kw_only(), py::arg("v_layout") = "transposed", py::arg("o_scale") = 1.0f);
  m.def("check_status", &check_status, "synchronise the current stream and raise if a launch reported a failure",
        py::arg("device_index") = -1);
  m.def("_forward", &forward, "the package's operator: a list of outputs, None (something is wrong with the call) or an error code");
  m.def("_quantize", &quantize, "the package's quantize_e4m3, the same way");
  m.def("_set_status_word", &set_status_word);
  m.def("abi_version", [] { return fa8_version(); }, "version of the C ABI the module was linked against");
}
