// Torch extension module with the function the reference's compiled module
// exports: gmm(a, b, c, batch_sizes, trans_a, trans_b) -> None
// (reference: csrc/ops.cu:7-9 binding grouped_gemm::GroupedGemm,
// csrc/grouped_gemm.cu:470-564).  It repeats the reference's argument checks as
// TORCH_CHECKs, takes the current CUDA stream and a workspace from torch's
// caching allocator, and hands raw pointers to the C ABI (include/b200gmm.h).
// All arithmetic lives in libb200gmm.so; nothing here touches the data.
// Beside it, gmm_autograd: the same product as a node of the autograd graph
// (reference: grouped_gemm/ops.py:8-29), for ops.gmm.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <mutex>
#include <unordered_map>

#include "b200gmm.h"

namespace {

// One status word per device: the kernels OR B200GMM_STATUS_* bits into it.
at::Tensor status_word(const c10::Device& device) {
  static std::mutex mu;
  static std::unordered_map<int, at::Tensor> words;
  std::lock_guard<std::mutex> lock(mu);
  auto it = words.find(device.index());
  if (it == words.end()) {
    it = words.emplace(device.index(),
                       at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(device))).first;
  }
  return it->second;
}

// Checks a product's arguments and returns the columns of its result.
int64_t check_product(const at::Tensor& a, const at::Tensor& b, const at::Tensor& c, const at::Tensor& batch_sizes, bool trans_a,
                      bool trans_b) {
  // Same checks, in the same order, as csrc/grouped_gemm.cu:476-540.
  TORCH_CHECK(!(trans_a && trans_b), "only one of trans_a / trans_b may be set");
  TORCH_CHECK(batch_sizes.is_cuda() || batch_sizes.is_cpu(), "batch_sizes must be a CPU or CUDA tensor");
  TORCH_CHECK(batch_sizes.dim() == 1, "batch_sizes must be 1-D");
  TORCH_CHECK(batch_sizes.scalar_type() == at::kLong, "batch_sizes must be int64");
  TORCH_CHECK(a.is_cuda(), "a must be a CUDA tensor");
  TORCH_CHECK(a.dim() == 2, "a must be 2-D");
  TORCH_CHECK(a.scalar_type() == at::kBFloat16, "a must be bfloat16");
  TORCH_CHECK(b.is_cuda() && c.is_cuda(), "b and c must be CUDA tensors");
  TORCH_CHECK(b.scalar_type() == at::kBFloat16 && c.scalar_type() == at::kBFloat16,
              "b and c must be bfloat16");
  const int64_t z = batch_sizes.size(0);
  int64_t n = 0;
  if (trans_a) {
    TORCH_CHECK(b.dim() == 2, "b must be 2-D when trans_a is set");
    TORCH_CHECK(c.dim() == 3, "c must be 3-D when trans_a is set");
    TORCH_CHECK(b.size(0) == a.size(0), "a and b must have the same number of rows");
    TORCH_CHECK(c.size(0) == z && c.size(1) == a.size(1) && c.size(2) == b.size(1),
                "c must be [num_experts, a.shape[1], b.shape[1]]");
    n = b.size(1);
  } else {
    TORCH_CHECK(b.dim() == 3, "b must be 3-D");
    TORCH_CHECK(c.dim() == 2, "c must be 2-D");
    const int64_t hidden_in = trans_b ? b.size(2) : b.size(1);
    n = trans_b ? b.size(1) : b.size(2);
    TORCH_CHECK(hidden_in == a.size(1), "contraction dimensions of a and b differ");
    TORCH_CHECK(z == b.size(0), "need one batch size per expert");
    // The reference leaves c's 2-D shape unchecked; a short c would be written
    // out of bounds, so it is checked here.
    TORCH_CHECK(c.size(0) == a.size(0) && c.size(1) == n, "c must be [a.shape[0], hidden_out]");
  }
  TORCH_CHECK(a.is_contiguous() && b.is_contiguous() && c.is_contiguous(), "a, b and c must be contiguous");
  TORCH_CHECK(a.device() == b.device() && a.device() == c.device(), "a, b and c must be on one device");
  if (batch_sizes.is_cuda()) {
    TORCH_CHECK(batch_sizes.device() == a.device(), "batch_sizes must be on a's device or on the CPU");
    TORCH_CHECK(batch_sizes.is_contiguous(), "batch_sizes must be contiguous");
  }
  TORCH_CHECK(z <= B200GMM_MAX_EXPERTS, b200gmm_strerror(B200GMM_ELIMIT));
  return n;
}

// batch_sizes as the library wants it.  It reads host batch sizes in pageable memory before the
// call returns (as an argument of the launch, or staged by an asynchronous copy).  Pinned
// memory it reads later, on the stream, when the caller may already have changed or freed
// it: take a pageable copy.
at::Tensor readable_sizes(const at::Tensor& batch_sizes) {
  if (batch_sizes.is_cuda()) return batch_sizes;
  at::Tensor sizes = batch_sizes.contiguous();
  return sizes.is_pinned() ? sizes.clone() : sizes;
}

at::Tensor workspace(const at::Tensor& a, int64_t z, size_t* bytes) {
  // Integers go into the messages below as std::to_string(...): streaming an int
  // into a TORCH_CHECK message has been seen to crash inside the iostream number
  // facets when libstdc++ versions are mixed; strings are always fine.
  const int rc = b200gmm_workspace_bytes(static_cast<int>(z), bytes);
  TORCH_CHECK(rc == 0, "b200gmm_workspace_bytes: ", b200gmm_strerror(rc), " (code ", std::to_string(rc), ")");
  return at::empty({static_cast<int64_t>(*bytes)}, at::TensorOptions().dtype(at::kByte).device(a.device()));
}

void gmm(at::Tensor a, at::Tensor b, at::Tensor c, at::Tensor batch_sizes, bool trans_a, bool trans_b) {
  const int64_t n = check_product(a, b, c, batch_sizes, trans_a, trans_b), z = batch_sizes.size(0);
  batch_sizes = readable_sizes(batch_sizes);
  c10::cuda::CUDAGuard guard(a.device());
  size_t ws_bytes = 0;
  at::Tensor ws = workspace(a, z, &ws_bytes);
  at::Tensor status = status_word(a.device());
  const int rc = b200gmm_run(a.data_ptr(), b.data_ptr(), c.data_ptr(), batch_sizes.data_ptr<int64_t>(),
                             batch_sizes.is_cuda() ? 1 : 0, static_cast<int>(z), a.size(0), a.size(1), n, trans_a ? 1 : 0,
                             trans_b ? 1 : 0, ws.data_ptr(), ws_bytes, reinterpret_cast<uint32_t*>(status.data_ptr<int>()),
                             at::cuda::getCurrentCUDAStream(a.device().index()).stream());
  TORCH_CHECK(rc == 0, "b200gmm_run: ", b200gmm_strerror(rc), " (code ", std::to_string(rc), ")");
}

// Both gradients of gmm(a, b, .., false, trans_b), given that of its result.
void gmm_gradients(const at::Tensor& a, const at::Tensor& b, const at::Tensor& grad, const at::Tensor& a_grad,
                   const at::Tensor& b_grad, const at::Tensor& batch_sizes, bool trans_b) {
  check_product(grad, b, a_grad, batch_sizes, false, !trans_b);
  check_product(trans_b ? grad : a, trans_b ? a : grad, b_grad, batch_sizes, true, false);
  const at::Tensor sizes = readable_sizes(batch_sizes);
  const int64_t z = sizes.size(0);
  c10::cuda::CUDAGuard guard(a.device());
  size_t ws_bytes = 0;
  at::Tensor ws = workspace(a, z, &ws_bytes);
  at::Tensor status = status_word(a.device());
  const int rc = b200gmm_run_gradients(a.data_ptr(), b.data_ptr(), grad.data_ptr(), a_grad.data_ptr(), b_grad.data_ptr(),
                                       sizes.data_ptr<int64_t>(), sizes.is_cuda() ? 1 : 0, static_cast<int>(z), a.size(0),
                                       a.size(1), grad.size(1), trans_b ? 1 : 0, ws.data_ptr(), ws_bytes,
                                       reinterpret_cast<uint32_t*>(status.data_ptr<int>()),
                                       at::cuda::getCurrentCUDAStream(a.device().index()).stream());
  TORCH_CHECK(rc == 0, "b200gmm_run_gradients: ", b200gmm_strerror(rc), " (code ", std::to_string(rc), ")");
}

// The reference's GroupedGemm (grouped_gemm/ops.py:8-29) as a native autograd function.
// A call of a few hundred rows is bound by the host: with the function in Python the
// training step of 512 rows (4 experts, k = n = 128) took 99 us, natively 74 us.  The saved tensors go through
// the graph's own hooks and version checks; forward-mode, vmap and second derivatives
// are as undefined as they are for the Python function.
struct GmmFunction : public torch::autograd::Function<GmmFunction> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& a, const at::Tensor& b,
                            const at::Tensor& batch_sizes, bool trans_b) {
    ctx->saved_data["trans_b"] = trans_b;
    ctx->save_for_backward({a, b, batch_sizes});
    at::Tensor c = at::empty({a.size(0), b.size(trans_b ? 1 : 2)}, a.options());
    gmm(a, b, c, batch_sizes, false, trans_b);
    return c;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const torch::autograd::variable_list saved = ctx->get_saved_variables();
    const at::Tensor &a = saved[0], &b = saved[1], &batch_sizes = saved[2];
    const bool trans_b = ctx->saved_data["trans_b"].toBool();
    const bool want_a = ctx->needs_input_grad(0), want_b = ctx->needs_input_grad(1);
    at::Tensor agrad, bgrad;
    if (want_a || want_b) {
      const at::Tensor grad = grads[0].contiguous();
      const at::Tensor& lhs = trans_b ? grad : a;
      const at::Tensor& rhs = trans_b ? a : grad;
      if (want_a) agrad = at::empty({grad.size(0), b.size(trans_b ? 2 : 1)}, grad.options());
      if (want_b) bgrad = at::empty({batch_sizes.size(0), lhs.size(1), rhs.size(1)}, lhs.options());
      if (want_a && want_b) gmm_gradients(a, b, grad, agrad, bgrad, batch_sizes, trans_b);
      else if (want_a) gmm(grad, b, agrad, batch_sizes, false, !trans_b);  // the other orientation of b (ops.py:19-22)
      else gmm(lhs, rhs, bgrad, batch_sizes, true, false);                 // in b's own layout (ops.py:24-28)
    }
    return {agrad, bgrad, at::Tensor(), at::Tensor()};
  }
};

at::Tensor gmm_autograd(const at::Tensor& a, const at::Tensor& b, const at::Tensor& batch_sizes, bool trans_b) {
  TORCH_CHECK(a.dim() == 2 && b.dim() == 3 && batch_sizes.dim() == 1, "a must be 2-D, b 3-D and batch_sizes 1-D");
  return GmmFunction::apply(a, b, batch_sizes, trans_b);
}

at::Tensor device_status(int64_t device_index) {
  return status_word(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device_index)));
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  m.def("gmm", &gmm, "Grouped GEMM into caller-provided c (B200, libb200gmm).", py::arg("a"), py::arg("b"),
        py::arg("c"), py::arg("batch_sizes"), py::arg("trans_a"), py::arg("trans_b"));
  m.def("gmm_autograd", &gmm_autograd, "Grouped GEMM (trans_a=False) as an autograd function.", py::arg("a"),
        py::arg("b"), py::arg("batch_sizes"), py::arg("trans_b"));
  m.def("device_status", &device_status, "Per-device status word tensor (int32[1]).",
        py::arg("device_index"));
}
