// The autograd node of the whole op: moba_b200_op_forward / moba_b200_op_backward between torch
// tensors, without the interpreter. At [1,1000,4,64] a step is nine launches, 85 us of kernels;
// as a Python autograd function its host side took 128 us (62 of them for the function itself: the
// backward runs on another thread, which waits for the interpreter lock).
//
// Saves q, k, v, out and the workspace that holds the index, the global log2-sum-exp and the
// per-slot marker. The gate receives no gradient. The C entry points come in as addresses from
// whoever loaded the library.
//
// Stands in for MoBAAttentionFunction of the reference (src/moba/kernels/attention.py:53-110) where
// the routing is the op's own.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include "../../include/moba_b200.h"

namespace {

decltype(&moba_b200_op_forward) op_forward = nullptr;
decltype(&moba_b200_op_backward) op_backward = nullptr;
decltype(&moba_b200_last_error) last_error = nullptr;

void check(int rc, const char* what) {
  if (rc >= 0) return;
  TORCH_CHECK_VALUE(rc != MOBA_B200_EINVAL && rc != MOBA_B200_EUNSUPPORTED, what, ": ", last_error());
  TORCH_CHECK(false, what, ": ", last_error());
}

// Functions of shapes, dtype and configuration only.
struct Plan : torch::CustomClassHolder {
  moba_b200_problem problem;
  int64_t keep_bytes, forward_bytes, backward_bytes;
};

at::Tensor bytes(const at::Tensor& like, int64_t n) { return at::empty({n}, like.options().dtype(at::kByte)); }

struct Attention : torch::autograd::Function<Attention> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& q_in, const at::Tensor& k_in,
                            const at::Tensor& v_in, const c10::intrusive_ptr<Plan>& plan,
                            const std::optional<at::Tensor>& cu_seqlens) {
    const c10::cuda::CUDAGuard guard(q_in.device());
    const at::Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous();
    at::Tensor out = at::empty_like(q);
    const at::Tensor keep = bytes(q, plan->keep_bytes), scratch = bytes(q, plan->forward_bytes);
    check(op_forward(&plan->problem, q.data_ptr(), k.data_ptr(), v.data_ptr(),
                     cu_seqlens ? cu_seqlens->data_ptr<int32_t>() : nullptr, keep.data_ptr(), scratch.data_ptr(),
                     out.data_ptr(), 1, c10::cuda::getCurrentCUDAStream().stream()),
          "moba_forward");
    ctx->save_for_backward({q, k, v, out, keep, cu_seqlens.value_or(at::Tensor())});
    ctx->saved_data["plan"] = c10::IValue::make_capsule(plan);
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &q = saved[0], &k = saved[1], &v = saved[2], &out = saved[3], &keep = saved[4], &cu_seqlens = saved[5];
    const auto plan = c10::static_intrusive_pointer_cast<Plan>(ctx->saved_data["plan"].toCapsule());
    const c10::cuda::CUDAGuard guard(q.device());
    const at::Tensor dout = grads[0].to(q.scalar_type()).contiguous();
    const at::Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
    const at::Tensor scratch = bytes(q, plan->backward_bytes);
    check(op_backward(&plan->problem, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), dout.data_ptr(),
                      cu_seqlens.defined() ? cu_seqlens.data_ptr<int32_t>() : nullptr, keep.data_ptr(), scratch.data_ptr(),
                      dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), c10::cuda::getCurrentCUDAStream().stream()),
          "moba_backward");
    return {dq, dk, dv, at::Tensor(), at::Tensor()};
  }
};

}  // namespace

PYBIND11_MODULE(_autograd, m) {
  py::class_<Plan, c10::intrusive_ptr<Plan>>(m, "Plan").def(py::init([](uintptr_t problem, int64_t keep, int64_t forward, int64_t backward) {
    auto plan = c10::make_intrusive<Plan>();
    plan->problem = *reinterpret_cast<const moba_b200_problem*>(problem);
    plan->keep_bytes = keep;
    plan->forward_bytes = forward;
    plan->backward_bytes = backward;
    return plan;
  }));
  m.def("bind", [](uintptr_t forward, uintptr_t backward, uintptr_t error) {
    op_forward = reinterpret_cast<decltype(op_forward)>(forward);
    op_backward = reinterpret_cast<decltype(op_backward)>(backward);
    last_error = reinterpret_cast<decltype(last_error)>(error);
  });
  m.def("attention",
        [](const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const c10::intrusive_ptr<Plan>& plan,
           const std::optional<at::Tensor>& cu_seqlens) {
          return Attention::apply(q, k, v, plan, cu_seqlens);
        },
        py::call_guard<py::gil_scoped_release>());
}
