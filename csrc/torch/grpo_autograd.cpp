// The GRPO loss on CUDA tensors as a C++ autograd node: allocations, launches and the node without the interpreter.
//
// What bounds a call is the host: 64 x 384 tokens keep the GPU busy for 11 us (five launches, torch's ones for the
// upstream gradient among them), while the same node written in Python, with ctypes for the launches, took 108 us for
// advantages, loss and gradient. As a node of C++ they take 76 us: 8 for the advantages, 14 for the loss, 46 in
// torch.autograd.grad, which takes 39 for a plain torch.sum.
//
// The launchers live in libka_sm100.so; `bind` gets their addresses from the loaded library, so that both sides use the
// same copy of it.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

using AdvantagesFn = int (*)(const float*, float*, int, int, float, void*);
using LossFn = int (*)(const float*, const float*, const float*, const float*, const void*, int, int, int, float, float, float,
                       int, float*, float*, float*, float*, void*);
using GradFn = int (*)(const float*, const float*, const float*, float*, int, int, void*);
AdvantagesFn g_advantages = nullptr;
LossFn g_loss = nullptr;
GradFn g_grad = nullptr;

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// A kernel reads the memory, so a tensor without any (a transform's wrapper) is refused.
void check_plain(const Tensor& t) {
  TORCH_CHECK(t.has_storage() && t.is_cuda(), "the GRPO operators take tensors that are all on the CPU or all on a CUDA device");
}

Tensor floats(const Tensor& t) {
  check_plain(t);
  return t.to(at::kFloat).contiguous();
}

struct GrpoLoss : public torch::autograd::Function<GrpoLoss> {
  static variable_list forward(AutogradContext* ctx, const Tensor& logp_new, const Tensor& logp_old, const OptTensor& logp_ref,
                               const Tensor& adv, const OptTensor& mask, double eps_low, double eps_high, double beta,
                               bool seq_mean, bool with_stats) {
    ctx->set_materialize_grads(false);
    const c10::cuda::CUDAGuard guard(logp_new.device());
    const Tensor ln = floats(logp_new), lo = floats(logp_old), a = floats(adv);
    Tensor lr, m;
    if (logp_ref) lr = floats(*logp_ref);
    if (mask) {
      // bytes and floats are read as they are, anything else is converted first
      m = *mask;
      check_plain(m);
      if (m.scalar_type() != at::kBool && m.scalar_type() != at::kByte && m.scalar_type() != at::kFloat) m = m.to(at::kByte);
      m = m.contiguous();
    }
    const int n_seq = static_cast<int>(ln.size(0)), seq_len = static_cast<int>(ln.size(1));
    const auto f32 = ln.options();
    const Tensor raw = at::empty_like(ln);
    const Tensor ws = at::empty({4 * static_cast<int64_t>(n_seq) + 3}, f32);     // per sequence, then the statistics
    const Tensor loss = at::empty({}, f32);
    Tensor out;
    if (with_stats) out = at::empty({3}, f32);
    float* w = ws.data_ptr<float>();
    const int rc = g_loss(ln.data_ptr<float>(), lo.data_ptr<float>(), lr.defined() ? lr.data_ptr<float>() : nullptr,
                          a.data_ptr<float>(), m.defined() ? m.data_ptr() : nullptr,
                          m.defined() && m.scalar_type() == at::kFloat, n_seq, seq_len, static_cast<float>(eps_low),
                          static_cast<float>(eps_high), static_cast<float>(beta), seq_mean, raw.data_ptr<float>(), w,
                          loss.data_ptr<float>(), with_stats ? out.data_ptr<float>() : w + 4 * static_cast<int64_t>(n_seq),
                          stream_of(ln));
    TORCH_CHECK(rc == 0, "ka_grpo_loss_fwd failed (", rc, ")");
    ctx->save_for_backward({raw, ws});
    if (!with_stats) return {loss};
    ctx->mark_non_differentiable({out});
    return {loss, out};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list result(10);
    if (!grads[0].defined()) return result;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &raw = saved[0], &ws = saved[1];
    const c10::cuda::CUDAGuard guard(raw.device());
    const Tensor up = floats(grads[0]);
    const Tensor grad = at::empty_like(raw);
    const int64_t n_seq = raw.size(0);
    const int rc = g_grad(raw.data_ptr<float>(), ws.data_ptr<float>() + 3 * n_seq, up.data_ptr<float>(), grad.data_ptr<float>(),
                          static_cast<int>(n_seq), static_cast<int>(raw.size(1)), stream_of(raw));
    TORCH_CHECK(rc == 0, "ka_grpo_loss_bwd failed (", rc, ")");
    result[0] = grad;
    return result;
  }
};

std::vector<Tensor> grpo_loss(const Tensor& logp_new, const Tensor& logp_old, const OptTensor& logp_ref, const Tensor& adv,
                              const OptTensor& mask, double eps_low, double eps_high, double beta, bool seq_mean,
                              bool with_stats) {
  return GrpoLoss::apply(logp_new, logp_old, logp_ref, adv, mask, eps_low, eps_high, beta, seq_mean, with_stats);
}

Tensor group_advantages(const Tensor& rewards, int64_t group, double eps) {
  const at::NoGradGuard no_grad;
  const c10::cuda::CUDAGuard guard(rewards.device());
  const Tensor r = floats(rewards);
  const Tensor adv = at::empty_like(r);
  const int rc = g_advantages(r.data_ptr<float>(), adv.data_ptr<float>(), static_cast<int>(r.numel() / group),
                              static_cast<int>(group), static_cast<float>(eps), stream_of(r));
  TORCH_CHECK(rc == 0, "grpo advantages failed (", rc, ")");
  return adv;
}

void bind(uintptr_t advantages, uintptr_t loss, uintptr_t grad) {
  g_advantages = reinterpret_cast<AdvantagesFn>(advantages);
  g_loss = reinterpret_cast<LossFn>(loss);
  g_grad = reinterpret_cast<GradFn>(grad);
}

}  // namespace

PYBIND11_MODULE(_ka_torch, m) {
  m.def("bind", &bind);
  // the interpreter is free while a launch waits for room in the queue
  m.def("grpo_loss", &grpo_loss, py::call_guard<py::gil_scoped_release>());
  m.def("group_advantages", &group_advantages, py::call_guard<py::gil_scoped_release>());
}
