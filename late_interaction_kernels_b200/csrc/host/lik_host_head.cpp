// Native host path of the document head (maxsim_from_hidden): the chained forward, the backward on the winning tokens,
// and the autograd node.
#include "lik_host.h"

#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <mutex>

namespace lik_host {

namespace {

using OptTensor = std::optional<Tensor>;
using torch::autograd::SavedVariable;

bool half_type(at::ScalarType t) { return t == at::kBFloat16 || t == at::kHalf; }

struct Winners {
  Tensor argmax, rows, counts, bitmap, prefix;
};
// the distinct winners of every document as a compact document (lik_hidden_winners)
Winners winners(const Tensor& argmax, int64_t nq, int64_t nd, int64_t lq, int64_t ld, int64_t slots) {
  const auto dev = argmax.device();
  const c10::cuda::CUDAGuard guard(dev);
  const auto opt = at::TensorOptions().device(dev);
  const int64_t words = (ld + 31) / 32;
  Winners w;
  w.argmax = at::empty(argmax.sizes(), opt.dtype(at::kInt));
  w.rows = at::empty({nd * slots}, opt.dtype(at::kLong));
  w.counts = at::empty({nd}, opt.dtype(at::kInt));
  w.bitmap = at::empty({nd, words}, opt.dtype(at::kInt));
  w.prefix = at::empty({nd, words}, opt.dtype(at::kInt));
  check(lik_hidden_winners((const int32_t*)argmax.data_ptr(), (int)nq, (int)nd, (int)lq, (int)ld, (int)slots, (int32_t*)w.argmax.data_ptr(),
                           (int64_t*)w.rows.data_ptr(), (int32_t*)w.counts.data_ptr(), (uint32_t*)w.bitmap.data_ptr(),
                           (int32_t*)w.prefix.data_ptr(), status_ptr(dev), c10::cuda::getCurrentCUDAStream(dev.index()).stream()),
        "lik_hidden_winners");
  return w;
}

// Only winning tokens carry gradient (fused_head.py:332-456 gathers H_d at the winners too): the distinct winners of every
// document, in token order, form a short "compact" document of at most Nq * Lq tokens.  Those rows of H are gathered and
// projected again, the deterministic backward kernels run on the compact documents (with the document-side normalise
// Jacobian), the three GEMMs of the linear layer see the winner rows alone, and one pass writes grad_H: a winner's row or
// zeros.  No host synchronisation; cost follows the winners, apart from that one pass over grad_H.
std::tuple<Tensor, Tensor, Tensor, Tensor> head_backward(const Tensor& g, const Tensor& Q, const Tensor& H, const Tensor& W, const Tensor& b,
                                                         const Tensor& argmax, bool normalize, bool need_q, bool need_h, bool need_w, bool need_b) {
  const int64_t nq = Q.size(0), lq = Q.size(1), d_out = Q.size(2), nd = H.size(0), ld = H.size(1), dm = H.size(2);
  const auto dt = common_dtype(Q, H);
  need_b = need_b && b.defined();
  const bool need_d = need_h || need_w || need_b;
  const int64_t slots = std::max<int64_t>(1, std::min(nq * lq, ld));
  const c10::cuda::CUDAGuard guard(Q.device());
  const Winners w = winners(argmax, nq, nd, lq, ld, slots);
  const Tensor H_rows = H.reshape({nd * ld, dm}).index_select(0, w.rows);
  const Tensor P_rows = at::linear(H_rows.to(dt), W.to(dt), b.defined() ? OptTensor(b.to(dt)) : std::nullopt);
  Pairing p;
  const Side q = padded_side(Q, dt, Tensor(), Tensor(), Tensor());
  const Side d = padded_side(P_rows.view({nd, slots, d_out}), dt, Tensor(), w.counts, Tensor());
  auto [gq, gp] = backward(q, d, p, g, w.argmax.view({nq * nd, lq}), normalize ? LIK_NORM_D : LIK_NORM_NONE, true, at::kFloat, need_q, need_d);
  Tensor gQ, gH, gW, gb;
  if (need_q) gQ = gq.view(Q.sizes()).to(Q.scalar_type());
  if (need_d) {
    // 16-bit models: the linear layer's gradient GEMMs take 16-bit operands with fp32 accumulation, as its forward does
    const auto gt = half_type(dt) ? dt : at::kFloat;
    const Tensor gpl = gp.to(gt);
    if (need_h) {
      const Tensor g_rows = at::mm(gpl, W.to(gt)).to(H.scalar_type());
      gH = at::empty(H.sizes(), H.options());
      const int64_t row_bytes = dm * (int64_t)gH.element_size();
      if (row_bytes % 16 == 0) {
        check(lik_hidden_scatter_rows(g_rows.data_ptr(), row_bytes, (int)nd, (int)ld, (int)slots, (const uint32_t*)w.bitmap.data_ptr(),
                                      (const int32_t*)w.prefix.data_ptr(), gH.data_ptr(), c10::cuda::getCurrentCUDAStream(Q.device().index()).stream()),
              "lik_hidden_scatter_rows");
      } else {
        gH.zero_();
        const Tensor live = (at::arange(slots, w.counts.options()).unsqueeze(0) < w.counts.unsqueeze(1)).reshape({-1});
        gH.view({nd * ld, dm}).index_copy_(0, w.rows.masked_select(live), g_rows.index({live}));
      }
    }
    if (need_w) gW = at::mm(gpl.t(), H_rows.to(gt)).to(W.scalar_type());
    if (need_b) gb = gp.sum(0).to(b.scalar_type());
  }
  return {gQ, gH, gW, gb};
}

// projection chained into the scoring MMA (lik_maxsim_hidden_fwd); nothing when the kernel does not take the problem
std::optional<std::tuple<Tensor, Tensor>> head_forward(const Side& q, const Side& h, const Tensor& w, const Tensor& bias, bool normalize, bool save_argmax) {
  const auto dt = q.data.scalar_type();
  if (!half_type(dt) || h.data.scalar_type() != dt || w.scalar_type() != dt || (bias.defined() && bias.scalar_type() != dt) || w.stride(1) != 1)
    return std::nullopt;
  const auto dev = q.data.device();
  const c10::cuda::CUDAGuard guard(dev);
  const auto opt = at::TensorOptions().device(dev);
  const int64_t ns = q.n_seq * h.n_seq;
  lik_hidden_fwd_args a{};
  a.q = q.c_struct();
  a.h = h.c_struct();
  a.w = w.data_ptr();
  a.w_stride = w.stride(0);
  a.bias = bias.defined() ? bias.data_ptr() : nullptr;
  a.dtype = dtype_code(dt);
  a.d_model = (int32_t)w.size(1);
  a.d_out = (int32_t)w.size(0);
  a.normalize = normalize ? LIK_NORM_D : LIK_NORM_NONE;
  a.argmax_stride = (int32_t)q.max_len;
  a.status = status_ptr(dev);
  if (ns == 0 || !lik_maxsim_hidden_fwd_supported(&a)) return std::nullopt;
  Tensor scores = at::empty({ns}, opt.dtype(at::kFloat)), argmax, ws;
  if (save_argmax) argmax = at::empty({ns, q.max_len}, opt.dtype(at::kInt));
  a.scores = (float*)scores.data_ptr();
  a.argmax = save_argmax ? (int32_t*)argmax.data_ptr() : nullptr;
  const size_t bytes = lik_maxsim_hidden_fwd_workspace(&a);
  if (bytes) {
    ws = at::empty({(int64_t)bytes}, opt.dtype(at::kByte));
    a.workspace = ws.data_ptr();
    a.workspace_bytes = bytes;
  }
  check(lik_maxsim_hidden_fwd(&a, c10::cuda::getCurrentCUDAStream(dev.index()).stream()), "lik_maxsim_hidden_fwd");
  return std::make_tuple(scores, argmax);
}

struct MaxSimFromHiddenBackward : public torch::autograd::Node {
  SavedVariable q, h, w, b, argmax;
  bool normalize = true;

  std::string name() const override { return "MaxSimFromHiddenBackward"; }
  void release_variables() override {
    const std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&q, &h, &w, &b, &argmax}) v->reset_data();
  }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list out(4);
    if (!grads[0].defined()) return out;
    Tensor Q, H, W, B, winners;
    {
      // (before the autograd keys are switched off: unpacking may run the caller's hooks)
      const std::lock_guard<std::mutex> lock(mutex_);
      Q = q.unpack();
      H = h.unpack();
      W = w.unpack();
      B = b.unpack();
      winners = argmax.unpack();
    }
    at::AutoDispatchBelowADInplaceOrView below;
    std::tie(out[0], out[1], out[2], out[3]) = head_backward(grads[0], Q, H, W, B, winners, normalize, task_should_compute_output(0),
                                                             task_should_compute_output(1), task_should_compute_output(2), task_should_compute_output(3));
    return out;
  }
};

// maxsim_from_hidden on the chained kernel, autograd-aware; None when the kernel does not take the problem
OptTensor maxsim_from_hidden(const Tensor& Q_, const Tensor& H_, const Tensor& W_, const OptTensor& b_, const OptTensor& mask, bool normalize) {
  // (strided inputs are copied once, outside the node: the backward reads the same copies)
  const Tensor Q = Q_.contiguous(), H = H_.contiguous(), W = W_.contiguous(), b = b_ ? b_->contiguous() : Tensor(), dm = mask ? *mask : Tensor();
  require_device(Q.device(), {{"H_d", &H}, {"W", &W}, {"b", &b}, {"d_mask", &dm}});
  const bool grad = at::GradMode::is_enabled() && (Q.requires_grad() || H.requires_grad() || W.requires_grad() || (b.defined() && b.requires_grad()));
  const auto dt = common_dtype(Q, H);
  if (!half_type(dt)) return std::nullopt;
  if (grad) require_no_tangent({&Q, &H, &W, &b});
  Tensor scores, argmax;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    auto got = head_forward(padded_side(Q, dt, Tensor(), Tensor(), Tensor()), padded_side(H, dt, dm, Tensor(), Tensor()),
                            W.to(dt).contiguous(), b.defined() ? b.to(dt).contiguous() : b, normalize, grad);
    if (!got) return std::nullopt;
    std::tie(scores, argmax) = *got;
    scores = scores.view({Q.size(0), H.size(0)});
  }
  if (grad) {
    auto node = std::shared_ptr<MaxSimFromHiddenBackward>(new MaxSimFromHiddenBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(Q, H, W, b));
    node->q = SavedVariable(Q, false);
    node->h = SavedVariable(H, false);
    node->w = SavedVariable(W, false);
    node->b = SavedVariable(b, false);
    node->argmax = SavedVariable(argmax, false);
    node->normalize = normalize;
    torch::autograd::set_history(scores, node);
  }
  return scores;
}

std::optional<std::tuple<Tensor, OptTensor>> head_forward_py(const pybind11::tuple& q, const pybind11::tuple& h, const Tensor& w, const OptTensor& bias,
                                                             bool normalize, bool save_argmax) {
  auto got = head_forward(side_of(q), side_of(h), w, bias ? *bias : Tensor(), normalize, save_argmax);
  if (!got) return std::nullopt;
  auto [s, a] = *got;
  return std::make_tuple(s, a.defined() ? OptTensor(a) : std::nullopt);
}

std::vector<OptTensor> head_backward_py(const Tensor& g, const Tensor& Q, const Tensor& H, const Tensor& W, const OptTensor& b, const Tensor& argmax,
                                        bool normalize, bool need_q, bool need_h, bool need_w, bool need_b) {
  auto [a, h, w, c] = head_backward(g, Q, H, W, b ? *b : Tensor(), argmax, normalize, need_q, need_h, need_w, need_b);
  std::vector<OptTensor> out;
  for (const Tensor& t : {a, h, w, c}) out.push_back(t.defined() ? OptTensor(t) : std::nullopt);
  return out;
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> winners_py(const Tensor& argmax, int64_t nq, int64_t nd, int64_t lq, int64_t ld, int64_t slots) {
  const Winners w = winners(argmax, nq, nd, lq, ld, slots);
  return {w.argmax, w.rows, w.counts, w.bitmap, w.prefix};
}

}  // namespace

void bind_head(pybind11::module_& m) {
  m.def("maxsim_from_hidden", torch::wrap_pybind_function_no_gil(&maxsim_from_hidden));
  m.def("hidden_forward", torch::wrap_pybind_function(&head_forward_py));
  m.def("hidden_backward", torch::wrap_pybind_function_no_gil(&head_backward_py));
  m.def("hidden_winners", torch::wrap_pybind_function_no_gil(&winners_py));
}

}  // namespace lik_host
