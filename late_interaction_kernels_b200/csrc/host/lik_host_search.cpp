// Native host path of top-k search over dense documents (maxsim_topk / retrieve).
#include "lik_host.h"

#include <torch/csrc/utils/pybind.h>

namespace lik_host {

namespace {

using OptTensor = std::optional<Tensor>;

// The k best documents of every query in one pass of the fused kernel; nothing when it does not take the problem.
// Q [Nq, Lq, d], D [Nd, Ld, d], masks [Nq, Lq] / [Nd, Ld].
std::optional<std::tuple<Tensor, Tensor>> topk(const Tensor& Q, const Tensor& D, int64_t k, const OptTensor& q_mask, const OptTensor& d_mask,
                                               bool normalize, bool largest) {
  const auto dev = Q.device();
  const Tensor qm = q_mask ? *q_mask : Tensor(), dm = d_mask ? *d_mask : Tensor();
  require_device(dev, {{"D", &D}, {"q_mask", &qm}, {"d_mask", &dm}});
  at::AutoDispatchBelowADInplaceOrView below;
  const c10::cuda::CUDAGuard guard(dev);
  const auto dt = common_dtype(Q, D);
  const Side q = padded_side(Q, dt, qm, Tensor(), Tensor());
  const Side d = padded_side(D, dt, dm, Tensor(), Tensor());
  lik_fwd_args a{};
  a.q = q.c_struct();
  a.d = d.c_struct();
  a.dtype = dtype_code(dt);
  a.dim = (int32_t)q.dim();
  a.pairing = LIK_PAIR_CROSS;
  a.normalize = normalize ? LIK_NORM_BOTH : LIK_NORM_NONE;
  a.argmax_stride = (int32_t)q.max_len;
  a.status = status_ptr(dev);
  lik_topk_spec t{};
  t.k = (int32_t)k;
  t.largest = largest;
  // (whether the kernel takes the problem does not depend on where the results go, but validation wants an address)
  t.out_scores = (float*)a.status;
  t.out_index = (int64_t*)a.status;
  if (!lik_maxsim_fwd_topk_supported(&a, &t)) return std::nullopt;
  const auto opt = at::TensorOptions().device(dev);
  const Tensor scores = at::empty({q.n_seq, k}, opt.dtype(at::kFloat)), index = at::empty({q.n_seq, k}, opt.dtype(at::kLong));
  t.out_scores = (float*)scores.data_ptr();
  t.out_index = (int64_t*)index.data_ptr();
  const Tensor ws = at::empty({std::max<int64_t>(1, (int64_t)lik_maxsim_fwd_topk_workspace(&a, &t))}, opt.dtype(at::kByte));
  a.workspace = ws.data_ptr();
  a.workspace_bytes = (size_t)ws.numel();
  check(lik_maxsim_fwd_topk(&a, &t, c10::cuda::getCurrentCUDAStream(dev.index()).stream()), "lik_maxsim_fwd_topk");
  return std::make_tuple(scores, index);
}

}  // namespace

void bind_search(pybind11::module_& m) { m.def("topk", torch::wrap_pybind_function_no_gil(&topk)); }

}  // namespace lik_host
