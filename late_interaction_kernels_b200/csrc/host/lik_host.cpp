// Native host path of the scoring operators: from the caller's tensors to the launches, and the autograd node.
//
// A small training step is bound by what the host does per call, not by its kernels: with this path in Python (argument
// structs through ctypes, a Python autograd function whose backward takes the interpreter lock in the engine's thread) a
// 16 x 16 step took 222 us of which the kernels ran 44.  Here a call is one crossing from Python into C++.
#include "lik_host.h"

#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <mutex>

namespace lik_host {

namespace {
void value_error(const std::string& what) { throw pybind11::value_error(what); }

template <typename T = void>
T* opt_ptr(const Tensor& t) {
  return t.defined() && t.numel() ? (T*)t.data_ptr() : nullptr;
}
}  // namespace

lik_seqs Side::c_struct() const {
  lik_seqs s{};
  const bool rows = data.size(0) > 0;
  s.data = data.numel() ? data.data_ptr() : nullptr;
  s.row_stride = rows ? data.stride(0) : data.size(1);
  s.n_rows = data.size(0);
  s.n_seq = (int32_t)n_seq;
  s.max_len = (int32_t)max_len;
  s.seq_stride = seq_stride;
  s.cu = cu.defined() ? (const int32_t*)cu.data_ptr() : nullptr;
  s.lens = lens.defined() ? (const int32_t*)lens.data_ptr() : nullptr;
  s.mask = mask.defined() ? (const uint8_t*)mask.data_ptr() : nullptr;
  s.scale = scale.defined() ? (const float*)scale.data_ptr() : nullptr;
  s.scale_scalar = 1.0f;
  return s;
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return LIK_F32;
    case at::kHalf: return LIK_F16;
    case at::kBFloat16: return LIK_BF16;
    case at::kFloat8_e4m3fn: return LIK_E4M3;
    default: value_error(std::string("dtype ") + c10::toString(t) + " is not supported (float32, float16, bfloat16, float8_e4m3fn)");
  }
  return -1;
}

// Element type both operands are brought to before the kernel runs: the same type is kept, mixed inputs become bf16 if
// either side is bf16 and fp16 otherwise (_utils.py:137-148).
at::ScalarType common_dtype(const Tensor& a, const Tensor& b) {
  if (a.scalar_type() == b.scalar_type()) return a.scalar_type();
  return a.scalar_type() == at::kBFloat16 || b.scalar_type() == at::kBFloat16 ? at::kBFloat16 : at::kHalf;
}

void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + " failed (status " + std::to_string(rc) + "): " + lik_last_error());
}

void require_device(const at::Device& dev, std::initializer_list<std::pair<const char*, const Tensor*>> tensors) {
  for (const auto& [name, t] : tensors)
    if (t->defined() && t->device() != dev)
      value_error(std::string(name) + " must be on the same device as the queries; got " + t->device().str() + " vs " + dev.str() + ".");
}

void require_no_tangent(std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(), "MaxSim scores have no forward-mode derivative.");
}

// One status word per device for the life of the process (never freed: the CUDA context may be gone before statics are).
Tensor status_tensor(int64_t index) {
  static std::mutex mutex;
  static auto* words = new std::array<Tensor, 64>();
  TORCH_CHECK(index >= 0 && index < 64, "device ordinal ", index, " not supported");
  std::lock_guard<std::mutex> lock(mutex);
  Tensor& t = (*words)[index];
  if (!t.defined()) t = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::Device(at::kCUDA, (c10::DeviceIndex)index)));
  return t;
}
int32_t* status_ptr(const at::Device& dev) {
  static std::array<std::atomic<int32_t*>, 64> cached{};
  const int i = dev.index();
  if (i >= 0 && i < 64)
    if (int32_t* p = cached[i].load(std::memory_order_acquire)) return p;
  int32_t* p = (int32_t*)status_tensor(i).data_ptr();
  cached[i].store(p, std::memory_order_release);
  return p;
}

Tensor byte_mask(const Tensor& mask) {
  if (!mask.defined()) return mask;
  Tensor m = mask.contiguous();
  const auto t = m.scalar_type();
  return t == at::kBool || t == at::kByte || t == at::kChar ? m : m.ne(0);
}

Side padded_side(const Tensor& x, at::ScalarType dt, const Tensor& mask, const Tensor& lens, const Tensor& scale) {
  Side s;
  Tensor c = x.scalar_type() == dt ? x : x.to(dt);
  if (!c.is_contiguous()) c = c.contiguous();
  s.n_seq = c.size(0);
  s.max_len = s.seq_stride = c.size(1);
  s.data = c.view({s.n_seq * s.max_len, c.size(2)});
  s.mask = byte_mask(mask);
  if (s.mask.defined() && s.mask.numel() != s.n_seq * s.max_len) value_error("a token mask does not have one entry per token");
  s.lens = lens;
  s.scale = scale;
  return s;
}

Side packed_side(const Tensor& x, at::ScalarType dt, const Tensor& cu, int64_t max_len) {
  Side s;
  s.data = (x.scalar_type() == dt ? x : x.to(dt)).contiguous();
  s.cu = cu;
  s.n_seq = cu.numel() - 1;
  s.max_len = max_len;
  return s;
}

std::tuple<Tensor, Tensor> forward(const Side& q, const Side& d, const Pairing& p, int normalize, bool save_argmax, int64_t stride, int engine) {
  const auto dev = q.data.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t ns = p.n_scores(q, d);
  const auto opt = at::TensorOptions().device(dev);
  Tensor scores = at::empty({ns}, opt.dtype(at::kFloat)), argmax;
  if (save_argmax) argmax = at::empty({ns, stride}, opt.dtype(at::kInt));
  if (ns == 0) return {scores, argmax};
  lik_fwd_args a{};
  a.q = q.c_struct();
  a.d = d.c_struct();
  a.dtype = dtype_code(q.data.scalar_type());
  a.dim = (int32_t)q.dim();
  a.pairing = p.kind;
  a.group = (int32_t)p.group;
  if (p.kind == LIK_PAIR_LIST) {
    a.pair_q = opt_ptr<const int32_t>(p.pair_q);
    a.pair_d = opt_ptr<const int32_t>(p.pair_d);
    a.n_pairs = p.pair_q.numel();
  }
  a.normalize = normalize;
  a.engine = engine;
  a.scores = (float*)scores.data_ptr();
  a.argmax = opt_ptr<int32_t>(argmax);
  a.argmax_stride = (int32_t)stride;
  a.status = status_ptr(dev);
  const size_t bytes = lik_maxsim_fwd_workspace(&a);
  Tensor ws;
  if (bytes) {
    ws = at::empty({(int64_t)bytes}, opt.dtype(at::kByte));
    a.workspace = ws.data_ptr();
    a.workspace_bytes = bytes;
  }
  check(lik_maxsim_fwd(&a, c10::cuda::getCurrentCUDAStream(dev.index()).stream()), "lik_maxsim_fwd");
  return {scores, argmax};
}

std::tuple<Tensor, Tensor> backward(const Side& q, const Side& d, const Pairing& p, const Tensor& grad_scores, const Tensor& argmax, int normalize,
                                    bool deterministic, at::ScalarType grad_dtype, bool need_q, bool need_d) {
  const auto dev = q.data.device();
  const c10::cuda::CUDAGuard guard(dev);
  const auto opt = at::TensorOptions().device(dev).dtype(grad_dtype);
  const int64_t dim = q.dim();
  Tensor gq, gd;
  const int64_t ns = p.n_scores(q, d);
  if (ns == 0 || argmax.numel() == 0) {
    if (need_q) gq = at::zeros({q.data.size(0), dim}, opt);
    if (need_d) gd = at::zeros({d.data.size(0), dim}, opt);
    return {gq, gd};
  }
  if (need_q) gq = at::empty({q.data.size(0), dim}, opt);
  if (need_d) gd = at::empty({d.data.size(0), dim}, opt);
  const Tensor g = grad_scores.contiguous().to(at::kFloat);
  lik_bwd_args a{};
  a.q = q.c_struct();
  a.d = d.c_struct();
  a.dtype = dtype_code(q.data.scalar_type());
  a.dim = (int32_t)dim;
  a.pairing = p.kind;
  a.group = (int32_t)p.group;
  if (p.kind == LIK_PAIR_LIST) {
    a.pair_q = opt_ptr<const int32_t>(p.pair_q);
    a.pair_d = opt_ptr<const int32_t>(p.pair_d);
    a.n_pairs = p.pair_q.numel();
  }
  a.normalize = normalize;
  a.deterministic = deterministic;
  a.grad_scores = (const float*)g.data_ptr();
  a.argmax = (const int32_t*)argmax.data_ptr();
  a.argmax_stride = (int32_t)argmax.size(-1);
  a.grad_dtype = dtype_code(grad_dtype);
  a.grad_q = opt_ptr(gq);
  a.grad_d = opt_ptr(gd);
  a.status = status_ptr(dev);
  const size_t bytes = lik_maxsim_bwd_workspace(&a);
  Tensor ws;
  if (bytes) {
    ws = at::empty({(int64_t)bytes}, opt.dtype(at::kByte));
    a.workspace = ws.data_ptr();
    a.workspace_bytes = bytes;
  }
  check(lik_maxsim_bwd(&a, c10::cuda::getCurrentCUDAStream(dev.index()).stream()), "lik_maxsim_bwd");
  return {gq, gd};
}

// ---------------------------------------------------------------------------------------------
// Autograd: one node for every layout.  Its backward runs in the engine's thread without the interpreter lock.
// ---------------------------------------------------------------------------------------------
namespace {

using torch::autograd::SavedVariable;

// What a differentiable scoring call is made of besides Q and D.
struct Problem {
  Tensor q_mask, d_mask, q_lens, d_lens;        // padded layouts
  Tensor cu_q, cu_d;                            // packed layouts
  Pairing pairing;
  int64_t max_q = 0, max_d = 0;                 // packed layouts
  int normalize = LIK_NORM_NONE;
  bool deterministic = true;
};

// Both sides as the kernels take them.  Padded inputs are [.., L, d]: leading dimensions are one list of sequences.
std::pair<Side, Side> sides(const Tensor& Q, const Tensor& D, const Problem& pr, at::ScalarType dt) {
  if (pr.cu_q.defined()) return {packed_side(Q, dt, pr.cu_q, pr.max_q), packed_side(D, dt, pr.cu_d, pr.max_d)};
  auto flat = [](const Tensor& x) {
    if (x.dim() == 3) return x;
    return x.dim() == 2 ? x.unsqueeze(0) : x.contiguous().view({x.size(0) * x.size(1), x.size(2), x.size(3)});
  };
  return {padded_side(flat(Q), dt, pr.q_mask, pr.q_lens, Tensor()), padded_side(flat(D), dt, pr.d_mask, pr.d_lens, Tensor())};
}

struct MaxSimBackward : public torch::autograd::Node {
  SavedVariable q, d, q_mask, d_mask, q_lens, d_lens, cu_q, cu_d, pair_q, pair_d, argmax;
  Problem scalars;  // its tensors are empty: they live in the saved variables

  std::string name() const override { return "MaxSimBackward"; }
  void release_variables() override {
    const std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&q, &d, &q_mask, &d_mask, &q_lens, &d_lens, &cu_q, &cu_d, &pair_q, &pair_d, &argmax}) v->reset_data();
  }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list out(2);
    if (!grads[0].defined()) return out;
    const bool need_q = task_should_compute_output(0), need_d = task_should_compute_output(1);
    if (!need_q && !need_d) return out;
    Tensor Q, D, winners;
    Problem pr = scalars;
    {
      // Unpacking may run the caller's hooks (activation checkpointing computes the forward again in one), so it comes
      // before the autograd keys are switched off.
      const std::lock_guard<std::mutex> lock(mutex_);
      Q = q.unpack();
      D = d.unpack();
      winners = argmax.unpack();
      pr.q_mask = q_mask.unpack();
      pr.d_mask = d_mask.unpack();
      pr.q_lens = q_lens.unpack();
      pr.d_lens = d_lens.unpack();
      pr.cu_q = cu_q.unpack();
      pr.cu_d = cu_d.unpack();
      pr.pairing.pair_q = pair_q.unpack();
      pr.pairing.pair_d = pair_d.unpack();
    }
    at::AutoDispatchBelowADInplaceOrView below;
    const auto dt = common_dtype(Q, D);
    auto [sq, sd] = sides(Q, D, pr, dt);
    auto [gq, gd] = backward(sq, sd, pr.pairing, grads[0], winners, pr.normalize, pr.deterministic, dt, need_q, need_d);
    if (need_q) out[0] = gq.view(Q.sizes()).to(Q.scalar_type());
    if (need_d) out[1] = gd.view(D.sizes()).to(D.scalar_type());
    return out;
  }
};

// Scores of a problem, reshaped to `shape`, attached to the graph when a gradient is wanted.  What the backward needs is
// kept in the layout the kernels read: strided inputs and masks of wider types are copied once, outside the node, and the
// caller may overwrite what they were copied from.
Tensor scored(const Tensor& Q_, const Tensor& D_, Problem pr, at::IntArrayRef shape) {
  const Tensor Q = Q_.contiguous(), D = D_.contiguous();
  pr.q_mask = byte_mask(pr.q_mask);
  pr.d_mask = byte_mask(pr.d_mask);
  const bool grad = at::GradMode::is_enabled() && (Q.requires_grad() || D.requires_grad());
  if (grad) require_no_tangent({&Q, &D});
  Tensor scores, argmax;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [sq, sd] = sides(Q, D, pr, common_dtype(Q, D));
    // (saved winners in rows of whole 16-byte groups: the backward reads four at a time)
    std::tie(scores, argmax) = forward(sq, sd, pr.pairing, pr.normalize, grad, (sq.max_len + 3) & ~int64_t(3), 0);
    scores = scores.view(shape);
  }
  if (grad) {
    auto node = std::shared_ptr<MaxSimBackward>(new MaxSimBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(Q, D));
    node->q = SavedVariable(Q, false);
    node->d = SavedVariable(D, false);
    node->q_mask = SavedVariable(pr.q_mask, false);
    node->d_mask = SavedVariable(pr.d_mask, false);
    node->q_lens = SavedVariable(pr.q_lens, false);
    node->d_lens = SavedVariable(pr.d_lens, false);
    node->cu_q = SavedVariable(pr.cu_q, false);
    node->cu_d = SavedVariable(pr.cu_d, false);
    node->pair_q = SavedVariable(pr.pairing.pair_q, false);
    node->pair_d = SavedVariable(pr.pairing.pair_d, false);
    node->argmax = SavedVariable(argmax, false);
    Problem& s = node->scalars;
    s.pairing.kind = pr.pairing.kind;
    s.pairing.group = pr.pairing.group;
    s.max_q = pr.max_q;
    s.max_d = pr.max_d;
    s.normalize = pr.normalize;
    s.deterministic = pr.deterministic;
    torch::autograd::set_history(scores, node);
  }
  return scores;
}

using OptTensor = std::optional<Tensor>;
Tensor opt(const OptTensor& t) { return t ? *t : Tensor(); }
bool on(const Tensor& t, const at::Device& dev) { return !t.defined() || t.device() == dev; }

// maxsim / maxsim_pairs / MaxSimScorer on padded inputs.  Returns None when an argument is not what the operator takes;
// the caller then says what is wrong.
std::optional<Tensor> maxsim(const Tensor& Q, const Tensor& D, const OptTensor& q_mask, const OptTensor& d_mask, bool normalize, bool deterministic) {
  const auto dev = Q.device();
  Problem pr;
  pr.q_mask = opt(q_mask);
  pr.d_mask = opt(d_mask);
  const int64_t qd = Q.dim(), dd = D.dim();
  if (!Q.is_cuda() || !on(D, dev) || !on(pr.q_mask, dev) || !on(pr.d_mask, dev)) return std::nullopt;
  if (qd < 2 || qd > 3 || dd < 2 || dd > 4 || (dd == 4 && qd != 3) || Q.size(-1) != D.size(-1)) return std::nullopt;
  const int64_t nq = qd == 3 ? Q.size(0) : 1, lq = Q.size(-2);
  const int64_t nd = dd >= 3 ? D.size(dd - 3) : 1;
  if (dd == 4) {
    if (D.size(0) != nq) return std::nullopt;
    if (pr.q_mask.defined() && pr.q_mask.sizes() != at::IntArrayRef({nq, lq})) return std::nullopt;
    if (pr.d_mask.defined() && pr.d_mask.sizes() != D.sizes().slice(0, 3)) return std::nullopt;
    pr.pairing.kind = LIK_PAIR_GROUPED;
    pr.pairing.group = nd;
    if (nq == 0 || nd == 0) return at::zeros({nq, nd}, at::TensorOptions().device(dev).dtype(at::kFloat));
  }
  pr.normalize = normalize ? LIK_NORM_BOTH : LIK_NORM_NONE;
  pr.deterministic = deterministic;
  c10::SmallVector<int64_t, 2> shape;
  if (qd == 3) shape.push_back(nq);
  if (dd >= 3) shape.push_back(nd);
  return scored(Q, D, pr, shape);
}

// candidate lists with length vectors: queries [B, Lq, d], documents [B, C, Ld, d], int32 lengths
Tensor maxsim_padded(const Tensor& Q, const Tensor& D, const Tensor& q_lens, const Tensor& d_lens) {
  require_device(Q.device(), {{"documents", &D}, {"query_lengths", &q_lens}, {"doc_lengths", &d_lens}});
  Problem pr;
  pr.q_lens = q_lens;
  pr.d_lens = d_lens;
  pr.pairing.kind = LIK_PAIR_GROUPED;
  pr.pairing.group = D.size(1);
  return scored(Q, D, pr, {D.size(0), D.size(1)});
}

// offsets and pair indices as the kernels take them: int32 beside the embeddings
Tensor as_int(const Tensor& t, const at::Device& dev) { return t.to(dev, at::kInt).contiguous(); }

int64_t longest(const Tensor& cu) {  // one device-to-host copy
  return cu.numel() <= 1 ? 0 : (cu.slice(0, 1) - cu.slice(0, 0, -1)).max().item<int64_t>();
}

// packed batches: every query against every document, or a pair list
Tensor maxsim_packed(const Tensor& Q, const Tensor& D, const Tensor& cu_q, const Tensor& cu_d, const OptTensor& pair_q, const OptTensor& pair_d,
                     std::optional<int64_t> max_q, std::optional<int64_t> max_d) {
  const auto dev = Q.device();
  require_device(dev, {{"D_packed", &D}});
  Problem pr;
  pr.cu_q = as_int(cu_q, dev);
  pr.cu_d = as_int(cu_d, dev);
  const bool grad = at::GradMode::is_enabled() && (Q.requires_grad() || D.requires_grad());
  // the longest query sizes the query tiles (and the saved winners); the longest document is only needed by the backward
  const bool none = pair_q && pair_q->numel() == 0;  // nothing to score, nothing to wait for
  pr.max_q = max_q ? *max_q : (none ? 0 : longest(pr.cu_q));
  pr.max_d = max_d ? *max_d : (grad && !none ? longest(pr.cu_d) : 0);
  if (pair_q) {
    pr.pairing.kind = LIK_PAIR_LIST;
    pr.pairing.pair_q = as_int(*pair_q, dev);
    pr.pairing.pair_d = as_int(*pair_d, dev);
    return scored(Q, D, pr, {pr.pairing.pair_q.numel()});
  }
  return scored(Q, D, pr, {pr.cu_q.numel() - 1, pr.cu_d.numel() - 1});
}

// e4m3 inputs: D [.., Ld, d] with one (kd) or no leading candidate dimension folded in; fp32 scales per token or absent
Tensor maxsim_fp8(const Tensor& Q, const Tensor& D, const OptTensor& q_scale, const OptTensor& d_scale, const OptTensor& q_mask, const OptTensor& d_mask,
                  int64_t group) {
  const Tensor qm = opt(q_mask), dm = opt(d_mask), qs = opt(q_scale), ds = opt(d_scale);
  require_device(Q.device(), {{"D", &D}, {"scale_Q", &qs}, {"scale_D", &ds}, {"q_mask", &qm}, {"d_mask", &dm}});
  at::AutoDispatchBelowADInplaceOrView below;
  Pairing p;
  p.kind = group > 0 ? LIK_PAIR_GROUPED : LIK_PAIR_CROSS;
  p.group = group;
  const Side q = padded_side(Q, Q.scalar_type(), qm, Tensor(), qs);
  const Side d = padded_side(D, D.scalar_type(), dm, Tensor(), ds);
  const int64_t cols = group > 0 ? group : d.n_seq;
  return std::get<0>(forward(q, d, p, LIK_NORM_NONE, false, q.max_len, 0)).view({q.n_seq, cols});
}

// ---- the launch helpers themselves, for the Python modules that describe their sides one by one ----
}  // namespace
Side side_of(const pybind11::tuple& t) {
  auto tensor = [&](int i) { return t[i].is_none() ? Tensor() : t[i].cast<Tensor>(); };
  Side s;
  s.data = tensor(0);
  s.n_seq = t[1].cast<int64_t>();
  s.max_len = t[2].cast<int64_t>();
  s.seq_stride = t[3].cast<int64_t>();
  s.cu = tensor(4);
  s.lens = tensor(5);
  s.mask = tensor(6);
  s.scale = tensor(7);
  return s;
}
namespace {
Pairing pairing_of(int kind, int64_t group, const OptTensor& pq, const OptTensor& pd) {
  Pairing p;
  p.kind = kind;
  p.group = group;
  p.pair_q = opt(pq);
  p.pair_d = opt(pd);
  return p;
}
std::tuple<Tensor, OptTensor> forward_py(const pybind11::tuple& q, const pybind11::tuple& d, int kind, int64_t group, const OptTensor& pq,
                                         const OptTensor& pd, int normalize, bool save_argmax, int64_t stride, int engine) {
  const Side sq = side_of(q), sd = side_of(d);
  pybind11::gil_scoped_release nogil;
  auto [s, a] = forward(sq, sd, pairing_of(kind, group, pq, pd), normalize, save_argmax, stride, engine);
  return {s, a.defined() ? OptTensor(a) : std::nullopt};
}
std::tuple<OptTensor, OptTensor> backward_py(const pybind11::tuple& q, const pybind11::tuple& d, const Tensor& g, const Tensor& argmax, int kind,
                                             int64_t group, const OptTensor& pq, const OptTensor& pd, int normalize, bool deterministic,
                                             pybind11::object grad_dtype, bool need_q, bool need_d) {
  const Side sq = side_of(q), sd = side_of(d);
  const auto gdt = grad_dtype.is_none() ? sq.data.scalar_type() : torch::python::detail::py_object_to_dtype(grad_dtype);
  pybind11::gil_scoped_release nogil;
  auto [gq, gd] = backward(sq, sd, pairing_of(kind, group, pq, pd), g, argmax, normalize, deterministic, gdt, need_q, need_d);
  return {gq.defined() ? OptTensor(gq) : std::nullopt, gd.defined() ? OptTensor(gd) : std::nullopt};
}

}  // namespace
}  // namespace lik_host

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using namespace lik_host;
  m.doc() = "Native host path of the MaxSim operators (torch tensors in, launches of liblik_b200.so out).";
  m.attr("abi") = LIK_HOST_ABI;  // looked for in the file when the build decides whether it is up to date
  m.def("maxsim", torch::wrap_pybind_function_no_gil(&maxsim));
  m.def("maxsim_padded", torch::wrap_pybind_function_no_gil(&maxsim_padded));
  m.def("maxsim_packed", torch::wrap_pybind_function_no_gil(&maxsim_packed));
  m.def("maxsim_fp8", torch::wrap_pybind_function_no_gil(&maxsim_fp8));
  m.def("forward", torch::wrap_pybind_function(&forward_py));
  m.def("backward", torch::wrap_pybind_function(&backward_py));
  bind_head(m);
  bind_search(m);
  m.def("status_word", torch::wrap_pybind_function_no_gil(&status_tensor));
}
