// What the files of the native host path share: one side of a problem as tensors, and the launch helpers that turn it
// into the argument structs of the C ABI.
#pragma once

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <initializer_list>
#include <optional>
#include <string>
#include <tuple>
#include <utility>

#include "lik_b200.h"

namespace lik_host {

using at::Tensor;

// One side of a MaxSim problem (the tensors behind a lik_seqs).  Undefined tensors are absent options.
struct Side {
  Tensor data;  // [n_rows, dim], last dimension contiguous
  int64_t n_seq = 0, max_len = 0, seq_stride = 0;
  Tensor cu, lens, mask, scale;  // int32 [n_seq + 1]; int32 [n_seq]; one byte per row; fp32 per row

  int64_t dim() const { return data.size(1); }
  lik_seqs c_struct() const;
};

int dtype_code(at::ScalarType t);  // lik_dtype; raises ValueError for a type without a kernel
at::ScalarType common_dtype(const Tensor& a, const Tensor& b);
void check(int rc, const char* what);
// every tensor's address goes to a kernel on `dev`: raises ValueError for a (defined) one that is somewhere else
void require_device(const at::Device& dev, std::initializer_list<std::pair<const char*, const Tensor*>> tensors);
// differentiable calls have no forward mode: raises NotImplementedError for an input that carries a tangent
void require_no_tangent(std::initializer_list<const Tensor*> tensors);
int32_t* status_ptr(const at::Device& dev);
Tensor status_tensor(int64_t index);

// [N, L, d] -> padded side; masks are taken as they come (any integer type, nonzero = valid)
Side padded_side(const Tensor& x, at::ScalarType dt, const Tensor& mask, const Tensor& lens, const Tensor& scale);
Side packed_side(const Tensor& x, at::ScalarType dt, const Tensor& cu, int64_t max_len);
Tensor byte_mask(const Tensor& mask);

struct Pairing {
  int kind = LIK_PAIR_CROSS;
  int64_t group = 0;
  Tensor pair_q, pair_d;  // int32, LIK_PAIR_LIST
  int64_t n_scores(const Side& q, const Side& d) const {
    return kind == LIK_PAIR_CROSS ? q.n_seq * d.n_seq : (kind == LIK_PAIR_GROUPED ? d.n_seq : pair_q.numel());
  }
};

// scores fp32 [n_scores], argmax int32 [n_scores, stride] (undefined unless asked for)
std::tuple<Tensor, Tensor> forward(const Side& q, const Side& d, const Pairing& p, int normalize, bool save_argmax, int64_t stride, int engine);
// gradients in grad_dtype, [n_rows, dim] each (undefined unless asked for)
std::tuple<Tensor, Tensor> backward(const Side& q, const Side& d, const Pairing& p, const Tensor& grad_scores, const Tensor& argmax, int normalize,
                                    bool deterministic, at::ScalarType grad_dtype, bool need_q, bool need_d);

// a side as the Python modules hand it over: (data, n_seq, max_len, seq_stride, cu, lens, mask, scale)
Side side_of(const pybind11::tuple& t);

void bind_head(pybind11::module_& m);
void bind_search(pybind11::module_& m);

}  // namespace lik_host
