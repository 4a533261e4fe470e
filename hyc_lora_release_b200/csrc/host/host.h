// Native host path: the operator wrappers of this package on at::Tensor, so that a call costs its launches and
// little else.  The same work in Python (argument checks, allocations, ctypes marshalling) cost 10-15 us per
// launch, more than most kernels of a short sequence run for.
#pragma once
#include <torch/extension.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <array>
#include <initializer_list>
#include <optional>
#include <stdexcept>
#include <string>
#include <vector>
#include "../../../include/hyc.h"

namespace hyc_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

struct Error : std::runtime_error { using std::runtime_error::runtime_error; };
void check(int rc, const char* what);

// makes the device of `t` current for the scope and hands out torch's current stream there
struct OnDevice {
  c10::cuda::CUDAGuard guard;
  void* stream;
  explicit OnDevice(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.get_device()).stream()) {}
};

void require_cuda(std::initializer_list<const Tensor*> ts);      // null entries are skipped
// the same for what the blocks take as lists: everything that a kernel reads by its address alone (index lists are moved
// to the device by the operators that read them)
struct SameDevice {
  const Tensor& first;
  SameDevice& with(const Tensor& t) { if (t.defined() && t.scalar_type() != at::kLong) require_cuda({&first, &t}); return *this; }
  SameDevice& with(const OptTensor& t) { return t.has_value() ? with(*t) : *this; }
  SameDevice& with(const std::vector<Tensor>& ts) { for (const Tensor& t : ts) with(t); return *this; }
};
void check_q(int64_t q);
inline const Tensor* opt(const OptTensor& t) { return t.has_value() && t->defined() ? &*t : nullptr; }
inline bool given(const OptTensor& t) { return t.has_value() && t->defined(); }
// (what is there already is returned without a trip through the dispatcher, which costs more than half a launch)
inline Tensor bf16c(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? t.contiguous() : t.to(at::kBFloat16).contiguous(); }
// a per-channel vector as the kernels read it: contiguous bf16, of any shape
inline Tensor vec(const Tensor& s) {
  if (s.scalar_type() == at::kBFloat16 && s.is_contiguous()) return s;
  return s.to(at::kBFloat16).reshape({-1}).contiguous();
}
inline Tensor empty(at::IntArrayRef sz, const Tensor& like, at::ScalarType ty = at::kBFloat16) {
  return at::detail::empty_cuda(sz, ty, like.device(), std::nullopt);
}
// Tensors that are kept and dropped together, in one allocation (an allocation and its release cost the host 0.8 us, a tensor more on
// the same storage 0.2; a layer step made seventy).  Each starts on a 256-byte boundary, none overlap.  SHARED only for what no caller
// gets hold of (the temporaries of a call, what the record of a layer step keeps): a tensor on a storage with others keeps them alive, is
// written to a file with them and frees them when its storage is emptied, so whatever is handed out has a storage of its own (which costs
// a small call: top-k save and restore of [1,8,64,64] 12.8 us, 10.5 with one storage; the norm with its saves 7.3, 5.7).
enum class Keep { OWN, SHARED };
struct Want { at::DimVector sizes; at::ScalarType type; };
template <size_t N>
std::array<Tensor, N> together(const Tensor& like, const Want (&wants)[N], Keep keep = Keep::SHARED) {
  if (keep == Keep::OWN) {
    std::array<Tensor, N> out;
    for (size_t i = 0; i < N; ++i) out[i] = empty(wants[i].sizes, like, wants[i].type);
    return out;
  }
  int64_t at[N], bytes = 0;
  for (size_t i = 0; i < N; ++i) {
    at[i] = bytes;
    bytes += (c10::multiply_integers(wants[i].sizes) * (int64_t)c10::elementSize(wants[i].type) + 255) / 256 * 256;
  }
  const Tensor all = empty({bytes}, like, at::kByte);
  std::array<Tensor, N> out;
  for (size_t i = 0; i < N; ++i) {
    out[i] = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(all.storage()), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                      c10::scalarTypeToTypeMeta(wants[i].type));
    c10::TensorImpl* t = out[i].unsafeGetTensorImpl();
    t->set_storage_offset(at[i] / (int64_t)c10::elementSize(wants[i].type));
    t->set_sizes_contiguous(wants[i].sizes);
  }
  return out;
}
inline void* data(const Tensor& t) { return t.defined() && t.numel() ? t.data_ptr() : nullptr; }
inline void* data(const OptTensor& t) { return given(t) ? data(*t) : nullptr; }
Tensor scale_vec(const Tensor& s, int64_t n);

// ---- operators (host_ops.cpp)
std::tuple<Tensor, OptTensor> quant(const Tensor& x, const Tensor& s, int64_t q_bit, const OptTensor& z, const OptTensor& channel,
                                    const OptTensor& out_q, const OptTensor& out_xo);
Tensor dequant(const Tensor& q, const Tensor& s, int64_t q_bit, const OptTensor& z, const OptTensor& channel, const OptTensor& xo,
               const OptTensor& out);
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> topk_compress(const Tensor& x, int64_t k, int64_t q_bit, const Tensor& row_cols = {},
                                                                 Keep keep = Keep::OWN);
void topk_compress_into(const Tensor& x, int64_t k, int64_t q_bit, const Tensor& val, const Tensor& col, const Tensor& q,
                        const Tensor& s, const Tensor& z);
Tensor topk_restore(const Tensor& val, const Tensor& col, const Tensor& q, const Tensor& s, const Tensor& z,
                    at::IntArrayRef shape, int64_t q_bit, const OptTensor& out, const Tensor& row_cols = {});
Tensor topk_softmax_backward(const Tensor& val, const Tensor& col, const Tensor& q, const Tensor& s, const Tensor& z,
                             at::IntArrayRef shape, int64_t q_bit, const Tensor& grad, const OptTensor& out, double scale);
Tensor prune_sparse(const Tensor& x, double thr, const OptTensor& thr_dev);
Tensor prune_restore(const Tensor& idx, const Tensor& val, int64_t numel);
std::tuple<Tensor, Tensor, Tensor> prune_tiled(const Tensor& x, double thr, int64_t capacity, const Tensor& row_cols = {}, Keep keep = Keep::OWN);
Tensor prune_tiled_restore(const Tensor& words, const Tensor& directory, at::IntArrayRef shape, const OptTensor& out, const Tensor& row_cols = {});
std::tuple<Tensor, Tensor, Tensor> silu_forward(const Tensor& xa1, const Tensor& b1, const Tensor& x1, const Tensor& s1,
                                                const Tensor& xa2, const Tensor& b2, const Tensor& x2, const Tensor& s2, int64_t q_bit);
std::tuple<Tensor, Tensor, Tensor> silu_backward(const Tensor& xa1, const Tensor& b1, const Tensor& q1, const Tensor& s1,
                                                 const Tensor& xa2, const Tensor& b2, const Tensor& q2, const Tensor& s2,
                                                 const Tensor& grad_o, int64_t q_bit);
std::tuple<Tensor, Tensor, Tensor, Tensor, OptTensor> rmsnorm_save(const Tensor& x, const Tensor& w, double eps, int64_t q_bit,
                                                                   const Tensor& sx, const OptTensor& idx, const OptTensor& sy, Keep keep = Keep::OWN);
Tensor rmsnorm_backward_packed(const Tensor& dy, const Tensor& qx, const Tensor& sx, const OptTensor& xo, const OptTensor& idx,
                               const Tensor& w, const Tensor& rstd, int64_t q_bit, const OptTensor& res);
Tensor softmax_backward(const Tensor& y, const Tensor& g, double scale);
Tensor softmax_forward(const Tensor& scores, double scale, const OptTensor& mask, bool inplace);
Tensor rope(const Tensor& x, const Tensor& cos, const Tensor& sin, bool backward, bool inplace);
Tensor dequant_lora_add(const Tensor& q, const Tensor& s, const Tensor& xa, const Tensor& b, int64_t q_bit);
Tensor dequant_nf4(const Tensor& packed, const Tensor& code, const Tensor& absmax, const OptTensor& code2, const OptTensor& absmax2,
                   int64_t blocksize2, double offset, int64_t blocksize, at::IntArrayRef shape);

// ---- GEMMs and the two halves of the layer (host_blocks.cpp)
struct RopeTables {                              // [>= seq, >= d / 2], bf16 or fp32, the same row stride
  Tensor cos, sin;
  int f32() const { return cos.scalar_type() == at::kFloat ? 1 : 0; }
};
RopeTables rope_tables(const Tensor& cos, const Tensor& sin, int64_t seq, int64_t d);
Tensor lora_grad_a(const Tensor& q, const Tensor& scale, const Tensor& gm, int64_t r2, int64_t q_bit);
void bind_ops(pybind11::module_& m);
void bind_blocks(pybind11::module_& m);

}  // namespace hyc_host
