#include "host.h"

namespace hyc_host {

void check(int rc, const char* what) {
  if (rc == HYC_OK) return;
  std::string msg = std::string(what) + ": " + hyc_strerror(rc);
  if (rc == HYC_ERR_LAUNCH) msg += " [cudaError " + std::to_string(hyc_last_cuda_error()) + "]";
  throw Error(msg);
}

void require_cuda(std::initializer_list<const Tensor*> ts) {
  const Tensor* first = nullptr;
  for (const Tensor* t : ts) {
    if (t == nullptr) continue;
    if (!t->is_cuda()) throw std::runtime_error("this operator runs only on CUDA tensors (sm_100a kernels); there is no CPU path");
    if (first == nullptr) first = t;
    else if (t->device() != first->device())
      throw std::runtime_error("the tensors of one call live on different devices (" + first->device().str() + " and " + t->device().str() + ")");
  }
}

void check_q(int64_t q) { TORCH_CHECK_VALUE(q == 2 || q == 4 || q == 8, "quantize_bit must be 2, 4 or 8"); }

Tensor scale_vec(const Tensor& s, int64_t n) {
  const Tensor v = vec(s);
  TORCH_CHECK_VALUE(v.numel() == n, "per-channel scale with ", v.numel(), " entries for ", n,
                    " channels (per-tensor scales cannot be quantized with)");
  return v;
}

// length of the rows of a tensor that is taken as rows; a caller divides by it
static int64_t row_length(const Tensor& t) {
  const int64_t n = t.size(-1);
  TORCH_CHECK_VALUE(n > 0, "the last dimension is empty (shape ", t.sizes(), ")");
  return n;
}

// [B, M, N] (or [B, heads, M, d], which becomes [B, M, heads*d]) -> bf16 with one row stride
static Tensor rows_view(const Tensor& x_in) {
  Tensor x = x_in;
  if (x.dim() == 4) x = x.transpose(1, 2).reshape({x.size(0), x.size(2), -1});
  TORCH_CHECK_VALUE(x.dim() == 3, "expected a [B, M, N] or [B, heads, M, d] tensor, got shape ", x_in.sizes());
  if (x.scalar_type() != at::kBFloat16) x = x.to(at::kBFloat16);
  const int64_t M = x.size(1), N = x.size(2);
  if (x.stride(2) != 1 || (x.size(0) > 1 && x.stride(0) != M * x.stride(1)) || x.stride(1) < N || x.stride(1) % 8 != 0 ||
      reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0)
    x = x.contiguous();
  return x;
}

// a caller's buffer that a kernel writes by its address
static const Tensor& buffer(const Tensor& t, at::IntArrayRef shape, at::ScalarType type, const Tensor& like, const char* what) {
  TORCH_CHECK_VALUE(t.numel() >= c10::multiply_integers(shape) && t.scalar_type() == type && t.is_contiguous() && t.device() == like.device(), what,
                    ": expected a contiguous ", type, " buffer for ", shape, " on ", like.device(), ", got ", t.scalar_type(), " ", t.sizes(),
                    " on ", t.device());
  return t;
}

static Tensor index_of(const Tensor& channel, const Tensor& like) {
  if (channel.scalar_type() == at::kLong && channel.device() == like.device()) return channel.contiguous();
  return channel.to(like.device(), at::kLong).contiguous();
}

std::tuple<Tensor, OptTensor> quant(const Tensor& x_in, const Tensor& s_in, int64_t q_bit, const OptTensor& z, const OptTensor& channel,
                                    const OptTensor& out_q, const OptTensor& out_xo) {
  require_cuda({&x_in, &s_in});
  check_q(q_bit);
  OnDevice on(x_in);
  const Tensor x = rows_view(x_in);
  const int64_t B = x.size(0), M = x.size(1), N = x.size(2), rows = B * M;
  TORCH_CHECK_VALUE(N % 32 == 0, "the hidden size must be a multiple of 32");
  const Tensor s = scale_vec(s_in, N);
  Tensor zt, idx;
  if (given(z)) zt = z->scalar_type() == at::kChar && z->is_contiguous() ? *z : z->reshape({-1}).to(at::kChar).contiguous();
  int64_t k = 0;
  if (given(channel)) { idx = index_of(*channel, x); k = idx.numel(); }
  Tensor q = given(out_q) ? buffer(*out_q, {B, M, N * q_bit / 8}, at::kByte, x, "codes") : empty({B, M, N * q_bit / 8}, x, at::kByte);
  OptTensor xo = out_xo;
  if (k && given(out_q)) {
    TORCH_CHECK_VALUE(given(xo), "a buffer for the outlier values is needed beside the one for the codes");
    buffer(*xo, {B, M, k}, at::kBFloat16, x, "outlier values");
  }
  if (!given(out_q) && given(channel)) xo = empty({B, M, k}, x);
  if (rows > 0)
    check(hyc_quant_pack(data(x), rows, (int)N, x.stride(1), data(s), (const int8_t*)data(zt), k ? (const int64_t*)data(idx) : nullptr,
                         (int)k, data(q), k ? data(xo) : nullptr, (int)q_bit, on.stream), "hyc_quant_pack");
  return {q, xo};
}

Tensor dequant(const Tensor& q_in, const Tensor& s_in, int64_t q_bit, const OptTensor& z, const OptTensor& channel, const OptTensor& xo_in,
               const OptTensor& out) {
  require_cuda({&q_in, &s_in});
  check_q(q_bit);
  OnDevice on(q_in);
  TORCH_CHECK_VALUE(q_in.dim() == 3, "expected [B, M, bytes] codes, got shape ", q_in.sizes());
  const int64_t B = q_in.size(0), M = q_in.size(1), N = s_in.size(-1);
  const Tensor q = q_in.contiguous(), s = scale_vec(s_in, N);
  Tensor zt, idx, xo;
  if (given(z)) zt = z->scalar_type() == at::kChar && z->is_contiguous() ? *z : z->reshape({-1}).to(at::kChar).contiguous();
  Tensor x = given(out) ? buffer(*out, {B, M, N}, at::kBFloat16, q, "out") : empty({B, M, N}, q);
  if (B * M == 0) return x;
  int64_t k = 0;
  if (given(channel)) {
    idx = index_of(*channel, q);
    k = idx.numel();
    xo = bf16c(*xo_in);
  }
  check(hyc_unpack_dequant(data(q), B * M, (int)N, data(s), (const int8_t*)data(zt), k ? (const int64_t*)data(idx) : nullptr, (int)k,
                           k ? data(xo) : nullptr, data(x), N, (int)q_bit, on.stream), "hyc_unpack_dequant");
  return x;
}

// ---- attention map, per-row top-k
void topk_compress_into(const Tensor& x, int64_t k, int64_t q_bit, const Tensor& val, const Tensor& col, const Tensor& q,
                        const Tensor& s, const Tensor& z) {
  const int64_t S = row_length(x), rows = x.numel() / S;
  require_cuda({&x});
  check_q(q_bit);
  OnDevice on(x);
  const Tensor xb = bf16c(x);
  check(hyc_softmax_topk_compress(data(xb), rows, (int)S, (int)k, k ? data(val) : nullptr, k ? (uint16_t*)data(col) : nullptr, data(q),
                                  data(s), (int8_t*)data(z), (int)q_bit, on.stream), "hyc_softmax_topk_compress");
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> topk_compress(const Tensor& x, int64_t k, int64_t q_bit, const Tensor& row_cols, Keep keep) {
  const int64_t S = row_length(x), rows = x.numel() / S;
  require_cuda({&x});
  check_q(q_bit);
  const auto [q, val, col, s, z] = together(x, {{{rows, S * q_bit / 8}, at::kByte}, {{rows, k}, at::kBFloat16}, {{rows, k}, at::kShort},
                                                {{rows, S / 64}, at::kBFloat16}, {{rows, S / 64}, at::kChar}}, keep);
  if (row_cols.defined()) {
    OnDevice on(x);
    check(hyc_softmax_topk_compress_cols(data(x), rows, (int)S, (const uint16_t*)data(row_cols), (int)k, k ? data(val) : nullptr,
                                         k ? (uint16_t*)data(col) : nullptr, data(q), data(s), (int8_t*)data(z), (int)q_bit, on.stream),
          "hyc_softmax_topk_compress_cols");
  } else {
    topk_compress_into(x, k, q_bit, val, col, q, s, z);
  }
  return {val, col, q, s, z};
}

Tensor topk_restore(const Tensor& val, const Tensor& col, const Tensor& q, const Tensor& s, const Tensor& z,
                    at::IntArrayRef shape, int64_t q_bit, const OptTensor& out, const Tensor& row_cols) {
  OnDevice on(q);
  Tensor x = given(out) ? *out : empty(shape, q);
  const int64_t k = val.size(1);
  if (row_cols.defined()) {
    check(hyc_softmax_topk_restore_cols(k ? data(val) : nullptr, k ? (const uint16_t*)data(col) : nullptr, (int)k, data(q), data(s),
                                        (const int8_t*)data(z), q.size(0), (int)shape.back(), (const uint16_t*)data(row_cols), data(x), (int)q_bit,
                                        on.stream), "hyc_softmax_topk_restore_cols");
    return x;
  }
  check(hyc_softmax_topk_restore(k ? data(val) : nullptr, k ? (const uint16_t*)data(col) : nullptr, (int)k, data(q), data(s),
                                 (const int8_t*)data(z), q.size(0), (int)shape.back(), data(x), (int)q_bit, on.stream), "hyc_softmax_topk_restore");
  return x;
}

Tensor topk_softmax_backward(const Tensor& val, const Tensor& col, const Tensor& q, const Tensor& s, const Tensor& z,
                             at::IntArrayRef shape, int64_t q_bit, const Tensor& grad, const OptTensor& out, double scale) {
  require_cuda({&grad, &q});
  OnDevice on(q);
  const Tensor g = bf16c(grad);
  TORCH_CHECK_VALUE(g.sizes() == shape, "the gradient must have the map's shape ", shape);
  // (a buffer of another layout or type receives a copy)
  const bool direct = !given(out) || (out->numel() == c10::multiply_integers(shape) && out->scalar_type() == at::kBFloat16 && out->is_contiguous() && out->device() == q.device());
  Tensor o = given(out) && direct ? *out : empty(shape, q);
  auto result = [&]() { return direct ? o : out->copy_(o); };
  const int64_t k = val.size(1);
  const int rc = hyc_softmax_topk_restore_bwd(k ? data(val) : nullptr, k ? (const uint16_t*)data(col) : nullptr, (int)k, data(q), data(s),
                                              (const int8_t*)data(z), q.size(0), (int)shape.back(), data(g), data(o), (int)q_bit,
                                              (float)scale, on.stream);
  if (rc == HYC_ERR_UNSUPPORTED) {      // shape outside the fused kernel: restore, then the softmax backward in place
    Tensor a = topk_restore(val, col, q, s, z, shape, q_bit, std::nullopt);
    check(hyc_softmax_bwd(data(a), data(g), data(o), a.numel() / shape.back(), (int)shape.back(), (float)scale, on.stream), "hyc_softmax_bwd");
    return result();
  }
  check(rc, "hyc_softmax_topk_restore_bwd");
  return result();
}

// ---- attention map, threshold prune
// thr_dev: the threshold as a one-element tensor on the device of x (then `thr` is not read), which spares the call its first
// wait for the device: 102 -> 83 us for save and restore of [2,32,696,696]
Tensor prune_sparse(const Tensor& x, double thr, const OptTensor& thr_dev) {
  require_cuda({&x, opt(thr_dev)});
  OnDevice on(x);
  const Tensor xf = bf16c(x);
  const int64_t numel = xf.numel();
  const size_t ws_bytes = hyc_softmax_prune_workspace_bytes(numel);
  Tensor ws = empty({(int64_t)((ws_bytes + 7) / 8)}, x, at::kLong), t;
  if (given(thr_dev)) {
    TORCH_CHECK_VALUE(thr_dev->numel() == 1, "the threshold must have one element");
    t = thr_dev->to(at::kFloat);
    check(hyc_softmax_prune_count_dev(data(xf), numel, (const float*)data(t), data(ws), ws_bytes, on.stream), "hyc_softmax_prune_count_dev");
  } else {
    check(hyc_softmax_prune_count(data(xf), numel, (float)thr, data(ws), ws_bytes, on.stream), "hyc_softmax_prune_count");
  }
  const int64_t nnz = ws.narrow(0, 0, 1).item<int64_t>();
  Tensor idx = empty({1, nnz}, x, at::kLong), val = empty({nnz}, x);
  if (t.defined())
    check(hyc_softmax_prune_fill_dev(data(xf), numel, (const float*)data(t), data(ws), (int64_t*)data(idx), data(val), nnz, on.stream),
          "hyc_softmax_prune_fill_dev");
  else
    check(hyc_softmax_prune_fill(data(xf), numel, (float)thr, data(ws), (int64_t*)data(idx), data(val), nnz, on.stream), "hyc_softmax_prune_fill");
  Tensor sp = at::_sparse_coo_tensor_unsafe(idx, val, {numel}, val.options().layout(at::kSparse));
  return sp._coalesced_(true);      // the fill writes ascending indices
}

Tensor prune_restore(const Tensor& idx_in, const Tensor& val_in, int64_t numel) {
  require_cuda({&idx_in, &val_in});
  OnDevice on(val_in);
  const Tensor idx = idx_in.reshape({-1}).contiguous(), val = bf16c(val_in);
  Tensor out = empty({numel}, val);
  check(hyc_softmax_prune_restore((const int64_t*)data(idx), data(val), idx.numel(), data(out), numel, on.stream), "hyc_softmax_prune_restore");
  return out;
}

std::tuple<Tensor, Tensor, Tensor> prune_tiled(const Tensor& x, double thr, int64_t capacity, const Tensor& row_cols, Keep keep) {
  require_cuda({&x});
  OnDevice on(x);
  const Tensor xf = bf16c(x);
  const int64_t numel = xf.numel();
  const auto [dir, nnz, words] = together(x, {{{(int64_t)(hyc_softmax_prune_tiled_directory_bytes(numel) / 4)}, at::kInt}, {{1}, at::kLong},
                                              {{capacity}, at::kInt}}, keep);
  if (row_cols.defined())
    check(hyc_softmax_prune_tiled_cols(data(xf), numel, (int)x.size(-1), (const uint16_t*)data(row_cols), (float)thr, (uint32_t*)data(words), capacity,
                                       data(dir), (int64_t*)data(nnz), on.stream), "hyc_softmax_prune_tiled_cols");
  else
    check(hyc_softmax_prune_tiled(data(xf), numel, (float)thr, (uint32_t*)data(words), capacity, data(dir), (int64_t*)data(nnz), on.stream),
          "hyc_softmax_prune_tiled");
  return {words, dir, nnz};
}

Tensor prune_tiled_restore(const Tensor& words, const Tensor& directory, at::IntArrayRef shape, const OptTensor& out, const Tensor& row_cols) {
  OnDevice on(words);
  Tensor x = given(out) ? *out : empty(shape, words);
  if (row_cols.defined()) {
    check(hyc_softmax_prune_tiled_restore_cols((const uint32_t*)data(words), words.numel(), data(directory), (int)shape.back(),
                                               (const uint16_t*)data(row_cols), data(x), x.numel(), on.stream), "hyc_softmax_prune_tiled_restore_cols");
    return x;
  }
  check(hyc_softmax_prune_tiled_restore((const uint32_t*)data(words), words.numel(), data(directory), data(x), x.numel(), on.stream),
        "hyc_softmax_prune_tiled_restore");
  return x;
}

// ---- fused LoRA-SiLU-Hadamard
// [R, N] LoRA-B operand -> the [N, R] row-major matrix the kernels read; ``lora_B.weight.T`` is a view of exactly that storage
// (only its memory is read)
static Tensor b_transposed(const Tensor& b) {
  TORCH_CHECK_VALUE(b.dim() == 2, "LoRA B must be [R, N]");
  if (b.scalar_type() == at::kBFloat16 && b.stride(0) == 1 && b.stride(1) == b.size(0)) return b;
  return b.t().to(at::kBFloat16).contiguous();
}

static void check_fused(int64_t q_bit, int64_t n, int64_t r, std::initializer_list<const Tensor*> ts) {
  require_cuda(ts);
  check_q(q_bit);
  TORCH_CHECK_VALUE(n % 32 == 0, "N must be a multiple of 32");
  TORCH_CHECK_VALUE(r == 16, "LoRA rank must be 16");
}

std::tuple<Tensor, Tensor, Tensor> silu_forward(const Tensor& xa1, const Tensor& b1, const Tensor& x1, const Tensor& s1,
                                                const Tensor& xa2, const Tensor& b2, const Tensor& x2, const Tensor& s2, int64_t q_bit) {
  TORCH_CHECK_VALUE(x1.dim() == 3, "expected [B, M, N] main branches, got shape ", x1.sizes());
  const int64_t B = x1.size(0), M = x1.size(1), N = x1.size(2), R = b1.size(0);
  check_fused(q_bit, N, R, {&xa1, &b1, &x1, &s1, &xa2, &b2, &x2, &s2});
  OnDevice on(x1);
  const Tensor x1c = bf16c(x1), x2c = bf16c(x2), a1 = bf16c(xa1), a2 = bf16c(xa2), bt1 = b_transposed(b1), bt2 = b_transposed(b2),
               sc1 = scale_vec(s1, N), sc2 = scale_vec(s2, N);
  Tensor q1 = empty({B, M, N * q_bit / 8}, x1, at::kByte), q2 = empty({B, M, N * q_bit / 8}, x1, at::kByte), o = empty({B, M, N}, x1);
  check(hyc_fused_lora_silu_hadamard_fwd(data(a1), data(bt1), data(x1c), data(sc1), data(a2), data(bt2), data(x2c), data(sc2), data(q1),
                                         data(q2), data(o), B * M, (int)N, (int)R, (int)q_bit, on.stream), "hyc_fused_lora_silu_hadamard_fwd");
  return {q1, q2, o};
}

std::tuple<Tensor, Tensor, Tensor> silu_backward(const Tensor& xa1, const Tensor& b1, const Tensor& q1, const Tensor& s1,
                                                 const Tensor& xa2, const Tensor& b2, const Tensor& q2, const Tensor& s2,
                                                 const Tensor& grad_o, int64_t q_bit) {
  TORCH_CHECK_VALUE(grad_o.dim() == 3, "expected a [B, M, N] gradient, got shape ", grad_o.sizes());
  const int64_t B = grad_o.size(0), M = grad_o.size(1), N = grad_o.size(2), R = b1.size(0);
  check_fused(q_bit, N, R, {&xa1, &b1, &q1, &s1, &xa2, &b2, &q2, &s2, &grad_o});
  OnDevice on(grad_o);
  const Tensor g = bf16c(grad_o), a1 = bf16c(xa1), a2 = bf16c(xa2), bt1 = b_transposed(b1), bt2 = b_transposed(b2),
               sc1 = scale_vec(s1, N), sc2 = scale_vec(s2, N), q1c = q1.contiguous(), q2c = q2.contiguous();
  Tensor o = empty({B, M, N}, g), gg = empty({B, M, N}, g), gu = empty({B, M, N}, g);
  check(hyc_fused_lora_silu_hadamard_bwd(data(a1), data(bt1), data(q1c), data(sc1), data(a2), data(bt2), data(q2c), data(sc2), data(g),
                                         data(o), data(gg), data(gu), B * M, (int)N, (int)R, (int)q_bit, on.stream),
        "hyc_fused_lora_silu_hadamard_bwd");
  return {o, gg, gu};
}

Tensor dequant_lora_add(const Tensor& q, const Tensor& s, const Tensor& xa, const Tensor& b, int64_t q_bit) {
  require_cuda({&q, &s, &xa, &b});
  check_q(q_bit);
  OnDevice on(q);
  const int64_t B = q.size(0), M = q.size(1), N = s.size(-1);
  const Tensor sc = scale_vec(s, N), xac = bf16c(xa), bt = b_transposed(b), qc = q.contiguous();
  Tensor y = empty({B, M, N}, q);
  if (B * M)
    check(hyc_dequant_lora_add(data(qc), data(sc), data(xac), data(bt), data(y), B * M, (int)N, (int)xac.size(-1), (int)q_bit, on.stream),
          "hyc_dequant_lora_add");
  return y;
}

// ---- norms, softmax, rotary embedding
std::tuple<Tensor, Tensor, Tensor, Tensor, OptTensor> rmsnorm_save(const Tensor& x, const Tensor& w_in, double eps, int64_t q_bit,
                                                                   const Tensor& sx_in, const OptTensor& idx_in, const OptTensor& sy_in, Keep keep) {
  const int64_t N = row_length(x), rows = x.numel() / N;
  require_cuda({&x, &w_in, &sx_in});
  check_q(q_bit);
  OnDevice on(x);
  const Tensor xc = bf16c(x), w = bf16c(w_in);
  const Tensor sx = scale_vec(sx_in, N);
  Tensor idx, sy;
  int64_t k = 0;
  if (given(idx_in)) { idx = index_of(*idx_in, x); k = idx.numel(); }
  if (given(sy_in)) sy = scale_vec(*sy_in, N);
  TORCH_CHECK_VALUE(w.numel() == N, "norm weight with ", w.numel(), " entries for ", N, " channels");
  at::DimVector qs(xc.sizes()), os = qs, none = {0};
  qs.back() = N * q_bit / 8;
  os.back() = k;
  const Tensor y = empty(xc.sizes(), x);
  const auto [rstd, qx, xo, codes_y] = together(x, {{{rows}, at::kFloat}, {qs, at::kByte}, {os, at::kBFloat16}, {sy.defined() ? qs : none, at::kByte}},
                                                    keep);
  OptTensor qy;
  if (sy.defined()) qy = codes_y;
  if (rows)
    check(hyc_rmsnorm_fwd_save(data(xc), data(w), (float)eps, rows, (int)N, data(sx), k ? (const int64_t*)data(idx) : nullptr, (int)k,
                               data(sy), data(y), (float*)data(rstd), data(qx), k ? data(xo) : nullptr, data(qy), (int)q_bit, on.stream),
          "hyc_rmsnorm_fwd_save");
  return {y, rstd, xo, qx, qy};
}

Tensor rmsnorm_backward_packed(const Tensor& dy, const Tensor& qx, const Tensor& sx_in, const OptTensor& xo_in, const OptTensor& idx_in,
                               const Tensor& w_in, const Tensor& rstd, int64_t q_bit, const OptTensor& res_in) {
  const int64_t N = row_length(dy), rows = dy.numel() / N;
  require_cuda({&dy, &qx, &sx_in, &w_in, &rstd});
  OnDevice on(dy);
  const Tensor dyc = bf16c(dy), sx = scale_vec(sx_in, N), w = bf16c(w_in), q = qx.contiguous(), rs = rstd.contiguous();
  TORCH_CHECK_VALUE(w.numel() == N, "norm weight with ", w.numel(), " entries for ", N, " channels");
  Tensor idx, xo, res;
  int64_t k = 0;
  if (given(idx_in)) { idx = index_of(*idx_in, dy); k = idx.numel(); }
  if (k) xo = bf16c(*xo_in);
  if (given(res_in)) res = bf16c(*res_in);
  Tensor dx = empty(dyc.sizes(), dyc);
  if (rows)
    check(hyc_rmsnorm_bwd_packed(data(dyc), data(q), data(sx), k ? (const int64_t*)data(idx) : nullptr, (int)k, data(xo), data(w),
                                 (const float*)data(rs), data(res), data(dx), rows, (int)N, (int)q_bit, on.stream), "hyc_rmsnorm_bwd_packed");
  return dx;
}

Tensor softmax_backward(const Tensor& y, const Tensor& g, double scale) {
  const int64_t S = row_length(y);
  require_cuda({&y, &g});
  OnDevice on(y);
  const Tensor yc = bf16c(y), gc = bf16c(g);
  Tensor o = at::empty_like(yc);
  check(hyc_softmax_bwd(data(yc), data(gc), data(o), yc.numel() / S, (int)S, (float)scale, on.stream), "hyc_softmax_bwd");
  return o;
}

Tensor softmax_forward(const Tensor& scores, double scale, const OptTensor& mask, bool inplace) {
  require_cuda({&scores, opt(mask)});
  TORCH_CHECK_VALUE(scores.dim() == 4, "scores must be [batch, heads, n, S]");
  TORCH_CHECK_VALUE(!inplace || (scores.scalar_type() == at::kBFloat16 && scores.is_contiguous()), "inplace needs contiguous bf16 scores");
  OnDevice on(scores);
  const Tensor sc = bf16c(scores);
  const int64_t b = sc.size(0), h = sc.size(1), n = sc.size(2), S = sc.size(3);
  Tensor out = inplace ? sc : at::empty_like(sc), mk;
  int64_t mb = 0, mh = 0, mr = 0;
  if (given(mask)) {
    mk = mask->to(at::kBFloat16);
    TORCH_CHECK_VALUE(mk.dim() == 4 && mk.size(3) == S && mk.size(2) == n && (mk.size(0) == 1 || mk.size(0) == b) &&
                      (mk.size(1) == 1 || mk.size(1) == h), "attention_mask must be [b or 1, h or 1, n, S]");
    auto strides = [&]() { mb = mk.size(0) == 1 ? 0 : mk.stride(0); mh = mk.size(1) == 1 ? 0 : mk.stride(1); mr = mk.stride(2); };
    if (mk.stride(3) != 1) mk = mk.contiguous();
    strides();
    if (((mb | mh | mr) & 7) || (reinterpret_cast<uintptr_t>(mk.data_ptr()) & 15)) { mk = mk.contiguous(); strides(); }
  }
  check(hyc_softmax_fwd_scale_mask(data(sc), (float)scale, data(mk), mb, mh, mr, (int)h, (int)n, data(out), b * h * n, (int)S, on.stream),
        "hyc_softmax_fwd_scale_mask");
  return out;
}

Tensor rope(const Tensor& x, const Tensor& cos_in, const Tensor& sin_in, bool backward, bool inplace) {
  require_cuda({&x, &cos_in, &sin_in});
  TORCH_CHECK_VALUE(x.dim() == 4, "expected a [batch, seq_len, n_heads, head_dim] tensor");
  OnDevice on(x);
  const int64_t batch = x.size(0), seq = x.size(1), heads = x.size(2), d = x.size(3);
  const auto [cos, sin] = rope_tables(cos_in, sin_in, seq, d);
  const Tensor xc = bf16c(x);
  Tensor out = inplace || xc.data_ptr() != x.data_ptr() ? xc : at::empty_like(xc);
  check(hyc_rope(data(xc), heads * d, data(out), heads * d, data(cos), data(sin), cos.stride(0), cos.scalar_type() == at::kFloat ? 1 : 0,
                 batch * seq, (int)seq, (int)heads, (int)d, backward ? 1 : 0, on.stream), "hyc_rope");
  return out.view({batch, seq, heads, d});
}

Tensor dequant_nf4(const Tensor& packed, const Tensor& code, const Tensor& absmax, const OptTensor& code2, const OptTensor& absmax2,
                   int64_t blocksize2, double offset, int64_t blocksize, at::IntArrayRef shape) {
  require_cuda({&packed, &code, &absmax, opt(code2), opt(absmax2)});
  OnDevice on(packed);
  Tensor out = empty(shape, packed);
  const bool nested = given(code2);
  check(hyc_dequant_nf4(data(packed), (const float*)data(code), nested ? nullptr : (const float*)data(absmax),
                        nested ? (const uint8_t*)data(absmax) : nullptr, (const float*)data(code2), (const float*)data(absmax2),
                        (int)blocksize2, (float)offset, out.numel(), (int)blocksize, data(out), on.stream), "hyc_dequant_nf4");
  return out;
}

void bind_ops(pybind11::module_& m) {
  m.def("quant", &quant);
  m.def("dequant", &dequant);
  m.def("topk_compress", [](const Tensor& x, int64_t k, int64_t q_bit) { return topk_compress(x, k, q_bit); });
  m.def("topk_compress_into", &topk_compress_into);
  m.def("topk_restore", [](const Tensor& v, const Tensor& c, const Tensor& q, const Tensor& s, const Tensor& z, std::vector<int64_t> shape,
                           int64_t q_bit, const OptTensor& out) { return topk_restore(v, c, q, s, z, shape, q_bit, out); });
  m.def("topk_softmax_backward", [](const Tensor& v, const Tensor& c, const Tensor& q, const Tensor& s, const Tensor& z,
                                    std::vector<int64_t> shape, int64_t q_bit, const Tensor& g, const OptTensor& out, double scale) {
    return topk_softmax_backward(v, c, q, s, z, shape, q_bit, g, out, scale); });
  m.def("prune_sparse", &prune_sparse, pybind11::arg("x"), pybind11::arg("thr"), pybind11::arg("thr_dev") = pybind11::none());
  m.def("prune_restore", &prune_restore);
  m.def("prune_tiled", [](const Tensor& x, double thr, int64_t capacity) { return prune_tiled(x, thr, capacity); });
  m.def("prune_tiled_restore", [](const Tensor& w, const Tensor& d, std::vector<int64_t> shape, const OptTensor& out) {
    return prune_tiled_restore(w, d, shape, out); });
  m.def("silu_forward", &silu_forward);
  m.def("silu_backward", &silu_backward);
  m.def("dequant_lora_add", &dequant_lora_add);
  m.def("rmsnorm_save", [](const Tensor& x, const Tensor& w, double eps, int64_t q_bit, const Tensor& sx, const OptTensor& idx, const OptTensor& sy) {
    return rmsnorm_save(x, w, eps, q_bit, sx, idx, sy); });
  m.def("rmsnorm_backward_packed", &rmsnorm_backward_packed);
  m.def("softmax_backward", &softmax_backward);
  m.def("softmax_forward", &softmax_forward);
  m.def("rope", &rope);
  m.def("dequant_nf4", [](const Tensor& p, const Tensor& code, const Tensor& absmax, const OptTensor& code2, const OptTensor& absmax2,
                          int64_t bs2, double offset, int64_t bs, std::vector<int64_t> shape) {
    return dequant_nf4(p, code, absmax, code2, absmax2, bs2, offset, bs, shape); });
}

}  // namespace hyc_host
