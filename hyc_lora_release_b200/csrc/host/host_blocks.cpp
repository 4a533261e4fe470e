// The two halves of the fused decoder layer in steady state (statistics calibrated), as fixed launch sequences.
// What each step is and which rounding points it has is documented in mlp.py and attention.py, which own the
// calibration branch and the weight records.
#include "host.h"
#include <algorithm>
#include <array>
#include <climits>
#include <cmath>

namespace hyc_host {

static int* status_ptr(const Tensor& st) { return (int*)st.data_ptr(); }

// what the kernels read by address and stride alone: a contiguous bf16 matrix of the size that the product needs
static void expect(const Tensor& t, int64_t rows, int64_t cols, const char* what) {
  TORCH_CHECK(t.dim() == 2 && t.size(0) == rows && t.size(1) == cols && t.scalar_type() == at::kBFloat16 && t.is_contiguous(), what,
              ": expected a contiguous bf16 [", rows, ", ", cols, "] matrix, got ", t.scalar_type(), " ", t.sizes(), " with strides ", t.strides());
}
static void expect_factor(const Tensor& b, int64_t rows, const char* what) {      // any strides
  TORCH_CHECK(b.dim() == 2 && b.size(0) == rows && b.size(1) == 16 && b.scalar_type() == at::kBFloat16, what, ": expected a bf16 [", rows,
              ", 16] factor, got ", b.scalar_type(), " ", b.sizes());
}

// a LoRA-B factor as the kernels load it: contiguous and on a 16-byte boundary (one that is a slice of a flat buffer is copied)
static Tensor factor(const Tensor& b) {
  const Tensor c = b.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0 ? c : c.clone();
}

// a frozen projection: a bf16 matrix, or 4-bit codes, which become one for the product that uses it or are read by it as they are
struct FrozenWeight {
  Tensor plain;
  Tensor packed, code, absmax;
  OptTensor code2, absmax2;
  int64_t blocksize2 = 1, blocksize = 64;
  double offset = 0;
  std::vector<int64_t> shape;
  hyc_nf4_weight codes() const {
    const bool nested = given(code2);
    return {data(packed), (const float*)data(code), nested ? nullptr : (const float*)data(absmax), nested ? (const uint8_t*)data(absmax) : nullptr,
            (const float*)data(code2), (const float*)data(absmax2), (int)blocksize, (int)blocksize2, (float)offset};
  }
};
// what a product gets of it
struct Weight {
  Tensor m;
  const FrozenWeight* f = nullptr;          // m undefined: the codes
  Weight(const Tensor& t) : m(t) {}
  explicit Weight(const FrozenWeight* w) : f(w) {}
  int64_t size(int i) const { return f ? f->shape[i] : m.size(i); }
  hyc_nf4_weight codes() const { return f ? f->codes() : hyc_nf4_weight{}; }
};
static void expect(const Weight& w, int64_t rows, int64_t cols, const Tensor& like, const char* what) {
  if (!w.f) return expect(w.m, rows, cols, what);
  TORCH_CHECK(w.size(0) == rows && w.size(1) == cols, what, ": expected a [", rows, ", ", cols, "] weight, got ", w.f->shape);
  require_cuda({&like, &w.f->packed, &w.f->code, &w.f->absmax, opt(w.f->code2), opt(w.f->absmax2)});
}

// sum of a_i op(b_i) (+ residual), one to four K segments
struct Segment { const Tensor* a; Weight b; };
static Tensor gemm(std::initializer_list<Segment> segs, int form, const Tensor* residual, const Tensor& status) {
  const Tensor& a = *segs.begin()->a;
  OnDevice on(a);
  const int64_t M = a.size(0), N = segs.begin()->b.size(form & HYC_GEMM_B_KN ? 1 : 0);
  const void *pa[4], *pb[4];
  hyc_nf4_weight codes[4];
  bool coded = false;
  int k[4], n = 0;
  for (const Segment& s : segs) {
    pa[n] = data(*s.a); pb[n] = data(s.b.m); codes[n] = s.b.codes(); k[n] = (int)s.a->size(1);
    coded = coded || s.b.f != nullptr;
    ++n;
  }
  Tensor d = empty({M, N}, a);
  if (coded)
    check(hyc_gemm_segments_nf4_tcgen05(n, pa, pb, codes, k, (int)M, (int)N, form, residual ? data(*residual) : nullptr, data(d),
                                        status_ptr(status), on.stream), "hyc_gemm_segments_nf4_tcgen05");
  else
    check(hyc_gemm_segments_tcgen05(n, pa, pb, k, (int)M, (int)N, form, residual ? data(*residual) : nullptr, data(d),
                                  status_ptr(status), on.stream), "hyc_gemm_segments_tcgen05");
  return d;
}

// The forward LoRA-A products stay library calls, batched where they share the left operand (stride 0): saved codes
// behind them depend on every bit of their results, and with 2-bit codes one that flips moves a value by a third of its
// range.  The backward products go through the kernel below.
static Tensor lora_a_products(const Tensor& x2, const Tensor& stacked) {
  return at::bmm(x2.unsqueeze(0).expand({stacked.size(0), -1, -1}), stacked);
}

// rank-16 products (one launch for up to three operands)
struct Skinny {
  hyc_skinny_job jobs[3] = {};
  int count = 0;
  // x [T, n]
  Skinny& on(const Tensor& x) {
    hyc_skinny_job& j = jobs[count++];
    j.x = data(x); j.ldx = x.stride(0); j.n = (int)x.size(1);
    return *this;
  }
  // y (columns [col, col + 16) of a row of ld elements) = x w, then `pad` zero columns
  Skinny& rows(const void* w, int64_t ld_w, const Tensor& y, int64_t offset, int64_t ld_y, int pad = 0) {
    hyc_skinny_job& j = jobs[count - 1];
    j.w[j.n_w] = w; j.ld_w = ld_w;
    j.y[j.n_w++] = (char*)y.data_ptr() + offset * 2;
    j.ld_y = ld_y; j.y_pad = pad;
    return *this;
  }
  // z = x^T xa
  Skinny& cols(const void* xa, int64_t ld_xa, void* z, bool transposed = false) {
    hyc_skinny_job& j = jobs[count - 1];
    j.xa = xa; j.ld_xa = ld_xa; j.z = z; j.z_transposed = transposed ? 1 : 0;
    return *this;
  }
  void run(int64_t T, const Tensor& like, const Tensor& status, void* stream) {
    const size_t bytes = hyc_skinny_workspace_bytes(count, jobs, (int)T);
    Tensor ws = empty({(int64_t)(bytes / 4)}, like, at::kFloat);
    check(hyc_skinny_products(count, jobs, (int)T, data(ws), bytes, status_ptr(status), stream), "hyc_skinny_products");
  }
};
static const char* at_row(const Tensor& t, int64_t i) { return (const char*)t.data_ptr() + i * t.stride(0) * t.element_size(); }

// the q, k and v projections with the saves of their main branches in one launch: -> {y, codes} of each
static std::array<std::pair<Tensor, Tensor>, 3> qkv_lora_save(const Tensor& x, const std::vector<Weight>& w, const Tensor& xa3,
                                                              const std::array<const Tensor*, 3>& b, const std::array<const Tensor*, 3>& scale,
                                                              int64_t q_bit, const Tensor& status, Keep keep_codes) {
  OnDevice on(x);
  const int64_t T = x.size(0), K = x.size(1);
  std::array<std::pair<Tensor, Tensor>, 3> out;
  const int64_t n0 = w[0].size(0), n1 = w[1].size(0), n2 = w[2].size(0);
  // (the projections themselves are gone behind the attention kernel, the codes stay for the backward pass)
  const auto y3 = together(x, {{{T, n0}, at::kBFloat16}, {{T, n1}, at::kBFloat16}, {{T, n2}, at::kBFloat16}});
  const auto q3 = together(x, {{{T, n0 * q_bit / 8}, at::kByte}, {{T, n1 * q_bit / 8}, at::kByte}, {{T, n2 * q_bit / 8}, at::kByte}}, keep_codes);
  Tensor keep[6];
  const void *wp[3], *xp[3], *bp[3], *sp[3];
  void *qp[3], *yp[3];
  hyc_nf4_weight codes[3];
  int n[3];
  for (int i = 0; i < 3; ++i) {
    n[i] = (int)w[i].size(0);
    codes[i] = w[i].codes();
    out[i] = {y3[i], q3[i]};
    keep[2 * i] = vec(*scale[i]);
    keep[2 * i + 1] = factor(*b[i]);
    wp[i] = data(w[i].m); xp[i] = (const char*)xa3.data_ptr() + i * T * 16 * 2; bp[i] = data(keep[2 * i + 1]); sp[i] = data(keep[2 * i]);
    yp[i] = data(out[i].first); qp[i] = data(out[i].second);
  }
  if (w[0].f || w[1].f || w[2].f)
    check(hyc_linears_lora_save_fwd_nf4_tcgen05(data(x), (int)T, (int)K, 3, wp, codes, n, xp, bp, sp, qp, yp, (int)q_bit, status_ptr(status), on.stream),
          "hyc_linears_lora_save_fwd_nf4_tcgen05");
  else
    check(hyc_linears_lora_save_fwd_tcgen05(data(x), (int)T, (int)K, 3, wp, n, xp, bp, sp, qp, yp, (int)q_bit, status_ptr(status), on.stream),
        "hyc_linears_lora_save_fwd_tcgen05");
  return out;
}

Tensor lora_grad_a(const Tensor& q, const Tensor& scale, const Tensor& gm, int64_t r2, int64_t q_bit) {
  require_cuda({&q, &scale, &gm});
  OnDevice on(q);
  const int64_t T = q.size(0), H = scale.numel();
  Tensor out = empty({r2, H}, q);
  const size_t nbytes = hyc_lora_grad_a_workspace_bytes((int)T, (int)H, (int)r2);
  Tensor ws;
  if (nbytes > 0) ws = empty({(int64_t)(nbytes / 4)}, q, at::kFloat);
  check(hyc_lora_grad_a_dequant(data(q), data(scale), data(gm), gm.stride(0), (int)r2, (int)T, (int)H, (int)q_bit, data(out), data(ws),
                                nbytes, on.stream), "hyc_lora_grad_a_dequant");
  return out;
}

// the matrices of up to four weights, one launch for all that are codes.  Called directly before the product that reads them:
// what fits of the matrices is then still in L2
static std::vector<Tensor> matrices(std::initializer_list<const FrozenWeight*> ws) {
  std::vector<Tensor> out;
  hyc_nf4_job jobs[4] = {};
  int n = 0;
  for (const FrozenWeight* f : ws) {
    if (f->plain.defined()) { out.push_back(f->plain); continue; }
    require_cuda({&f->packed, &f->code, &f->absmax, opt(f->code2), opt(f->absmax2)});
    out.push_back(empty(f->shape, f->packed));
    const bool nested = given(f->code2);
    jobs[n++] = {data(f->packed), (const float*)data(f->code), nested ? nullptr : (const float*)data(f->absmax),
                 nested ? (const uint8_t*)data(f->absmax) : nullptr, (const float*)data(f->code2), (const float*)data(f->absmax2),
                 data(out.back()), out.back().numel(), (int)f->blocksize, (int)f->blocksize2, (float)f->offset};
  }
  if (n) {
    OnDevice on(out[0]);
    check(hyc_dequant_nf4_many(n, jobs, on.stream), "hyc_dequant_nf4_many");
  }
  return out;
}

// The same for a product of T rows: the codes as they are where it takes them (gate and up: where it takes both) and is faster for it
// (the rule and its figures: tc_split.cu).  recorded: the product becomes part of a capture.
enum class Use { QKV, O, GATE_UP, DOWN, GRAD_DOWN, GRAD_X };
static std::vector<Weight> weights(std::initializer_list<const FrozenWeight*> ws, int64_t T, Use use, bool recorded) {
  const bool backward = use == Use::GRAD_DOWN || use == Use::GRAD_X;
  bool coded = false, refused = T > INT_MAX;
  int64_t sum0 = 0, rows = 0, cols = 0;
  for (const FrozenWeight* f : ws) {
    const at::IntArrayRef shape = f->plain.defined() ? f->plain.sizes() : at::IntArrayRef(f->shape);
    if (shape.size() != 2) { refused = true; break; }
    sum0 += rows = shape[0];
    cols = shape[1];
    if (f->plain.defined()) { refused = refused || use == Use::GATE_UP; continue; }
    const hyc_nf4_weight c = f->codes();
    coded = true;
    refused = refused || !hyc_nf4_product_supported(&c, (int)T, (int)cols);
    if (refused) break;
  }
  if (coded && !refused) {
    // outputs side by side and depth (64: the LoRA products that ride along)
    const int kind = use == Use::GATE_UP ? HYC_NF4_GATE_UP : (use == Use::GRAD_DOWN ? HYC_NF4_GRAD_DOWN : (use == Use::QKV || use == Use::O ? HYC_GEMM_FIXED_ORDER : 0));
    const int64_t n = backward ? cols : (use == Use::GATE_UP ? rows : sum0), k = (backward ? sum0 : cols) + (use == Use::QKV || use == Use::GATE_UP ? 0 : 64);
    refused = !hyc_nf4_product_pays(kind, (int)T, (int)std::min<int64_t>(n, INT_MAX), (int)std::min<int64_t>(k, INT_MAX), recorded);
  }
  std::vector<Weight> out;
  if (!coded || refused) {
    for (const Tensor& m : matrices(ws)) out.emplace_back(m);
  } else {
    for (const FrozenWeight* f : ws) f->plain.defined() ? out.emplace_back(f->plain) : out.emplace_back(f);
  }
  return out;
}

// ------------------------------------------------------------------ MLP half
struct MlpForward { Tensor x_out, rstd, xm_o, xm_q, xn_q, q1, q2, gs, us, gu_xa, down_xa64; };

static MlpForward mlp_forward(const Tensor& x_medium, const std::vector<Tensor>& w, const std::vector<Tensor>& stats,
                                       const OptTensor& bias_d, int64_t q, double eps, const Tensor& status, const std::vector<Weight>& gate_up,
                                       const Weight* wd_now, const FrozenWeight* wd_later, bool recorded, Keep keep) {
  const Weight &wg = gate_up[0], &wu = gate_up[1];
  const Tensor &norm_w = w[0], &agu_t = w[6], &ad_cols = w[7], &bd_cols = w[8];
  const Tensor &xm_idx = stats[0], &xm_scale = stats[1], &xn_scale = stats[2];
  const int64_t B = x_medium.size(0), M = x_medium.size(1), H = x_medium.size(2), T = B * M, I = wg.size(0);
  expect(wg, I, H, x_medium, "gate projection");
  expect(wu, I, H, x_medium, "up projection");
  expect_factor(w[4], I, "gate lora_B");
  expect_factor(w[5], I, "up lora_B");
  expect(bd_cols, H, 64, "down lora_B");
  const Tensor gs = scale_vec(stats[3], I), us = scale_vec(stats[4], I);
  SameDevice{x_medium}.with(w).with(wg.m).with(wu.m).with(stats).with(bias_d).with(status);
  OnDevice on(x_medium);
  const Tensor bg = factor(w[4]), bu = factor(w[5]);
  auto [x_norm, rstd, xm_o, xm_q, xn_q] = rmsnorm_save(x_medium, norm_w, eps, q, xm_scale, xm_idx, xn_scale, keep);
  const Tensor xn2 = x_norm.view({T, H});
  const Tensor gu_xa = lora_a_products(xn2, agu_t);
  const char* xa = (const char*)gu_xa.data_ptr();
  const auto [q1, q2] = together(x_norm, {{{B, M, I * q / 8}, at::kByte}, {{B, M, I * q / 8}, at::kByte}}, keep);
  const Tensor had = empty({T, I}, x_norm);
  if (wg.f) {
    const hyc_nf4_weight codes[2] = {wg.codes(), wu.codes()};
    check(hyc_mlp_gateup_fwd_nf4_tcgen05(data(xn2), codes, (int)T, (int)H, (int)I, xa, data(bg), 16, 1, xa + T * 16 * 2, data(bu), 16, 1, data(gs),
                                         data(us), data(q1), data(q2), data(had), nullptr, nullptr, (int)q, status_ptr(status), on.stream),
          "hyc_mlp_gateup_fwd_nf4_tcgen05");
  } else {
    check(hyc_mlp_gateup_fwd_tcgen05(data(xn2), data(wg.m), data(wu.m), (int)T, (int)H, (int)I, xa, data(bg), 16, 1, xa + T * 16 * 2, data(bu), 16, 1,
                                     data(gs), data(us), data(q1), data(q2), data(had), nullptr, nullptr, (int)q, status_ptr(status), on.stream),
          "hyc_mlp_gateup_fwd_tcgen05");
  }
  const Tensor down_xa64 = at::mm(had, ad_cols);
  const Tensor res = bf16c(x_medium);
  const Weight wd = wd_later ? weights({wd_later}, T, Use::DOWN, recorded)[0] : *wd_now;
  if (!wd.f) require_cuda({&x_medium, &wd.m});
  expect(wd, H, I, x_medium, "down projection");
  Tensor x_out = gemm({{&had, wd}, {&down_xa64, bd_cols}}, 0, &res, status);
  if (given(bias_d)) x_out.add_(bias_d->to(at::kBFloat16));
  return {x_out.view({B, M, H}), rstd, xm_o, xm_q, *xn_q, q1, q2, gs, us, gu_xa, down_xa64};
}

// up to and including the six LoRA gradients: -> had, ggu, gm64, grad_bd, grad_ad, ga, grad_bgu
static std::vector<Tensor> mlp_backward_lora(const Tensor& g, const Weight& wd, const std::vector<Tensor>& w, const std::vector<Tensor>& saved, int64_t q,
                                             const Tensor& status) {
  const Tensor& ad_rows = w[4];
  const Tensor &gate_q = saved[0], &gate_s = saved[1], &up_q = saved[2], &up_s = saved[3], &gu_xa = saved[4], &down_xa = saved[5],
               &xn_q = saved[6], &xn_scale = saved[7];
  const int64_t T = g.size(0), H = g.size(1), I = wd.size(1);
  expect(wd, H, I, g, "down projection");
  expect_factor(w[1], I, "gate lora_B");
  expect_factor(w[2], I, "up lora_B");
  expect_factor(w[3], H, "down lora_B");
  expect(ad_rows, 64, I, "down lora_A");
  SameDevice{g}.with(wd.m).with(w).with(saved).with(status);
  OnDevice on(g);
  const Tensor bg = factor(w[1]), bu = factor(w[2]), bd = factor(w[3]);
  const auto [gdm64, gm64] = together(g, {{{T, 64}, at::kBFloat16}, {{T, 64}, at::kBFloat16}});
  Tensor grad_bd = empty({H, 16}, g), grad_ad = empty({16, I}, g), grad_bgu = empty({2, I, 16}, g);
  Skinny().on(g).rows(data(bd), 16, gdm64, 0, 64, 48).cols(data(down_xa), down_xa.stride(0), data(grad_bd)).run(T, g, status, on.stream);
  Tensor had = empty({T, I}, g), ggu = empty({2, T, I}, g);
  char* gp = (char*)ggu.data_ptr();
  const char* xa = (const char*)gu_xa.data_ptr();
  if (wd.f) {
    const hyc_nf4_weight codes = wd.codes();
    check(hyc_mlp_graddown_bwd_nf4_tcgen05(data(g), &codes, (int)T, (int)H, (int)I, data(gdm64), data(ad_rows), 64, xa, data(bg), 16, 1,
                                           xa + T * 16 * 2, data(bu), 16, 1, data(gate_q), data(gate_s), data(up_q), data(up_s), nullptr, nullptr, 0,
                                           data(had), gp, gp + T * I * 2, (int)q, status_ptr(status), on.stream), "hyc_mlp_graddown_bwd_nf4_tcgen05");
  } else {
    check(hyc_mlp_graddown_bwd_tcgen05(data(g), data(wd.m), (int)T, (int)H, (int)I, data(gdm64), data(ad_rows), 64, xa, data(bg), 16, 1,
                                       xa + T * 16 * 2, data(bu), 16, 1, data(gate_q), data(gate_s), data(up_q), data(up_s), nullptr, nullptr, 0,
                                       data(had), gp, gp + T * I * 2, (int)q, status_ptr(status), on.stream), "hyc_mlp_graddown_bwd_tcgen05");
  }
  // g_gate Bg | g_up Bu side by side, the two B gradients and grad_ad, each operand read once
  const Tensor g0 = ggu[0], g1 = ggu[1];
  Skinny().on(g0).rows(data(bg), 16, gm64, 0, 64).cols(xa, 16, data(grad_bgu))
          .on(g1).rows(data(bu), 16, gm64, 16, 64, 32).cols(xa + T * 32, 16, (char*)data(grad_bgu) + I * 32)
          .on(had).cols(data(gdm64), 64, data(grad_ad), true).run(T, g, status, on.stream);
  Tensor ga = lora_grad_a(xn_q.view({T, -1}), vec(xn_scale), gm64, 32, q);
  return {had, ggu, gm64, grad_bd, grad_ad, ga, grad_bgu};
}

static Tensor mlp_backward_x(const Tensor& g, const Tensor& ggu, const Tensor& gm64, const std::vector<Weight>& gate_up, const std::vector<Tensor>& w,
                             const std::vector<Tensor>& saved, at::IntArrayRef shape, int64_t q, const Tensor& status) {
  const Weight &wg = gate_up[0], &wu = gate_up[1];
  const Tensor &agu_rows = w[0], &norm_w = w[1];
  expect(wg, ggu.size(2), g.size(1), g, "gate projection");
  expect(wu, ggu.size(2), g.size(1), g, "up projection");
  expect(agu_rows, 64, g.size(1), "gate and up lora_A");
  SameDevice{g}.with(ggu).with(gm64).with(wg.m).with(wu.m).with(w).with(saved).with(status);
  const Tensor g0 = ggu[0], g1 = ggu[1];
  Tensor grad_xn = gemm({{&g0, wg}, {&g1, wu}, {&gm64, agu_rows}}, HYC_GEMM_B_KN, nullptr, status);
  return rmsnorm_backward_packed(grad_xn.view(shape), saved[0], saved[1], saved[2], saved[3], norm_w, saved[4], q, g.view(shape));
}

// ------------------------------------------------------------------ attention half
static Tensor heads(const Tensor& x2, int64_t B, int64_t M, int64_t n) { return x2.view({B, M, n, -1}).transpose(1, 2); }
static Tensor hidden(const Tensor& xh) { return xh.transpose(1, 2).reshape({xh.size(0) * xh.size(2), xh.size(1) * xh.size(3)}); }
static Tensor repeat_kv(const Tensor& x, int64_t n) {
  if (n == 1) return x;
  const auto b = x.size(0), h = x.size(1), m = x.size(2), d = x.size(3);
  return x.unsqueeze(2).expand({b, h, n, m, d}).reshape({b, h * n, m, d});
}
static Tensor repeat_kv_backward(const Tensor& g, int64_t n) {
  if (n == 1) return g;
  return g.reshape({g.size(0), g.size(1) / n, n, g.size(2), g.size(3)}).sum(2);
}
// [B, n, M, K] @ [B, n, K, d] written straight into the hidden layout
static Tensor matmul_to_hidden(const Tensor& a4, const Tensor& b4) {
  const int64_t B = a4.size(0), n = a4.size(1), M = a4.size(2), d = b4.size(3);
  Tensor out = empty({B, M, n, d}, a4);
  for (int64_t b = 0; b < B; ++b) {
    Tensor o = out[b].transpose(0, 1);
    at::bmm_out(o, a4[b], b4[b]);
  }
  return out.view({B * M, n * d});
}

// additive mask as the attention kernels take it: bf16, [b or 1, h or 1, M, M], strides in multiples of 8 elements
struct MaskView { Tensor t; int64_t b = 0, h = 0, row = 0; };
static MaskView mask_view(const OptTensor& mask, int64_t B, int64_t nh, int64_t M) {
  MaskView v;
  if (!given(mask)) return v;
  v.t = mask->to(at::kBFloat16);
  TORCH_CHECK_VALUE(v.t.dim() == 4 && v.t.size(3) == M && v.t.size(2) == M && (v.t.size(0) == 1 || v.t.size(0) == B) &&
                    (v.t.size(1) == 1 || v.t.size(1) == nh), "attention_mask must be [b or 1, h or 1, n, S]");
  auto strides = [&]() { v.b = v.t.size(0) == 1 ? 0 : v.t.stride(0); v.h = v.t.size(1) == 1 ? 0 : v.t.stride(1); v.row = v.t.stride(2); };
  strides();
  if (v.t.stride(3) != 1 || ((v.b | v.h | v.row) & 7) || (reinterpret_cast<uintptr_t>(v.t.data_ptr()) & 15)) { v.t = v.t.contiguous(); strides(); }
  return v;
}
static bool attn_kernels_take(int64_t M, int64_t d) { return d == 128 && M % 8 == 0 && M <= 4096; }

RopeTables rope_tables(const Tensor& cos_in, const Tensor& sin_in, int64_t seq, int64_t d) {
  RopeTables t{cos_in.dim() == 2 ? cos_in : cos_in.squeeze(), sin_in.dim() == 2 ? sin_in : sin_in.squeeze()};
  TORCH_CHECK_VALUE(t.cos.dim() == 2 && t.sin.sizes() == t.cos.sizes(), "cos / sin must squeeze to [seq_len, head_dim] tables");
  if (seq > t.cos.size(0)) {
    PyErr_SetString(PyExc_AssertionError, "the rotary tables are shorter than the sequence");
    throw pybind11::error_already_set();
  }
  TORCH_CHECK_VALUE(t.cos.size(1) >= d / 2, "cos / sin tables are narrower than head_dim / 2");
  if (t.cos.scalar_type() != at::kBFloat16 && t.cos.scalar_type() != at::kFloat) t.cos = t.cos.to(at::kFloat);
  if (t.sin.scalar_type() != t.cos.scalar_type()) t.sin = t.sin.to(t.cos.scalar_type());
  if (t.cos.stride(1) != 1 || t.sin.stride(1) != 1 || t.sin.stride(0) != t.cos.stride(0)) { t.cos = t.cos.contiguous(); t.sin = t.sin.contiguous(); }
  return t;
}
// Projections and head geometry have to agree: the kernels take rows of heads * d elements as they are told
static void check_geometry(const std::array<int64_t, 3>& widths, int64_t nh, int64_t d, int64_t nkv) {
  if (nh < 1 || nkv < 1 || d < 1 || nh % nkv != 0)
    throw std::runtime_error("invalid head geometry: " + std::to_string(nh) + " heads, " + std::to_string(nkv) + " key/value heads of " + std::to_string(d));
  for (int i = 0; i < 3; ++i)
    if (widths[i] != (i == 0 ? nh : nkv) * d)
      throw std::runtime_error(std::string("the ") + "qkv"[i] + " projection has " + std::to_string(widths[i]) + " outputs, not " +
                               std::to_string(i == 0 ? nh : nkv) + " heads of " + std::to_string(d));
}
// q and k (contiguous [rows, heads*d]) in place
static void rope_pair(const Tensor& q, int64_t nh, const Tensor& k, int64_t nkv, const RopeTables& t, int64_t seq, int64_t d, bool backward,
                      void* stream) {
  check(hyc_rope_pair(data(q), (int)nh, data(k), (int)nkv, data(t.cos), data(t.sin), t.cos.stride(0), t.f32(), q.size(0), (int)seq, (int)d,
                      backward ? 1 : 0, stream), "hyc_rope_pair");
}

// the q, k, v projections with their saves, rotary embedding, scores and probabilities
using MapForward = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, OptTensor, OptTensor, int64_t, int64_t>;
// row_cols (wanted if not null): how far each row of the probabilities reaches; what lies behind is zero and then not written.
// Left undefined where the rows are whole
static MapForward attn_forward_map(const Tensor& x, const std::vector<Weight>& qkv, const std::vector<Tensor>& w, const std::vector<Tensor>& stats, const RopeTables& tables,
                                   const OptTensor& mask, int64_t nh, int64_t d, int64_t nkv, int64_t q, double eps, const Tensor& status,
                                   Keep keep, Tensor* row_cols = nullptr) {
  const Tensor &norm_w = w[0], &bq = w[1], &bk = w[2], &bv = w[3], &aqkv_t = w[4];
  const Tensor &x_idx = stats[0], &x_scale = stats[1], &xn_scale = stats[2], &q_scale = stats[3], &k_scale = stats[4], &v_scale = stats[5];
  check_geometry({qkv[0].size(0), qkv[1].size(0), qkv[2].size(0)}, nh, d, nkv);
  for (int i = 0; i < 3; ++i) {
    const char* const names[3][2] = {{"q projection", "q lora_B"}, {"k projection", "k lora_B"}, {"v projection", "v lora_B"}};
    expect(qkv[i], qkv[i].size(0), x.size(2), x, names[i][0]);
    expect_factor(w[1 + i], qkv[i].size(0), names[i][1]);
    scale_vec(stats[3 + i], qkv[i].size(0));
  }
  for (const Weight& f : qkv) SameDevice{x}.with(f.m);
  SameDevice{x}.with(w).with(stats).with(tables.cos).with(tables.sin).with(mask).with(status);
  OnDevice on(x);
  const int64_t B = x.size(0), M = x.size(1), H = x.size(2), T = B * M, rep = nh / nkv;
  auto [x_norm, rstd, x_o, x_q, xn_q] = rmsnorm_save(x, norm_w, eps, q, x_scale, x_idx, xn_scale, keep);
  const Tensor xn2 = x_norm.view({T, H});
  const Tensor xa3 = lora_a_products(xn2, aqkv_t);
  auto p3 = qkv_lora_save(xn2, qkv, xa3, {&bq, &bk, &bv}, {&q_scale, &k_scale, &v_scale}, q, status, keep);
  const auto &[qy, q_q] = p3[0];
  const auto &[ky, k_q] = p3[1];
  const auto &[vy, v_q] = p3[2];
  rope_pair(qy, nh, ky, nkv, tables, M, d, false, on.stream);
  if (attn_kernels_take(M, d)) {
    // one kernel from q, k, v to the probabilities, o and the codes of o
    const MaskView mv = mask_view(mask, B, nh, M);
    Tensor cls, a = empty({B, nh, M, M}, x_norm), o2 = empty({T, nh * d}, x_norm), o_q = empty({T, nh * d * q / 8}, x_norm, at::kByte);
    const Tensor os = scale_vec(stats[6], nh * d);
    int64_t cls_b = 0, cls_h = 0;
    if (mv.t.defined()) {
      const int64_t nb = mv.t.size(0), nhm = mv.t.size(1);
      cls = empty({(int64_t)hyc_attn_mask_class_bytes((int)nb, (int)nhm, (int)M)}, x_norm, at::kByte);
      check(hyc_attn_mask_class(data(mv.t), mv.b, mv.h, mv.row, (int)nb, (int)nhm, (int)M, data(cls), on.stream), "hyc_attn_mask_class");
      cls_b = nb == 1 ? 0 : nhm;
      cls_h = nhm == 1 ? 0 : 1;
      // (a mask per head with grouped heads: the backward kernels read the whole map)
      if (row_cols && !(cls_h != 0 && nh != nkv)) *row_cols = empty({B * nh * M}, x_norm, at::kShort);
    }
    check(hyc_attn_fwd_cols_tcgen05(data(qy), data(ky), data(vy), (int)B, (int)M, (int)nh, (int)nkv, (int)d, (float)(1.0 / std::sqrt((double)d)),
                               data(mv.t), mv.b, mv.h, mv.row, data(cls), cls_b, cls_h, data(a), row_cols ? (uint16_t*)data(*row_cols) : nullptr,
                               data(o2), data(os), data(o_q), (int)q, status_ptr(status), on.stream), "hyc_attn_fwd_cols_tcgen05");
    return {a, o2, rstd, x_o, x_q, *xn_q, q_q, k_q, v_q, xa3, o_q, cls, cls_b, cls_h};
  }
  const Tensor kh = repeat_kv(heads(ky, B, M, nkv), rep), vh = repeat_kv(heads(vy, B, M, nkv), rep);
  Tensor scores = at::matmul(heads(qy, B, M, nh), kh.transpose(-2, -1));
  const Tensor a = softmax_forward(scores, 1.0 / std::sqrt((double)d), mask, true);
  const Tensor o2 = matmul_to_hidden(a, vh);
  return {a, o2, rstd, x_o, x_q, *xn_q, q_q, k_q, v_q, xa3, std::nullopt, std::nullopt, 0, 0};
}

// o projection with residual and the save of its input
static std::vector<Tensor> attn_forward_out(const Tensor& x, const Tensor& o2, const Weight& wo, const Tensor& ao_cols, const Tensor& bo_cols,
                                            const Tensor& o_scale, const OptTensor& o_codes, const OptTensor& bias_o, int64_t q, const Tensor& status) {
  expect(wo, x.size(2), o2.size(1), x, "o projection");
  expect(bo_cols, x.size(2), 64, "o lora_B");
  SameDevice{x}.with(o2).with(wo.m).with(ao_cols).with(bo_cols).with(o_scale).with(o_codes).with(bias_o).with(status);
  const int64_t B = x.size(0), M = x.size(1), H = x.size(2), T = B * M;
  const Tensor o_xa64 = at::mm(o2, ao_cols);
  const Tensor res = bf16c(x);
  Tensor x_medium = gemm({{&o2, wo}, {&o_xa64, bo_cols}}, HYC_GEMM_FIXED_ORDER, &res, status);
  if (given(bias_o)) x_medium.add_(bias_o->to(at::kBFloat16));
  const Tensor o_q = given(o_codes) ? *o_codes : std::get<0>(quant(o2.view({B, M, -1}), o_scale, q, std::nullopt, std::nullopt, std::nullopt, std::nullopt));
  return {x_medium.view({B, M, H}), o_q.view({T, -1}), o_xa64};
}

static Tensor rebuild(const Tensor& codes, const Tensor& scale, const Tensor& xa, const Tensor& b, int64_t q) {
  const int64_t T = codes.size(0);
  return dequant_lora_add(codes.view({1, T, -1}), scale, xa.view({1, T, -1}), b.t(), q).view({T, -1});
}

// o projection backward: -> grad_bo, grad_ao, grad_o2
static std::vector<Tensor> attn_backward_out(const Tensor& g, const Weight& wo, const Tensor& bo_in, const Tensor& ao_rows, const Tensor& o_xa,
                                             const Tensor& o_q, const Tensor& o_scale, int64_t q, const Tensor& status) {
  expect(wo, g.size(1), wo.size(1), g, "o projection");
  expect_factor(bo_in, g.size(1), "o lora_B");
  expect(ao_rows, 64, wo.size(1), "o lora_A");
  SameDevice{g}.with(wo.m).with(bo_in).with(ao_rows).with(o_xa).with(o_q).with(o_scale).with(status);
  OnDevice on(g);
  const int64_t T = g.size(0);
  const Tensor bo = factor(bo_in);
  Tensor gm64 = empty({T, 64}, g), grad_bo = empty({g.size(1), 16}, g);
  Skinny().on(g).rows(data(bo), 16, gm64, 0, 64, 48).cols(data(o_xa), o_xa.stride(0), data(grad_bo)).run(T, g, status, on.stream);
  Tensor grad_ao = lora_grad_a(o_q, vec(o_scale), gm64, 16, q);
  Tensor grad_o2 = gemm({{&g, wo}, {&gm64, ao_rows}}, HYC_GEMM_B_KN, nullptr, status);
  return {grad_bo, grad_ao, grad_o2};
}

// the map's backward.  `a`: the restored map; `topk`: the five tensors of the top-k form (the softmax backward then
// restores once more on chip), empty for the pruned form.  -> grad_q, grad_k, grad_v [T, n*d] after the inverse
// rotation
static std::vector<Tensor> attn_backward_map(const Tensor& grad_o2, Tensor a, const std::vector<Tensor>& topk, int64_t map_q_bit,
                                                const std::vector<Tensor>& saved, const std::vector<Tensor>& w, const RopeTables& tables,
                                                int64_t B, int64_t M, int64_t nh, int64_t d, int64_t nkv, int64_t q,
                                                const OptTensor& cls, int64_t cls_b, int64_t cls_h, const Tensor& status, Keep keep) {
  const Tensor &q_q = saved[0], &q_s = saved[1], &q_xa = saved[2], &k_q = saved[3], &k_s = saved[4], &k_xa = saved[5], &v_q = saved[6],
               &v_s = saved[7], &v_xa = saved[8];
  check_geometry({w[0].size(0), w[1].size(0), w[2].size(0)}, nh, d, nkv);
  for (int i = 0; i < 3; ++i) expect_factor(w[i], w[i].size(0), "lora_B of q, k or v");
  SameDevice{grad_o2}.with(a).with(topk).with(saved).with(w).with(tables.cos).with(tables.sin).with(cls).with(status);
  OnDevice on(grad_o2);
  const int64_t T = B * M, rep = nh / nkv;
  const double scale = 1.0 / std::sqrt((double)d);
  if (attn_kernels_take(M, d)) {
    // q, k (rotated) and v from their codes in one launch
    const auto rebuilt = together(grad_o2, {{{T, nh * d}, at::kBFloat16}, {{T, nkv * d}, at::kBFloat16}, {{T, nkv * d}, at::kBFloat16}});
    Tensor held[9];
    const void *cp[3], *sp[3], *xp[3], *bp[3];
    void* yp[3];
    int n[3];
    for (int i = 0; i < 3; ++i) {
      n[i] = (int)((i == 0 ? nh : nkv) * d);
      cp[i] = data(held[3 * i] = saved[3 * i].contiguous()); sp[i] = data(held[3 * i + 1] = vec(saved[3 * i + 1]));
      xp[i] = data(saved[3 * i + 2]); bp[i] = data(held[3 * i + 2] = factor(w[i])); yp[i] = data(rebuilt[i]);
    }
    check(hyc_rebuild_qkv(cp, sp, xp, bp, yp, n, data(tables.cos), data(tables.sin), tables.cos.stride(0), tables.f32(), T, (int)M, (int)q, on.stream),
          "hyc_rebuild_qkv");
    const Tensor &q2 = rebuilt[0], &k2 = rebuilt[1], &v2 = rebuilt[2];
    Tensor gs = empty({B, nh, M, M}, grad_o2);
    const auto [gq, gk, gv] = together(grad_o2, {{{T, nh * d}, at::kBFloat16}, {{T, nkv * d}, at::kBFloat16}, {{T, nkv * d}, at::kBFloat16}}, keep);
    check(hyc_attn_bwd_tcgen05(data(q2), data(k2), data(v2), data(grad_o2), data(a), data(gs), (int)B, (int)M, (int)nh, (int)nkv, (int)d,
                               (float)scale, data(cls), cls_b, cls_h, data(gq), data(gk), data(gv), status_ptr(status), on.stream),
          "hyc_attn_bwd_tcgen05");
    rope_pair(gq, nh, gk, nkv, tables, M, d, true, on.stream);
    return {gq, gk, gv};
  }
  const Tensor grad_oh = heads(grad_o2, B, M, nh);
  Tensor v2 = rebuild(v_q, v_s, v_xa, w[2], q);
  Tensor grad_v = rep == 1 ? matmul_to_hidden(a.transpose(-2, -1), grad_oh)
                           : hidden(repeat_kv_backward(at::matmul(a.transpose(-2, -1), grad_oh), rep));
  Tensor grad_a = at::matmul(grad_oh, repeat_kv(heads(v2, B, M, nkv), rep).transpose(-2, -1));
  v2.reset();
  Tensor grad_s;
  if (!topk.empty()) {
    const std::vector<int64_t> shape(a.sizes().begin(), a.sizes().end());
    a.reset();
    grad_s = topk_softmax_backward(topk[0], topk[1], topk[2], topk[3], topk[4], shape, map_q_bit, grad_a, std::nullopt, scale);
  } else {
    grad_s = softmax_backward(a, grad_a, scale);
    a.reset();
  }
  grad_a.reset();
  Tensor q2 = rebuild(q_q, q_s, q_xa, w[0], q);
  rope(q2.view({B, M, nh, d}), tables.cos, tables.sin, false, true);
  Tensor grad_k = rep == 1 ? matmul_to_hidden(grad_s.transpose(-2, -1), heads(q2, B, M, nh))
                           : hidden(repeat_kv_backward(at::matmul(grad_s.transpose(-2, -1), heads(q2, B, M, nh)), rep));
  q2.reset();
  Tensor k2 = rebuild(k_q, k_s, k_xa, w[1], q);
  rope(k2.view({B, M, nkv, d}), tables.cos, tables.sin, false, true);
  Tensor grad_q = matmul_to_hidden(grad_s, repeat_kv(heads(k2, B, M, nkv), rep));
  rope_pair(grad_q, nh, grad_k, nkv, tables, M, d, true, on.stream);
  return {grad_q, grad_k, grad_v};
}

// LoRA gradients of q/k/v: -> gmq [T, 64], ga [48, H], grad_bq, grad_bk, grad_bv
static std::vector<Tensor> attn_backward_lora(const std::vector<Tensor>& grads, const std::vector<Tensor>& b_in, const Tensor& qkv_xa, const Tensor& xn_q,
                                              const Tensor& xn_scale, int64_t q, const Tensor& status) {
  for (int i = 0; i < 3; ++i) expect_factor(b_in[i], grads[i].size(1), "lora_B of q, k or v");
  SameDevice{grads[0]}.with(grads).with(b_in).with(qkv_xa).with(xn_q).with(xn_scale).with(status);
  OnDevice on(grads[0]);
  const int64_t T = grads[0].size(0);
  Tensor gmq = empty({T, 64}, grads[0]), gb[3], b[3];
  Skinny s;
  for (int i = 0; i < 3; ++i) {
    gb[i] = empty({grads[i].size(1), 16}, grads[0]);
    b[i] = factor(b_in[i]);
    s.on(grads[i]).rows(data(b[i]), 16, gmq, 16 * i, 64, i == 2 ? 16 : 0).cols(at_row(qkv_xa, i), 16, data(gb[i]));
  }
  s.run(T, gmq, status, on.stream);
  Tensor ga = lora_grad_a(xn_q.view({T, -1}), vec(xn_scale), gmq, 48, q);
  return {gmq, ga, gb[0], gb[1], gb[2]};
}

static Tensor attn_backward_x(const Tensor& g, const std::vector<Tensor>& grads, const Tensor& gmq, const std::vector<Weight>& qkv, const std::vector<Tensor>& w,
                              const std::vector<Tensor>& saved, at::IntArrayRef shape, int64_t q, const Tensor& status) {
  const Tensor &aqkv_rows = w[0], &norm_w = w[1];
  for (int i = 0; i < 3; ++i) {
    expect(qkv[i], grads[i].size(1), g.size(1), g, "q, k or v projection");
    SameDevice{g}.with(qkv[i].m);
  }
  expect(aqkv_rows, 64, g.size(1), "lora_A of q, k and v");
  SameDevice{g}.with(grads).with(gmq).with(w).with(saved).with(status);
  Tensor grad_xn = gemm({{&grads[0], qkv[0]}, {&grads[1], qkv[1]}, {&grads[2], qkv[2]}, {&gmq, aqkv_rows}}, HYC_GEMM_B_KN, nullptr, status);
  return rmsnorm_backward_packed(grad_xn.view(shape), saved[0], saved[1], saved[2], saved[3], norm_w, saved[4], q, g.view(shape));
}

// ------------------------------------------------------------------ the whole layer
// Forward and backward of a calibrated layer as one call each: between the launches there is then no Python (attribute and
// dictionary look-ups, argument conversion), which cost more than the kernels of a short sequence run for.
// 128 tokens, Llama-2-7B, bf16 weights, host work per forward + backward: 863 us as ten calls.

enum { PQ, PK, PV, PO, PGATE, PUP, PDOWN, PROJECTIONS };
enum { AQKV_T, AQKV_ROWS, AO_COLS, AO_ROWS, BO_COLS, AGU_T, AGU_ROWS, AD_ROWS, AD_COLS, BD_COLS, PADS };

// What a tensor was: the same memory, seen the same way, nothing written since.  Holding the storage keeps its address from
// being handed out again, so that an adapter whose `.data` was replaced cannot look unchanged.
struct Stamp {
  c10::Storage storage;
  int64_t offset = 0;
  uint32_t version = 0;
  at::ScalarType type = at::kBFloat16;
  at::DimVector sizes, strides;
  static uint32_t version_of(const Tensor& t) { return t.is_inference() ? 0u : (uint32_t)t._version(); }
  static Stamp of(const Tensor& t) {
    return {t.storage(), t.storage_offset(), version_of(t), t.scalar_type(), at::DimVector(t.sizes()), at::DimVector(t.strides())};
  }
  bool fits(const Tensor& t) const {
    return t.storage().unsafeGetStorageImpl() == storage.unsafeGetStorageImpl() && t.storage_offset() == offset && version_of(t) == version &&
           t.scalar_type() == type && t.sizes() == at::IntArrayRef(sizes) && t.strides() == at::IntArrayRef(strides);
  }
};

// The stream capture that work on the device of `t` is being recorded into, 0 if it runs.  What is computed inside a capture holds
// nothing until the graph is replayed, and a replay computes anew only what was recorded: copies of things that change between
// replays (adapters) are made inside each capture that reads them, and made again outside of it.
static int64_t capture_of(const Tensor& t) {
  if (!t.is_cuda()) return 0;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(c10::cuda::getCurrentCUDAStream(t.get_device()).stream(), &status, &id) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  return status == cudaStreamCaptureStatusNone ? 0 : (int64_t)id;
}

struct LayerPlan {
  Tensor norm1, norm2;
  FrozenWeight w[PROJECTIONS];
  Tensor lora[2 * PROJECTIONS];                 // A, B of each projection
  OptTensor bias_o, bias_d;
  std::vector<Tensor> pad;                      // what AttnWeights.padded / MLPWeights.padded make of the LoRA factors
  Stamp pad_of[2 * PROJECTIONS];
  int64_t pad_capture = 0;                      // where it is fresh: the capture that the calls are recorded into, 0 if they run
  std::vector<Tensor> stats_in, stats;          // calibrated statistics as given, and as the kernels read them
  std::vector<Stamp> stats_of;

  // false: the padded factors are out of date, or a weight is no longer what it was checked to be
  bool fresh() const {
    if ((int)pad.size() != PADS || pad_capture != capture_of(lora[0])) return false;
    for (const FrozenWeight& f : w)
      if (f.plain.defined() && f.plain.scalar_type() != at::kBFloat16) return false;
    for (const OptTensor* b : {&bias_o, &bias_d})
      if (given(*b) && (*b)->scalar_type() != at::kBFloat16) return false;
    for (int i = 0; i < 2 * PROJECTIONS; ++i)
      if (lora[i].scalar_type() != at::kBFloat16 || !pad_of[i].fits(lora[i])) return false;
    return true;
  }
  void set_padded(const std::vector<Tensor>& p) {
    TORCH_CHECK_VALUE((int)p.size() == PADS, "LayerPlan: ", (int)PADS, " padded factors expected");
    pad = p;
    for (int i = 0; i < 2 * PROJECTIONS; ++i) pad_of[i] = Stamp::of(lora[i]);
    pad_capture = capture_of(lora[0]);
  }
  // A statistic that the kernels read where it lies is looked up once.  One that has to be converted is converted on every
  // call: the copy could not follow a write that bumps no version (through `.data`, or to an inference tensor).
  void set_stats(const std::vector<Tensor>& s) {
    stats_in.resize(s.size());
    stats.resize(s.size());
    stats_of.resize(s.size());
    for (size_t i = 0; i < s.size(); ++i) {
      if (stats_in[i].defined() && s[i].unsafeGetTensorImpl() == stats_in[i].unsafeGetTensorImpl() && stats_of[i].fits(s[i])) continue;
      Tensor now = s[i].scalar_type() == at::kLong ? s[i].contiguous() : vec(s[i]);
      const bool in_place = now.storage().unsafeGetStorageImpl() == s[i].storage().unsafeGetStorageImpl();
      stats[i] = std::move(now);
      stats_in[i] = in_place ? s[i] : Tensor();
      if (in_place) stats_of[i] = Stamp::of(s[i]);
    }
  }
};

// order of the statistics
enum { X_IDX, X_SCALE, XN1_SCALE, Q_SCALE, K_SCALE, V_SCALE, O_SCALE, XM_IDX, XM_SCALE, XN2_SCALE, GATE_SCALE, UP_SCALE, STATS };

struct LayerSaved {
  MlpForward mlp;
  Tensor rstd, x_o, x_q, xn_q, q_q, k_q, v_q, xa3, o_q, o_xa64;
  std::vector<Tensor> map;                      // top-k form: five tensors; pruned form: words, directory, nnz
  OptTensor cls;
  int64_t cls_b = 0, cls_h = 0;
  Tensor row_cols;                              // how far the rows of the map reach; undefined: they are whole
  std::vector<Tensor> stats;
  RopeTables tables;
  int64_t B, M, H, nh, d, nkv, q_attn, q_mlp, map_q;    // map_q = 0: pruned form
  at::ScalarType x_type;
};

static std::pair<Tensor, std::shared_ptr<LayerSaved>> layer_forward(LayerPlan& p, const Tensor& x_in, const std::vector<Tensor>& stats, const Tensor& cos,
                                                                    const Tensor& sin, const OptTensor& mask, int64_t nh, int64_t d, int64_t nkv,
                                                                    int64_t q_attn, int64_t q_mlp, int64_t map_q, int64_t map_k, double threshold,
                                                                    int64_t capacity, double eps, const Tensor& status) {
  at::AutoDispatchBelowADInplaceOrView below;
  TORCH_CHECK_VALUE((int)stats.size() == STATS, "layer_forward: ", (int)STATS, " statistics expected");
  TORCH_CHECK_VALUE(x_in.dim() == 3, "expected a [B, M, H] input, got shape ", x_in.sizes());
  require_cuda({&x_in, &status});
  p.set_stats(stats);
  const std::vector<Tensor>& st = p.stats;
  const Tensor x = bf16c(x_in);
  auto s = std::make_shared<LayerSaved>();
  s->B = x.size(0); s->M = x.size(1); s->H = x.size(2);
  s->nh = nh; s->d = d; s->nkv = nkv; s->q_attn = q_attn; s->q_mlp = q_mlp; s->map_q = map_q;
  s->stats = st;
  s->x_type = x_in.scalar_type();
  s->tables = rope_tables(cos, sin, s->M, d);
  const bool recorded = p.pad_capture != 0;
  Tensor x_medium;
  {
    Tensor a, o2;
    OptTensor o_codes;
    std::vector<Weight> w = weights({&p.w[PQ], &p.w[PK], &p.w[PV]}, s->B * s->M, Use::QKV, recorded);
    // where the save and the restore know how to leave out what the mask rules out (tiles of 128 columns: not in maps of one tile).
    // us of the attention kernel, save and restore without / with, 5 % kept: causal [4,32,1024,1024] top-k 364 / 300, pruned 254 / 231,
    // [4,32,256,256] 41 / 40 and 42 / 41; a mask that rules out nothing, which is not known here, 396 / 392 and 304 / 308
    const bool cols = s->M > 128 && (map_q == 0 ? s->M % 256 == 0 : hyc_softmax_topk_cols_supported((int)s->M, (int)map_k) == 1);
    std::tie(a, o2, s->rstd, s->x_o, s->x_q, s->xn_q, s->q_q, s->k_q, s->v_q, s->xa3, o_codes, s->cls, s->cls_b, s->cls_h) = attn_forward_map(
        x, w, {p.norm1, p.lora[2 * PQ + 1], p.lora[2 * PK + 1], p.lora[2 * PV + 1], p.pad[AQKV_T]},
        {st[X_IDX], st[X_SCALE], st[XN1_SCALE], st[Q_SCALE], st[K_SCALE], st[V_SCALE], st[O_SCALE]}, s->tables, mask, nh, d, nkv, q_attn, eps, status, Keep::SHARED, cols ? &s->row_cols : nullptr);
    w.clear();
    if (map_q > 0) {
      auto [val, col, q, sc, z] = topk_compress(a, map_k, map_q, s->row_cols, Keep::SHARED);
      s->map = {val, col, q, sc, z};
    } else {
      auto [words, directory, nnz] = prune_tiled(a, threshold, capacity, s->row_cols, Keep::SHARED);
      s->map = {words, directory, nnz};
    }
    a.reset();
    auto out = attn_forward_out(x, o2, weights({&p.w[PO]}, s->B * s->M, Use::O, recorded)[0], p.pad[AO_COLS], p.pad[BO_COLS], st[O_SCALE], o_codes, p.bias_o, q_attn, status);
    x_medium = out[0]; s->o_q = out[1]; s->o_xa64 = out[2];
  }
  std::vector<Weight> w = weights({&p.w[PGATE], &p.w[PUP]}, s->B * s->M, Use::GATE_UP, recorded);
  s->mlp = mlp_forward(x_medium, {p.norm2, Tensor(), Tensor(), Tensor(), p.lora[2 * PGATE + 1], p.lora[2 * PUP + 1],
                                  p.pad[AGU_T], p.pad[AD_COLS], p.pad[BD_COLS]},
                       {st[XM_IDX], st[XM_SCALE], st[XN2_SCALE], st[GATE_SCALE], st[UP_SCALE]}, p.bias_d, q_mlp, eps, status, w, nullptr, &p.w[PDOWN], recorded, Keep::SHARED);
  Tensor y = std::move(s->mlp.x_out);
  s->mlp.x_out = Tensor();
  return {y.to(s->x_type), s};
}

// -> grad_x and the fourteen LoRA gradients (A, B of q, k, v, o, gate, up, down).  hook: see mlp.mlp_backward; refresh: makes the
// padded factors again
static std::vector<Tensor> layer_backward(const LayerPlan& p, const Tensor& grad_y, LayerSaved& s, const pybind11::object& hook,
                                          const pybind11::object& refresh, const Tensor& overflow, const Tensor& status) {
  // the steps run below the dispatch keys of autograd and version counting, the hook above them: it is the caller's code, and
  // an update in place that it makes has to bump the versions that fresh() goes by
  std::optional<at::AutoDispatchBelowADInplaceOrView> below(std::in_place);
  const std::vector<Tensor>& st = s.stats;
  const int64_t T = s.B * s.M;
  const std::vector<int64_t> shape = {s.B, s.M, s.H};
  const bool recorded = p.pad_capture != 0;
  require_cuda({&grad_y, &s.rstd});
  OnDevice on(s.rstd);
  std::vector<Tensor> out(1 + 2 * PROJECTIONS);
  auto lora = [&](int proj, const Tensor& a, const Tensor& b) { out[1 + 2 * proj] = a; out[2 + 2 * proj] = b; };
  auto report = [&](std::initializer_list<std::pair<const char*, int>> which) {
    if (hook.is_none()) return;
    pybind11::dict d;
    for (const auto& [name, proj] : which) {
      d[(std::string("grad_a") + name).c_str()] = out[1 + 2 * proj];
      d[(std::string("grad_b") + name).c_str()] = out[2 + 2 * proj];
    }
    below.reset();
    hook(d);
    below.emplace();
  };
  Tensor g_medium;
  {
    const Tensor g = bf16c(grad_y).view({T, s.H});
    const MlpForward& m = s.mlp;
    auto r = mlp_backward_lora(g, weights({&p.w[PDOWN]}, T, Use::GRAD_DOWN, recorded)[0], {Tensor(), p.lora[2 * PGATE + 1], p.lora[2 * PUP + 1], p.lora[2 * PDOWN + 1], p.pad[AD_ROWS]},
                               {m.q1, m.gs, m.q2, m.us, m.gu_xa, m.down_xa64, m.xn_q, st[XN2_SCALE]}, s.q_mlp, status);
    lora(PGATE, r[5].narrow(0, 0, 16), r[6].select(0, 0));
    lora(PUP, r[5].narrow(0, 16, 16), r[6].select(0, 1));
    lora(PDOWN, r[4], r[3]);
    report({{"g", PGATE}, {"u", PUP}, {"d", PDOWN}});
    r[0].reset();
    g_medium = mlp_backward_x(g, r[1], r[2], weights({&p.w[PGATE], &p.w[PUP]}, T, Use::GRAD_X, recorded), {p.pad[AGU_ROWS], p.norm2},
                              {m.xm_q, st[XM_SCALE], m.xm_o, st[XM_IDX], m.rstd}, shape, s.q_mlp, status).view({T, s.H});
  }
  if (!hook.is_none() && !p.fresh()) {           // the hook of the MLP half changed factors of this one
    below.reset();
    refresh();
    below.emplace();
  }
  std::vector<Tensor> grads;
  {
    auto r = attn_backward_out(g_medium, weights({&p.w[PO]}, T, Use::GRAD_X, recorded)[0], p.lora[2 * PO + 1], p.pad[AO_ROWS], s.o_xa64, s.o_q, st[O_SCALE], s.q_attn, status);
    lora(PO, r[1], r[0]);
    const std::vector<int64_t> a_shape = {s.B, s.nh, s.M, s.M};
    const bool topk = s.map_q > 0;
    Tensor a = topk ? topk_restore(s.map[0], s.map[1], s.map[2], s.map[3], s.map[4], a_shape, s.map_q, std::nullopt, s.row_cols)
                    : prune_tiled_restore(s.map[0], s.map[1], a_shape, std::nullopt, s.row_cols);
    grads = attn_backward_map(r[2], std::move(a), topk ? s.map : std::vector<Tensor>(), s.map_q,
                              {s.q_q, st[Q_SCALE], s.xa3.select(0, 0), s.k_q, st[K_SCALE], s.xa3.select(0, 1), s.v_q, st[V_SCALE], s.xa3.select(0, 2)},
                              {p.lora[2 * PQ + 1], p.lora[2 * PK + 1], p.lora[2 * PV + 1]}, s.tables, s.B, s.M, s.nh, s.d, s.nkv, s.q_attn,
                              s.cls, s.cls_b, s.cls_h, status, Keep::SHARED);
    if (!topk)
      check(hyc_prune_overflow_flag((const int64_t*)data(s.map[2]), s.map[0].numel(), (int*)data(overflow), on.stream), "hyc_prune_overflow_flag");
  }
  auto r = attn_backward_lora(grads, {p.lora[2 * PQ + 1], p.lora[2 * PK + 1], p.lora[2 * PV + 1]}, s.xa3, s.xn_q, st[XN1_SCALE], s.q_attn, status);
  for (int i = 0; i < 3; ++i) lora(PQ + i, r[1].narrow(0, 16 * i, 16), r[2 + i]);
  report({{"q", PQ}, {"k", PK}, {"v", PV}, {"o", PO}});
  out[0] = attn_backward_x(g_medium, grads, r[0], weights({&p.w[PQ], &p.w[PK], &p.w[PV]}, T, Use::GRAD_X, recorded), {p.pad[AQKV_ROWS], p.norm1},
                           {s.x_q, st[X_SCALE], s.x_o, st[X_IDX], s.rstd}, shape, s.q_attn, status).to(s.x_type);
  return out;
}

void bind_blocks(pybind11::module_& m) {
  m.def("lora_grad_a", &lora_grad_a);
  m.def("capture_of", &capture_of);
  m.def("mlp_forward", [](const Tensor& x, const std::vector<Tensor>& w, const std::vector<Tensor>& stats, const OptTensor& bias_d, int64_t q,
                          double eps, const Tensor& st) {
    const Weight wd(w[3]);
    MlpForward f = mlp_forward(x, w, stats, bias_d, q, eps, st, {Weight(w[1]), Weight(w[2])}, &wd, nullptr, false, Keep::OWN);
    return std::vector<Tensor>{f.x_out, f.rstd, f.xm_o, f.xm_q, f.xn_q, f.q1, f.q2, f.gs, f.us, f.gu_xa, f.down_xa64}; });
  m.def("mlp_backward_lora", [](const Tensor& g, const std::vector<Tensor>& w, const std::vector<Tensor>& saved, int64_t q, const Tensor& st) {
    return mlp_backward_lora(g, w[0], w, saved, q, st); });
  m.def("mlp_backward_x", [](const Tensor& g, const Tensor& ggu, const Tensor& gm64, const std::vector<Tensor>& w, const std::vector<Tensor>& saved,
                             std::vector<int64_t> shape, int64_t q, const Tensor& st) { return mlp_backward_x(g, ggu, gm64, {Weight(w[0]), Weight(w[1])}, {w[2], w[3]}, saved, shape, q, st); });
  m.def("attn_forward_map", [](const Tensor& x, const std::vector<Tensor>& w, const std::vector<Tensor>& stats, const Tensor& cos, const Tensor& sin,
                               const OptTensor& mask, int64_t nh, int64_t d, int64_t nkv, int64_t q, double eps, const Tensor& st) {
    return attn_forward_map(x, {Weight(w[1]), Weight(w[2]), Weight(w[3])}, {w[0], w[4], w[5], w[6], w[7]}, stats, rope_tables(cos, sin, x.size(1), d), mask, nh, d, nkv, q, eps, st, Keep::OWN); });
  m.def("attn_forward_out", [](const Tensor& x, const Tensor& o2, const Tensor& wo, const Tensor& ao_cols, const Tensor& bo_cols, const Tensor& o_scale,
                               const OptTensor& o_codes, const OptTensor& bias_o, int64_t q, const Tensor& st) {
    return attn_forward_out(x, o2, wo, ao_cols, bo_cols, o_scale, o_codes, bias_o, q, st); });
  m.def("attn_backward_out", [](const Tensor& g, const Tensor& wo, const Tensor& bo, const Tensor& ao_rows, const Tensor& o_xa, const Tensor& o_q,
                                const Tensor& o_scale, int64_t q, const Tensor& st) {
    return attn_backward_out(g, wo, bo, ao_rows, o_xa, o_q, o_scale, q, st); });
  m.def("attn_backward_map", [](const Tensor& grad_o2, const Tensor& a, const std::vector<Tensor>& topk, int64_t map_q_bit, const std::vector<Tensor>& saved,
                                const std::vector<Tensor>& w, const Tensor& cos, const Tensor& sin, int64_t B, int64_t M, int64_t nh, int64_t d,
                                int64_t nkv, int64_t q, const OptTensor& cls, int64_t cls_b, int64_t cls_h, const Tensor& st) {
    return attn_backward_map(grad_o2, a, topk, map_q_bit, saved, w, rope_tables(cos, sin, M, d), B, M, nh, d, nkv, q, cls, cls_b, cls_h, st, Keep::OWN); });
  m.def("attn_backward_lora", &attn_backward_lora);
  m.def("attn_backward_x", [](const Tensor& g, const std::vector<Tensor>& grads, const Tensor& gmq, const std::vector<Tensor>& w,
                              const std::vector<Tensor>& saved, std::vector<int64_t> shape, int64_t q, const Tensor& st) {
    return attn_backward_x(g, grads, gmq, {Weight(w[0]), Weight(w[1]), Weight(w[2])}, {w[3], w[4]}, saved, shape, q, st); });
  pybind11::class_<FrozenWeight>(m, "FrozenWeight")
      .def(pybind11::init([](const Tensor& w) { FrozenWeight f; f.plain = w; return f; }))
      .def(pybind11::init([](const Tensor& packed, const Tensor& code, const Tensor& absmax, const OptTensor& code2, const OptTensor& absmax2,
                             int64_t blocksize2, double offset, int64_t blocksize, std::vector<int64_t> shape) {
        return FrozenWeight{Tensor(), packed, code, absmax, code2, absmax2, blocksize2, blocksize, offset, std::move(shape)}; }));
  pybind11::class_<LayerSaved, std::shared_ptr<LayerSaved>>(m, "LayerSaved");
  pybind11::class_<LayerPlan>(m, "LayerPlan")
      .def(pybind11::init([](const Tensor& norm1, const Tensor& norm2, const std::vector<FrozenWeight>& w, const std::vector<Tensor>& lora,
                             const OptTensor& bias_o, const OptTensor& bias_d) {
        TORCH_CHECK_VALUE(w.size() == PROJECTIONS && lora.size() == 2 * PROJECTIONS, "LayerPlan: seven weights and fourteen LoRA factors expected");
        auto p = std::make_unique<LayerPlan>();
        p->norm1 = norm1; p->norm2 = norm2; p->bias_o = bias_o; p->bias_d = bias_d;
        std::copy(w.begin(), w.end(), p->w);
        std::copy(lora.begin(), lora.end(), p->lora);
        return p; }))
      .def("fresh", &LayerPlan::fresh)
      .def("set_padded", &LayerPlan::set_padded)
      .def("forward", &layer_forward)
      .def("backward", &layer_backward);
}

}  // namespace hyc_host
