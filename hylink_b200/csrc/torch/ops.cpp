// Autograd functions of the training step over the kernels of csrc/train: what surrounds the GEMMs and the attention
// of a transformer block, the language-model head with its loss, the mixture-of-experts layer; the optimizers; and the
// launches of emulated collectives and of the landing reduce. Products that gelu or its gradient follows go through the kernel of
// train/expert_gemm.cu where that pays, and so do an expert layer's others; the rest of the GEMMs are torch's own (cuBLAS), the
// attention between the two halves of a block is whatever torch's scaled_dot_product_attention picks.
//
// A block is cut in two around the attention:
//   blockPre:   x1 = x + y; h = layer norm(x1); q, k, v = h Wqkv^T + b     (y: the branch of the block before)
//   blockPost:  x2 = x1 + a Wproj^T + b; h = layer norm(x2); y2 = gelu(h Wfc^T + b) Wout^T + b;  returns x2, y2
// The add of y2 is left to the next block's (or the final) layer norm, which reads x2 anyway.
#include <ATen/ATen.h>
#include <ATen/SavedTensorHooks.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/python.h>

#include "hylink/hylink_ext.h"
#include "train/train_kernels.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;
namespace train = hl::train;

void ok(hlResult_t r, const char* what) {
  if (r != hlSuccess) TORCH_CHECK(false, "hylink ", what, ": ", hlGetErrorString(r), " (", hlGetLastError(), ")");
}
int code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kHalf: return hlFloat16;
    case at::kBFloat16: return hlBfloat16;
    default: TORCH_CHECK(false, "hylink: training kernels take fp16 and bf16 tensors");
  }
}
cudaStream_t streamOf(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
Tensor floats(const Tensor& like, at::IntArrayRef sizes) { return at::empty(sizes, like.options().dtype(at::kFloat)); }
bool aligned(const Tensor& t) { return ((uintptr_t)t.data_ptr() & 15) == 0; }
// What the kernels' 16-byte packets need of whatever comes from outside (tokens, weights, incoming gradients, what saved-tensor
// hooks give back): contiguous, and on a 16-byte boundary. Parameters that are views into one flat buffer start anywhere.
Tensor dense(const Tensor& t) {
  const Tensor c = t.contiguous();
  return aligned(c) ? c : c.clone();
}
// Rows of a [..., width] tensor as one matrix.
Tensor rowsOf(const Tensor& t) { return dense(t).view({-1, t.size(-1)}); }

// The gradients below are computed by kernels that autograd does not see into. Where a caller asks for a backward pass that
// can be differentiated again (create_graph; gradient mode is on inside it then), a node runs its forward once more as plain
// operations on aliases of its inputs, and lets autograd write that backward pass. Aliases, because an input may depend on
// another one (the head's weight is also the embedding), and the gradients wanted here are those of the node alone.
bool wantsGraph() { return at::GradMode::is_enabled(); }
Tensor viewOf(const Tensor& t) { return t.defined() ? t.view_as(t) : t; }
// d(outs)/d(inputs) applied to `grads`; undefined for inputs that need no gradient.
variable_list recorded(const variable_list& outs, const variable_list& grads, const variable_list& inputs) {
  variable_list o, g, wanted, result(inputs.size());
  for (size_t i = 0; i < outs.size(); ++i)
    if (outs[i].requires_grad() && grads[i].defined()) {
      o.push_back(outs[i]);
      g.push_back(grads[i]);
    }
  for (const Tensor& t : inputs)
    if (t.defined() && t.requires_grad()) wanted.push_back(t);
  if (o.empty() || wanted.empty()) return result;
  const variable_list got = torch::autograd::grad(o, wanted, g, true, true, true);
  for (size_t i = 0, k = 0; i < inputs.size(); ++i)
    if (inputs[i].defined() && inputs[i].requires_grad()) result[i] = got[k++];
  return result;
}
Tensor plus(const Tensor& a, const Tensor& b) { return a.defined() ? (b.defined() ? a + b : a) : b; }

// Whether any of the inputs [from, to] of a node (its tensors in order, absent ones not counted) is to get a gradient: the
// products of frozen weights are left out.
bool needed(AutogradContext* ctx, size_t from, size_t to) {
  for (size_t i = from; i <= to; ++i)
    if (ctx->needs_input_grad(i)) return true;
  return false;
}
bool needed(AutogradContext* ctx, size_t i) { return needed(ctx, i, i); }

// Column-sum partials collected over a backward pass and added up in one launch.
class Columns {
 public:
  explicit Columns(const Tensor& like) : like_(like) {}
  Tensor add(const float* src, int rows, int64_t width) {
    Tensor out = at::empty({width}, like_.options());
    segs_[n_++] = {src, out.data_ptr(), rows, (int)width};
    return out;
  }
  void finish() { ok(train::finishColumns(code(like_), segs_, n_, streamOf(like_)), "column sums"); }

 private:
  Tensor like_;
  train::ColSegment segs_[train::kMaxColSegments];
  int n_ = 0;
};

struct Normed {
  Tensor sum, out, mean, rstd;
};
// Layer norm of x + y (y may be undefined). Forward stays with torch's kernels: their results are what the layers above
// see, and a 24-layer model turns a last-bit difference in one mean into rounding noise everywhere.
Normed normForward(const Tensor& x, const Tensor& y, const Tensor& gamma, const Tensor& beta, double eps) {
  Normed r;
  r.sum = y.defined() ? at::add(x, y) : x;
  std::tie(r.out, r.mean, r.rstd) = at::native_layer_norm(r.sum, {x.size(-1)}, gamma, beta, eps);
  return r;
}
// Returns dx; `partials` becomes [3][parts][width].
Tensor normBackward(const Tensor& dh, const Tensor& x_, const Tensor& mean, const Tensor& rstd, const Tensor& gamma_, const Tensor& residual,
                    bool dx_sums, Tensor* partials, int* parts) {
  const Tensor x = dense(x_), gamma = dense(gamma_);
  const int64_t width = x.size(-1), rows = x.numel() / width;
  *parts = train::layerNormPartials(rows);
  *partials = floats(x, {3, *parts, width});
  Tensor dx = at::empty_like(x);
  ok(train::layerNormBackward(code(x), dh.data_ptr(), x.data_ptr(), mean.data_ptr<float>(), rstd.data_ptr<float>(), gamma.data_ptr(),
                              residual.defined() ? residual.data_ptr() : nullptr, dx.data_ptr(), dx_sums, partials->data_ptr<float>(), rows, (int)width,
                              streamOf(x)),
     "layer norm backward");
  return dx;
}

class AddNorm : public torch::autograd::Function<AddNorm> {
 public:
  static Variable forward(AutogradContext* ctx, const Variable& x_, const std::optional<Variable>& y_, const Variable& gamma, const Variable& beta, double eps) {
    c10::cuda::CUDAGuard dg(x_.device());
    const Tensor x = dense(x_), y = y_ ? dense(*y_) : Tensor();
    Normed n = normForward(x, y, gamma, beta, eps);
    ctx->save_for_backward({n.sum, n.mean, n.rstd, gamma, x_, y_ ? *y_ : Tensor(), beta});
    ctx->saved_data["y"] = y.defined();
    ctx->saved_data["eps"] = eps;
    return n.out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    c10::cuda::CUDAGuard dg(s[0].device());
    if (wantsGraph()) {
      const Tensor gamma = viewOf(s[3]), x = viewOf(s[4]), y = viewOf(s[5]), beta = viewOf(s[6]);
      variable_list r = recorded({at::layer_norm(plus(x, y), {x.size(-1)}, gamma, beta, ctx->saved_data["eps"].toDouble())}, g, {x, y, gamma, beta});
      r.emplace_back();
      return r;
    }
    Tensor parts;
    int np;
    const int64_t w = s[0].size(-1);
    Tensor dx = normBackward(dense(g[0]), s[0], s[1], s[2], s[3], Tensor(), false, &parts, &np);
    Columns cols(s[3]);
    const float* p = parts.data_ptr<float>();
    Tensor dgamma = cols.add(p, np, w), dbeta = cols.add(p + np * w, np, w);
    cols.finish();
    return {dx, ctx->saved_data["y"].toBool() ? dx : Tensor(), dgamma, dbeta, Tensor()};
  }
};

class BlockPre : public torch::autograd::Function<BlockPre> {
 public:
  static variable_list forward(AutogradContext* ctx, const Variable& x_, const std::optional<Variable>& y_, const Variable& gamma, const Variable& beta,
                               const Variable& w, const Variable& b, int64_t heads, double eps) {
    c10::cuda::CUDAGuard dg(x_.device());
    const Tensor x = dense(x_), y = y_ ? dense(*y_) : Tensor();
    const int64_t batch = x.size(0), seq = x.size(1), width = x.size(2), hd = w.size(0) / 3 / heads;
    Normed n = normForward(x, y, gamma, beta, eps);
    const Tensor h = n.out.view({-1, width});
    const Tensor qkv = at::addmm(b, h, w.t()).view({batch, seq, 3, heads, hd}).permute({2, 0, 3, 1, 4});
    ctx->save_for_backward({n.sum, n.mean, n.rstd, gamma, h, w, beta, b});
    ctx->saved_data["y"] = y.defined();
    ctx->saved_data["eps"] = eps;
    return {n.sum, qkv[0], qkv[1], qkv[2]};   // without y the sum is the input itself
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &gamma = s[3], &h = s[4], &w = s[5];
    c10::cuda::CUDAGuard dg(x.device());
    const int64_t batch = x.size(0), seq = x.size(1), width = x.size(2);
    const int64_t heads = g[1].size(1), hd = g[1].size(3), rows = batch * seq, n3 = 3 * heads * hd;
    if (wantsGraph()) {
      const variable_list in = {viewOf(x), viewOf(gamma), viewOf(s[6]), viewOf(w), viewOf(s[7])};
      const Tensor n = at::layer_norm(in[0], {width}, in[1], in[2], ctx->saved_data["eps"].toDouble());
      const Tensor qkv = at::linear(n, in[3], in[4]).view({batch, seq, 3, heads, hd}).permute({2, 0, 3, 1, 4});
      const variable_list r = recorded({qkv[0], qkv[1], qkv[2]}, {g[1], g[2], g[3]}, in);
      const Tensor dx = plus(g[0], r[0]);
      return {dx, ctx->saved_data["y"].toBool() ? dx : Tensor(), r[1], r[2], r[3], r[4], Tensor(), Tensor()};
    }
    Tensor dqkv = at::empty({rows, n3}, x.options());
    const int sp = train::stripPartials(rows);
    Tensor bias_parts = floats(x, {sp, n3});
    train::Strided4 gs[3];
    Tensor keep[3];
    for (int i = 0; i < 3; ++i) {
      Tensor t = g[1 + i];
      if (t.stride(3) != 1 || t.stride(0) % 8 || t.stride(1) % 8 || t.stride(2) % 8 || ((uintptr_t)t.data_ptr() & 15)) t = t.contiguous();
      keep[i] = t;
      gs[i] = {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
    }
    ok(train::packQkvGradient(code(x), gs, dqkv.data_ptr(), bias_parts.data_ptr<float>(), batch, seq, (int)heads, (int)hd, streamOf(x)),
       "attention gradient");
    const size_t y = ctx->saved_data["y"].toBool();
    Tensor dw, dx, dgamma, dbeta, parts;
    if (needed(ctx, 3 + y)) dw = at::mm(dqkv.t(), h);
    Columns cols(gamma);
    if (needed(ctx, 0, 2 + y)) {
      int np;
      dx = normBackward(at::mm(dqkv, w), x, s[1], s[2], gamma, dense(g[0]), false, &parts, &np);
      const float* p = parts.data_ptr<float>();
      dgamma = cols.add(p, np, width);
      dbeta = cols.add(p + np * width, np, width);
    }
    Tensor db = cols.add(bias_parts.data_ptr<float>(), sp, n3);
    cols.finish();
    return {dx, ctx->saved_data["y"].toBool() ? dx : Tensor(), dgamma, dbeta, dw, db, Tensor(), Tensor()};
  }
};

// Products with gelu, or its gradient, in the own kernel's epilogue. `out` [groups][n][m] or [n][m]; see GemmSpec.
train::GemmSpec product(const Tensor& a, bool a_mn, const Tensor& b, bool b_mn, const Tensor& out, int64_t k, int ragged = train::kGemmWhole,
                        int epilogue = train::kGemmStore, const Tensor& aux = Tensor()) {
  return {a.data_ptr(), b.data_ptr(), out.data_ptr(), aux.defined() ? aux.data_ptr() : nullptr, (int)out.size(-1), (int)out.size(-2), (int)k,
          a_mn, b_mn, ragged, epilogue};
}
void products(const train::GemmSpec* specs, int n, const Tensor& like, const Tensor& count = Tensor()) {
  ok(train::expertGemm(code(like), specs, n, like.dim() == 3 ? (int)like.size(0) : 1, count.defined() ? count.data_ptr<int>() : nullptr, streamOf(like)),
     "grouped product");
}
// What the own kernel takes of an operand besides its place: anything else is left to the library, errors among it.
bool operand(const Tensor& t, const Tensor& like, at::IntArrayRef sizes) {
  return t.sizes() == sizes && t.scalar_type() == like.scalar_type() && t.device() == like.device() && t.layout() == at::kStrided;
}
bool captured(const Tensor& t) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(streamOf(t), &status) == cudaSuccess && status != cudaStreamCaptureStatusNone;
}
// `alone`: nothing else holds multiprocessors for long while the call runs. A product's tiles are dealt out beforehand to as many CTAs as
// an empty GPU holds, one per multiprocessor; those that find theirs taken start when the others are done. Beside a kernel on 16 (32) of
// them, us own / library: a block's second half forward 241 / 204 (294 / 280), backward 388 / 343 (521 / 499), experts of 8 x 1024 x 1024 x 4096
// forward 198 / 146 (216 / 206), backward 347 / 280 (372 / 382); alone 179 / 194, 304 / 323, 134 / 140, 220 / 267. Gradient
// all-reduces of a job of several ranks are such kernels.
bool ownExperts(const Tensor& h, const Tensor& w1, const Tensor& w2, bool alone) {
  if (!alone || h.dim() != 3 || w1.dim() != 3 || !h.is_cuda() || (h.scalar_type() != at::kBFloat16 && h.scalar_type() != at::kHalf)) return false;
  const int64_t experts = h.size(0), width = h.size(2), hidden = w1.size(2);
  return operand(w1, h, {experts, width, hidden}) && operand(w2, h, {experts, hidden, width}) &&
         train::expertGemmPays(experts * h.size(1), width, hidden, captured(h)) && train::gemmRuns(code(h));
}
// The first product of a block's MLP, or gelu's gradient with the product before it: `weight` and `matrix` are its operands, the result [rows][hidden].
bool ownMlp(const Tensor& matrix, const Tensor& weight, at::IntArrayRef sizes, int64_t rows, int64_t width, int64_t hidden, bool alone) {
  return alone && matrix.is_cuda() && operand(weight, matrix, sizes) && train::mlpGemmPays(rows, width, hidden) && train::gemmRuns(code(matrix));
}

class BlockPost : public torch::autograd::Function<BlockPost> {
 public:
  static variable_list forward(AutogradContext* ctx, const Variable& x_, const Variable& a_, const Variable& wp, const Variable& bp,
                               const Variable& gamma, const Variable& beta, const Variable& wf, const Variable& bf, const Variable& wo,
                               const Variable& bo, double eps, bool alone) {
    c10::cuda::CUDAGuard dg(x_.device());
    const Tensor x = dense(x_), a = rowsOf(a_);
    const int64_t width = x.size(-1);
    const Tensor p = at::addmm(bp, a, wp.t());
    Normed n = normForward(x, p.view(x.sizes()), gamma, beta, eps);
    const Tensor h = n.out.view({-1, width});
    Tensor u, act;
    if (wf.dim() == 2 && operand(bf, h, {wf.size(0)}) && ownMlp(h, wf, {wf.size(0), width}, h.size(0), width, wf.size(0), alone)) {
      u = at::empty({h.size(0), wf.size(0)}, h.options());
      act = at::empty_like(u);
      const Tensor w = dense(wf), bias = bf.contiguous();
      train::GemmSpec p = product(w, false, h, false, u, width, train::kGemmWhole, train::kGemmGelu, act);
      p.bias = bias.data_ptr();
      products(&p, 1, h);
    } else {
      u = at::addmm(bf, h, wf.t());
      act = at::empty_like(u);
      ok(train::geluForward(code(u), u.data_ptr(), act.data_ptr(), u.numel(), streamOf(u)), "gelu");
    }
    const Tensor y = at::addmm(bo, act, wo.t()).view(x.sizes());
    ctx->save_for_backward({a_, wp, n.sum, n.mean, n.rstd, gamma, h, wf, u, act, wo, beta, bf, bo});
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["alone"] = alone;
    return {n.sum, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &wp = s[1], &x2 = s[2], &gamma = s[5], &h = s[6], &wf = s[7], &act = s[9], &wo = s[10];
    c10::cuda::CUDAGuard dg(x2.device());
    const int64_t width = x2.size(-1), rows = x2.numel() / width;
    if (wantsGraph()) {
      const variable_list in = {viewOf(x2), viewOf(gamma), viewOf(s[11]), viewOf(wf), viewOf(s[12]), viewOf(wo), viewOf(s[13])};
      const Tensor n = at::layer_norm(in[0], {width}, in[1], in[2], ctx->saved_data["eps"].toDouble());
      const variable_list r = recorded({at::linear(at::gelu(at::linear(n, in[3], in[4]), "tanh"), in[5], in[6])}, {g[1]}, in);
      const Tensor dx = plus(g[0], r[0]), d = dx.reshape({rows, width}), a = s[0].reshape({rows, -1});
      return {dx, at::mm(d, wp).view(s[0].sizes()), at::mm(d.t(), a), d.sum(0), r[1], r[2], r[3], r[4], r[5], r[6], Tensor(), Tensor()};
    }
    const Tensor a = rowsOf(s[0]), u = dense(s[8]);
    const int64_t hidden = u.size(1);
    const int dt = code(x2), sp = train::stripPartials(rows);
    cudaStream_t st = streamOf(x2);
    TORCH_CHECK(g[1].defined(), "hylink: the block's branch has no gradient");
    const Tensor gy = rowsOf(g[1]);
    const bool own = operand(u, gy, {rows, hidden}) && ownMlp(gy, wo, {width, hidden}, rows, width, hidden, ctx->saved_data["alone"].toBool());
    const int fcp = own ? train::gemmPartials(rows) : sp;
    Tensor out_parts = floats(x2, {sp, width}), fc_parts = floats(x2, {fcp, hidden}), parts;
    Tensor dwo, dwf, dwp, da, dx, dgamma, dbeta, dbp, dbf;
    Columns cols(gamma);
    ok(train::columnSums(dt, gy.data_ptr(), out_parts.data_ptr<float>(), rows, (int)width, st), "bias gradient");
    Tensor dbo = cols.add(out_parts.data_ptr<float>(), sp, width);
    if (needed(ctx, 8)) dwo = at::mm(gy.t(), act);
    if (needed(ctx, 0, 7)) {
      Tensor du = at::empty_like(u);
      if (own) {
        const Tensor w = dense(wo);
        train::GemmSpec p = product(w, true, gy, false, du, width, train::kGemmWhole, train::kGemmGeluGradient, u);
        p.columns = fc_parts.data_ptr<float>();
        products(&p, 1, gy);
      } else {
        const Tensor dact = at::mm(gy, wo);
        ok(train::geluBackward(dt, dact.data_ptr(), u.data_ptr(), du.data_ptr(), fc_parts.data_ptr<float>(), rows, (int)hidden, st), "gelu backward");
      }
      dbf = cols.add(fc_parts.data_ptr<float>(), fcp, hidden);
      if (needed(ctx, 6)) dwf = at::mm(du.t(), h);
      if (needed(ctx, 0, 5)) {
        int np;
        dx = normBackward(at::mm(du, wf), x2, s[3], s[4], gamma, dense(g[0]), true, &parts, &np);
        const Tensor dxr = dx.view({rows, width});
        if (needed(ctx, 2)) dwp = at::mm(dxr.t(), a);
        if (needed(ctx, 1)) da = at::mm(dxr, wp).view(s[0].sizes());
        const float* p = parts.data_ptr<float>();
        dgamma = cols.add(p, np, width);
        dbeta = cols.add(p + np * width, np, width);
        dbp = cols.add(p + 2 * np * width, np, width);
      }
    }
    cols.finish();
    return {dx, da, dwp, dbp, dgamma, dbeta, dwf, dbf, dwo, dbo, Tensor(), Tensor()};
  }
};

// logits = h W^T and their mean cross entropy. The vocabulary is padded to a multiple of 64: an odd leading dimension
// keeps cuBLAS off the tensor-memory kernels (8192 x 50257 x 1024 in bf16 on B200: 7.43 ms against 0.60 for the logits,
// 4.71 against 0.55 for the weight gradient); padding the weight is a copy of 0.04 ms.
// The input gradient sums over the vocabulary. While torch allows reduced-precision reductions (its default) and the
// vocabulary is no multiple of eight, that sum is the library's product over exactly the vocabulary, as the plain modules
// call it: its rounding is part of what a training run with them gives. Switched off, or with an even vocabulary, it is
// one pass over the padded operands (zero behind the vocabulary on both sides), summed in fp32 and rounded once.
// 8192 x 50257 x 1024: 5.6 ms against 0.56. The padded pass everywhere would be nearer to fp32 (first-step gradients of
// the 24-layer model 1.37e-2 from an fp32 model, 1.71e-2 with the plain modules), but from the second step on its
// gradients are 3 % away from those of the plain modules, where two runs of these differ by 0.8 %.
bool reducedPrecisionSums(at::ScalarType t) {
  const auto& ctx = at::globalContext();
  return (t == at::kBFloat16 ? ctx.allowBF16ReductionCuBLAS() : ctx.allowFP16ReductionCuBLAS()) == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK;
}
// d [rows][padded], zero behind `vocab`; w [padded][width].
Tensor headInputGradient(const Tensor& d, const Tensor& w, int64_t vocab) {
  if (vocab % 8 == 0 || !reducedPrecisionSums(d.scalar_type())) return at::mm(d, w);
  return at::mm(d.narrow(1, 0, vocab), w.narrow(0, 0, vocab));
}

class HeadLoss : public torch::autograd::Function<HeadLoss> {
 public:
  static Variable forward(AutogradContext* ctx, const Variable& h_, const Variable& w, const Variable& targets_) {
    c10::cuda::CUDAGuard dg(h_.device());
    const Tensor h = rowsOf(h_), targets = targets_.reshape({-1}).contiguous();
    const int64_t vocab = w.size(0), padded = (vocab + 63) / 64 * 64, rows = h.size(0);
    TORCH_CHECK_VALUE(targets.scalar_type() == at::kLong && targets.device() == h.device() && targets.numel() == rows, "hylink: ", rows,
                      " rows and ", targets.numel(), " targets");
    Tensor wpad = w;
    if (padded != vocab || !w.is_contiguous()) {
      wpad = at::empty({padded, w.size(1)}, w.options());
      wpad.narrow(0, 0, vocab).copy_(w);
      if (padded != vocab) wpad.narrow(0, vocab, padded - vocab).zero_();
    }
    Tensor logits = at::mm(h, wpad.t());
    Tensor lse = floats(h, {rows}), row_loss = floats(h, {rows}), loss = floats(h, {2});
    ok(train::crossEntropyForward(code(h), logits.data_ptr(), padded, targets.data_ptr<int64_t>(), rows, (int)vocab, -100, lse.data_ptr<float>(),
                                  row_loss.data_ptr<float>(), loss.data_ptr<float>(), streamOf(h)),
       "cross entropy");
    ctx->save_for_backward({h_, wpad, targets, logits, lse, loss, w});
    return loss.select(0, 0).clone();
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &wpad = s[1], &targets = s[2], &lse = s[4], &loss = s[5];
    c10::cuda::CUDAGuard dg(s[0].device());
    const int64_t vocab = s[6].size(0);
    if (wantsGraph()) {
      const variable_list in = {viewOf(s[0]), viewOf(s[6])};
      const Tensor z = at::linear(in[0], in[1]).to(at::kFloat).reshape({-1, vocab});
      variable_list r = recorded({at::cross_entropy_loss(z, targets, {}, at::Reduction::Mean, -100)}, g, in);
      r.emplace_back();
      return r;
    }
    const Tensor h = rowsOf(s[0]), logits = dense(s[3]);
    const Tensor grad = g[0].to(at::kFloat).contiguous();
    Tensor dlogits = at::empty_like(logits);
    ok(train::crossEntropyBackward(code(h), logits.data_ptr(), logits.size(1), targets.data_ptr<int64_t>(), h.size(0), (int)vocab, -100,
                                   lse.data_ptr<float>(), loss.data_ptr<float>(), grad.data_ptr<float>(), dlogits.data_ptr(), streamOf(h)),
       "cross entropy backward");
    Tensor dw, dh;
    if (needed(ctx, 1)) dw = at::mm(dlogits.narrow(1, 0, vocab).t(), h);
    if (needed(ctx, 0)) dh = headInputGradient(dlogits, wpad, vocab).view(s[0].sizes());
    return {dh, dw, Tensor()};
  }
};

// ---- top-1 mixture of experts
struct Routed {
  Tensor logits, expert, gate, row_of, token_of, count, send;
};
Routed moeRouted(const Tensor& x, const Tensor& router, int64_t capacity) {
  const int64_t tokens = x.size(0), width = x.size(1), experts = router.size(0);
  const auto ints = x.options().dtype(at::kInt);
  Routed r;
  r.logits = at::mm(x, router.t());
  r.expert = at::empty({tokens}, ints);
  r.row_of = at::empty({tokens}, ints);
  r.token_of = at::empty({experts * capacity}, ints);
  r.count = at::empty({experts}, ints);
  r.gate = floats(x, {tokens});
  r.send = at::empty({experts * capacity, width}, x.options());
  ok(train::moeRoute(code(x), r.logits.data_ptr(), (int)tokens, (int)experts, (int)capacity, r.expert.data_ptr<int>(), r.gate.data_ptr<float>(),
                     r.row_of.data_ptr<int>(), r.token_of.data_ptr<int>(), r.count.data_ptr<int>(), streamOf(x)),
     "MoE routing");
  ok(train::moeGather(x.data_ptr(), r.token_of.data_ptr<int>(), r.send.data_ptr(), (int)(experts * capacity), (int)width, streamOf(x)), "MoE dispatch");
  return r;
}
// {dx, drouter (where it is needed)}; dres may be undefined.
std::pair<Tensor, Tensor> moeRoutedBackward(const Tensor& x, const Tensor& router_, const Tensor& logits, const Tensor& expert, const Tensor& gate,
                                            const Tensor& row_of, const Tensor& dres, const Tensor& dsend, const Tensor& dgate, bool router_needed) {
  const Tensor router = dense(router_);
  const int64_t tokens = x.size(0), width = x.size(1), experts = router.size(0);
  Tensor dx = at::empty_like(x);
  if (router_needed && tokens > 0 && train::moeTokensAndRouterFits((int)experts)) {   // (no tokens: a gradient of zeros, by the product below)
    const int parts = train::moeRouterPartials((int)tokens);
    Tensor partials = floats(x, {parts, experts * width});
    ok(train::moeTokensAndRouter(code(x), dres.defined() ? dres.data_ptr() : nullptr, dsend.data_ptr(), row_of.data_ptr<int>(), logits.data_ptr(),
                                 expert.data_ptr<int>(), gate.data_ptr<float>(), dgate.data_ptr<float>(), router.data_ptr(), x.data_ptr(), dx.data_ptr(),
                                 partials.data_ptr<float>(), (int)tokens, (int)width, (int)experts, streamOf(x)),
       "MoE token gradient");
    Columns cols(x);
    Tensor drouter = cols.add(partials.data_ptr<float>(), parts, experts * width).view({experts, width});
    cols.finish();
    return {dx, drouter};
  }
  Tensor dlogits = at::empty_like(logits);
  ok(train::moeTokenGradient(code(x), dres.defined() ? dres.data_ptr() : nullptr, dsend.data_ptr(), row_of.data_ptr<int>(), logits.data_ptr(),
                             expert.data_ptr<int>(), gate.data_ptr<float>(), dgate.data_ptr<float>(), router.data_ptr(), dx.data_ptr(),
                             dlogits.data_ptr(), (int)tokens, (int)width, (int)experts, streamOf(x)),
     "MoE token gradient");
  if (!train::moeRouterFits((int)experts)) dx.addmm_(dlogits, router);
  return {dx, router_needed ? at::mm(dlogits.t(), x) : Tensor()};
}
struct Expert {
  Tensor u, act, out;
  bool own = false;   // by the own products: the backward pass follows, whatever it would choose itself
};
// h: [experts][rows][width]. `count`: rows of each expert in use (the others are zeros), undefined where that is not known; results
// of rows out of use may be anything then.
Expert moeExpert(const Tensor& h_, const Tensor& w1_, const Tensor& w2_, const Tensor& count, bool alone) {
  Expert e;
  if ((e.own = ownExperts(h_, w1_, w2_, alone))) {
    const Tensor h = dense(h_), w1 = dense(w1_), w2 = dense(w2_);
    e.u = at::empty({h.size(0), h.size(1), w1.size(2)}, h.options());
    e.act = at::empty_like(e.u);
    e.out = at::empty_like(h);
    const train::GemmSpec first = product(w1, true, h, false, e.u, h.size(2), train::kGemmRaggedN, train::kGemmGelu, e.act);
    products(&first, 1, h, count);
    const train::GemmSpec second = product(w2, true, e.act, false, e.out, w1.size(2), train::kGemmRaggedN);
    products(&second, 1, h, count);
    return e;
  }
  e.u = at::bmm(h_, w1_);
  e.act = at::empty_like(e.u);
  ok(train::geluForward(code(e.u), e.u.data_ptr(), e.act.data_ptr(), e.u.numel(), streamOf(e.u)), "gelu");
  e.out = at::bmm(e.act, w2_);
  return e;
}
// {dh, dw1, dw2}, those that are needed
variable_list moeExpertBackward(const Tensor& h_, const Tensor& w1_, const Tensor& w2_, const Tensor& u_, const Tensor& act_, const Tensor& dout_,
                                bool own, const Tensor& count, bool h_needed, bool w1_needed, bool w2_needed) {
  Tensor dh, dw1, dw2;
  if (own) {
    // nothing else looks at these between the hooks that gave them back and the kernel
    const bool fit = h_.dim() == 3 && w1_.dim() == 3 && operand(h_, dout_, dout_.sizes()) && operand(w1_, h_, {h_.size(0), h_.size(2), w1_.size(2)}) &&
                     operand(w2_, h_, {h_.size(0), w1_.size(2), h_.size(2)}) && operand(u_, h_, {h_.size(0), h_.size(1), w1_.size(2)}) &&
                     operand(act_, h_, u_.sizes()) &&
                     (!count.defined() || (count.scalar_type() == at::kInt && count.device() == h_.device() && count.numel() == h_.size(0) && count.is_contiguous()));
    TORCH_CHECK(fit, "hylink: the experts' saved tensors have come back with other sizes, types or places");
    const Tensor h = dense(h_), w1 = dense(w1_), w2 = dense(w2_), u = dense(u_), act = dense(act_), dout = dense(dout_);
    const int64_t rows = h.size(1), width = h.size(2), hidden = w1.size(2);
    train::GemmSpec specs[2];
    int n = 0;
    Tensor du;
    if (h_needed || w1_needed) {
      du = at::empty_like(u);
      specs[n++] = product(w2, false, dout, false, du, width, train::kGemmRaggedN, train::kGemmGeluGradient, u);
    }
    if (w2_needed) {
      dw2 = at::empty_like(w2);
      specs[n++] = product(dout, true, act, true, dw2, rows, train::kGemmRaggedK);
    }
    if (n) products(specs, n, h, count);
    n = 0;
    if (h_needed) {                                  // the longer tiles first
      dh = at::empty_like(h);
      specs[n++] = product(w1, false, du, false, dh, hidden, train::kGemmRaggedN);
    }
    if (w1_needed) {
      dw1 = at::empty_like(w1);
      specs[n++] = product(du, true, h, true, dw1, rows, train::kGemmRaggedK);
    }
    if (n) products(specs, n, h, count);
    return {dh, dw1, dw2};
  }
  if (w2_needed) dw2 = at::bmm(act_.transpose(1, 2), dout_);
  if (h_needed || w1_needed) {
    Tensor dact = at::bmm(dout_, w2_.transpose(1, 2));
    const Tensor u = dense(u_);
    Tensor du = at::empty_like(u);
    ok(train::geluBackward(code(u), dact.data_ptr(), u.data_ptr(), du.data_ptr(), nullptr, u.size(0) * u.size(1), (int)u.size(2), streamOf(u)),
       "gelu backward");
    if (w1_needed) dw1 = at::bmm(h_.transpose(1, 2), du);
    if (h_needed) dh = at::bmm(du, w1_.transpose(1, 2));
  }
  return {dh, dw1, dw2};
}
Tensor moeCombined(const Tensor& x, const Tensor& gate, const Tensor& rows, const Tensor& row_of) {
  Tensor y = at::empty_like(x);
  ok(train::moeCombine(code(x), x.data_ptr(), gate.data_ptr<float>(), rows.data_ptr(), row_of.data_ptr<int>(), y.data_ptr(), (int)x.size(0),
                       (int)x.size(1), streamOf(x)),
     "MoE combine");
  return y;
}
// {drows, dgate}; with `whole`, dgate is zero for tokens without a row, which matters where it leaves this file: autograd's anomaly
// check and hooks read all of it
std::pair<Tensor, Tensor> moeCombinedBackward(const Tensor& dy, const Tensor& gate, const Tensor& rows, const Tensor& token_of, bool whole = true) {
  Tensor drows = at::empty_like(rows), dgate = whole ? at::zeros_like(gate) : at::empty_like(gate);
  const int width = (int)rows.size(-1);
  ok(train::moeRowGradient(code(rows), dy.data_ptr(), gate.data_ptr<float>(), rows.data_ptr(), token_of.data_ptr<int>(), drows.data_ptr(),
                           dgate.data_ptr<float>(), (int)(rows.numel() / width), width, streamOf(rows)),
     "MoE row gradient");
  return {drows, dgate};
}

// The same as plain operations, for a recorded backward pass: with the routing as it was chosen.
Tensor plainGate(const Tensor& x, const Tensor& router, const Tensor& expert) {
  return at::softmax(at::linear(x, router).to(at::kFloat), -1).gather(1, expert.to(at::kLong).unsqueeze(1)).squeeze(1);
}
Tensor plainRows(const Tensor& from, const Tensor& index) {
  const Tensor i = index.to(at::kLong);
  return from.index_select(0, i.clamp_min(0)).masked_fill((i < 0).unsqueeze(1), 0);
}
Tensor plainExperts(const Tensor& h, const Tensor& w1, const Tensor& w2) { return at::bmm(at::gelu(at::bmm(h, w1), "tanh"), w2); }
Tensor plainCombined(const Tensor& x, const Tensor& gate, const Tensor& rows, const Tensor& row_of) {
  return x + gate.unsqueeze(1).to(x.scalar_type()) * plainRows(rows.reshape({-1, x.size(1)}), row_of);
}

// The whole layer where the experts are all here: one node instead of a dozen. (Host time of a layer of 1072 tokens,
// forward and backward: 300 us in pieces, 210 in one.)
class MoeLayer : public torch::autograd::Function<MoeLayer> {
 public:
  static Variable forward(AutogradContext* ctx, const Variable& x_, const Variable& router, const Variable& w1, const Variable& w2, int64_t capacity,
                          bool alone) {
    c10::cuda::CUDAGuard dg(x_.device());
    const Tensor x = dense(x_);
    const Routed r = moeRouted(x, router, capacity);
    const Tensor h = r.send.view({router.size(0), capacity, x.size(1)});
    // Hooks on saved tensors see all of them, and may scale what they keep by its largest value: rows out of use are computed then (zeros).
    const Tensor count = at::SavedTensorDefaultHooks::get_hooks() ? Tensor() : r.count;
    const Expert e = moeExpert(h, w1, w2, count, alone);
    ctx->save_for_backward({x_, router, w1, w2, r.logits, r.expert, r.gate, r.row_of, r.token_of, h, e.u, e.act, e.out, count});
    ctx->saved_data["own"] = e.own;
    return moeCombined(x, r.gate, e.out, r.row_of);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &router = s[1], &w1 = s[2], &w2 = s[3], &h = s[9];
    c10::cuda::CUDAGuard dg(s[0].device());
    if (wantsGraph()) {
      const variable_list in = {viewOf(s[0]), viewOf(router), viewOf(w1), viewOf(w2)};
      const Tensor out = plainExperts(plainRows(in[0], s[8]).view(h.sizes()), in[2], in[3]);
      variable_list r = recorded({plainCombined(in[0], plainGate(in[0], in[1], s[5]), out, s[7])}, g, in);
      r.resize(6);
      return r;
    }
    const Tensor x = dense(s[0]), rows = dense(s[12]);
    const Tensor dy = dense(g[0]);
    const auto [drows, dgate] = moeCombinedBackward(dy, s[6], rows, s[8], false);
    const variable_list e = moeExpertBackward(h, w1, w2, s[10], s[11], drows, ctx->saved_data["own"].toBool(), s[13], needed(ctx, 0), needed(ctx, 2),
                                              needed(ctx, 3));
    if (!needed(ctx, 0, 1)) return {Tensor(), Tensor(), e[1], e[2], Tensor(), Tensor()};
    const Tensor dsend = e[0].defined() ? e[0] : at::zeros_like(h);   // the router alone
    const auto [dx, drouter] = moeRoutedBackward(x, router, s[4], s[5], s[6], s[7], dy, dsend, dgate, needed(ctx, 1));
    return {dx, drouter, e[1], e[2], Tensor(), Tensor()};
  }
};

// In pieces, with the tokens travelling between ranks in between. Dispatch returns x again (the residual path: its
// gradient then joins the others in one pass), the dispatch buffer, the gates, and the maps token -> row and row -> token.
class MoeDispatch : public torch::autograd::Function<MoeDispatch> {
 public:
  static variable_list forward(AutogradContext* ctx, const Variable& x_, const Variable& router, int64_t capacity) {
    c10::cuda::CUDAGuard dg(x_.device());
    const Tensor x = dense(x_);
    const Routed r = moeRouted(x, router, capacity);
    ctx->save_for_backward({x_, router, r.logits, r.expert, r.gate, r.row_of, r.token_of});
    ctx->saved_data["rows"] = router.size(0) * capacity;
    // Without a gradient for the tokens the exchange of the rows needs none either, and a rank that takes the plain path (one
    // without tokens) must find its peers in as many exchanges as it has itself.
    if (x_.requires_grad()) ctx->mark_non_differentiable({r.row_of, r.token_of});
    else ctx->mark_non_differentiable({r.row_of, r.token_of, r.send});
    ctx->set_materialize_grads(false);
    return {x, r.send, r.gate, r.row_of, r.token_of};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    c10::cuda::CUDAGuard dg(s[0].device());
    if (wantsGraph()) {
      const variable_list in = {viewOf(s[0]), viewOf(s[1])};
      const variable_list r = recorded({plainRows(in[0], s[6]), plainGate(in[0], in[1], s[3])}, {g[1], g[2]}, in);
      return {plus(g[0], r[0]), r[1], Tensor()};
    }
    const Tensor x = dense(s[0]), &gate = s[4];
    const Tensor dres = g[0].defined() ? dense(g[0]) : Tensor();
    const Tensor dsend = g[1].defined() ? dense(g[1]) : at::zeros({ctx->saved_data["rows"].toInt(), x.size(1)}, x.options());
    const Tensor dgate = g[2].defined() ? dense(g[2]) : at::zeros_like(gate);
    const auto [dx, drouter] = moeRoutedBackward(x, s[1], s[2], s[3], gate, s[5], dres, dsend, dgate, needed(ctx, 1));
    return {dx, drouter, Tensor()};
  }
};

// out = gelu(h W1) W2, per expert.
class MoeExperts : public torch::autograd::Function<MoeExperts> {
 public:
  static Variable forward(AutogradContext* ctx, const Variable& h, const Variable& w1, const Variable& w2, bool alone) {
    c10::cuda::CUDAGuard dg(h.device());
    const Expert e = moeExpert(h, w1, w2, Tensor(), alone);
    ctx->save_for_backward({h, w1, w2, e.u, e.act});
    ctx->saved_data["own"] = e.own;
    return e.out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    c10::cuda::CUDAGuard dg(s[0].device());
    if (wantsGraph()) {
      const variable_list in = {viewOf(s[0]), viewOf(s[1]), viewOf(s[2])};
      variable_list r = recorded({plainExperts(in[0], in[1], in[2])}, g, in);
      r.emplace_back();
      return r;
    }
    variable_list r = moeExpertBackward(s[0], s[1], s[2], s[3], s[4], dense(g[0]), ctx->saved_data["own"].toBool(), Tensor(), needed(ctx, 0),
                                        needed(ctx, 1), needed(ctx, 2));
    r.emplace_back();
    return r;
  }
};

// y = x + gate * rows[row_of] for the tokens that have a row.
class MoeCombine : public torch::autograd::Function<MoeCombine> {
 public:
  static Variable forward(AutogradContext* ctx, const Variable& x_, const Variable& gate, const Variable& rows_, const Variable& row_of,
                          const Variable& token_of) {
    c10::cuda::CUDAGuard dg(x_.device());
    const Tensor x = dense(x_), rows = dense(rows_);
    ctx->save_for_backward({gate, rows_, token_of, row_of});
    return moeCombined(x, gate, rows, row_of);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    c10::cuda::CUDAGuard dg(s[1].device());
    if (wantsGraph()) {
      const variable_list in = {viewOf(s[0]), viewOf(s[1])};
      const variable_list r = recorded({plainCombined(at::zeros_like(g[0]), in[0], in[1], s[3])}, g, in);
      return {g[0], r[0], r[1], Tensor(), Tensor()};
    }
    const Tensor dy = dense(g[0]);
    const auto [drows, dgate] = moeCombinedBackward(dy, s[0], dense(s[1]), s[2]);
    return {dy, dgate, drows, Tensor(), Tensor()};
  }
};

// Whether anything hangs on the nodes that accumulate these parameters' gradients (a recorded step would not call it).
bool accumulationHooks(const std::vector<Tensor>& params) {
  for (const Tensor& p : params) {
    const auto node = torch::autograd::impl::try_get_grad_accumulator(p);
    if (node && !(node->pre_hooks().empty() && node->post_hooks().empty() && node->tensor_pre_hooks().empty())) return true;
  }
  return false;
}

// One AdamW step on lists of tensors. False (and nothing done) unless all are contiguous CUDA tensors of one type that
// the kernel takes.
bool multiAdamW(const std::vector<Tensor>& weights, const std::vector<Tensor>& grads, const std::vector<Tensor>& ms, const std::vector<Tensor>& vs,
                const std::vector<Tensor>& steps, double lr, double beta1, double beta2, double decay, double eps) {
  const size_t n = weights.size();
  if (n == 0 || grads.size() != n || ms.size() != n || vs.size() != n || steps.size() != n) return false;
  const auto type = weights[0].scalar_type();
  if (type != at::kBFloat16 && type != at::kHalf && type != at::kFloat) return false;
  const c10::Device device = weights[0].device();
  std::vector<train::AdamWTensor> list(n);
  for (size_t i = 0; i < n; ++i) {
    for (const Tensor* t : {&weights[i], &grads[i], &ms[i], &vs[i]})
      if (t->device() != device || !device.is_cuda() || t->scalar_type() != type || t->layout() != at::kStrided || !t->is_contiguous() ||
          t->numel() != weights[i].numel())
        return false;
    if (steps[i].device() != device || steps[i].scalar_type() != at::kFloat || steps[i].numel() != 1) return false;
    list[i] = {weights[i].data_ptr(), ms[i].data_ptr(), vs[i].data_ptr(), grads[i].data_ptr(), steps[i].data_ptr<float>(), weights[i].numel()};
  }
  c10::cuda::CUDAGuard dg(device);
  at::_foreach_add_(steps, 1);
  ok(train::multiAdamW(type == at::kFloat ? (int)hlFloat32 : code(weights[0]), list.data(), (int)n, lr, beta1, beta2, decay, eps,
                       streamOf(weights[0])),
     "AdamW");
  for (size_t i = 0; i < n; ++i)   // autograd has to know that these were written
    for (const Tensor* t : {&weights[i], &ms[i], &vs[i]}) t->unsafeGetTensorImpl()->bump_version();
  return true;
}

// False (and nothing done) for a shard that the kernel does not take: it wants packets of contiguous CUDA tensors.
bool shardedAdamW(const Tensor& grad, const Tensor& weight, const std::optional<Tensor>& master, const Tensor& m, const Tensor& v, int64_t ranks,
                  double keep, double beta1, double beta2, double step, double correction2, double eps) {
  const int64_t n = weight.numel();
  const auto type = weight.scalar_type();
  const auto fits = [&](const Tensor& t, at::ScalarType want) {
    return t.scalar_type() == want && t.device() == weight.device() && t.layout() == at::kStrided && t.is_contiguous() && t.numel() == n && aligned(t);
  };
  if (!weight.is_cuda() || n % 8 || (type != at::kBFloat16 && type != at::kHalf && type != at::kFloat) || !fits(weight, type) || !fits(grad, type) ||
      !fits(m, at::kFloat) || !fits(v, at::kFloat) || (master && (type == at::kFloat || !fits(*master, at::kFloat))))
    return false;
  c10::cuda::CUDAGuard dg(weight.device());
  const train::AdamWArgs a = {(float)ranks, (float)keep, (float)beta1, (float)(1 - beta1), (float)beta2, (float)(1 - beta2), (float)step, (float)correction2, (float)eps};
  const int dt = weight.scalar_type() == at::kFloat ? (int)hlFloat32 : code(weight);
  ok(train::shardedAdamW(dt, grad.data_ptr(), weight.data_ptr(), master ? master->data_ptr<float>() : nullptr, m.data_ptr<float>(),
                         v.data_ptr<float>(), n, a, streamOf(weight)),
     "sharded AdamW");
  return true;
}

// ---- calls whose cost on the host is most of a small one: argument lists are taken apart here, not in Python
int typeCode(at::ScalarType t) {
  switch (t) {
    case at::kChar: return hlInt8;
    case at::kByte: return hlUint8;
    case at::kInt: return hlInt32;
    case at::kLong: return hlInt64;
    case at::kHalf: return hlFloat16;
    case at::kFloat: return hlFloat32;
    case at::kDouble: return hlFloat64;
    case at::kBFloat16: return hlBfloat16;
    default: TORCH_CHECK(false, "hylink: unsupported dtype ", t);
  }
}
// The two calls below are launches of a few microseconds, so their arguments are read by hand: through pybind11's
// converters (a vector of optional tensors, a dtype) an empty emulated collective of eight ranks took 1.4 us on the
// host, of two 0.8; read by hand 0.28 and 0.22.
template <typename F>
PyObject* native(const char* name, Py_ssize_t want, Py_ssize_t got, F&& body) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(want == got, name, " takes ", want, " arguments, not ", got);
  return PyLong_FromLong(body());
  END_HANDLE_TH_ERRORS
}
long long whole(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1. && PyErr_Occurred()) throw python_error();
  return v;
}
const Tensor& tensor(PyObject* o) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), "hylink: expected a tensor, got ", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
// A list or tuple as it is, anything else as a list of its items.
py::object sequence(PyObject* o) {
  PyObject* s = PySequence_Fast(o, "hylink: expected a sequence of tensors");
  if (!s) throw python_error();
  return py::reinterpret_steal<py::object>(s);
}

// One collective of an emulated group on the current stream; returns the library's result code. Arguments: group, ranks,
// kind, inputs, outputs, count, segment strides, wire type or None, operator, scale, root, algorithm, CTAs.
PyObject* emuRun(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  return native("emu_run", 14, nargs, [&]() -> long {
    const int nranks = (int)whole(args[1]);
    void* bufs[2][8] = {{nullptr}, {nullptr}};
    int dt[2] = {-1, -1};
    for (int k = 0; k < 2; ++k) {
      if (args[3 + k] == Py_None) continue;
      const py::object list = sequence(args[3 + k]);
      const Py_ssize_t n = PySequence_Fast_GET_SIZE(list.ptr());
      PyObject** items = PySequence_Fast_ITEMS(list.ptr());
      TORCH_CHECK(nranks <= 8 && n <= nranks, "hylink: more buffers than ranks");
      TORCH_CHECK(n > 0, "hylink: no buffers");
      dt[k] = typeCode(tensor(items[0]).scalar_type());
      for (Py_ssize_t i = 0; i < n; ++i)
        if (items[i] != Py_None) bufs[k][i] = tensor(items[i]).data_ptr();
    }
    if (dt[0] < 0) dt[0] = (int)hlFloat32;
    if (dt[1] < 0) dt[1] = dt[0];
    int wire = dt[0];
    if (args[8] != Py_None) {
      TORCH_CHECK_TYPE(THPDtype_Check(args[8]), "hylink: the wire type is a torch.dtype");
      wire = typeCode(reinterpret_cast<THPDtype*>(args[8])->scalar_type);
    }
    const hlEmu_t group = reinterpret_cast<hlEmu_t>((uintptr_t)whole(args[0]));
    const int kind = (int)whole(args[2]), op = (int)whole(args[9]), root = (int)whole(args[11]), algo = (int)whole(args[12]), ctas = (int)whole(args[13]);
    const size_t count = (size_t)whole(args[5]), in_stride = (size_t)whole(args[6]), out_stride = (size_t)whole(args[7]);
    const float scale = (float)real(args[10]);
    py::gil_scoped_release others;   // a launch waits while the stream's queue is full
    return (long)hlEmuCollective(group, kind, bufs[0], bufs[1], count, in_stride, out_stride, dt[0], dt[1], wire, op, scale, root, algo, ctas,
                                 c10::cuda::getCurrentCUDAStream().stream());
  });
}

// Destination, sources, operator, scale, accumulate, CTAs.
PyObject* reduceLanding(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  return native("reduce_landing", 6, nargs, [&]() -> long {
    const Tensor& dst = tensor(args[0]);
    TORCH_CHECK_VALUE(dst.is_cuda(), "reduce_landing needs a CUDA destination");
    const py::object list = sequence(args[1]);
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(list.ptr());
    c10::SmallVector<const void*, 8> p;
    for (Py_ssize_t i = 0; i < n; ++i) {
      const Tensor& s = tensor(PySequence_Fast_ITEMS(list.ptr())[i]);
      TORCH_CHECK_VALUE(s.numel() == dst.numel() && s.scalar_type() == dst.scalar_type(), "sources must match the destination's size and dtype");
      TORCH_CHECK_VALUE(s.is_cuda() || s.is_pinned(), "host sources must be pinned");
      p.push_back(s.data_ptr());
    }
    const int accumulate = PyObject_IsTrue(args[4]);
    if (accumulate < 0) throw python_error();
    void* const to = dst.data_ptr();
    const size_t count = (size_t)dst.numel();
    const auto type = (hlDataType_t)typeCode(dst.scalar_type());
    const auto op = (hlRedOp_t)whole(args[2]);
    const float scale = (float)real(args[3]);
    const int ctas = (int)whole(args[5]);
    py::gil_scoped_release others;
    return (long)hlReduceLanding(to, p.data(), (int)p.size(), accumulate != 0, count, type, op, scale, ctas, c10::cuda::getCurrentCUDAStream().stream());
  });
}
PyMethodDef kNativeCalls[] = {{"emu_run", (PyCFunction)(void*)emuRun, METH_FASTCALL, nullptr},
                              {"reduce_landing", (PyCFunction)(void*)reduceLanding, METH_FASTCALL, nullptr},
                              {nullptr, nullptr, 0, nullptr}};

}  // namespace

// A product whose operands never arrive, and whose waits end after this time: for tests of what is reported then.
void productWithoutOperands(const Tensor& a, double limit_ms) {
  TORCH_CHECK(a.dim() == 2 && a.is_cuda() && a.is_contiguous() && a.size(1) % 8 == 0 && a.size(0) % 8 == 0, "hylink: a matrix of whole packets");
  c10::cuda::CUDAGuard dg(a.device());
  const Tensor out = at::empty({a.size(0), a.size(0)}, a.options());
  const train::GemmSpec p = product(a, false, a, false, out, a.size(1));
  ok(train::expertGemm(code(a), &p, 1, 1, nullptr, streamOf(a), (uint64_t)(limit_ms * 1e6), false), "grouped product");
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.attr("max_norm_width") = train::kMaxNormWidth;
  m.attr("max_rows") = train::kMaxRows;
  m.def("add_norm", [](const Tensor& x, const std::optional<Tensor>& y, const Tensor& gamma, const Tensor& beta, double eps) {
    return AddNorm::apply(x, y, gamma, beta, eps);
  });
  m.def("block_pre", [](const Tensor& x, const std::optional<Tensor>& y, const Tensor& gamma, const Tensor& beta, const Tensor& w, const Tensor& b,
                        int64_t heads, double eps) { return BlockPre::apply(x, y, gamma, beta, w, b, heads, eps); });
  // `alone`: see ownExperts
  using py::arg;
  m.def("block_post", [](const Tensor& x, const Tensor& a, const Tensor& wp, const Tensor& bp, const Tensor& gamma, const Tensor& beta,
                         const Tensor& wf, const Tensor& bf, const Tensor& wo, const Tensor& bo, double eps, bool alone) {
    return BlockPost::apply(x, a, wp, bp, gamma, beta, wf, bf, wo, bo, eps, alone);
  }, arg(), arg(), arg(), arg(), arg(), arg(), arg(), arg(), arg(), arg(), arg(), arg("alone") = true);
  m.def("moe_layer", [](const Tensor& x, const Tensor& router, const Tensor& w1, const Tensor& w2, int64_t capacity, bool alone) {
    return MoeLayer::apply(x, router, w1, w2, capacity, alone);
  }, arg(), arg(), arg(), arg(), arg(), arg("alone") = true);
  m.def("check_products", [](int device) { ok(train::gemmStatus(device, true), "products"); });
  m.def("product_without_operands", &productWithoutOperands);
  m.def("multi_adamw", &multiAdamW);
  m.def("accumulation_hooks", &accumulationHooks);
  m.def("moe_dispatch", [](const Tensor& x, const Tensor& router, int64_t capacity) { return MoeDispatch::apply(x, router, capacity); });
  m.def("moe_experts", [](const Tensor& h, const Tensor& w1, const Tensor& w2, bool alone) { return MoeExperts::apply(h, w1, w2, alone); }, arg(), arg(),
        arg(), arg("alone") = true);
  m.def("moe_combine", [](const Tensor& x, const Tensor& gate, const Tensor& rows, const Tensor& row_of, const Tensor& token_of) {
    return MoeCombine::apply(x, gate, rows, row_of, token_of);
  });
  m.def("sharded_adamw", &shardedAdamW);
  if (PyModule_AddFunctions(m.ptr(), kNativeCalls)) throw py::error_already_set();
  m.def("head_loss", [](const Tensor& h, const Tensor& w, const Tensor& targets) { return HeadLoss::apply(h, w, targets); });
}
