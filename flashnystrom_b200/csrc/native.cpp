// The eager path of flash_nystrom_attention and of the module in C++: argument checks, allocations, the autograd nodes and the
// calls of the C ABI.  Host time of a forward and backward pass (us, the autograd functions in Python / this): the op 185 / 111,
// with the convolution residual 340 / 150 (about 50 of each are the launches), the module at B=4, N=4096, 8 heads of 64
// 816 / 466; inference through the op 48 / 24.  (A pass of that module among others: 793 / 479.)
//
// attention() only takes calls that it can see through completely: plain CUDA tensors of one device and dtype in one of the
// two layouts, no dispatch mode, no forward-mode tangent (tracing and functorch transforms the caller sees).  For anything
// else it returns nothing and the caller goes on in Python, which accepts or refuses it as ever.
#include <torch/extension.h>

#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/autocast_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <cmath>
#include <cstdlib>

#include "../../include/flashnystrom_b200.h"

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

std::atomic<uint32_t> g_flags{0};
PyObject* g_debug = nullptr;     // called with (dO, dQ, dK, dV, step2, k2inv) when FNB_BWD_DEBUG is set

void check(int rc) { TORCH_CHECK(rc == 0, "flashnystrom_b200: ", fnb_last_error(), " (status ", rc, ")"); }

constexpr int kNoLayout = -1;
int layout_of(const at::Tensor& t) {
  if (t.is_contiguous()) return FNB_LAYOUT_BHND;
  return t.transpose(1, 2).is_contiguous() ? FNB_LAYOUT_BNHD : kNoLayout;
}
int dtype_of(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return FNB_F32;
    case at::kHalf: return FNB_F16;
    case at::kBFloat16: return FNB_BF16;
    default: return -1;
  }
}
// shapes that take the (B, N, H, D) layout: the tensor-core kernels' own
bool takes_bnhd(int dtype, int64_t D, int64_t m, uint32_t flags) {
  return !(flags & FNB_FLAG_FORCE_GENERIC) && dtype != FNB_F32 && ((D == 64 && m <= 64) || (D == 128 && m <= 128));
}
at::Tensor empty_in(const at::Tensor& like, int layout) {
  const int64_t B = like.size(0), H = like.size(1), N = like.size(2), D = like.size(3);
  return layout == FNB_LAYOUT_BNHD ? at::empty_strided({B, H, N, D}, {N * H * D, D, H * D, 1}, like.options())
                                   : at::empty({B, H, N, D}, like.options());
}
at::Tensor to_layout(const at::Tensor& t, int layout) {
  if (layout_of(t) == layout) return t;
  return layout == FNB_LAYOUT_BNHD ? t.transpose(1, 2).contiguous().transpose(1, 2) : t.contiguous();
}

// The FP32 tensors that the backward needs, in one buffer: lse1, q~, k~, K2, lse2, iterates, K2inv, Bmat, lse3, step2 (the order of
// fnb_fwd_args), each on a 256-byte step.
struct Saved {
  int64_t offset[10], floats;
  Saved(int64_t BH, int64_t N, int64_t D, int64_t m, int64_t J) {
    const int64_t n[10] = {N, m * D, m * D, m * m, m, (J + 1) * m * m, m * m, m * D, m, m * D};
    floats = 0;
    for (int i = 0; i < 10; ++i) {
      offset[i] = floats;
      floats += (BH * n[i] + 63) / 64 * 64;
    }
  }
};

struct Call {
  fnb_shape shape;
  int layout;
  at::Tensor status;       // the device's status word
};
fnb_shape shape_of(at::IntArrayRef sizes, int dtype, int64_t m, int64_t J, double kappa, int layout, uint32_t flags) {
  fnb_shape s{};
  s.batch = sizes[0]; s.heads = sizes[1]; s.seq_len = sizes[2]; s.head_dim = (int32_t)sizes[3];
  s.num_landmarks = (int32_t)m; s.newton_iter = (int32_t)J; s.dtype = dtype;
  s.kappa_star = (float)kappa; s.flags = flags; s.layout = layout;
  return s;
}
at::Tensor bytes(size_t n, const at::Tensor& like) {
  return at::empty({(int64_t)std::max<size_t>(n, 256)}, like.options().dtype(at::kByte));
}
// (with the tensors' device current: workspace sizes follow its SM count)
at::Tensor run_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const Call& c, at::Tensor& saved) {
  const Saved parts(c.shape.batch * c.shape.heads, c.shape.seq_len, c.shape.head_dim, c.shape.num_landmarks, c.shape.newton_iter);
  at::Tensor out = empty_in(q, c.layout);
  saved = at::empty({parts.floats}, q.options().dtype(at::kFloat));
  at::Tensor ws = bytes(fnb_fwd_workspace_bytes(&c.shape), q);
  float* s = saved.data_ptr<float>();
  fnb_fwd_args a{};
  a.shape = c.shape;
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.out = out.data_ptr();
  float** to[10] = {&a.lse1, &a.q_landmarks, &a.k_landmarks, &a.k2, &a.lse2, &a.ns_iterates, &a.k2_inv, &a.bmat, &a.lse3, &a.step2};
  for (int i = 0; i < 10; ++i) *to[i] = s + parts.offset[i];
  a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
  a.device = q.device().index();
  a.stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  a.device_status = c.status.data_ptr<int32_t>();
  check(fnb_forward(&a));
  return out;
}

at::Tensor run_conv(const at::Tensor& v, int layout, const at::Tensor& w32, const at::Tensor* base, bool transposed) {
  at::Tensor result = empty_in(v, layout);
  fnb_conv_args a{};
  a.batch = v.size(0); a.heads = v.size(1); a.seq_len = v.size(2); a.head_dim = (int32_t)v.size(3);
  a.kernel_size = (int32_t)w32.size(1); a.dtype = dtype_of(v); a.layout = layout;
  a.v = v.data_ptr(); a.base = base ? base->data_ptr() : nullptr; a.result = result.data_ptr(); a.weight = w32.data_ptr<float>();
  a.transposed = transposed ? 1 : 0; a.device = v.device().index();
  a.stream = c10::cuda::getCurrentCUDAStream(v.device().index()).stream();
  check(fnb_conv_residual(&a));
  return result;
}
at::Tensor run_conv_dweight(const at::Tensor& v, const at::Tensor& g, int layout, int64_t ks) {
  at::Tensor dw = at::empty({v.size(1), ks}, v.options().dtype(at::kFloat));
  at::Tensor ws = bytes(fnb_conv_dweight_workspace_bytes(v.size(0), v.size(1), v.size(2), (int32_t)ks), v);
  fnb_conv_dw_args a{};
  a.batch = v.size(0); a.heads = v.size(1); a.seq_len = v.size(2); a.head_dim = (int32_t)v.size(3);
  a.kernel_size = (int32_t)ks; a.dtype = dtype_of(v); a.layout = layout;
  a.v = v.data_ptr(); a.d_out = g.data_ptr(); a.d_weight = dw.data_ptr<float>();
  a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel(); a.device = v.device().index();
  a.stream = c10::cuda::getCurrentCUDAStream(v.device().index()).stream();
  check(fnb_conv_residual_dweight(&a));
  return dw;
}
// the taps take part rounded to the tensors' dtype
at::Tensor rounded_taps(const at::Tensor& weight, const at::Tensor& v) {
  return weight.detach().to(v.scalar_type()).to(at::kFloat).contiguous();
}

// Attention, with the convolution residual where a weight is given (its gradient with respect to v is then added to the
// attention's in the convolution kernel).
struct AttentionNode : torch::autograd::Function<AttentionNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                            const std::optional<at::Tensor>& weight, const Call& c) {
    at::Tensor saved;
    at::Tensor out = run_forward(q, k, v, c, saved);
    // (a gradient of the taps alone needs v and nothing else of the attention)
    const bool inputs = q.requires_grad() || k.requires_grad() || v.requires_grad();
    variable_list keep = inputs ? variable_list{v, q, k, saved} : variable_list{v};
    if (weight) {
      at::Tensor w32 = rounded_taps(*weight, v);
      out = run_conv(v, c.layout, w32, &out, false);
      keep.push_back(w32);
      ctx->saved_data["weight_dtype"] = (int64_t)weight->scalar_type();
    }
    ctx->save_for_backward(keep);
    ctx->saved_data["conv"] = weight.has_value();
    ctx->saved_data["m"] = (int64_t)c.shape.num_landmarks;
    ctx->saved_data["J"] = (int64_t)c.shape.newton_iter;
    ctx->saved_data["kappa"] = (double)c.shape.kappa_star;
    ctx->saved_data["status"] = c.status;
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list kept = ctx->get_saved_variables();
    const bool conv = ctx->saved_data["conv"].toBool(), inputs = kept.size() > 2;
    const at::Tensor& v = kept[0];
    at::Tensor g = grads[0];
    TORCH_CHECK(g.defined() && g.is_cuda() && g.dim() == 4, "dO must be a 4D CUDA tensor (flashnystrom_b200 has no CPU path)");
    const int dtype = dtype_of(g);
    TORCH_CHECK(dtype >= 0, "Supported dtypes: float32, float16, bfloat16");
    c10::cuda::CUDAGuard guard(g.device());
    const int64_t m = ctx->saved_data["m"].toInt();
    const uint32_t flags = g_flags.load();
    int layout = layout_of(v);
    if (layout != FNB_LAYOUT_BNHD || !takes_bnhd(dtype, g.size(3), m, flags)) layout = FNB_LAYOUT_BHND;
    g = to_layout(g, layout);
    for (size_t i = 0; i < (inputs ? 3 : 1); ++i)
      TORCH_CHECK(kept[i].scalar_type() == g.scalar_type() && kept[i].device() == g.device() && kept[i].sizes() == g.sizes() &&
                      layout_of(kept[i]) == layout,
                  "a saved q, k or v does not match dO in shape, dtype, device or layout");
    variable_list result(5);
    if (inputs) attention_backward(ctx, kept[1], kept[2], v, kept[3], g, layout, m, flags, result);
    if (conv) {
      const at::Tensor& w32 = kept.back();
      TORCH_CHECK(w32.scalar_type() == at::kFloat && w32.device() == g.device() && w32.dim() == 2 && w32.size(0) == g.size(1) && w32.is_contiguous(),
                  "the saved convolution weights do not match dO");
      if (ctx->needs_input_grad(2)) result[2] = run_conv(g, layout, w32, &result[2], true);
      if (ctx->needs_input_grad(3))
        result[3] = run_conv_dweight(v, g, layout, w32.size(1)).to((at::ScalarType)ctx->saved_data["weight_dtype"].toInt());
    }
    return result;
  }

  static void attention_backward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, at::Tensor saved,
                                 const at::Tensor& g, int layout, int64_t m, uint32_t flags, variable_list& result) {
    const int64_t J = ctx->saved_data["J"].toInt();
    const Saved parts(g.size(0) * g.size(1), g.size(2), g.size(3), m, J);
    TORCH_CHECK(saved.device() == g.device() && saved.scalar_type() == at::kFloat && saved.dim() == 1 && saved.numel() == parts.floats &&
                    saved.is_contiguous(),
                "the saved tensors do not match dO");
    if (reinterpret_cast<uintptr_t>(saved.data_ptr()) & 15u) saved = saved.clone();   // (a saved-tensor hook may hand it back anywhere)
    const at::Tensor status = ctx->saved_data["status"].toTensor();
    fnb_bwd_args a{};
    a.shape = shape_of(g.sizes(), dtype_of(g), m, J, ctx->saved_data["kappa"].toDouble(), layout, flags);
    check(fnb_check_shape(&a.shape));
    at::Tensor dq = empty_in(g, layout), dk = empty_in(g, layout), dv = empty_in(g, layout);
    at::Tensor ws = bytes(fnb_bwd_workspace_bytes(&a.shape), g);
    const float* s = saved.data_ptr<float>();
    a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.d_out = g.data_ptr();
    a.lse1 = s + parts.offset[0]; a.q_landmarks = s + parts.offset[1]; a.k_landmarks = s + parts.offset[2]; a.k2 = s + parts.offset[3];
    a.ns_iterates = s + parts.offset[5]; a.k2_inv = s + parts.offset[6]; a.bmat = s + parts.offset[7]; a.lse3 = s + parts.offset[8];
    a.step2 = s + parts.offset[9];
    a.dq = dq.data_ptr(); a.dk = dk.data_ptr(); a.dv = dv.data_ptr();
    a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel(); a.device = g.device().index();
    a.stream = c10::cuda::getCurrentCUDAStream(g.device().index()).stream();
    a.device_status = status.data_ptr<int32_t>();
    check(fnb_backward(&a));
    if (std::getenv("FNB_BWD_DEBUG") && std::getenv("FNB_BWD_DEBUG")[0] && g_debug) {
      py::gil_scoped_acquire gil;
      const int64_t BH = g.size(0) * g.size(1), D = g.size(3);
      py::reinterpret_borrow<py::object>(g_debug)(g, dq, dk, dv, saved.narrow(0, parts.offset[9], BH * m * D),
                                                  saved.narrow(0, parts.offset[6], BH * m * m));
    }
    result[0] = dq;
    result[1] = dk;
    result[2] = dv;
  }
};

// The three projections of the module as one node.  q, k and v come out as the (B, H, N, D) views of (B, N, H D) products; the
// backward is written in differentiable operators, as that of three torch linears is, with the gradients of x added up in the
// products.
at::Tensor head_split(const at::Tensor& x2, const at::Tensor& w, int64_t B, int64_t N, int64_t H) {
  const int64_t dim = w.size(0), D = dim / H;
  at::Tensor t = at::empty_strided({B, H, N, D}, {N * dim, D, dim, 1}, x2.options());
  at::Tensor flat = t.as_strided({B * N, dim}, {dim, 1});
  at::mm_out(flat, x2, w.t());
  return t;
}
at::Tensor rows_of(const at::Tensor& t) { return t.transpose(1, 2).reshape({t.size(0) * t.size(2), t.size(1) * t.size(3)}); }

// Both nodes keep what a gradient that is wanted takes, as a torch linear does: its input for the weight's, its weight for the
// input's.  (The rest may be changed in place, and is not held.)
bool wants(const at::Tensor& t) { return t.requires_grad(); }
at::Tensor kept_if(bool keep, const at::Tensor& t) { return keep ? t : at::Tensor(); }

struct ProjectionsNode : torch::autograd::Function<ProjectionsNode> {
  static variable_list forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& wq, const at::Tensor& wk, const at::Tensor& wv,
                               int64_t H) {
    const int64_t B = x.size(0), N = x.size(1);
    const at::Tensor x2 = x.view({B * N, x.size(2)});
    ctx->save_for_backward({kept_if(wants(wq) || wants(wk) || wants(wv), x), kept_if(wants(x), wq), kept_if(wants(x), wk), kept_if(wants(x), wv)});
    return {head_split(x2, wq, B, N, H), head_split(x2, wk, B, N, H), head_split(x2, wv, B, N, H)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list kept = ctx->get_saved_variables();
    const at::Tensor x2 = kept[0].defined() ? kept[0].reshape({-1, kept[0].size(-1)}) : at::Tensor();
    variable_list result(5);
    at::Tensor dx;
    for (int i = 0; i < 3; ++i) {
      const at::Tensor g = rows_of(grads[i]);
      if (ctx->needs_input_grad(0)) dx = i == 0 ? at::mm(g, kept[1]) : at::addmm(dx, g, kept[1 + i]);
      if (ctx->needs_input_grad(1 + i)) result[1 + i] = at::mm(g.t(), x2);
    }
    if (dx.defined()) result[0] = dx.view({grads[0].size(0), grads[0].size(2), dx.size(1)});
    return result;
  }
};

// The output projection of (B, H, N, D) tensors, likewise.
at::Tensor project_out(const at::Tensor& o, const at::Tensor& w) {
  return at::mm(rows_of(o), w.t()).view({o.size(0), o.size(2), w.size(0)});
}
struct OutputNode : torch::autograd::Function<OutputNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& o, const at::Tensor& w) {
    ctx->save_for_backward({kept_if(wants(w), o), kept_if(wants(o), w)});
    ctx->saved_data["heads"] = o.size(1);
    at::Tensor y = at::empty({o.size(0), o.size(2), w.size(0)}, o.options());
    at::Tensor flat = y.as_strided({o.size(0) * o.size(2), w.size(0)}, {w.size(0), 1});
    at::mm_out(flat, rows_of(o), w.t());
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list kept = ctx->get_saved_variables();
    const at::Tensor &o = kept[0], &w = kept[1];
    const int64_t B = grads[0].size(0), N = grads[0].size(1), H = ctx->saved_data["heads"].toInt();
    const at::Tensor g = grads[0].reshape({B * N, -1});
    variable_list result(2);
    if (ctx->needs_input_grad(0)) result[0] = at::mm(g, w).view({B, N, H, w.size(1) / H}).transpose(1, 2);
    if (ctx->needs_input_grad(1)) result[1] = at::mm(g.t(), rows_of(o));
    return result;
  }
};

bool plain(const at::Tensor& t) { return t.is_cuda() && t.layout() == at::kStrided && !at::isTensorSubclassLike(t) && !t.is_neg() && !t.is_conj(); }
bool has_tangent(const at::Tensor& t) { return t._fw_grad(0).defined(); }

// taps for B x H slices
bool takes_taps(const at::Tensor& w, const at::Tensor& like, int64_t B, int64_t H) {
  return plain(w) && w.device() == like.device() && at::isFloatingType(w.scalar_type()) && w.dim() == 2 && w.size(0) == H && w.size(1) % 2 == 1 &&
         w.size(1) <= 127 && !has_tangent(w) && B * H <= 65535;
}
bool takes_numbers(int64_t m, int64_t J, double kappa) {
  return m >= 1 && m <= INT32_MAX && J >= 1 && J <= INT32_MAX && std::isfinite(kappa);
}

// (without the interpreter's lock, with the tensors' device current, all of it checked)
at::Tensor run_attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const std::optional<at::Tensor>& weight, const Call& c) {
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad() || (weight && weight->requires_grad())))
    return AttentionNode::apply(q, k, v, weight, c);
  at::Tensor saved;
  at::Tensor out = run_forward(q, k, v, c, saved);
  return weight ? run_conv(v, c.layout, rounded_taps(*weight, v), &out, false) : out;
}

// out, or nothing where the call is not one for this path
std::optional<at::Tensor> attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, int64_t m, int64_t J, double kappa,
                                    const std::optional<at::Tensor>& weight, const at::Tensor& status) {
  if (c10::impl::dispatch_mode_enabled()) return std::nullopt;
  for (const at::Tensor* t : {&q, &k, &v})
    if (!plain(*t) || t->dim() != 4 || t->scalar_type() != q.scalar_type() || t->sizes() != q.sizes() || t->device() != q.device() || has_tangent(*t))
      return std::nullopt;
  const int dtype = dtype_of(q);
  if (dtype < 0 || q.numel() == 0 || !takes_numbers(m, J, kappa)) return std::nullopt;
  if (status.device() != q.device()) return std::nullopt;
  const uint32_t flags = g_flags.load();
  int layout = layout_of(q);
  if (layout == FNB_LAYOUT_BNHD && !takes_bnhd(dtype, q.size(3), m, flags)) return std::nullopt;
  if (layout == kNoLayout || layout_of(k) != layout || layout_of(v) != layout) return std::nullopt;
  if (weight && !takes_taps(*weight, q, q.size(0), q.size(1))) return std::nullopt;
  for (const at::Tensor* t : {&q, &k, &v})
    if (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15u) return std::nullopt;
  Call c{shape_of(q.sizes(), dtype, m, J, kappa, layout, flags), layout, status};
  if (fnb_check_shape(&c.shape)) return std::nullopt;
  py::gil_scoped_release nogil;
  c10::cuda::CUDAGuard guard(q.device());
  return run_attention(q, k, v, weight, c);
}

// The module's forward: projections, attention, output projection.  The caller has seen to it that the projections are plain
// bias-free linears without hooks.
std::optional<at::Tensor> module_forward(const at::Tensor& x, const at::Tensor& wq, const at::Tensor& wk, const at::Tensor& wv, const at::Tensor& wo,
                                         int64_t H, int64_t m, int64_t J, double kappa, const std::optional<at::Tensor>& conv,
                                         const at::Tensor& status) {
  if (c10::impl::dispatch_mode_enabled() || at::autocast::is_autocast_enabled(at::kCUDA)) return std::nullopt;
  const int64_t dim = x.dim() == 3 ? x.size(2) : 0;
  for (const at::Tensor* t : {&x, &wq, &wk, &wv, &wo})
    if (!plain(*t) || t->scalar_type() != x.scalar_type() || t->device() != x.device() || !t->is_contiguous() || has_tangent(*t)) return std::nullopt;
  for (const at::Tensor* t : {&wq, &wk, &wv, &wo})
    if (t->dim() != 2 || t->size(0) != dim || t->size(1) != dim) return std::nullopt;
  const uint32_t flags = g_flags.load();
  if (dim == 0 || x.numel() == 0 || H < 1 || dim % H || dtype_of(x) < 0 || !takes_numbers(m, J, kappa) || !takes_bnhd(dtype_of(x), dim / H, m, flags))
    return std::nullopt;
  if (status.device() != x.device() || (conv && !takes_taps(*conv, x, x.size(0), H))) return std::nullopt;
  const int64_t B = x.size(0), N = x.size(1);
  const int layout = H == 1 || N == 1 ? FNB_LAYOUT_BHND : FNB_LAYOUT_BNHD;      // (head-split views of one head or row are contiguous)
  const Call c{shape_of({B, H, N, dim / H}, dtype_of(x), m, J, kappa, layout, flags), layout, status};
  if (fnb_check_shape(&c.shape)) return std::nullopt;      // (refused further on; nothing has been formed yet)
  py::gil_scoped_release nogil;
  c10::cuda::CUDAGuard guard(x.device());
  variable_list qkv;
  if (at::GradMode::is_enabled() && (x.requires_grad() || wq.requires_grad() || wk.requires_grad() || wv.requires_grad())) {
    qkv = ProjectionsNode::apply(x, wq, wk, wv, H);
  } else {
    at::AutoGradMode off(false);
    const at::Tensor x2 = x.view({B * N, dim});
    for (const at::Tensor* w : {&wq, &wk, &wv}) qkv.push_back(head_split(x2, *w, B, N, H));
  }
  const at::Tensor o = run_attention(qkv[0], qkv[1], qkv[2], conv, c);
  if (at::GradMode::is_enabled() && (o.requires_grad() || wo.requires_grad())) return OutputNode::apply(o, wo);
  return project_out(o, wo);
}

}  // namespace

PYBIND11_MODULE(_native, mod) {
  mod.def("attention", &attention);
  mod.def("module_forward", &module_forward);
  mod.def("set_flags", [](uint32_t flags) { g_flags = flags; });
  mod.def("set_debug", [](py::object f) { g_debug = f.release().ptr(); });
}
