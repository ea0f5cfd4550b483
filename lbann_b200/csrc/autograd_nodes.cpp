// Autograd nodes of the layers that every model is made of, as C++ (forward, backward and the
// launches of their kernels).
//
// A kernel of a small layer runs for 3-10 us; composed in Python, a linear layer's forward and
// backward took 185 us of host time (argument checks, views and three GEMM wrappers at 20-30 us
// each), a convolution + batch norm 280 us, an attention 165 us: every model step that is not
// replayed as a CUDA graph was bound by it.  The nodes here do the same work in the same order.
// Inputs that the backward pass needs go through save_for_backward (saved-tensor hooks and
// version checks apply as before); weights are not inputs in that sense: their 16-bit copies and
// gradient buffers belong to the weight handle, which outlives the step, and weight gradients
// are accumulated into those buffers (the reference's destination-scale / gradient-scale
// contract, include/lbann/optimizers/optimizer_impl.hpp:208-290).  The weights' master tensors
// are passed along so that an output requires a gradient when only a weight does.
//
// Tensors that a node allocates for one launch are released behind it on the same stream, which
// is what the caching allocator orders reuse by.
#include <ATen/cuda/CUDAContext.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>
#include <cstdlib>

#include "abi.h"

extern "C" {          // a change here raises LB_ABI_VERSION
int lb_gemm_tc(const void*, const void*, void*, const float*, int, int, int, int, long long, long long, long long,
               long long, long long, long long, int, int, int, int, float, float, int, int, float, int, void*);
int lb_splitk_offer(void*, long long);
int lb_sm_count();
int lb_outer_accum(const void*, const void*, float*, int, int, long long, float, float, int, void*);
int lb_grad_prep(const void*, const void*, void*, float*, long long, int, long long, int, float, int, void*);
int lb_pad_rows(const void*, void*, long long, int, long long, int, void*);
int lb_unary(const void*, const void*, void*, long long, int, int, float, float, int, void*);
int lb_binary(const void*, const void*, const void*, void*, void*, long long, int, int, int, void*);
int lb_attention_fwd(const void*, const void*, const void*, void*, float*, int, int, int, int, const long long*,
                     const long long*, const long long*, const long long*, float, int, int, void*);
int lb_attention_bwd(const void*, const void*, const void*, const void*, const void*, const float*, float*, void*,
                     void*, void*, int, int, int, int, const long long*, const long long*, const long long*,
                     const long long*, const long long*, const long long*, const long long*, const long long*, float,
                     int, int, void*);
int lb_conv_fwd_halo_tc(const void*, const void*, void*, const float*, const int*, const long long*, const long long*,
                        int, int, float, float, int, float, const void*, void*);
long long lb_conv_wgrad_ws(const int*);
int lb_conv_wgrad_tc(const void*, const void*, float*, float*, const int*, const long long*, const long long*,
                     long long, long long, long long, int, float, void*);
int lb_upsample_zero(const void*, void*, const int*, void*);
int lb_pack_filter(const float*, void*, void*, int, int, int, int, int, int, void*);
int lb_bn_fused_fwd(const void*, const float*, const float*, void*, float*, float*, float*, float*, long long, int,
                    float, float, float, float, int, float, int, void* const*, void* const*, int, int, long long,
                    unsigned*, void*);
int lb_bn_fused_bwd(const void*, const void*, const void*, const float*, const float*, void*, float*, float*, float*,
                    long long, int, float, float, float, int, float, int, void* const*, void* const*, int, int,
                    long long, unsigned*, void*);
int lb_embedding_fwd(const void*, int, const float*, void*, int*, long long, int, long long, long long, int, void*);
int lb_embedding_bwd(const int*, const void*, float*, long long, int, int, void*);
int lb_layer_norm_fwd(const void*, const float*, const float*, void*, float*, float*, long long, int, float, int,
                      void*);
int lb_layer_norm_bwd(const void*, const void*, const float*, const float*, const float*, void*, float*, float*,
                      long long, int, int, void*);
}

namespace {

using at::Tensor;
using std::optional;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
namespace py = pybind11;

std::atomic<long long> g_launches{0}, g_offers{0};

PyObject* g_native_error = nullptr;      // lbann_b200.ops.native.NativeError

[[noreturn]] void fail(const std::string& what) {      // from backward's threads too
  py::gil_scoped_acquire gil;
  PyErr_SetString(g_native_error ? g_native_error : PyExc_RuntimeError, what.c_str());
  throw py::error_already_set();
}
void check(int rc, const char* what) {
  if (rc) fail(std::string(what) + " failed with code " + std::to_string(rc));
}
void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }
int code(at::ScalarType t) {
  if (t == at::kHalf) return 0;
  if (t == at::kBFloat16) return 1;
  if (t == at::kFloat) return 2;
  fail("unsupported dtype");
}
const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* fptr(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
// A gradient buffer that a kernel adds to as a dense run of floats.
float* dense_grad(const Tensor& t) {
  TORCH_CHECK(!t.defined() || t.is_contiguous(), "gradient buffers of scales and biases must be contiguous");
  return fptr(t);
}
Tensor fp32(const Tensor& t) { return !t.defined() || t.scalar_type() == at::kFloat ? t : t.to(at::kFloat); }

// What a node keeps besides saved tensors: the weight's copies and gradient buffer, the handles
// whose mark_ready() has to run (data-parallel steps only), its scalars, and the owner of the
// memory that addresses among them point into.
struct State : torch::CustomClassHolder {
  Tensor w, w2, wgrad, bgrad, scale;
  Tensor written;            // host flags of gradients that a step's only writer overwrites: set behind the write
  py::object wh, bh, owner;
  std::vector<int64_t> i;
  std::vector<double> f;
  ~State() override {
    if (wh || bh || owner) {
      py::gil_scoped_acquire gil;
      wh = py::object();
      bh = py::object();
      owner = py::object();
    }
  }
};
c10::intrusive_ptr<State> state_of(AutogradContext* ctx) {
  return c10::static_intrusive_pointer_cast<State>(ctx->saved_data["s"].toCapsule());
}
void keep(AutogradContext* ctx, const c10::intrusive_ptr<State>& s) {
  ctx->saved_data["s"] = c10::IValue::make_capsule(s);
}
void mark_ready(const py::object& handle) {
  if (!handle) return;
  py::gil_scoped_acquire gil;
  handle.attr("mark_ready")();
}
// A handle is kept only where a data-parallel context has asked to hear about its gradient.
py::object listening(const py::object& handle) {
  if (handle.is_none() || !py::hasattr(handle, "on_grad_ready") || handle.attr("on_grad_ready").is_none())
    return py::object();
  return handle;
}
Tensor opt(const optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }

// ---------------------------------------------------------------------------------- split-K
bool splitk_disabled() {
  const char* e = std::getenv("LBANN_DISABLE_SPLITK");
  return e && *e && std::string(e) != "0";
}
// Lends scratch to the next product of this thread (csrc/tc_pipeline.cuh): only to outputs of at
// most half a wave of 128 x 256 tiles.
Tensor offer_splitk(int64_t rows, int64_t cols, const Tensor& like) {
  if (rows * cols > 74 * 128 * 256 || splitk_disabled()) return Tensor();
  const int64_t bn = cols > 128 ? 256 : 128;
  Tensor ws = at::empty({(int64_t)lb_sm_count() * 128 * bn}, like.options().dtype(at::kFloat));
  check(lb_splitk_offer(ws.data_ptr(), ws.numel() * 4), "lb_splitk_offer");
  ++g_offers;
  return ws;
}

// ------------------------------------------------------------------------------------- GEMM
// `t` or a copy whose rows start on 16-byte boundaries with a legal pitch.  A matrix expanded over
// the batch (stride 0) is copied too: to the launch a batch stride of 0 means dense matrices.
Tensor tma_ready(const Tensor& t) {
  const int64_t nd = t.dim();
  if (t.stride(nd - 1) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && t.stride(nd - 2) % 8 == 0 &&
      (nd == 2 || (t.stride(0) % 8 == 0 && (t.stride(0) > 0 || t.size(0) == 1))))
    return t;
  auto shape = t.sizes().vec();
  const int64_t cols = shape[nd - 1], pitch = (cols + 7) / 8 * 8;
  shape[nd - 1] = pitch;
  if (t.stride(nd - 1) == 1 && t.numel() > 0 && t.element_size() == 2 &&
      (nd == 2 || t.stride(0) == t.size(1) * t.stride(1))) {
    Tensor buf = at::empty(shape, t.options());
    check(lb_pad_rows(t.data_ptr(), buf.data_ptr(), t.numel() / cols, cols, t.stride(nd - 2), pitch, stream()),
          "lb_pad_rows");
    ++g_launches;
    return pitch == cols ? buf : buf.narrow(nd - 1, 0, cols);
  }
  Tensor buf = at::zeros(shape, t.options());
  Tensor view = buf.narrow(nd - 1, 0, cols);
  view.copy_(t);
  return view;
}

Tensor gemm(Tensor a, Tensor b, bool ta, bool tb, const Tensor& out_, at::ScalarType out_dtype, double alpha,
            double beta, Tensor bias, bool bias_per_row, int64_t act, double act_param, int64_t bn_hint) {
  const bool batched = a.dim() == 3;
  const int64_t nd = a.dim();
  const int64_t M = a.size(ta ? nd - 1 : nd - 2), K = a.size(ta ? nd - 2 : nd - 1), N = b.size(tb ? nd - 2 : nd - 1);
  const int64_t nb = batched ? a.size(0) : 1;
  if (a.scalar_type() != at::kHalf && a.scalar_type() != at::kBFloat16) a = a.to(at::kBFloat16);
  if (b.scalar_type() != a.scalar_type()) b = b.to(a.scalar_type());
  a = tma_ready(a);
  b = tma_ready(b);
  Tensor out = out_;
  if (!out.defined()) {
    out = batched ? at::empty({nb, M, N}, a.options().dtype(out_dtype)) : at::empty({M, N}, a.options().dtype(out_dtype));
    if (beta != 0.0) out.zero_();
  }
  TORCH_CHECK_VALUE(out.stride(-1) == 1, "gemm: output must have unit stride in its last dimension");
  bias = fp32(bias);
  Tensor scratch = K >= 512 ? offer_splitk(M * nb, N, a) : Tensor();
  check(lb_gemm_tc(a.data_ptr(), b.data_ptr(), out.data_ptr(), fptr(bias), M, N, K, nb, a.stride(-2), b.stride(-2),
                   out.stride(-2), batched ? a.stride(0) : 0, batched ? b.stride(0) : 0, batched ? out.stride(0) : 0,
                   ta ? 1 : 0, tb ? 0 : 1, code(a.scalar_type()), code(out.scalar_type()), alpha, beta,
                   bias_per_row ? 2 : 1, act, act_param, bn_hint, stream()),
        "lb_gemm_tc");
  ++g_launches;
  return out;
}
Tensor mm(const Tensor& a, const Tensor& b, bool ta, bool tb) {
  return gemm(a, b, ta, tb, Tensor(), a.scalar_type(), 1.0, 0.0, Tensor(), false, 0, 0.0, 0);
}

// ---------------------------------------------------------------- shared pieces of backward
Tensor unary_raw(int64_t op, const Tensor& x, const Tensor& dy, double p0, double p1, int64_t mode) {
  Tensor out = at::empty_like(x);
  check(lb_unary(x.data_ptr(), ptr(dy), out.data_ptr(), x.numel(), op, mode, p0, p1, code(x.scalar_type()), stream()),
        "lb_unary");
  ++g_launches;
  return out;
}
Tensor same_strides(const Tensor& dy, const Tensor& x) {
  if (dy.strides() == x.strides()) return dy;
  return at::empty_like(x).copy_(dy);
}
// What the products of a layer's backward read, from the dense rows of dy (csrc/grad_prep.cu):
// dy * act'(.) where `y`, the layer's output, is given, with a row pitch that TMA takes; the bias
// gradient (may be undefined) receives the column sums on the way.
Tensor grad_prep(const Tensor& dy, const Tensor& y, int64_t act, double p, const Tensor& bgrad) {
  const int64_t C = dy.size(-1), rows = dy.numel() / C, pitch = (C + 7) / 8 * 8;
  const bool copy = y.defined() || pitch != C;
  if (!copy && !bgrad.defined()) return dy;
  Tensor sums = bgrad;
  const bool direct = bgrad.defined() && bgrad.scalar_type() == at::kFloat && bgrad.is_contiguous() && bgrad.numel() == C;
  if (bgrad.defined() && !direct) sums = at::zeros({C}, dy.options().dtype(at::kFloat));
  Tensor g;
  if (copy) {
    auto shape = dy.sizes().vec();
    shape.back() = pitch;
    g = at::empty(shape, dy.options());
  }
  check(lb_grad_prep(dy.data_ptr(), ptr(y), copy ? g.data_ptr() : nullptr, fptr(sums), rows, C, pitch,
                     y.defined() ? act : 0, p, code(dy.scalar_type()), stream()),
        "lb_grad_prep");
  ++g_launches;
  if (bgrad.defined() && !direct) bgrad.add_(sums.narrow(0, 0, bgrad.numel()).view(bgrad.sizes()));
  if (!copy) return dy;
  return pitch == C ? g : g.narrow(-1, 0, C);
}
// grad[out, in] += dy^T x, or = with `overwrite`.  Mini-batches of at most 16 rows make this a rank-K
// update bound by the read-modify-write of grad (csrc/outer_accum.cu); the rest goes to the tensor
// cores, in the same tiles and splits either way (the error of a long reduction depends on them).
constexpr int64_t kTilesAsAdded = 1;
bool outer_rows(int64_t K) { return K == 1 || K == 2 || K == 4 || K == 8 || K == 16; }
void weight_grad(const Tensor& dy, const Tensor& x, const Tensor& grad, bool overwrite) {
  const int64_t K = dy.size(0);
  if (K == 0) {
    if (overwrite) grad.zero_();
    return;
  }
  const float beta = overwrite ? 0.f : 1.f;
  if (outer_rows(K) && dy.is_contiguous() && x.is_contiguous() && grad.scalar_type() == at::kFloat && grad.is_contiguous() &&
      x.size(1) % 4 == 0 && dy.scalar_type() == x.scalar_type()) {
    const int rc = lb_outer_accum(dy.data_ptr(), x.data_ptr(), fptr(grad), K, dy.size(1), x.size(1), 1.f, beta,
                                  code(x.scalar_type()), stream());
    if (rc != -2) {
      check(rc, "lb_outer_accum");
      ++g_launches;
      return;
    }
  }
  gemm(dy, x, true, false, grad, grad.scalar_type(), 1.0, beta, Tensor(), false, 0, 0.0, kTilesAsAdded);
}

// ----------------------------------------------------------------------------------- linear
struct LinearNode : torch::autograd::Function<LinearNode> {
  // state: w = 16-bit weight, wgrad, bgrad, written (may be undefined); i = {act, index into written}; f = {act_param}
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w_leaf, const optional<Tensor>& b_leaf,
                        const c10::intrusive_ptr<State>& s) {
    Tensor x2 = x.reshape({-1, x.size(-1)});
    if (!x2.is_contiguous()) x2 = x2.contiguous();
    // operands that need another row pitch are copied once for all three products (a few rows:
    // the weight gradient reads them dense)
    const Tensor xt = tma_ready(x2);
    s->w = tma_ready(s->w);
    Tensor y = gemm(xt, s->w, false, true, Tensor(), x.scalar_type(), 1.0, 0.0, opt(b_leaf), false, s->i[0], s->f[0], 0);
    keep(ctx, s);
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->save_for_backward({outer_rows(x2.size(0)) ? x2 : xt, s->i[0] ? y : Tensor()});
    auto shape = x.sizes().vec();
    shape.back() = s->w.size(0);
    return x.dim() == 2 ? y : y.reshape(shape);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = state_of(ctx);
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &y = saved[1];
    Tensor dy = g[0].reshape({-1, g[0].size(-1)});
    if (!dy.is_contiguous()) dy = dy.contiguous();
    dy = grad_prep(dy, y, s->i[0], s->f[0], s->bgrad);
    if (s->bgrad.defined()) mark_ready(s->bh);
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      dx = mm(dy, s->w, false, false);
      const auto shape = ctx->saved_data["shape"].toIntVector();
      if (shape.size() != 2) dx = dx.reshape(shape);
    }
    if (s->wgrad.defined()) {
      weight_grad(outer_rows(dy.size(0)) && !dy.is_contiguous() ? dy.contiguous() : dy, x2, s->wgrad, s->written.defined());
      if (s->written.defined()) s->written.data_ptr<bool>()[s->i[1]] = true;
      mark_ready(s->wh);
    }
    return {dx, Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ convolution
bool sample_dense(const Tensor& t) {     // [N, D, H, W, C]: only the sample stride may leave a gap
  const int64_t D = t.size(1), H = t.size(2), W = t.size(3), C = t.size(4);
  return t.stride(4) == 1 && t.stride(3) == C && t.stride(2) == W * C && t.stride(1) == H * W * C &&
         t.stride(0) >= D * H * W * C;
}
Tensor cl_view(const Tensor& x_) {       // [N, C, (D,) H, W] -> channels-last NDHWC view, copying if needed
  Tensor x = x_.dim() == 3 ? x_.unsqueeze(2) : x_;
  if (x.dim() == 4) return x.contiguous(at::MemoryFormat::ChannelsLast).permute({0, 2, 3, 1}).unsqueeze(1);
  Tensor v = x.permute({0, 2, 3, 4, 1});
  if (sample_dense(v)) return v;
  return x.contiguous(at::MemoryFormat::ChannelsLast3d).permute({0, 2, 3, 4, 1});
}
Tensor from_cl(const Tensor& y, int64_t ndim) {
  if (ndim == 5) return y.permute({0, 4, 1, 2, 3});
  if (ndim == 4) return y.squeeze(1).permute({0, 3, 1, 2});
  return y.squeeze(1).squeeze(1).permute({0, 2, 1});
}
Tensor pad_channels(const Tensor& t) {
  const int64_t C = t.size(-1);
  return C % 8 == 0 ? t : at::constant_pad_nd(t, {0, 8 - C % 8}, 0);
}

// geom = {kd, kh, kw, pd, ph, pw, sd, sh, sw, dd, dh, dw}
void fill_geom(int* out, const Tensor& x, int64_t Do, int64_t Ho, int64_t Wo, int64_t Kout, const int64_t* g) {
  const int64_t head[9] = {x.size(0), x.size(1), x.size(2), x.size(3), x.size(4), Do, Ho, Wo, Kout};
  for (int i = 0; i < 9; ++i) out[i] = (int)head[i];
  for (int i = 0; i < 12; ++i) out[9 + i] = (int)g[i];
}
// Element strides of N, D, H, W.  PyTorch keeps any stride for a dimension of one element ([N, C, 1, 1]
// as a reshape leaves it counts as channels-last with strides of 1); the launches want multiples
// of eight, so such a dimension gets the stride of a dense one.
struct Strides4 {
  long long v[4];
  explicit Strides4(const Tensor& t) {
    long long dense = t.size(4);
    for (int i = 3; i >= 0; --i) {
      v[i] = t.size(i) == 1 && t.stride(i) % 8 ? dense : t.stride(i);
      dense = v[i] * t.size(i);
    }
  }
};

Tensor conv_fwd(const Tensor& x, Tensor w, const Tensor& out_, at::ScalarType out_dtype, const int64_t* g, int64_t Do,
                int64_t Ho, int64_t Wo, double alpha, double beta, Tensor bias, int64_t act, double act_param,
                int64_t halo) {
  if (w.scalar_type() != x.scalar_type() || !w.is_contiguous()) w = w.to(x.scalar_type()).contiguous();
  const int64_t Kout = w.size(1), N = x.size(0);
  Tensor out = out_;
  if (!out.defined()) {
    out = at::empty({N, Do, Ho, Wo, Kout}, x.options().dtype(out_dtype));
    if (beta != 0.0) out.zero_();
  }
  int geom[21];
  fill_geom(geom, x, Do, Ho, Wo, Kout, g);
  const Strides4 xs(x), ys(out);
  bias = fp32(bias);
  Tensor scratch = x.size(4) * g[0] * g[1] * g[2] >= 512 ? offer_splitk(N * Do * Ho * Wo, Kout, x) : Tensor();
  check(lb_conv_fwd_halo_tc(x.data_ptr(), w.data_ptr(), out.data_ptr(), fptr(bias), geom, xs.v, ys.v,
                            code(x.scalar_type()), code(out.scalar_type()), alpha, beta, act, act_param,
                            reinterpret_cast<const void*>(halo), stream()),
        "lb_conv_fwd_halo_tc");
  ++g_launches;
  return out;
}

// Filter gradient, added into `out` (fp32, contiguous, Kout x C x kd x kh x kw).
void conv_wgrad(const Tensor& x, Tensor dy, const Tensor& out, const int64_t* g, double alpha) {
  TORCH_CHECK_VALUE(out.scalar_type() == at::kFloat && out.is_contiguous(),
                    "conv_wgrad: out must be a contiguous fp32 tensor");
  if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
  int geom[21];
  fill_geom(geom, x, dy.size(1), dy.size(2), dy.size(3), dy.size(4), g);
  const Strides4 xs(x), ys(dy);
  const long long taps = g[0] * g[1] * g[2], words = lb_conv_wgrad_ws(geom);     // -1: reported by the launch
  Tensor ws = words > 0 ? at::empty({words}, x.options().dtype(at::kFloat)) : Tensor();
  check(lb_conv_wgrad_tc(x.data_ptr(), dy.data_ptr(), fptr(out), fptr(ws), geom, xs.v, ys.v, 1, x.size(4) * taps, taps,
                         code(x.scalar_type()), alpha, stream()),
        "lb_conv_wgrad_tc");
  g_launches += 2;
}

// Zeros between the elements of dy (data gradient of a strided convolution); dy is dense NDHWC.
Tensor upsample_zero(const Tensor& dy, const int64_t* stride) {
  std::vector<int64_t> shape{dy.size(0)};
  for (int i = 0; i < 3; ++i) shape.push_back((dy.size(1 + i) - 1) * stride[i] + 1);
  shape.push_back(dy.size(4));
  int geom[8];
  for (int i = 0; i < 5; ++i) geom[i] = (int)dy.size(i);
  for (int i = 0; i < 3; ++i) geom[5 + i] = (int)stride[i];
  Tensor up = at::empty(shape, dy.options());
  Tensor src = reinterpret_cast<uintptr_t>(dy.data_ptr()) % 16 ? dy.clone() : dy;
  check(lb_upsample_zero(src.data_ptr(), up.data_ptr(), geom, stream()), "lb_upsample_zero");
  ++g_launches;
  return up;
}

struct ConvNode : torch::autograd::Function<ConvNode> {
  // state: w / w2 = filters of the forward / data-gradient product (w2 undefined: no data
  // gradient), wgrad, bgrad; i = {act, act whose gradient is applied here, Kout, Cin, geom[12]};
  // f = {act_param}
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w_leaf, const optional<Tensor>& b_leaf,
                        const c10::intrusive_ptr<State>& s) {
    const int64_t* g = s->i.data() + 4;
    const int64_t Kout = s->i[2], Kp = s->w.size(1);
    Tensor x_cl = pad_channels(cl_view(x)), bias = opt(b_leaf);
    if (bias.defined() && Kp != Kout) bias = at::constant_pad_nd(bias, {0, Kp - Kout}, 0);
    int64_t o[3];
    for (int i = 0; i < 3; ++i) o[i] = (x_cl.size(1 + i) + 2 * g[3 + i] - g[9 + i] * (g[i] - 1) - 1) / g[6 + i] + 1;
    Tensor y = conv_fwd(x_cl, s->w, Tensor(), x.scalar_type(), g, o[0], o[1], o[2], 1.0, 0.0, bias, s->i[0], s->f[0], 0);
    keep(ctx, s);
    ctx->saved_data["ndim"] = x.dim();
    ctx->save_for_backward({x_cl, s->i[1] ? y : Tensor()});
    return from_cl(Kp != Kout ? y.narrow(4, 0, Kout) : y, x.dim());
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto s = state_of(ctx);
    const auto saved = ctx->get_saved_variables();
    const Tensor &x_cl = saved[0], &y = saved[1];
    const int64_t ndim = ctx->saved_data["ndim"].toInt();
    const int64_t* g = s->i.data() + 4;
    const int64_t Kout = s->i[2], Cin = s->i[3], Kp = s->w.size(1), Cp = x_cl.size(4);
    Tensor dy = cl_view(grads[0]);
    if (Kp != Kout) dy = pad_channels(dy);
    if (!dy.is_contiguous()) dy = dy.contiguous();
    dy = grad_prep(dy, y, s->i[1], s->f[0], s->bgrad);
    if (s->bgrad.defined()) mark_ready(s->bh);
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      const bool unit = g[6] == 1 && g[7] == 1 && g[8] == 1;
      int64_t b[12];
      for (int i = 0; i < 3; ++i) {
        b[i] = g[i];
        b[3 + i] = g[9 + i] * (g[i] - 1) - g[3 + i];
        b[6 + i] = 1;
        b[9 + i] = g[9 + i];
      }
      dx = conv_fwd(unit ? dy : upsample_zero(dy, g + 6), s->w2, Tensor(), dy.scalar_type(), b, x_cl.size(1), x_cl.size(2),
                    x_cl.size(3), 1.0, 0.0, Tensor(), 0, 0.0, 0);
      dx = from_cl(Cp != Cin ? dx.narrow(4, 0, Cin) : dx, ndim);
    }
    if (s->wgrad.defined()) {
      if (Kp == Kout && Cp == Cin) {
        conv_wgrad(x_cl, dy, s->wgrad, g, 1.0);
      } else {
        Tensor tmp = at::zeros({Kp, Cp, g[0], g[1], g[2]}, s->wgrad.options());
        conv_wgrad(x_cl, dy, tmp, g, 1.0);
        s->wgrad.add_(tmp.narrow(0, 0, Kout).narrow(1, 0, Cin).reshape(s->wgrad.sizes()));
      }
      mark_ready(s->wh);
    }
    return {dx, Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------- batch norm
struct BatchNormNode : torch::autograd::Function<BatchNormNode> {
  // state: w / w2 = forward / backward workspaces, wgrad / bgrad = gradients of scale / bias;
  // i = {act, staging, pads, rank, world, slot stride, counters} (staging and pads are host arrays of
  // the group, which `owner` keeps until backward has run); f = {eps, decay, correction, count scale, act_param}
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const optional<Tensor>& scale_,
                        const optional<Tensor>& bias_, const optional<Tensor>& mean_, const optional<Tensor>& var_,
                        const c10::intrusive_ptr<State>& s) {
    const Tensor scale = opt(scale_), bias = opt(bias_), mean = opt(mean_), var = opt(var_);
    Tensor x_cl = cl_view(x);
    if (!x_cl.is_contiguous()) x_cl = x_cl.contiguous();
    const int64_t C = x_cl.size(4), rows = x_cl.numel() / C;
    Tensor y = at::empty_like(x_cl), stats = at::empty({2 * C}, x.options().dtype(at::kFloat));
    const auto& i = s->i;
    const auto& f = s->f;
    check(lb_bn_fused_fwd(x_cl.data_ptr(), fptr(scale), fptr(bias), y.data_ptr(), fptr(stats), fptr(mean), fptr(var),
                          fptr(s->w), rows, C, (float)(rows * f[3]), f[2], f[0], f[1], i[0], f[4], code(x.scalar_type()),
                          reinterpret_cast<void* const*>(i[1]), reinterpret_cast<void* const*>(i[2]), i[3], i[4], i[5],
                          reinterpret_cast<unsigned*>(i[6]), stream()),
          "lb_bn_fused_fwd");
    ++g_launches;
    s->scale = scale.defined() ? scale.detach() : scale;
    keep(ctx, s);
    ctx->saved_data["ndim"] = x.dim();
    ctx->save_for_backward({x_cl, stats, i[0] ? y : Tensor()});
    return from_cl(y, x.dim());
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto s = state_of(ctx);
    const auto saved = ctx->get_saved_variables();
    const Tensor &x_cl = saved[0], &stats = saved[1], &y = saved[2];
    Tensor dy = cl_view(grads[0]);
    if (!dy.is_contiguous()) dy = dy.contiguous();
    const int64_t C = x_cl.size(4), rows = x_cl.numel() / C;
    Tensor dx = at::empty_like(x_cl);
    const auto& i = s->i;
    const auto& f = s->f;
    check(lb_bn_fused_bwd(x_cl.data_ptr(), dy.data_ptr(), ptr(y), fptr(stats), fptr(s->scale), dx.data_ptr(),
                          dense_grad(s->wgrad), dense_grad(s->bgrad), fptr(s->w2), rows, C, (float)(rows * f[3]), f[2], f[0], i[0],
                          f[4], code(x_cl.scalar_type()), reinterpret_cast<void* const*>(i[1]),
                          reinterpret_cast<void* const*>(i[2]), i[3], i[4], i[5], reinterpret_cast<unsigned*>(i[6]),
                          stream()),
          "lb_bn_fused_bwd");
    ++g_launches;
    if (s->wgrad.defined()) mark_ready(s->wh);
    if (s->bgrad.defined()) mark_ready(s->bh);
    return {from_cl(dx, ctx->saved_data["ndim"].toInt()), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------- layer norm
struct LayerNormNode : torch::autograd::Function<LayerNormNode> {
  // state: scale, wgrad / bgrad = gradients of scale / bias; i = {cols}; f = {eps}
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const optional<Tensor>& scale_,
                        const optional<Tensor>& bias_, const c10::intrusive_ptr<State>& s) {
    Tensor xc = x.contiguous(), scale, bias;
    if (scale_.has_value()) scale = scale_->detach().reshape({-1});
    if (bias_.has_value()) bias = bias_->detach().reshape({-1});
    const int64_t cols = s->i[0], rows = xc.numel() / cols;
    Tensor y = at::empty_like(xc), stat = at::empty({2, rows}, x.options().dtype(at::kFloat));
    check(lb_layer_norm_fwd(xc.data_ptr(), fptr(scale), fptr(bias), y.data_ptr(), fptr(stat), fptr(stat) + rows, rows,
                            cols, s->f[0], code(x.scalar_type()), stream()),
          "lb_layer_norm_fwd");
    ++g_launches;
    s->scale = scale;
    keep(ctx, s);
    ctx->save_for_backward({xc, stat});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto s = state_of(ctx);
    const auto saved = ctx->get_saved_variables();
    const Tensor &xc = saved[0], &stat = saved[1];
    Tensor dy = grads[0].contiguous(), dx = at::empty_like(xc);
    const int64_t cols = s->i[0], rows = xc.numel() / cols;
    check(lb_layer_norm_bwd(xc.data_ptr(), dy.data_ptr(), fptr(s->scale), fptr(stat), fptr(stat) + rows, dx.data_ptr(),
                            dense_grad(s->wgrad), dense_grad(s->bgrad), rows, cols, code(xc.scalar_type()), stream()),
          "lb_layer_norm_bwd");
    ++g_launches;
    if (s->wgrad.defined()) mark_ready(s->wh);
    if (s->bgrad.defined()) mark_ready(s->bh);
    return {dx, Tensor(), Tensor(), Tensor()};
  }
};

// -------------------------------------------------------------------------------- embedding
struct EmbeddingNode : torch::autograd::Function<EmbeddingNode> {
  // state: wgrad; i = {padding index, dtype of the output}
  static int kind(const Tensor& idx) {
    return idx.scalar_type() == at::kInt ? 0 : (idx.scalar_type() == at::kLong ? 1 : 2);
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& idx, const Tensor& table, const c10::intrusive_ptr<State>& s) {
    auto shape = idx.sizes().vec();
    shape.push_back(table.size(1));
    const auto dt = s->i[1] == 0 ? at::kHalf : (s->i[1] == 1 ? at::kBFloat16 : at::kFloat);
    Tensor out = at::empty(shape, table.options().dtype(dt)), rows = at::empty({idx.numel()}, table.options().dtype(at::kInt));
    check(lb_embedding_fwd(idx.data_ptr(), kind(idx), fptr(table), out.data_ptr(), rows.data_ptr<int>(), idx.numel(),
                           table.size(1), table.size(0), s->i[0], s->i[1], stream()),
          "lb_embedding_fwd");
    ++g_launches;
    keep(ctx, s);
    ctx->save_for_backward({rows});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto s = state_of(ctx);
    const Tensor rows = ctx->get_saved_variables()[0];
    Tensor g = grads[0].contiguous();
    if (reinterpret_cast<uintptr_t>(g.data_ptr()) % 16) g = g.clone();
    check(lb_embedding_bwd(rows.data_ptr<int>(), g.data_ptr(), fptr(s->wgrad), rows.numel(), s->wgrad.size(1),
                           code(g.scalar_type()), stream()),
          "lb_embedding_bwd");
    ++g_launches;
    mark_ready(s->wh);
    return {Tensor(), Tensor(), Tensor()};
  }
};

// -------------------------------------------------------------------------------- attention
struct Attn {
  int64_t H;
  double scale;
  bool causal;
};
struct Strides3 {
  long long v[3];
  explicit Strides3(const Tensor& t) : v{t.stride(0), t.stride(1), 128} {}
};
Tensor attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Attn& a, Tensor& lse) {
  const int64_t B = q.size(0), Sq = q.size(1);
  Tensor o = at::empty({B, Sq, q.size(2)}, q.options());
  lse = at::empty({B, a.H, Sq}, q.options().dtype(at::kFloat));
  const Strides3 sq(q), sk(k), sv(v), so(o);
  check(lb_attention_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), fptr(lse), B, a.H, Sq, k.size(1), sq.v,
                         sk.v, sv.v, so.v, a.scale, a.causal, code(q.scalar_type()), stream()),
        "lb_attention_fwd");
  ++g_launches;
  return o;
}
void attn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, Tensor g, const Tensor& lse,
              const Tensor& dq, const Tensor& dk, const Tensor& dv, const Attn& a) {
  if (g.stride(2) != 1 || g.stride(1) % 8 || g.stride(0) % 8 || reinterpret_cast<uintptr_t>(g.data_ptr()) % 16)
    g = g.contiguous();
  Tensor delta = at::empty_like(lse);
  const Strides3 sq(q), sk(k), sv(v), so(o), sg(g), sdq(dq), sdk(dk), sdv(dv);
  check(lb_attention_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), g.data_ptr(), fptr(lse), fptr(delta),
                         dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), q.size(0), a.H, q.size(1), k.size(1), sq.v, sk.v,
                         sv.v, so.v, sg.v, sdq.v, sdk.v, sdv.v, a.scale, a.causal, code(q.scalar_type()), stream()),
        "lb_attention_bwd");
  g_launches += 2;
}
void keep_attn(AutogradContext* ctx, const Attn& a) {
  ctx->saved_data["H"] = a.H;
  ctx->saved_data["scale"] = a.scale;
  ctx->saved_data["causal"] = a.causal;
}
Attn attn_of(AutogradContext* ctx) {
  return {ctx->saved_data["H"].toInt(), ctx->saved_data["scale"].toDouble(), ctx->saved_data["causal"].toBool()};
}
struct AttentionNode : torch::autograd::Function<AttentionNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, int64_t H, double scale,
                        bool causal) {
    Tensor lse;
    const Attn a{H, scale, causal};
    Tensor o = attn_fwd(q, k, v, a, lse);
    ctx->save_for_backward({q, k, v, o, lse});
    keep_attn(ctx, a);
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    Tensor dq = at::empty(s[0].sizes(), s[0].options()), dk = at::empty(s[1].sizes(), s[1].options()),
           dv = at::empty(s[2].sizes(), s[2].options());
    attn_bwd(s[0], s[1], s[2], s[3], g[0], s[4], dq, dk, dv, attn_of(ctx));
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};
struct AttentionPackedNode : torch::autograd::Function<AttentionPackedNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, int64_t H, double scale, bool causal) {
    const int64_t E = qkv.size(2) / 3;
    Tensor lse;
    const Attn a{H, scale, causal};
    Tensor o = attn_fwd(qkv.narrow(2, 0, E), qkv.narrow(2, E, E), qkv.narrow(2, 2 * E, E), a, lse);
    ctx->save_for_backward({qkv, o, lse});
    keep_attn(ctx, a);
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor& qkv = s[0];
    const int64_t E = qkv.size(2) / 3;
    Tensor d = at::empty(qkv.sizes(), qkv.options());
    attn_bwd(qkv.narrow(2, 0, E), qkv.narrow(2, E, E), qkv.narrow(2, 2 * E, E), s[1], g[0], s[2], d.narrow(2, 0, E),
             d.narrow(2, E, E), d.narrow(2, 2 * E, E), attn_of(ctx));
    return {d, Tensor(), Tensor(), Tensor()};
  }
};

// ----------------------------------------------------------------------------- element-wise
struct UnaryNode : torch::autograd::Function<UnaryNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t op, double p0, double p1) {
    ctx->save_for_backward({x});
    ctx->saved_data["op"] = op;
    ctx->saved_data["p0"] = p0;
    ctx->saved_data["p1"] = p1;
    return unary_raw(op, x, Tensor(), p0, p1, 0);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor x = ctx->get_saved_variables()[0];
    return {unary_raw(ctx->saved_data["op"].toInt(), x, same_strides(g[0], x), ctx->saved_data["p0"].toDouble(),
                      ctx->saved_data["p1"].toDouble(), 1),
            Tensor(), Tensor(), Tensor()};
  }
};
Tensor binary_fwd(const Tensor& a, const Tensor& b, int64_t op) {
  Tensor out = at::empty_like(a);
  check(lb_binary(a.data_ptr(), b.data_ptr(), nullptr, out.data_ptr(), nullptr, a.numel(), op, 0, code(a.scalar_type()),
                  stream()),
        "lb_binary");
  ++g_launches;
  return out;
}
struct BinaryNode : torch::autograd::Function<BinaryNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, int64_t op, bool is_add) {
    ctx->saved_data["op"] = op;
    ctx->saved_data["add"] = is_add;
    ctx->save_for_backward({a, b});
    return binary_fwd(a, b, op);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    if (ctx->saved_data["add"].toBool()) return {g[0], g[0], Tensor(), Tensor()};      // no kernel, no copies
    const Tensor &a = s[0], &b = s[1];
    Tensor dy = same_strides(g[0], a), da = at::empty_like(a), db = at::empty_like(a);
    check(lb_binary(a.data_ptr(), b.data_ptr(), dy.data_ptr(), da.data_ptr(), db.data_ptr(), a.numel(),
                    ctx->saved_data["op"].toInt(), 1, code(a.scalar_type()), stream()),
          "lb_binary");
    ++g_launches;
    return {da, db, Tensor(), Tensor()};
  }
};
// relu(a + b): backward masks with the saved output, both inputs receive the same tensor
struct AddReluNode : torch::autograd::Function<AddReluNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, int64_t op, int64_t relu_op) {
    Tensor out = binary_fwd(a, b, op);
    ctx->saved_data["relu"] = relu_op;
    ctx->save_for_backward({out});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor out = ctx->get_saved_variables()[0];
    Tensor d = unary_raw(ctx->saved_data["relu"].toInt(), out, same_strides(g[0], out), 0.0, 0.0, 1);
    return {d, d, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------ Python entry points
// A launch waits for room in a full launch queue, so no entry point holds the interpreter's lock
// there: the threads that read the next mini-batch run on.
using NoGil = py::call_guard<py::gil_scoped_release>;

c10::intrusive_ptr<State> make_state(const optional<Tensor>& w, const optional<Tensor>& w2, const optional<Tensor>& wgrad,
                                     const optional<Tensor>& bgrad, const py::object& wh, const py::object& bh,
                                     std::vector<int64_t> i, std::vector<double> f) {
  auto s = c10::make_intrusive<State>();
  s->w = opt(w);
  s->w2 = opt(w2);
  s->wgrad = opt(wgrad);
  s->bgrad = opt(bgrad);
  s->wh = listening(wh);
  s->bh = listening(bh);
  s->i = std::move(i);
  s->f = std::move(f);
  return s;
}

}  // namespace

// ``t.backward(gradient)``, which imports PyTorch's symbolic shapes (1.4 s) to compare two shapes.
void backward(const Tensor& t, const Tensor& gradient) {
  TORCH_CHECK(t.sizes() == gradient.sizes(), "gradient of another shape");
  t.backward(gradient);
}

PYBIND11_MODULE(_lbann_autograd, m) {
  m.def("set_error_type", [](const py::object& t) { g_native_error = py::object(t).release().ptr(); });
  m.attr("abi_version") = LB_ABI_VERSION;
  m.def("launches", [] { return (long long)g_launches; });
  m.def("backward", torch::wrap_pybind_function_no_gil(backward));
  m.def("splitk_offers", [] { return (long long)g_offers; });
  m.def("gemm", [](const Tensor& a, const Tensor& b, bool ta, bool tb, const optional<Tensor>& out, int64_t out_code,
                   double alpha, double beta, const optional<Tensor>& bias, bool per_row, int64_t act, double act_param,
                   int64_t bn_hint) {
    const at::ScalarType dt = out_code == 2 ? at::kFloat : (out_code == 1 ? at::kBFloat16 : at::kHalf);
    at::AutoDispatchBelowAutograd guard;
    return gemm(a, b, ta, tb, opt(out), dt, alpha, beta, opt(bias), per_row, act, act_param, bn_hint);
  }, NoGil());
  m.def("conv_fwd", [](const Tensor& x, const Tensor& w, const optional<Tensor>& out, int64_t out_code,
                       const std::vector<int64_t>& g, const std::vector<int64_t>& dims, double alpha, double beta,
                       const optional<Tensor>& bias, int64_t act, double act_param, int64_t halo) {
    const at::ScalarType dt = out_code == 2 ? at::kFloat : (out_code == 1 ? at::kBFloat16 : at::kHalf);
    at::AutoDispatchBelowAutograd guard;
    return conv_fwd(x, w, opt(out), dt, g.data(), dims[0], dims[1], dims[2], alpha, beta, opt(bias), act, act_param,
                    halo);
  }, NoGil());
  m.def("conv_wgrad", [](const Tensor& x, const Tensor& dy, const Tensor& out, const std::vector<int64_t>& g,
                         double alpha) {
    at::AutoDispatchBelowAutograd guard;
    conv_wgrad(x, dy, out, g.data(), alpha);
  }, NoGil());
  m.def("pack_filter", [](const Tensor& w, int64_t Kout, int64_t Cin, int64_t taps, int64_t Kp, int64_t Cp,
                          int64_t dtype) {
    const auto o = w.options().dtype(dtype == 0 ? at::kHalf : at::kBFloat16).requires_grad(false);
    Tensor fwd = at::empty({taps, Kp, Cp}, o), dgrad = at::empty({taps, Cp, Kp}, o);
    check(lb_pack_filter(fptr(w), fwd.data_ptr(), dgrad.data_ptr(), Kout, Cin, taps, Kp, Cp, dtype, stream()),
          "lb_pack_filter");
    ++g_launches;
    return std::make_pair(fwd, dgrad);
  }, NoGil());
  m.def("weight_grad", [](const Tensor& dy, const Tensor& x, const Tensor& grad) {
    at::AutoDispatchBelowAutograd guard;
    weight_grad(dy, x, grad, false);
  }, NoGil());
  m.def("linear", [](const Tensor& x, const Tensor& w_leaf, const optional<Tensor>& b_leaf, const Tensor& w16,
                     const optional<Tensor>& wgrad, const optional<Tensor>& bgrad, const py::object& wh,
                     const py::object& bh, int64_t act, double act_param, const optional<Tensor>& written, int64_t at) {
    auto s = make_state(w16, {}, wgrad, bgrad, wh, bh, {act, at}, {act_param});
    s->written = opt(written);
    py::gil_scoped_release nogil;
    return LinearNode::apply(x, w_leaf, b_leaf, s);
  });
  m.def("convolution", [](const Tensor& x, const Tensor& w_leaf, const optional<Tensor>& b_leaf, const Tensor& fwd,
                          const optional<Tensor>& dgrad, const optional<Tensor>& wgrad, const optional<Tensor>& bgrad,
                          const py::object& wh, const py::object& bh, std::vector<int64_t> ints, double act_param) {
    auto s = make_state(fwd, dgrad, wgrad, bgrad, wh, bh, std::move(ints), {act_param});
    py::gil_scoped_release nogil;
    return ConvNode::apply(x, w_leaf, b_leaf, s);
  });
  m.def("batch_norm", [](const Tensor& x, const optional<Tensor>& scale, const optional<Tensor>& bias,
                         const optional<Tensor>& mean, const optional<Tensor>& var, const Tensor& ws_fwd,
                         const Tensor& ws_bwd, const optional<Tensor>& sgrad, const optional<Tensor>& bgrad,
                         const py::object& sh, const py::object& bh, std::vector<int64_t> ints, std::vector<double> f,
                         const py::object& owner) {
    auto s = make_state(ws_fwd, ws_bwd, sgrad, bgrad, sh, bh, std::move(ints), std::move(f));
    if (!owner.is_none()) s->owner = owner;
    py::gil_scoped_release nogil;
    return BatchNormNode::apply(x, scale, bias, mean, var, s);
  });
  m.def("layer_norm", [](const Tensor& x, const optional<Tensor>& scale, const optional<Tensor>& bias,
                         const optional<Tensor>& sgrad, const optional<Tensor>& bgrad, const py::object& sh,
                         const py::object& bh, int64_t cols, double eps) {
    auto s = make_state({}, {}, sgrad, bgrad, sh, bh, {cols}, {eps});
    py::gil_scoped_release nogil;
    return LayerNormNode::apply(x, scale, bias, s);
  });
  m.def("embedding", [](const Tensor& idx, const Tensor& table, const Tensor& wgrad, const py::object& wh,
                        int64_t padding, int64_t dtype) {
    auto s = make_state({}, {}, wgrad, {}, wh, py::none(), {padding, dtype}, {});
    py::gil_scoped_release nogil;
    return EmbeddingNode::apply(idx, table, s);
  });
  m.def("attention", [](const Tensor& q, const Tensor& k, const Tensor& v, int64_t H, double scale, bool causal) {
    return AttentionNode::apply(q, k, v, H, scale, causal);
  }, NoGil());
  m.def("attention_packed", [](const Tensor& qkv, int64_t H, double scale, bool causal) {
    return AttentionPackedNode::apply(qkv, H, scale, causal);
  }, NoGil());
  m.def("unary_raw", [](int64_t op, const Tensor& x, const optional<Tensor>& dy, double p0, double p1, int64_t mode) {
    at::AutoDispatchBelowAutograd guard;
    return unary_raw(op, x, opt(dy), p0, p1, mode);
  }, NoGil());
  m.def("unary", [](const Tensor& x, int64_t op, double p0, double p1) { return UnaryNode::apply(x, op, p0, p1); },
        NoGil());
  m.def("binary", [](const Tensor& a, const Tensor& b, int64_t op, bool is_add) {
    return BinaryNode::apply(a, b, op, is_add);
  }, NoGil());
  m.def("add_relu", [](const Tensor& a, const Tensor& b, int64_t op, int64_t relu_op) {
    return AddReluNode::apply(a, b, op, relu_op);
  }, NoGil());
}
