// Host side of the package in native code: operators on torch tensors and the autograd Functions of the training
// path, each a few allocations and calls into libmega_b200.so on the current stream.
//
// At the small shapes of the path the host is what a call costs: an operator through Python (checks, allocations,
// thirty converted arguments) takes 20 - 40 us, a Python autograd Function as much again each way, against 3 - 10 us
// of device time per launch.  Here an operator takes 3 - 5 us and the backward of a training pass runs in the
// autograd engine without the interpreter.
//
// fairseq/modules/norm_layer/{timestep_norm,sequence_norm}.py, fairseq/modules/fused_ops/*.py and
// fairseq/modules/moving_average_gated_attention.py:317-414 of the reference are what the Functions stand in for.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <algorithm>
#include <tuple>
#include <unordered_map>
#include <vector>

#include "mega_b200.h"

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

namespace {

PyObject* g_error = nullptr;   // the package's MegaError

void check(int status, const char* what) {
  if (status == MEGA_OK) return;
  std::string msg = std::string(what) + ": " + mega_status_string(status);
  if (status == MEGA_ERR_CUDA) msg += std::string(" (") + mega_last_cuda_error() + ")";
  if (g_error && PyGILState_Check()) {
    PyErr_SetString(g_error, msg.c_str());
    throw py::error_already_set();
  }
  throw std::runtime_error(msg);   // (a backward in the autograd engine's threads)
}

void on_cuda(const Tensor& t) {
  if (t.defined() && !t.is_cuda())
    throw std::runtime_error("mega_b200 ops run on CUDA tensors only (there is no CPU fallback)");
}
template <typename... Ts>
void on_cuda(const Tensor& t, const Ts&... rest) {
  on_cuda(t);
  on_cuda(rest...);
}

// The library takes pointers: what it reads behind one has to be there.
void expect(bool ok, const char* what) {
  if (!ok) throw py::value_error(what);
}
void expect_numel(const Tensor& t, int64_t n, const char* what) {
  if (t.defined() && t.numel() != n)
    throw py::value_error(std::string(what) + " has " + std::to_string(t.numel()) + " values, not " + std::to_string(n));
}

// device of the call and its current stream
struct Where {
  c10::cuda::CUDAGuard guard;
  void* stream;
  explicit Where(const Tensor& t) : guard(t.device()), stream(at::cuda::getCurrentCUDAStream(t.get_device()).stream()) {}
};

int dtype_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return MEGA_F32;
    case at::kBFloat16: return MEGA_BF16;
    case at::kHalf: return MEGA_F16;
    default: throw py::type_error("mega_b200 supports float32, bfloat16 and float16 activations");
  }
}

Tensor none() { return Tensor(); }
Tensor given(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

template <typename T = void>
T* ptr(const Tensor& t) {
  return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}
float* fptr(const Tensor& t) { return ptr<float>(t); }

// fp32, contiguous (parameters, statistics, states are small)
Tensor f32c(const Tensor& t) {
  if (!t.defined() || (t.scalar_type() == at::kFloat && t.is_contiguous())) return t;
  return t.detach().to(at::kFloat).contiguous();
}
// Parameters in fp32, contiguous, side by side: one launch for all that are not so already
std::vector<Tensor> f32_all(const std::vector<Tensor>& ts, void* stream) {
  std::vector<Tensor> out(ts.size());
  const void* src[8];
  float* dst[8];
  int64_t n[8], total = 0;
  int count = 0;
  auto half = [](const Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf; };
  for (const auto& t : ts) total += half(t) ? (t.numel() + 3) / 4 * 4 : 0;
  Tensor all;
  if (total) all = at::empty({total}, at::TensorOptions().dtype(at::kFloat).device(ts[0].device()));
  int64_t from = 0;
  int dt = -1;
  for (size_t i = 0; i < ts.size(); ++i) {
    const Tensor& t = ts[i];
    if (!half(t) || !t.is_contiguous() || (dt >= 0 && dtype_of(t) != dt) || count == 8) {
      out[i] = f32c(t);
      continue;
    }
    dt = dtype_of(t);
    out[i] = all.narrow(0, from, t.numel()).view(t.sizes());
    src[count] = t.data_ptr();
    dst[count] = fptr(all) + from;
    n[count++] = t.numel();
    from += (t.numel() + 3) / 4 * 4;
  }
  if (count) check(mega_to_float(src, dst, n, count, dt, stream), "to_float");
  return out;
}
// complex64 of `dims` dimensions as its interleaved floats; a real tensor has no imaginary part, unless it is (..., 2) fp32
// and so interleaved already
Tensor c64(const Tensor& t, int64_t dims) {
  if (!t.defined()) return t;
  Tensor d = t.detach();
  if (d.scalar_type() == at::kFloat && d.dim() > dims && d.size(-1) == 2) return d.contiguous();
  if (d.scalar_type() != at::kComplexFloat) d = d.to(at::kComplexFloat);
  return at::view_as_real(d.contiguous());
}

Tensor mask_u8(const Tensor& mask, int64_t bsz, int64_t length) {
  if (!mask.defined()) return mask;
  if (mask.dim() != 2 || mask.size(0) != bsz || mask.size(1) != length)
    throw py::value_error("padding_mask must be (batch, length) = (" + std::to_string(bsz) + ", " + std::to_string(length) + ")");
  return mask.scalar_type() == at::kBool ? mask.contiguous() : mask.ne(0).contiguous();
}

// uninitialised, strided like t (contiguous when t's strides leave gaps)
Tensor like(const Tensor& t) {
  if (t.is_contiguous()) return at::empty(t.sizes(), t.options().requires_grad(false));
  if (t.is_non_overlapping_and_dense()) return at::empty_strided(t.sizes(), t.strides(), t.options().requires_grad(false));
  return at::empty(t.sizes(), t.options().requires_grad(false));
}
Tensor floats(at::IntArrayRef size, const Tensor& t) {
  return at::empty(size, at::TensorOptions().dtype(at::kFloat).device(t.device()));
}
Tensor counts(int64_t n, const Tensor& t) { return at::empty({n}, at::TensorOptions().dtype(at::kLong).device(t.device())); }

#define STRIDES3(t) (t).stride(0), (t).stride(1), (t).stride(2)

// ------------------------------------------------------------------------------------------------ EMA
struct Coeffs {
  Tensor p, q, g;
};

void check_rows(int64_t rows, int64_t dim, bool bidir) {
  if (rows != (bidir ? 2 * dim : dim))
    throw py::value_error("coefficient rows " + std::to_string(rows) + " do not match embed_dim " + std::to_string(dim));
}
// p (K, N); q, gamma (K, N), complex ones interleaved; omega (D); a state (B, D, N)
void check_coeffs(const Tensor& p, const Tensor& q, const Tensor& g, const Tensor& omega, const Tensor& h, bool cplx, int64_t bsz,
                  int64_t dim, bool bidir) {
  expect(p.dim() >= 2, "coefficients must be (rows, ndim)");
  check_rows(p.size(0), dim, bidir);
  const int64_t m = cplx ? 2 : 1, n = p.size(1);
  expect_numel(p, p.size(0) * n, "p");
  expect_numel(q, p.numel() * m, "q");
  expect_numel(g, p.numel() * m, "gamma");
  expect_numel(omega, dim, "omega");
  expect_numel(h, bsz * dim * n * m, "the state");
}

Coeffs coeffs(const Tensor& alpha, const Tensor& delta, const Tensor& third, const Tensor& gamma, bool cplx, const Where& w) {
  const int64_t k = alpha.size(0), n = alpha.size(1);
  expect_numel(alpha, k * n, "alpha");
  expect_numel(delta, k * n, "delta");
  expect_numel(third, cplx ? k : k * n, cplx ? "theta" : "beta");
  expect_numel(gamma, cplx ? 2 * k * n : k * n, "gamma");
  const auto st = alpha.scalar_type();
  auto prep = [&](const Tensor& t) { return (t.scalar_type() == st ? t.detach() : t.detach().to(st)).contiguous(); };
  const Tensor a = prep(alpha), d = prep(delta), t = prep(third), g = prep(gamma);
  Tensor f = floats({(cplx ? 5 : 3) * k * n}, alpha);
  Coeffs c;
  c.p = f.narrow(0, 0, k * n).view({k, n});
  if (cplx) {
    c.q = f.narrow(0, k * n, 2 * k * n).view({k, n, 2});
    c.g = f.narrow(0, 3 * k * n, 2 * k * n).view({k, n, 2});
    check(mega_cema_coeffs(a.data_ptr(), d.data_ptr(), t.data_ptr(), g.data_ptr(), dtype_of(a), (int)k, (int)n, fptr(c.p),
                           fptr(c.q), fptr(c.g), w.stream), "cema_coeffs");
  } else {
    c.q = f.narrow(0, k * n, k * n).view({k, n});
    c.g = f.narrow(0, 2 * k * n, k * n).view({k, n});
    check(mega_ema_coeffs(a.data_ptr(), d.data_ptr(), t.data_ptr(), g.data_ptr(), dtype_of(a), (int)k, (int)n, fptr(c.p),
                          fptr(c.q), fptr(c.g), w.stream), "ema_coeffs");
  }
  return c;
}

// x (B, D, L); p (K, N), q / g (K, N) or interleaved (K, N, 2); states likewise
void run_ema(const Tensor& x, const Tensor& y, const Tensor& p, const Tensor& q, const Tensor& g, const Tensor& omega,
             const Tensor& mask, const Tensor& h_in, const Tensor& h_out, unsigned flags, int trunc, bool cplx, const Where& w) {
  const int B = (int)x.size(0), D = (int)x.size(1), L = (int)x.size(2), N = (int)p.size(1);
  auto fn = cplx ? mega_cema_fwd : mega_ema_fwd;
  check(fn(x.data_ptr(), y.data_ptr(), dtype_of(x), B, D, L, STRIDES3(x), STRIDES3(y), fptr(p), fptr(q), fptr(g), fptr(omega),
           N, ptr<uint8_t>(mask), fptr(h_in), fptr(h_out), flags, trunc, w.stream), cplx ? "cema_fwd" : "ema_fwd");
}

std::tuple<Tensor, OptTensor> ema_forward(const Tensor& x, const Tensor& p_, const Tensor& q_, const Tensor& g_,
                                          const Tensor& omega_, const OptTensor& mask_, const OptTensor& h_in_, bool want_state,
                                          int64_t flags, int64_t trunc, bool cplx, const OptTensor& out_) {
  on_cuda(x, p_, q_, g_, omega_, given(mask_), given(h_in_));
  const Where w(x);
  const int64_t bsz = x.size(0), dim = x.size(1);
  const Tensor p = f32c(p_), q = cplx ? c64(q_, 2) : f32c(q_), g = cplx ? c64(g_, 2) : f32c(g_), omega = f32c(omega_);
  const int64_t n = p.size(1);
  const Tensor mask = mask_u8(given(mask_), bsz, x.size(2));
  const Tensor h_in = cplx ? c64(given(h_in_), 3) : f32c(given(h_in_));
  check_coeffs(p, q, g, omega, h_in, cplx, bsz, dim, flags & MEGA_EMA_BIDIRECTIONAL);
  const Tensor y = out_.has_value() ? *out_ : like(x);
  expect(y.sizes() == x.sizes() && y.scalar_type() == x.scalar_type(), "out must be like x");
  Tensor h_out = want_state ? (cplx ? floats({bsz, dim, n, 2}, x) : floats({bsz, dim, n}, x)) : Tensor();
  run_ema(x, y, p, q, g, omega, mask, h_in, h_out, (unsigned)flags, (int)trunc, cplx, w);
  if (!want_state) return {y, std::nullopt};
  return {y, cplx ? at::view_as_complex(h_out) : h_out};
}

// y = silu(a) / its gradient over a dense tensor's memory
bool rows_of(const Tensor& t, int64_t cols, int64_t& rows) {
  const int64_t vec = 16 / t.element_size();
  if (!t.is_non_overlapping_and_dense() || t.numel() % cols != 0 || cols % vec != 0) return false;
  rows = t.numel() / cols;
  return true;
}

class EmaFn : public torch::autograd::Function<EmaFn> {
 public:
  // chan: x and y are (B, L, D) instead of (B, D, L)
  static Tensor forward(AutogradContext* ctx, Tensor x_, Tensor alpha, Tensor delta, Tensor third, Tensor gamma, Tensor omega,
                        OptTensor mask_, int64_t flags, int64_t trunc, bool cplx, bool silu, bool chan) {
    const Tensor x = chan ? x_.transpose(1, 2) : x_;
    on_cuda(x, alpha, delta, third, gamma, omega, given(mask_));
    expect(x.dim() == 3 && alpha.dim() >= 2, "x must have three dimensions, alpha (rows, ndim, 1)");
    check_rows(alpha.size(0), x.size(1), flags & MEGA_EMA_BIDIRECTIONAL);
    expect_numel(omega, x.size(1), "omega");
    const Where w(x);
    const Tensor mask = mask_u8(given(mask_), x.size(0), x.size(2));
    const Coeffs c = coeffs(alpha, delta, third, gamma, cplx, w);
    // (the result is a tensor of its own, not a view of one: a view made in here could not be changed in place)
    Tensor y_ = like(x_), y = chan ? y_.transpose(1, 2) : y_, out = y_;
    const auto f = f32_all({omega, alpha, delta, third}, w.stream);
    run_ema(x, y, c.p, c.q, c.g, f[0], mask, none(), none(), (unsigned)flags, (int)trunc, cplx, w);
    if (silu) {
      int64_t rows;
      if (rows_of(y_, x.size(1), rows)) {
        out = like(y_);
        check(mega_gate_silu(y_.data_ptr(), x.size(1), nullptr, 0, out.data_ptr(), x.size(1), dtype_of(y), rows, (int)x.size(1),
                             w.stream), "gate_silu");
      } else {
        out = at::silu(y_);
      }
    }
    ctx->save_for_backward({x_, f[1], f[2], f[3], f[0], mask, c.p, c.q, c.g, silu ? y : Tensor()});
    ctx->saved_data["flags"] = flags;
    ctx->saved_data["trunc"] = trunc;
    ctx->saved_data["cplx"] = cplx;
    ctx->saved_data["chan"] = chan;
    ctx->saved_data["types"] = std::vector<int64_t>{(int64_t)alpha.scalar_type(), (int64_t)delta.scalar_type(),
                                                    (int64_t)third.scalar_type(), (int64_t)gamma.scalar_type(),
                                                    (int64_t)omega.scalar_type()};
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const bool chan = ctx->saved_data["chan"].toBool();
    const Tensor x = chan ? s[0].transpose(1, 2) : s[0];
    const Tensor &alpha = s[1], &delta = s[2], &third = s[3], &omega = s[4], &mask = s[5], &p = s[6], &q = s[7], &g = s[8], &y = s[9];
    const unsigned flags = (unsigned)ctx->saved_data["flags"].toInt();
    const int trunc = (int)ctx->saved_data["trunc"].toInt();
    const bool cplx = ctx->saved_data["cplx"].toBool();
    const auto types = ctx->saved_data["types"].toIntVector();
    const Where w(x);
    Tensor dy = chan ? grads[0].transpose(1, 2) : grads[0];
    if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
    if (y.defined()) {   // through the SiLU, in y's memory order
      if (dy.strides() != y.strides()) {
        Tensor t = like(y);
        t.copy_(dy);
        dy = t;
      }
      int64_t rows;
      if (rows_of(y, x.size(1), rows)) {
        Tensor d = like(y);
        const int64_t c = x.size(1);
        check(mega_gate_silu_bwd(dy.data_ptr(), c, y.data_ptr(), c, d.data_ptr(), c, nullptr, dtype_of(y), rows, (int)c, w.stream),
              "gate_silu_bwd");
        dy = d;
      } else {
        dy = at::silu_backward(dy, y);
      }
    }
    const int B = (int)x.size(0), D = (int)x.size(1), L = (int)x.size(2);
    const int64_t k = p.size(0), n = p.size(1), kn = k * n, m = cplx ? 2 : 1;
    Tensor dx = like(x);
    // dp, dq, dgamma_hat and domega in one piece (the library zeroes them together), the raw parameters' behind them
    const int64_t sums = kn * (1 + 2 * m), raw = cplx ? 4 * kn + k : 4 * kn;
    Tensor f = floats({sums + D + raw}, x);
    float* at_ = f.data_ptr<float>();
    float *dp = at_, *dq = at_ + kn, *dg = at_ + kn * (1 + m), *dom = at_ + sums, *da = dom + D, *dd = da + kn;
    if (cplx) {
      float *dgm = dd + kn, *dt = dgm + 2 * kn;
      check(mega_cema_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), dtype_of(x), B, D, L, STRIDES3(dy), STRIDES3(x), STRIDES3(dx),
                          fptr(p), fptr(q), fptr(g), fptr(omega), (int)n, ptr<uint8_t>(mask), flags, trunc, dp, dq, dg, dom, w.stream),
            "cema_bwd");
      check(mega_cema_coeffs_bwd(fptr(alpha), fptr(delta), fptr(third), fptr(q), dp, dq, dg, (int)k, (int)n, da, dd, dt, dgm, w.stream),
            "cema_coeffs_bwd");
    } else {
      float *db = dd + kn, *dgm = db + kn;
      check(mega_ema_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), dtype_of(x), B, D, L, STRIDES3(dy), STRIDES3(x), STRIDES3(dx),
                         fptr(p), fptr(q), fptr(g), fptr(omega), (int)n, ptr<uint8_t>(mask), nullptr, nullptr, flags, trunc, dp, dq, dg,
                         dom, nullptr, w.stream), "ema_bwd");
      check(mega_ema_coeffs_bwd(fptr(alpha), fptr(delta), fptr(third), dp, dq, dg, (int)k, (int)n, da, dd, db, dgm, w.stream), "ema_coeffs_bwd");
    }
    // (one conversion where the parameters share a type; none passes through another's)
    Tensor out = f.narrow(0, sums, D + raw);
    if (std::all_of(types.begin(), types.end(), [&](int64_t t) { return t == types[0]; })) out = out.to((at::ScalarType)types[0]);
    const int64_t base = out.storage_offset();
    auto part = [&](int64_t from, at::IntArrayRef size, at::IntArrayRef stride, int64_t type) {
      Tensor v = out.as_strided(size, stride, base + from);
      return v.scalar_type() == (at::ScalarType)type ? v : v.to((at::ScalarType)type);
    };
    auto like_param = [&](int64_t from, const Tensor& t, int64_t type) { return part(from, t.sizes(), t.strides(), type); };
    const Tensor g_om = like_param(0, omega, types[4]), g_a = like_param(D, alpha, types[0]), g_d = like_param(D + kn, delta, types[1]);
    const Tensor g_3 = like_param(D + (cplx ? 4 : 2) * kn, third, types[2]);
    const Tensor g_g = cplx ? part(D + 2 * kn, {k, n, 2}, {2 * n, 2, 1}, types[3]) : part(D + 3 * kn, {k, n}, {n, 1}, types[3]);
    return {chan ? dx.transpose(1, 2) : dx, g_a, g_d, g_3, g_g, g_om, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor ema_train(const Tensor& x, const Tensor& alpha, const Tensor& delta, const Tensor& third, const Tensor& gamma,
                 const Tensor& omega, const OptTensor& mask, int64_t flags, int64_t trunc, bool cplx, bool silu,
                 bool chan) {
  return EmaFn::apply(x, alpha, delta, third, gamma, omega, mask, flags, trunc, cplx, silu, chan);
}

// ------------------------------------------------------------------------------------------------ norms
struct NormParams {
  Tensor gamma, beta, count, mean, var;
};

// The type that parameters share when the library reads it, else fp32: none of them passes through a narrower one.
at::ScalarType common_type(std::initializer_list<Tensor> ts) {
  at::ScalarType type = at::kFloat;
  bool first = true;
  for (const auto& t : ts) {
    if (!t.defined()) continue;
    const auto own = t.scalar_type();
    if ((own != at::kFloat && own != at::kBFloat16 && own != at::kHalf) || (!first && own != type)) return at::kFloat;
    type = own;
    first = false;
  }
  return type;
}
Tensor as_type(const Tensor& t, at::ScalarType type) {
  if (!t.defined()) return t;
  return (t.scalar_type() == type ? t.detach() : t.detach().to(type)).contiguous();
}

NormParams prepare(const Tensor& weight, const Tensor& bias, const Tensor& pc, const Tensor& pm, const Tensor& pl, int64_t bsz,
                   const Where& w) {
  const int64_t d = weight.size(0), g = pm.defined() ? pm.size(0) : 0;
  expect_numel(weight, d, "weight");
  expect_numel(bias, d, "bias");
  expect_numel(pm, g, "prior_mean");
  if (pm.defined()) expect_numel(pl, g, "prior_logv");
  expect(g <= d, "more prior means than features");
  const auto type = common_type({weight, bias, pm, pl});
  const Tensor wt = as_type(weight, type), b = as_type(bias, type), m = as_type(pm, type), l = as_type(pl, type);
  const Tensor c = pc.defined() ? pc.detach().to(at::kLong).contiguous() : pc;
  Tensor f = floats({2 * d + 2 * bsz * g}, weight);
  NormParams r;
  r.gamma = f.narrow(0, 0, d);
  r.beta = f.narrow(0, d, d);
  if (g) {
    r.mean = f.narrow(0, 2 * d, bsz * g).view({bsz, g});
    r.var = f.narrow(0, 2 * d + bsz * g, bsz * g).view({bsz, g});
    r.count = counts(bsz, weight);
  }
  check(mega_norm_prepare(ptr<int64_t>(c), ptr(m), ptr(l), wt.data_ptr(), b.data_ptr(), dtype_of(wt),
                          (int)(g ? bsz : 0), (int)g, (int)d, ptr<int64_t>(r.count), fptr(r.mean), fptr(r.var), fptr(r.gamma),
                          fptr(r.beta), w.stream), "norm_prepare");
  return r;
}

py::tuple norm_prepare(const Tensor& weight, const Tensor& bias, const OptTensor& pc, const OptTensor& pm, const OptTensor& pl,
                       int64_t bsz) {
  on_cuda(weight, bias, given(pc), given(pm), given(pl));
  const Where w(weight);
  const NormParams r = prepare(weight, bias, given(pc), given(pm), given(pl), bsz, w);
  if (!pm.has_value()) return py::make_tuple(r.gamma, r.beta);
  return py::make_tuple(r.gamma, r.beta, r.count, r.mean, r.var);
}

// (dweight, dbias, dprior_mean, dprior_logv), each in its parameter's type
std::vector<Tensor> finish(const Tensor& weight, const Tensor& bias, const Tensor& pm, const Tensor& logv, const float* dgamma,
                           const float* dbeta, const float* dpm, const float* dpv, int64_t bsz, int64_t g, const Where& w) {
  const int64_t d = weight.size(0);
  const auto type = common_type({weight, bias, pm, logv});
  Tensor out = at::empty({2 * d + 2 * g}, weight.options().requires_grad(false).dtype(type));
  const Tensor l = as_type(logv, type);
  char* at_ = static_cast<char*>(out.data_ptr());
  const int64_t es = out.element_size();
  check(mega_norm_finish(dpm, dpv, ptr(l), dgamma, dbeta, dtype_of(out), (int)(g ? bsz : 0), (int)g, (int)d,
                         g ? at_ + 2 * d * es : nullptr, g ? at_ + (2 * d + g) * es : nullptr, at_, at_ + d * es, w.stream),
        "norm_finish");
  auto own = [&](int64_t from, const Tensor& p) { return out.narrow(0, from, p.numel()).view(p.sizes()).to(p.scalar_type()); };
  std::vector<Tensor> r = {own(0, weight), own(d, bias)};
  if (g) {
    r.push_back(own(2 * d, pm));
    r.push_back(own(2 * d + g, logv));
  }
  return r;
}

constexpr int64_t kGridSequences = 65535;   // sequences that the kernels over time take in a launch

bool whole_rows(const Tensor& x) {   // contiguous channels in whole 16-byte pieces
  const int64_t es = x.element_size();
  return x.stride(2) == 1 && x.size(2) * es % 16 == 0 && x.stride(0) * es % 16 == 0 && x.stride(1) * es % 16 == 0 &&
         reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0;
}

std::tuple<Tensor, Tensor, Tensor, Tensor> timestep_norm_fwd(const Tensor& x, const Tensor& pc_, const Tensor& pm_, const Tensor& pv_,
                                                             const Tensor& gamma_, const Tensor& beta_, const OptTensor& mask_,
                                                             double eps, int64_t groups, const OptTensor& out_) {
  on_cuda(x, pc_, pm_, pv_, gamma_, beta_, given(mask_));
  const Where w(x);
  const int64_t bsz = x.size(0), length = x.size(1), dim = x.size(2), g = groups > 0 ? groups : dim;
  const Tensor pc = pc_.to(at::kLong).contiguous(), pm = f32c(pm_), pv = f32c(pv_), gamma = f32c(gamma_), beta = f32c(beta_);
  if (pm.dim() != 2 || pm.size(0) != bsz || pm.size(1) != g || pv.sizes() != pm.sizes())
    throw py::value_error("prev_mean/prev_var must be (batch, groups) = (" + std::to_string(bsz) + ", " + std::to_string(g) + ")");
  const Tensor mask = mask_u8(given(mask_), bsz, length);
  expect_numel(pc, bsz, "prev_count");
  expect_numel(gamma, dim, "gamma");
  expect_numel(beta, dim, "beta");
  const Tensor y = out_.has_value() ? *out_ : like(x);
  expect(y.sizes() == x.sizes() && y.scalar_type() == x.scalar_type(), "out must be like x");
  Tensor count = counts(bsz, x), st = floats({2, bsz, g}, x);
  Tensor mean = st.select(0, 0), var = st.select(0, 1);
  check(mega_timestep_norm_fwd(x.data_ptr(), y.data_ptr(), dtype_of(x), (int)bsz, (int)length, (int)dim, STRIDES3(x), STRIDES3(y),
                               ptr<int64_t>(pc), fptr(pm), fptr(pv), fptr(gamma), fptr(beta), ptr<uint8_t>(mask), (int)g, eps,
                               ptr<int64_t>(count), fptr(mean), fptr(var), w.stream), "timestep_norm_fwd");
  return {y, count, mean, var};
}

class TsnFn : public torch::autograd::Function<TsnFn> {
 public:
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor pcount, Tensor pmean, Tensor plogv, Tensor weight, Tensor bias,
                        OptTensor mask_, int64_t groups, double eps) {
    on_cuda(x, pcount, pmean, plogv, weight, bias, given(mask_));
    const Where w(x);
    const int64_t bsz = x.size(0), length = x.size(1), dim = x.size(2), g = groups > 0 ? groups : dim;
    expect_numel(weight, dim, "weight");
    expect_numel(pmean, g, "prior_mean");
    const NormParams r = prepare(weight, bias, pcount, pmean, plogv, bsz, w);
    const Tensor mask = mask_u8(given(mask_), bsz, length);
    const bool again = groups <= 0 && whole_rows(x) && bsz <= kGridSequences;
    Tensor y = like(x), count = counts(bsz, x);
    if (again) {   // the backward takes the statistics again: nothing is kept but the arguments
      Tensor st = floats({2, bsz, g}, x);
      check(mega_timestep_norm_fwd(x.data_ptr(), y.data_ptr(), dtype_of(x), (int)bsz, (int)length, (int)dim, STRIDES3(x), STRIDES3(y),
                                   ptr<int64_t>(r.count), fptr(r.mean), fptr(r.var), fptr(r.gamma), fptr(r.beta),
                                   ptr<uint8_t>(mask), (int)g, eps, ptr<int64_t>(count), fptr(st), fptr(st) + bsz * g, w.stream),
            "timestep_norm_fwd");
      ctx->save_for_backward({x, weight, plogv, r.gamma, mask, r.count, r.mean, r.var, bias, pmean});
    } else {
      Tensor st = floats({2, bsz, g}, x), cm = floats({bsz, length, g}, x), cr = floats({bsz, length, g}, x);
      Tensor gm = g != dim ? floats({bsz, length, g}, x) : Tensor();
      check(mega_timestep_norm_fwd_train(x.data_ptr(), y.data_ptr(), dtype_of(x), (int)bsz, (int)length, (int)dim, STRIDES3(x),
                                         STRIDES3(y), ptr<int64_t>(r.count), fptr(r.mean), fptr(r.var), fptr(r.gamma),
                                         fptr(r.beta), ptr<uint8_t>(mask), (int)g, eps, ptr<int64_t>(count), fptr(st),
                                         fptr(st) + bsz * g, fptr(cm), fptr(cr), fptr(gm), w.stream), "timestep_norm_fwd_train");
      ctx->save_for_backward({x, weight, plogv, r.gamma, mask, count, r.mean, Tensor(), bias, pmean, cm, cr, gm});
    }
    ctx->saved_data["again"] = again;
    ctx->saved_data["g"] = g;
    ctx->saved_data["eps"] = eps;
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &weight = s[1], &plogv = s[2], &gamma = s[3], &mask = s[4];
    const int64_t g = ctx->saved_data["g"].toInt();
    const Where w(x);
    const int64_t bsz = x.size(0), dim = x.size(2);
    Tensor dy = grads[0];
    if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
    const bool again = ctx->saved_data["again"].toBool();
    if (again && !whole_rows(dy)) dy = dy.contiguous();
    Tensor dx = like(x);
    Tensor f = floats({2 * dim + 2 * bsz * g}, x);
    float *dgamma = fptr(f), *dbeta = dgamma + dim, *dpm = dbeta + dim, *dpv = dpm + bsz * g;
    bool done = false;
    if (again) {
      const int rc = mega_timestep_norm_bwd_stats(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), dtype_of(x), (int)bsz, (int)x.size(1), (int)dim,
                                                  STRIDES3(dy), STRIDES3(x), STRIDES3(dx), nullptr, nullptr, ptr<int64_t>(s[5]),
                                                  fptr(s[6]), fptr(s[7]), fptr(gamma), ptr<uint8_t>(mask),
                                                  ctx->saved_data["eps"].toDouble(), dpm, dpv, dgamma, dbeta, w.stream);
      done = rc != MEGA_ERR_UNSUPPORTED;   // (the device had no scratch memory for it: with saves, as the other forms do)
      if (done) check(rc, "timestep_norm_bwd_stats");
    }
    if (!done) {
      Tensor count = s[5], cm, cr, gm;
      if (again) {
        const int64_t length = x.size(1);
        Tensor y = like(x), st = floats({2, bsz, g}, x);
        count = counts(bsz, x);
        cm = floats({bsz, length, g}, x);
        cr = floats({bsz, length, g}, x);
        check(mega_timestep_norm_fwd_train(x.data_ptr(), y.data_ptr(), dtype_of(x), (int)bsz, (int)length, (int)dim, STRIDES3(x),
                                           STRIDES3(y), ptr<int64_t>(s[5]), fptr(s[6]), fptr(s[7]), fptr(gamma), fptr(gamma),
                                           ptr<uint8_t>(mask), (int)g, ctx->saved_data["eps"].toDouble(), ptr<int64_t>(count),
                                           fptr(st), fptr(st) + bsz * g, fptr(cm), fptr(cr), nullptr, w.stream),
              "timestep_norm_fwd_train");
      } else {
        cm = s[10];
        cr = s[11];
        gm = s[12];
      }
      check(mega_timestep_norm_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), dtype_of(x), (int)bsz, (int)x.size(1), (int)dim,
                                   STRIDES3(dy), STRIDES3(x), STRIDES3(dx), nullptr, nullptr, fptr(s[6]), ptr<int64_t>(count),
                                   fptr(cm), fptr(cr), fptr(gm), fptr(gamma), ptr<uint8_t>(mask), (int)g, dpm, dpv, dgamma, dbeta,
                                   w.stream), "timestep_norm_bwd");
    }
    auto r = finish(weight, s[8], s[9], plogv, dgamma, dbeta, dpm, dpv, bsz, g, w);
    return {dx, Tensor(), r[2], r[3], r[0], r[1], Tensor(), Tensor(), Tensor()};
  }
};

Tensor timestep_norm_train(const Tensor& x, const Tensor& pc, const Tensor& pm, const Tensor& pl, const Tensor& weight,
                           const Tensor& bias, const OptTensor& mask, int64_t groups, double eps) {
  return TsnFn::apply(x, pc, pm, pl, weight, bias, mask, groups, eps);
}

// x (B, D, L), or (B, L, D) with length_last = false
struct Sqn {
  int64_t bsz, dim, length, sb, sd, sl;
};
Sqn sqn_view(const Tensor& x, bool length_last) {
  if (length_last) return {x.size(0), x.size(1), x.size(2), x.stride(0), x.stride(1), x.stride(2)};
  return {x.size(0), x.size(2), x.size(1), x.stride(0), x.stride(2), x.stride(1)};
}

void run_sqn(const Tensor& x, const Tensor& y, const Tensor& gamma, const Tensor& beta, const Tensor& mask, double eps,
             bool length_last, int64_t g, const Tensor& count, const Tensor& mean, const Tensor& rstd, const Where& w) {
  const Sqn a = sqn_view(x, length_last), o = sqn_view(y, length_last);
  check(mega_sequence_norm_fwd(x.data_ptr(), y.data_ptr(), dtype_of(x), (int)a.bsz, (int)a.dim, (int)a.length, a.sb, a.sd, a.sl, o.sb,
                               o.sd, o.sl, fptr(gamma), fptr(beta), ptr<uint8_t>(mask), (int)g, eps, ptr<int64_t>(count),
                               fptr(mean), fptr(rstd), w.stream), "sequence_norm_fwd");
}

std::tuple<Tensor, Tensor, Tensor, Tensor> sequence_norm_fwd(const Tensor& x, const Tensor& gamma_, const Tensor& beta_,
                                                             const OptTensor& mask_, double eps, bool length_last, int64_t groups,
                                                             const OptTensor& out_) {
  on_cuda(x, gamma_, beta_, given(mask_));
  const Where w(x);
  const Sqn a = sqn_view(x, length_last);
  const int64_t g = groups > 0 ? groups : a.dim;
  const Tensor mask = mask_u8(given(mask_), a.bsz, a.length);
  expect_numel(gamma_, a.dim, "gamma");
  expect_numel(beta_, a.dim, "beta");
  const Tensor y = out_.has_value() ? *out_ : like(x);
  expect(y.sizes() == x.sizes() && y.scalar_type() == x.scalar_type(), "out must be like x");
  Tensor count = counts(a.bsz, x), st = floats({2, a.bsz, g}, x);
  Tensor mean = st.select(0, 0), rstd = st.select(0, 1);
  run_sqn(x, y, f32c(gamma_), f32c(beta_), mask, eps, length_last, g, count, mean, rstd, w);
  return {y, count, mean, rstd};
}

class SqnFn : public torch::autograd::Function<SqnFn> {
 public:
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor weight, Tensor bias, OptTensor mask_, double eps, bool length_last,
                        int64_t groups) {
    on_cuda(x, weight, bias, given(mask_));
    const Where w(x);
    const Sqn a = sqn_view(x, length_last);
    const int64_t g = groups > 0 ? groups : a.dim;
    expect_numel(weight, a.dim, "weight");
    const NormParams r = prepare(weight, bias, none(), none(), none(), 0, w);
    const Tensor mask = mask_u8(given(mask_), a.bsz, a.length);
    Tensor y = like(x), count = counts(a.bsz, x), st = floats({2, a.bsz, g}, x);
    Tensor mean = st.select(0, 0), rstd = st.select(0, 1);
    run_sqn(x, y, r.gamma, r.beta, mask, eps, length_last, g, count, mean, rstd, w);
    ctx->save_for_backward({x, weight, r.gamma, mask, count, mean, rstd, bias});
    ctx->saved_data["ll"] = length_last;
    ctx->saved_data["g"] = g;
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &weight = s[1];
    const bool ll = ctx->saved_data["ll"].toBool();
    const Where w(x);
    Tensor dy = grads[0];
    if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
    Tensor dx = like(x);
    const Sqn a = sqn_view(x, ll), q = sqn_view(dy, ll), o = sqn_view(dx, ll);
    Tensor f = floats({2 * a.dim}, x);
    check(mega_sequence_norm_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), dtype_of(x), (int)a.bsz, (int)a.dim, (int)a.length, q.sb,
                                 q.sd, q.sl, a.sb, a.sd, a.sl, o.sb, o.sd, o.sl, ptr<int64_t>(s[4]), fptr(s[5]), fptr(s[6]),
                                 fptr(s[2]), ptr<uint8_t>(s[3]), (int)ctx->saved_data["g"].toInt(), fptr(f), fptr(f) + a.dim,
                                 w.stream), "sequence_norm_bwd");
    auto r = finish(weight, s[7], none(), none(), fptr(f), fptr(f) + a.dim, nullptr, nullptr, 0, 0, w);
    return {dx, r[0], r[1], Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor sequence_norm_train(const Tensor& x, const Tensor& weight, const Tensor& bias, const OptTensor& mask, double eps,
                           bool length_last, int64_t groups) {
  return SqnFn::apply(x, weight, bias, mask, eps, length_last, groups);
}

// ---------------------------------------------------------------------------------------- fused norm -> EMA
// (y, count, mean, var, h or None, xn or None)
py::tuple tsn_ema_forward(const Tensor& x, const Tensor& pc_, const Tensor& pm_, const Tensor& pv_, const Tensor& gamma_,
                          const Tensor& beta_, double eps, const Tensor& p_, const Tensor& q_, const Tensor& g_,
                          const Tensor& omega_, const OptTensor& mask_, const OptTensor& h_in_, bool want_state, bool silu,
                          bool want_normed, bool cplx) {
  on_cuda(x, pc_, pm_, pv_, gamma_, beta_, p_, q_, g_, omega_, given(mask_), given(h_in_));
  const Where w(x);
  const int64_t bsz = x.size(0), length = x.size(1), dim = x.size(2);
  const Tensor pc = pc_.to(at::kLong).contiguous(), pm = f32c(pm_), pv = f32c(pv_), gamma = f32c(gamma_), beta = f32c(beta_);
  const Tensor p = f32c(p_), q = cplx ? c64(q_, 2) : f32c(q_), g = cplx ? c64(g_, 2) : f32c(g_), omega = f32c(omega_);
  const Tensor h_in = cplx ? c64(given(h_in_), 3) : f32c(given(h_in_));
  const int64_t n = p.size(1);
  check_coeffs(p, q, g, omega, h_in, cplx, bsz, dim, false);
  expect_numel(pc, bsz, "prev_count");
  expect_numel(pm, bsz * dim, "prev_mean");
  expect_numel(pv, bsz * dim, "prev_var");
  expect_numel(gamma, dim, "gamma");
  expect_numel(beta, dim, "beta");
  const Tensor mask = mask_u8(given(mask_), bsz, length);
  Tensor y = like(x), xn = want_normed ? like(y) : Tensor();
  Tensor count = counts(bsz, x), st = floats({2, bsz, dim}, x);
  Tensor mean = st.select(0, 0), var = st.select(0, 1);
  Tensor h_out = want_state ? (cplx ? floats({bsz, dim, n, 2}, x) : floats({bsz, dim, n}, x)) : Tensor();
  auto fn = cplx ? mega_tsn_cema_fwd : mega_tsn_ema_fwd;
  check(fn(x.data_ptr(), y.data_ptr(), ptr(xn), dtype_of(x), (int)bsz, (int)length, (int)dim, STRIDES3(x), STRIDES3(y),
           ptr<int64_t>(pc), fptr(pm), fptr(pv), fptr(gamma), fptr(beta), eps, ptr<int64_t>(count), fptr(mean), fptr(var), fptr(p),
           fptr(q), fptr(g), fptr(omega), (int)n, ptr<uint8_t>(mask), fptr(h_in), fptr(h_out), silu ? MEGA_EMA_SILU : 0u,
           w.stream), cplx ? "tsn_cema_fwd" : "tsn_ema_fwd");
  py::object h = py::none(), nx = py::none();
  if (want_state) h = py::cast(cplx ? at::view_as_complex(h_out) : h_out);
  if (want_normed) nx = py::cast(xn);
  return py::make_tuple(y, count, mean, var, h, nx);
}

// y, or None outside the fused kernel's envelope
OptTensor sqn_ema_forward(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& p_, const Tensor& q_,
                          const Tensor& g_, const Tensor& omega_, const OptTensor& mask_, int64_t flags) {
  on_cuda(x, gamma, beta, p_, q_, g_, omega_, given(mask_));
  if (x.stride(2) != 1) return std::nullopt;
  const Where w(x);
  const Tensor p = f32c(p_), q = f32c(q_), g = f32c(g_), omega = f32c(omega_), ga = f32c(gamma), be = f32c(beta);
  check_coeffs(p, q, g, omega, none(), false, x.size(0), x.size(1), flags & MEGA_EMA_BIDIRECTIONAL);
  expect_numel(ga, x.size(1), "gamma");
  expect_numel(be, x.size(1), "beta");
  const Tensor mask = mask_u8(given(mask_), x.size(0), x.size(2));
  Tensor y = at::empty(x.sizes(), x.options().requires_grad(false));
  const int rc = mega_sqn_ema_fwd(x.data_ptr(), y.data_ptr(), dtype_of(x), (int)x.size(0), (int)x.size(1), (int)x.size(2), STRIDES3(x),
                                  STRIDES3(y), fptr(ga), fptr(be), eps, nullptr, nullptr, nullptr, fptr(p), fptr(q), fptr(g),
                                  fptr(omega), (int)p.size(1), ptr<uint8_t>(mask), (unsigned)flags, w.stream);
  if (rc == MEGA_ERR_UNSUPPORTED) return std::nullopt;
  check(rc, "sqn_ema_fwd");
  return y;
}

// ------------------------------------------------------------------------------------------------ the block
// Row-major matrix view of a tensor's last dimension with one row pitch; copied when it is none.
struct Rows {
  Tensor t;
  int64_t rows, cols, ld;
};
Rows rows_view(const Tensor& t) {
  const int64_t cols = t.size(-1);
  bool ok = t.dim() >= 2 && (t.stride(-1) == 1 || cols == 1);
  int64_t ld = cols;
  if (ok) {
    ld = t.size(-2) > 1 ? t.stride(-2) : std::max(cols, t.stride(-2));
    int64_t exp = ld;
    for (int64_t i = t.dim() - 2; i >= 0; --i) {
      if (t.size(i) != 1 && t.stride(i) != exp) ok = false;
      exp *= t.size(i);
    }
  }
  if (!ok || ld < cols) return {t.contiguous(), t.numel() / cols, cols, cols};
  return {t, t.numel() / cols, cols, ld};
}
Tensor fresh(const Tensor& t) { return at::empty(t.sizes(), t.options().requires_grad(false)); }

Tensor gate_silu(const Tensor& a, const OptTensor& b) {
  on_cuda(a, given(b));
  const Where w(a);
  const Rows ra = rows_view(a);
  Tensor y = fresh(a);
  Rows rb{Tensor(), 0, 0, 0};
  if (b.has_value()) rb = rows_view(*b);
  check(mega_gate_silu(ra.t.data_ptr(), ra.ld, ptr(rb.t), rb.ld, y.data_ptr(), ra.cols, dtype_of(a), ra.rows, (int)ra.cols, w.stream),
        "gate_silu");
  return y;
}

Tensor gate_mul_silu(const Tensor& a, const Tensor& r) {
  on_cuda(a, r);
  const Where w(a);
  const Rows ra = rows_view(a), rr = rows_view(r);
  Tensor y = fresh(a);
  check(mega_gate_mul_silu(ra.t.data_ptr(), ra.ld, rr.t.data_ptr(), rr.ld, y.data_ptr(), ra.cols, dtype_of(a), ra.rows, (int)ra.cols,
                           w.stream), "gate_mul_silu");
  return y;
}

Tensor gate_output(const Tensor& residual, const Tensor& u, const Tensor& hx, const Tensor& h_lin) {
  on_cuda(residual, u, hx, h_lin);
  const Where w(residual);
  const Rows r = rows_view(residual), ru = rows_view(u), rx = rows_view(hx), rh = rows_view(h_lin);
  Tensor y = fresh(residual);
  check(mega_gate_output(r.t.data_ptr(), r.ld, ru.t.data_ptr(), ru.ld, rx.t.data_ptr(), rx.ld, rh.t.data_ptr(), rh.ld, y.data_ptr(),
                         r.cols, dtype_of(residual), r.rows, (int)r.cols, w.stream), "gate_output");
  return y;
}

// rot: fp32 (positions, S / 2, 2), or None
std::tuple<Tensor, Tensor> gate_qk(const Tensor& z, const Tensor& gamma, const Tensor& beta, const OptTensor& rot, int64_t period,
                                   int64_t q_offset, double eps) {
  on_cuda(z, gamma, beta, given(rot));
  const Where w(z);
  const Rows r = rows_view(z);
  const Tensor g = f32c(gamma), b = f32c(beta);
  if (g.dim() != 2 || g.size(0) != 2 || g.size(1) != r.cols || b.sizes() != g.sizes())
    throw py::value_error("gate_qk: gamma and beta must be (2, " + std::to_string(r.cols) + ")");
  Tensor q = fresh(z), k = fresh(z);
  if (!rot.has_value()) {
    check(mega_gate_qk(r.t.data_ptr(), r.ld, fptr(g), fptr(b), q.data_ptr(), r.cols, k.data_ptr(), r.cols, dtype_of(z), r.rows,
                       (int)r.cols, eps, w.stream), "gate_qk");
    return {q, k};
  }
  Tensor t = rot->is_complex() ? at::view_as_real(*rot) : *rot;
  t = f32c(t);
  if (t.dim() != 3 || t.size(1) * 2 != r.cols || t.size(2) != 2)
    throw py::value_error("gate_qk_rotary: rot must be (positions, S / 2) complex or (positions, S / 2, 2) float");
  check(mega_gate_qk_rotary(r.t.data_ptr(), r.ld, fptr(g), fptr(b), fptr(t), (int)t.size(0), (int)period, (int)q_offset, q.data_ptr(),
                            r.cols, k.data_ptr(), r.cols, dtype_of(z), r.rows, (int)r.cols, eps, w.stream), "gate_qk_rotary");
  return {q, k};
}

Tensor softmax_fwd(const Tensor& x, bool causal) {
  on_cuda(x);
  const Where w(x);
  const Tensor xc = x.contiguous();
  const int64_t outer = xc.size(-2), inner = xc.size(-1);
  Tensor y = fresh(xc);
  check(mega_attention_softmax_fwd(xc.data_ptr(), y.data_ptr(), dtype_of(xc), xc.numel() / (outer * inner), outer, (int)inner, causal,
                                   w.stream), "attention_softmax_fwd");
  return y;
}

// the shapes that pointers into the projections' outputs rely on
void check_block(const Tensor& x, const Tensor& wv, const Tensor& wm, const Tensor& wh, const Tensor& gamma, const Tensor& beta,
                 const Tensor& bias, const Tensor& rot, int64_t period) {
  const int64_t d = x.size(2), s = gamma.size(1), e = wv.size(0);
  expect(wv.dim() == 2 && wv.size(1) == d && wm.dim() == 2 && wm.size(0) == 2 * d + s + e && wm.size(1) == d && wh.dim() == 2 &&
             wh.size(0) == d && wh.size(1) == e, "projections do not fit the block");
  expect(gamma.numel() == 2 * s && beta.numel() == 2 * s, "gamma and beta must be (2, zdim)");
  expect(period > 0 && x.size(0) * x.size(1) % period == 0, "chunks do not divide the sequence");
  expect(!bias.defined() || bias.numel() >= 2 * period - 1, "relative bias too short");
  expect(!rot.defined() || rot.numel() >= period * s, "rotary table too short");
}

// Training pass from the moving average to the output.  bias: learned relative bias (2 P - 1), or rot: rotary table
// (positions, S / 2, 2) with the causal mask; rows (b, t) sit at position t % period of their chunk.
class BlockFn : public torch::autograd::Function<BlockFn> {
 public:
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor xn, Tensor mx, Tensor wv, Tensor bv, Tensor wm, Tensor bm, Tensor wh,
                        Tensor gamma, Tensor beta, OptTensor bias_, OptTensor rot_, OptTensor mask_, int64_t period) {
    on_cuda(x, xn, mx, wv, bv, wm, bm, wh, gamma, beta, given(bias_), given(rot_), given(mask_));
    const Where w(x);
    const int64_t bsz = x.size(0), seq = x.size(1), d = x.size(2), rows = bsz * seq, s = gamma.size(1), e = wv.size(0);
    const int64_t f = 2 * d + s + e, nb = rows / period;
    check_block(x, wv, wm, wh, gamma, beta, given(bias_), given(rot_), period);
    const int dt = dtype_of(x);
    const int64_t es = x.element_size();
    const Tensor bias = given(bias_), rot = given(rot_);
    const Tensor x_ = x, xn_ = xn, mx_ = mx;
    x = x.contiguous();
    xn = xn.contiguous().view({rows, d});
    mx = mx.contiguous().view({rows, d});
    Tensor v_lin = at::addmm(bv, xn, wv.t());
    Tensor base = at::addmm(bm, mx, wm.t());
    char* bp = static_cast<char*>(base.data_ptr());
    char *u = bp, *z = bp + d * es, *r = z + s * es, *hx = r + e * es;
    Tensor v = fresh(v_lin);
    check(mega_gate_silu(v_lin.data_ptr(), e, nullptr, 0, v.data_ptr(), e, dt, rows, (int)e, w.stream), "gate_silu");
    const auto affine = f32_all({gamma, beta}, w.stream);
    const Tensor &ga = affine[0], &be = affine[1];
    Tensor q = at::empty({nb, period, s}, x.options().requires_grad(false)), k = fresh(q);
    if (rot.defined())
      check(mega_gate_qk_rotary(z, f, fptr(ga), fptr(be), fptr(rot), (int)rot.size(0), (int)period, 0, q.data_ptr(), s, k.data_ptr(), s,
                                dt, rows, (int)s, 1e-5, w.stream), "gate_qk_rotary");
    else
      check(mega_gate_qk(z, f, fptr(ga), fptr(be), q.data_ptr(), s, k.data_ptr(), s, dt, rows, (int)s, 1e-5, w.stream), "gate_qk");
    Tensor v3 = v.view({nb, period, e});
    Tensor wgt;
    {
      Tensor scores = at::bmm(q, k.transpose(1, 2));
      wgt = fresh(scores);
      if (rot.defined()) {
        check(mega_attention_softmax_fwd(scores.data_ptr(), wgt.data_ptr(), dt, nb, period, (int)period, 1, w.stream),
              "attention_softmax_fwd");
      } else {
        const Tensor mask = mask_u8(given(mask_), bsz, seq);
        const Tensor b = bias.scalar_type() == x.scalar_type() ? bias.detach().contiguous() : bias.detach().to(x.scalar_type()).contiguous();
        check(mega_attention_bias_softmax_fwd(scores.data_ptr(), wgt.data_ptr(), b.data_ptr(), (int)((b.size(0) + 1) / 2),
                                              ptr<uint8_t>(mask), dt, nb, (int)period, (int)period, w.stream),
              "attention_bias_softmax_fwd");
      }
    }
    Tensor attn = at::bmm(wgt, v3).view({rows, e});
    Tensor gated = fresh(attn);
    check(mega_gate_mul_silu(attn.data_ptr(), e, r, f, gated.data_ptr(), e, dt, rows, (int)e, w.stream), "gate_mul_silu");
    Tensor h_lin = at::mm(gated, wh.t());
    Tensor out = at::empty({bsz, seq, d}, x.options().requires_grad(false));
    check(mega_gate_output(x.data_ptr(), d, u, f, hx, f, h_lin.data_ptr(), d, out.data_ptr(), d, dt, rows, (int)d, w.stream), "gate_output");
    ctx->save_for_backward({x_, xn_, mx_, wv, wm, wh, ga, bias, rot, v_lin, base, q, k, v3, wgt, attn, gated, h_lin, bv, bm, gamma, beta,
                            rot.defined() ? Tensor() : mask_u8(given(mask_), bsz, seq)});
    ctx->saved_data["period"] = period;
    ctx->saved_data["types"] = std::vector<int64_t>{(int64_t)bv.scalar_type(), (int64_t)bm.scalar_type(), (int64_t)gamma.scalar_type(),
                                                    (int64_t)beta.scalar_type()};
    return out;
  }

  // The pass in torch operations, for a gradient that is to be differentiated again: the gradients of the inputs as
  // functions of the inputs.  (Through aliases of them: an input that another one was computed from gets its own share.)
  static variable_list differentiable(AutogradContext* ctx, const variable_list& sv, Tensor dout) {
    const int64_t period = ctx->saved_data["period"].toInt();
    std::vector<Tensor> in = {sv[0], sv[1], sv[2], sv[3], sv[18], sv[4], sv[19], sv[5], sv[20], sv[21], sv[7]};
    for (auto& t : in)
      if (t.defined()) t = t.view_as(t);
    const Tensor &x = in[0], &xn = in[1], &mx = in[2], &wv = in[3], &bv = in[4], &wm = in[5], &bm = in[6], &wh = in[7], &gamma = in[8],
                 &beta = in[9], &bias = in[10], &rot = sv[8], &mask = sv[22];
    const int64_t bsz = x.size(0), seq = x.size(1), d = x.size(2), s = gamma.size(1), e = wv.size(0), nb = bsz * seq / period;
    const auto type = x.scalar_type();
    const Tensor v = at::silu(at::linear(xn, wv, bv)).reshape({nb, period, e}), base = at::linear(mx, wm, bm);
    const Tensor u = base.narrow(2, 0, d), z = base.narrow(2, d, s), r = base.narrow(2, d + s, e), hx = base.narrow(2, d + s + e, d);
    const Tensor zn = z / z.norm(2, {-1}, true).clamp_min(1e-5);
    auto part = [&](int64_t i) {
      Tensor t = (zn * (gamma[i] + 1.0) + beta[i]).reshape({nb, period, s});
      if (!rot.defined()) return t.to(type);
      const Tensor w = rot.narrow(0, 0, period), f = t.to(at::kFloat).reshape({nb, period, s / 2, 2});
      const Tensor a = f.select(3, 0), b = f.select(3, 1), c = w.select(2, 0), i_ = w.select(2, 1);
      return at::stack({a * c - b * i_, a * i_ + b * c}, -1).flatten(2).to(type);
    };
    Tensor scores = at::bmm(part(0), part(1).transpose(1, 2));
    const auto where = scores.options().requires_grad(false);
    if (rot.defined()) {
      scores = scores.masked_fill(at::ones({period, period}, where.dtype(at::kBool)).triu(1), -INFINITY);
    } else {
      const Tensor at_ = at::arange(period, where.dtype(at::kLong));
      scores = scores + bias.index({at_.unsqueeze(0) - at_.unsqueeze(1) + (bias.size(0) + 1) / 2 - 1});
      if (mask.defined()) {
        const Tensor m = mask.reshape({nb, period}).to(at::kBool);
        scores = scores.masked_fill(m.logical_and(m.all(1, true).logical_not()).unsqueeze(1), -INFINITY);
      }
    }
    const Tensor attn = at::bmm(scores.to(at::kFloat).softmax(-1).to(type), v).reshape({bsz, seq, e});
    const Tensor h = at::silu(hx + at::linear(attn * at::silu(r), wh));
    const Tensor out = at::addcmul(x, u.sigmoid(), h - x);
    variable_list wanted, result(14);
    std::vector<size_t> place;
    for (size_t i = 0; i < in.size(); ++i)
      if (in[i].defined() && in[i].requires_grad()) {
        wanted.push_back(in[i]);
        place.push_back(i);
      }
    const auto g = torch::autograd::grad({out}, wanted, {dout}, true, true, true);
    for (size_t i = 0; i < place.size(); ++i) result[place[i]] = g[i];
    return result;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto sv = ctx->get_saved_variables();
    if (at::GradMode::is_enabled()) return differentiable(ctx, sv, grads[0].to(sv[0].scalar_type()));
    const Tensor x = sv[0].contiguous(), xn = sv[1].contiguous().flatten(0, 1), mx = sv[2].contiguous().flatten(0, 1);
    const Tensor &wv = sv[3], &wm = sv[4], &wh = sv[5], &ga = sv[6], &bias = sv[7], &rot = sv[8],
                 &v_lin = sv[9], &base = sv[10], &q = sv[11], &k = sv[12], &v3 = sv[13], &wgt = sv[14], &attn = sv[15], &gated = sv[16],
                 &h_lin = sv[17];
    const Where w(x);
    const int64_t period = ctx->saved_data["period"].toInt();
    const auto types = ctx->saved_data["types"].toIntVector();
    const int64_t bsz = x.size(0), seq = x.size(1), d = x.size(2), rows = bsz * seq, s = ga.size(1), e = wv.size(0), nb = rows / period;
    const int64_t f = base.size(1), nbias = bias.defined() ? bias.size(0) : 0;
    const int dt = dtype_of(x);
    const int64_t es = x.element_size();
    Tensor dout = grads[0];
    if (dout.scalar_type() != x.scalar_type()) dout = dout.to(x.scalar_type());
    dout = dout.contiguous();
    // every sum in one zeroed piece: bias gradients of v_proj and mx_proj, the (2, s) affine, the relative bias
    Tensor sums = at::zeros({e + f + 4 * s + nbias}, at::TensorOptions().dtype(at::kFloat).device(x.device()));
    float *sbv = fptr(sums), *sbm = sbv + e, *sg = sbm + f, *sb = sg + 2 * s, *srel = sb + 2 * s;
    Tensor dbase = fresh(base), dx = fresh(x);
    auto cut = [&](const Tensor& t, char*& u, char*& z, char*& r, char*& hx) {
      u = static_cast<char*>(t.data_ptr());
      z = u + d * es;
      r = z + s * es;
      hx = r + e * es;
    };
    char *u, *z, *r, *hx, *du, *dz, *dr, *dhx;
    cut(base, u, z, r, hx);
    cut(dbase, du, dz, dr, dhx);
    check(mega_gate_output_bwd(dout.data_ptr(), d, x.data_ptr(), d, u, f, hx, f, h_lin.data_ptr(), d, dx.data_ptr(), d, du, f, dhx, f, sbm,
                               sbm + d + s + e, dt, rows, (int)d, w.stream), "gate_output_bwd");
    const Tensor dh = dbase.narrow(1, d + s + e, d);
    Tensor dgated = at::mm(dh, wh);
    const bool need_xn = ctx->needs_input_grad(1), need_mx = ctx->needs_input_grad(2), need_wv = ctx->needs_input_grad(3),
               need_wm = ctx->needs_input_grad(5), need_wh = ctx->needs_input_grad(7);
    Tensor dwh = need_wh ? at::mm(dh.t(), gated) : Tensor();
    check(mega_gate_mul_silu_bwd(dgated.data_ptr(), e, attn.data_ptr(), e, r, f, dgated.data_ptr(), e, dr, f, sbm + d + s, dt, rows, (int)e,
                                 w.stream), "gate_mul_silu_bwd");
    const Tensor dattn = dgated.view({nb, period, e});
    Tensor dv = at::bmm(wgt.transpose(1, 2), dattn).view({rows, e});
    Tensor ds;
    {
      Tensor dw = at::bmm(dattn, v3.transpose(1, 2));
      ds = fresh(dw);
      check(mega_attention_softmax_bwd(dw.data_ptr(), wgt.data_ptr(), ds.data_ptr(), dt, nb, period, (int)period, rot.defined() ? 1 : 0,
                                       w.stream), "attention_softmax_bwd");
    }
    if (nbias)
      check(mega_attention_bias_grad(ds.data_ptr(), srel, (int)((nbias + 1) / 2), dt, nb, (int)period, (int)period, w.stream),
            "attention_bias_grad");
    Tensor dq = at::bmm(ds, k), dk = at::bmm(ds.transpose(1, 2), q);
    check(mega_gate_qk_bwd(z, f, fptr(ga), fptr(rot), rot.defined() ? (int)rot.size(0) : 0, (int)period, 0, dq.data_ptr(), s, dk.data_ptr(),
                           s, dz, f, sg, sb, sbm + d, dt, rows, (int)s, 1e-5, w.stream), "gate_qk_bwd");
    check(mega_gate_silu_bwd(dv.data_ptr(), e, v_lin.data_ptr(), e, dv.data_ptr(), e, sbv, dt, rows, (int)e, w.stream), "gate_silu_bwd");
    Tensor dxn = need_xn ? at::mm(dv, wv).view({bsz, seq, d}) : Tensor();
    Tensor dwv = need_wv ? at::mm(dv.t(), xn) : Tensor();
    Tensor dmx = need_mx ? at::mm(dbase, wm).view({bsz, seq, d}) : Tensor();
    Tensor dwm = need_wm ? at::mm(dbase.t(), mx) : Tensor();
    const auto own = wv.scalar_type();   // (one conversion where all share it; none passes through another's type)
    const bool same = std::all_of(types.begin(), types.end(), [&](int64_t t) { return t == (int64_t)own; }) &&
                      (!nbias || bias.scalar_type() == own);
    Tensor flat = same ? sums.to(own) : sums;
    auto part = [&](int64_t from, int64_t count, int64_t type) {
      Tensor t = flat.narrow(0, from, count);
      return t.scalar_type() == (at::ScalarType)type ? t : t.to((at::ScalarType)type);
    };
    return {dx, dxn, dmx, dwv, part(0, e, types[0]), dwm, part(e, f, types[1]), dwh, part(e + f, 2 * s, types[2]).view({2, s}),
            part(e + f + 2 * s, 2 * s, types[3]).view({2, s}),
            nbias ? part(e + f + 4 * s, nbias, (int64_t)bias.scalar_type()) : Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// Inference from the moving average to the output, chunked causal attention with rotary positions.  cache: the keys
// (before their rotation) and values come back too, as a decoding state keeps them.
std::tuple<Tensor, Tensor, Tensor> block_infer(Tensor x, Tensor xn, Tensor mx, const Tensor& wv, const Tensor& bv, const Tensor& wm,
                                               const Tensor& bm, const Tensor& wh, const Tensor& gamma, const Tensor& beta,
                                               const Tensor& rot, int64_t period, bool cache) {
  on_cuda(x, xn, mx, wv, bv, wm, bm, wh, gamma, beta, rot);
  check_block(x, wv, wm, wh, gamma, beta, none(), rot, period);
  const Where w(x);
  const int64_t bsz = x.size(0), seq = x.size(1), d = x.size(2), rows = bsz * seq, s = gamma.size(1), e = wv.size(0);
  const int64_t f = 2 * d + s + e, nb = rows / period;
  const int dt = dtype_of(x);
  const int64_t es = x.element_size();
  x = x.contiguous();
  const Tensor xn2 = xn.contiguous().view({rows, d}), mx2 = mx.contiguous().view({rows, d});
  // (score rows and reduction indices in whole 16-byte pieces: the library's products are several times faster on them;
  // the positions in between are of no row's causal range, and their values zero.  It takes a launch for each chunk, so at 32
  // chunks the two are level: 32 of 500 take 615 us with the pitch, 33 of 500 take 605 without)
  const int64_t pitch = period % 8 && nb <= 32 ? (period + 7) / 8 * 8 : period;
  Tensor v_lin = at::addmm(bv, xn2, wv.t()), v3 = v_lin.view({nb, period, e}), vp = v3;
  if (pitch != period) {
    vp = at::empty({nb, pitch, e}, x.options());
    vp.narrow(1, period, pitch - period).zero_();
    v3 = vp.narrow(1, 0, period);
    for (int64_t i = 0; i < nb; ++i)
      check(mega_gate_silu(static_cast<char*>(v_lin.data_ptr()) + i * period * e * es, e, nullptr, 0,
                           static_cast<char*>(vp.data_ptr()) + i * pitch * e * es, e, dt, period, (int)e, w.stream), "gate_silu");
  } else {
    check(mega_gate_silu(v_lin.data_ptr(), e, nullptr, 0, v_lin.data_ptr(), e, dt, rows, (int)e, w.stream), "gate_silu");
  }
  const Tensor base = at::addmm(bm, mx2, wm.t());
  char* bp = static_cast<char*>(base.data_ptr());
  char *u = bp, *z = bp + d * es, *r = z + s * es, *hx = r + e * es;
  const auto affine = f32_all({gamma, beta}, w.stream);
  const Tensor &ga = affine[0], &be = affine[1];
  Tensor q = at::empty({nb, pitch, s}, x.options()), k = fresh(q), raw;
  if (cache) raw = at::empty({bsz, seq, s}, x.options());
  check(mega_gate_qk_rotary_cache(z, f, fptr(ga), fptr(be), fptr(rot), (int)rot.size(0), (int)period, 0, (int)pitch, q.data_ptr(), s,
                                  k.data_ptr(), s, ptr(raw), dt, rows, (int)s, 1e-5, w.stream), "gate_qk_rotary");
  const Tensor scores = at::bmm(q, k.transpose(1, 2));
  Tensor wgt = fresh(scores);
  check(mega_attention_softmax_fwd(scores.data_ptr(), wgt.data_ptr(), dt, nb, pitch, (int)pitch, 1, w.stream), "attention_softmax_fwd");
  Tensor attn = at::bmm(wgt.narrow(1, 0, period), vp).view({rows, e});
  check(mega_gate_mul_silu(attn.data_ptr(), e, r, f, attn.data_ptr(), e, dt, rows, (int)e, w.stream), "gate_mul_silu");
  Tensor out = at::mm(attn, wh.t()).view({bsz, seq, d});
  check(mega_gate_output(x.data_ptr(), d, u, f, hx, f, out.data_ptr(), d, out.data_ptr(), d, dt, rows, (int)d, w.stream), "gate_output");
  return {out, raw, cache ? v3.reshape({bsz, seq, e}) : Tensor()};
}

Tensor block_train(const Tensor& x, const Tensor& xn, const Tensor& mx, const Tensor& wv, const Tensor& bv, const Tensor& wm,
                   const Tensor& bm, const Tensor& wh, const Tensor& gamma, const Tensor& beta, const OptTensor& bias,
                   const OptTensor& rot, const OptTensor& mask, int64_t period) {
  return BlockFn::apply(x, xn, mx, wv, bv, wm, bm, wh, gamma, beta, bias, rot, mask, period);
}

// ------------------------------------------------------------------------------------ single-token step
// TimestepNorm -> EMA on one token is one launch of 3 us, so the call is as fast as its host path: the same checks
// and the same library call took 6.6 us through the interpreter and ctypes, 2 us here.
//
// A plan is everything a step passes to the library, and what it was built from: it holds as long as the parameters
// (identity, version counters and storage: p.data = t, which is also how a module is moved, leaves the first two alone), the
// state tensors, the batch, the dtype and the options stay what they were.  The state tensors are updated in place, except
// the counts: one array is read, another written, and they alternate.
struct Names {
  PyObject *params, *modules, *groups, *bidirectional, *plan, *block_plan, *count, *mean, *var, *h, *key, *value, *key_mask,
      *forward, *hooks, *pre_hooks;
  Names() {
    auto s = [](const char* t) { return PyUnicode_InternFromString(t); };
    params = s("_parameters"); groups = s("num_groups"); bidirectional = s("bidirectional"); plan = s("_step_plan");
    modules = s("_modules"); block_plan = s("_block_plan"); key = s("prev_key"); value = s("prev_value");
    key_mask = s("prev_key_padding_mask"); forward = s("forward"); hooks = s("_forward_hooks"); pre_hooks = s("_forward_pre_hooks");
    count = s("prev_count"); mean = s("prev_mean"); var = s("prev_var"); h = s("prev_state");
  }
};
const Names& names() {
  static const Names* n = new Names;
  return *n;
}

int64_t version_of(const Tensor& t) { return (int64_t)t.unsafeGetTensorImpl()->version_counter().current_version(); }

// A parameter as it was when a plan was built; its storage stays as long as the plan, which may hold its address.
struct Mark {
  int64_t version;
  const void* at;
  c10::Storage storage;
  explicit Mark(const Tensor& t) : version(version_of(t)), at(t.data_ptr()), storage(t.storage()) {}
  bool holds(const Tensor& t) const { return version_of(t) == version && t.data_ptr() == at; }
};

struct StepPlan {
  std::vector<py::object> names, params;   // two of the norm, five of the layer
  std::vector<Mark> marks;
  py::object nkey, ekey, groups, activation;
  py::object count, count_next, mean, var, h;
  std::vector<Tensor> operands;            // gamma, beta, p, q, g, omega (fp32)
  bool kept = false;                       // (below)
  Tensor count_t, next_t, mean_t, var_t, h_t;
  int dtype, device, ndim, cplx, normed;
  int64_t batch, dim;
  double eps;
};

std::unique_ptr<StepPlan> step_plan(std::vector<py::object> names, std::vector<py::object> params, py::object nkey, py::object ekey,
                                    py::object groups, py::object activation, std::vector<py::object> state,
                                    std::vector<Tensor> operands, const Tensor& x, bool cplx, bool normed, double eps) {
  auto p = std::make_unique<StepPlan>();
  p->names = std::move(names);
  p->params = std::move(params);
  for (auto& t : p->params) p->marks.emplace_back(THPVariable_Unpack(t.ptr()));
  p->nkey = std::move(nkey); p->ekey = std::move(ekey); p->groups = std::move(groups); p->activation = std::move(activation);
  p->count = state[0]; p->count_next = state[1]; p->mean = state[2]; p->var = state[3]; p->h = state[4];
  p->count_t = THPVariable_Unpack(p->count.ptr()); p->next_t = THPVariable_Unpack(p->count_next.ptr());
  p->mean_t = THPVariable_Unpack(p->mean.ptr()); p->var_t = THPVariable_Unpack(p->var.ptr());
  p->h_t = THPVariable_Unpack(p->h.ptr());
  p->operands = std::move(operands);
  p->dtype = dtype_of(x); p->device = (int)x.get_device(); p->ndim = (int)p->operands[2].size(1);
  p->cplx = cplx; p->normed = normed; p->batch = x.size(0); p->dim = x.size(2); p->eps = eps;
  return p;
}

bool params_match(const StepPlan& p, PyObject* dict, size_t from, size_t to) {
  for (size_t i = from; i < to; ++i) {
    PyObject* t = PyDict_GetItemWithError(dict, p.names[i].ptr());
    if (t != p.params[i].ptr() || !p.marks[i].holds(THPVariable_Unpack(t))) return false;
  }
  return true;
}

// norm_ema_step(norm, move, x, incremental_state, activation, return_normed): the outputs, or None when the layer has
// no plan for this call
// A graph that holds a step works on the state's tensors, which whoever replays it has to keep, and on the plan's, which go
// with the plan: with the next generation, or a change of mode.  Those stay as long as the pole states then.
void keep_with_state(StepPlan& p) {
  using Kept = std::unordered_map<PyObject*, std::pair<py::object, std::vector<Tensor>>>;
  static Kept* const all = new Kept;
  PyObject* const h = p.h.ptr();
  auto& kept = (*all)[h];
  if (!kept.first) kept.first = py::weakref(h, py::cpp_function([h](py::handle) { all->erase(h); }));
  kept.second.insert(kept.second.end(), p.operands.begin(), p.operands.end());
  kept.second.push_back(p.count_t);
  kept.second.push_back(p.next_t);
  p.kept = true;
}

PyObject* norm_ema_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    if (n != 6) throw py::type_error("norm_ema_step takes 6 arguments");
    if (!THPVariable_Check(a[2]) || !PyDict_Check(a[3]) || at::GradMode::is_enabled()) Py_RETURN_NONE;
    const Names& k = names();
    const auto norm = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(a[0], nullptr));
    const auto move = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(a[1], nullptr));
    PyObject* held = move ? PyDict_GetItemWithError(move.ptr(), k.plan) : nullptr;
    if (!held || held == Py_None || !norm) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    StepPlan& p = *py::cast<StepPlan*>(py::handle(held));
    const Tensor& x = THPVariable_Unpack(a[2]);
    PyObject* ns = PyDict_GetItemWithError(a[3], p.nkey.ptr());
    PyObject* es = PyDict_GetItemWithError(a[3], p.ekey.ptr());
    PyObject* np = PyDict_GetItemWithError(norm.ptr(), k.params);
    PyObject* mp = PyDict_GetItemWithError(move.ptr(), k.params);
    const bool same = ns && es && np && mp && PyDict_Check(ns) && PyDict_Check(es) &&
                      PyDict_GetItemWithError(ns, k.mean) == p.mean.ptr() && PyDict_GetItemWithError(ns, k.var) == p.var.ptr() &&
                      PyDict_GetItemWithError(ns, k.count) == p.count.ptr() && PyDict_GetItemWithError(es, k.h) == p.h.ptr() &&
                      PyDict_GetItemWithError(norm.ptr(), k.groups) == p.groups.ptr() &&
                      PyDict_GetItemWithError(move.ptr(), k.bidirectional) == Py_False &&
                      PyObject_RichCompareBool(a[4], p.activation.ptr(), Py_EQ) == 1 && PyObject_IsTrue(a[5]) == p.normed &&
                      x.is_cuda() && x.get_device() == p.device && x.dim() == 3 && x.size(1) == 1 && x.size(0) == p.batch &&
                      x.size(2) == p.dim && x.is_contiguous() && x.scalar_type() != at::kDouble && x.is_floating_point() &&
                      dtype_of(x) == p.dtype && params_match(p, np, 0, 2) && params_match(p, mp, 2, p.params.size());
    if (!same) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)p.device);
    void* stream = at::cuda::getCurrentCUDAStream((c10::DeviceIndex)p.device).stream();
    // (the default stream cannot be captured; asking takes 0.4 us, a twentieth of a step)
    if (stream && !p.kept && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) keep_with_state(p);
    auto like = [&] { return Tensor(at::detail::empty_cuda(x.sizes(), x.scalar_type(), x.device(), std::nullopt)); };
    Tensor y = like(), xn = p.normed ? like() : Tensor();
    const auto& o = p.operands;
    const unsigned flags = p.activation.is_none() ? 0u : MEGA_EMA_SILU;
    const auto step = p.cplx ? mega_tsn_cema_step : mega_tsn_ema_step;
    check(step(x.data_ptr(), y.data_ptr(), ptr(xn), p.dtype, (int)p.batch, (int)p.dim, ptr<int64_t>(p.count_t), ptr<int64_t>(p.next_t),
               fptr(p.mean_t), fptr(p.var_t), fptr(o[0]), fptr(o[1]), p.eps, fptr(o[2]), fptr(o[3]), fptr(o[4]), fptr(o[5]), p.ndim,
               (float*)p.h_t.data_ptr(), flags, stream), "tsn_ema_step");
    std::swap(p.count, p.count_next);
    std::swap(p.count_t, p.next_t);
    if (PyDict_SetItem(ns, k.count, p.count.ptr()) != 0) return nullptr;
    PyObject* out = THPVariable_Wrap(std::move(y));
    if (!p.normed) return out;
    PyObject* second = THPVariable_Wrap(std::move(xn));
    PyObject* both = PyTuple_Pack(2, out, second);
    Py_XDECREF(out);
    Py_XDECREF(second);
    return both;
  } catch (py::error_already_set& e) {
    e.restore();
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// ------------------------------------------------------------------------------------ single-token step of a block
// Five launches of 3 - 6 us each: through the interpreter and ctypes a step took 31 us of host, more than the device.
//
// A plan belongs to a generation: to its running mean, a tensor that the steps update in place and that the state keeps
// from the first to the last of them.  The block's plans are found by it, so generations that are answered in turn keep
// theirs, and a plan goes, with the buffers of keys and values it holds, when the tensor does.
constexpr int kOwners = 7;
struct BlockPlan {
  mega_block_step_args args;
  PyObject* block;                         // (not owned: the plans live in the block's dictionary)
  py::object owners[kOwners];              // norm, move, then those a step stands for: v_proj, mx_proj, h_proj, attention, positions
  std::vector<std::pair<int, py::object>> names;   // of a parameter: owner (0: the block, 1 ...: the above), key
  std::vector<py::object> params;
  std::vector<Mark> marks;
  py::object submodules[kOwners];          // the owners' keys
  py::object nkey, ekey, akey;
  PyObject* mean;                          // (not owned: the plan goes with it)
  py::object count, count_next, var, h, last_key, last_value;
  Tensor keys, values;
  std::vector<py::object> keep;
  int64_t pos, chunk, batch, dim;
  int device;
  uintptr_t stream;
  at::ScalarType type;
};

std::shared_ptr<BlockPlan> block_plan(py::bytes args, std::vector<py::object> owners, std::vector<std::string> submodules,
                                      std::vector<std::pair<int, std::string>> names, std::vector<py::object> params,
                                      std::vector<py::object> state_keys, std::vector<py::object> state, const Tensor& keys,
                                      const Tensor& values, std::vector<py::object> keep, int64_t chunk, const Tensor& x,
                                      uintptr_t stream) {
  auto p = std::make_shared<BlockPlan>();
  const std::string raw = args;
  if (raw.size() != sizeof p->args || owners.size() != kOwners + 1 || submodules.size() != kOwners) throw py::value_error("block_plan");
  memcpy(&p->args, raw.data(), raw.size());
  auto word = [](const std::string& t) { return py::reinterpret_steal<py::object>(PyUnicode_InternFromString(t.c_str())); };
  p->block = owners[0].ptr();
  for (int i = 0; i < kOwners; ++i) p->owners[i] = owners[i + 1];
  for (int i = 0; i < kOwners; ++i) p->submodules[i] = word(submodules[i]);
  for (auto& n : names) p->names.emplace_back(n.first, word(n.second));
  p->params = std::move(params);
  for (auto& t : p->params) p->marks.emplace_back(THPVariable_Unpack(t.ptr()));
  p->nkey = state_keys[0]; p->ekey = state_keys[1]; p->akey = state_keys[2];
  p->count = state[0]; p->count_next = state[1]; p->mean = state[2].ptr(); p->var = state[3]; p->h = state[4];
  p->last_key = state[5]; p->last_value = state[6];
  p->keys = keys; p->values = values;
  p->keep = std::move(keep);
  p->pos = p->args.pos; p->chunk = chunk;
  p->batch = x.size(0); p->dim = x.size(2); p->device = (int)x.get_device(); p->stream = stream; p->type = x.scalar_type();
  return p;
}

// A block's plans.
struct BlockPlans {
  struct Entry {
    std::shared_ptr<BlockPlan> plan;
    py::object watch;   // weak reference to the mean
  };
  using Map = std::unordered_map<PyObject*, Entry>;
  std::shared_ptr<Map> plans = std::make_shared<Map>();
  py::object nkey;      // the norm's key in a state

  void add(std::shared_ptr<BlockPlan> p) {
    PyObject* const mean = p->mean;
    nkey = p->nkey;
    std::weak_ptr<Map> all = plans;
    py::object watch = py::weakref(mean, py::cpp_function([all, mean](py::handle) {
      if (auto m = all.lock()) m->erase(mean);
    }));
    (*plans)[mean] = Entry{std::move(p), std::move(watch)};
  }
};

py::object dict_of(PyObject* o) { return py::reinterpret_steal<py::object>(PyObject_GenericGetDict(o, nullptr)); }

// (an absent entry and None are the same)
bool holds(PyObject* dict, PyObject* key, PyObject* want) {
  PyObject* v = dict ? PyDict_GetItemWithError(dict, key) : nullptr;
  return (v ? v : Py_None) == want;
}

// whether a dictionary in a module's dictionary is empty
bool empty(PyObject* dict, PyObject* key) {
  PyObject* v = PyDict_GetItemWithError(dict, key);
  return v && PyDict_Check(v) && PyDict_Size(v) == 0;
}

// Whether the plan is one for this block, these inputs and this state.
bool block_matches(const BlockPlan& p, PyObject* blk, PyObject* block_dict, const Tensor& x, PyObject* inc) {
  const Names& k = names();
  if (blk != p.block || p.pos >= p.args.cap) return false;
  PyObject* ns = PyDict_GetItemWithError(inc, p.nkey.ptr());
  PyObject* es = PyDict_GetItemWithError(inc, p.ekey.ptr());
  PyObject* as = PyDict_GetItemWithError(inc, p.akey.ptr());
  if (as == Py_None) as = nullptr;
  if (!ns || !es || !PyDict_Check(ns) || !PyDict_Check(es) || (as && !PyDict_Check(as))) return false;
  if (!holds(ns, k.mean, p.mean) || !holds(ns, k.var, p.var.ptr()) || !holds(ns, k.count, p.count.ptr()) ||
      !holds(es, k.h, p.h.ptr()) || !holds(as, k.key, p.last_key.ptr()) || !holds(as, k.value, p.last_value.ptr()) ||
      !holds(as, k.key_mask, Py_None))
    return false;
  if (!x.is_cuda() || x.get_device() != p.device || x.dim() != 3 || x.size(1) != 1 || x.size(0) != p.batch || x.size(2) != p.dim ||
      x.scalar_type() != p.type || !x.is_contiguous())
    return false;
  PyObject* subs = PyDict_GetItemWithError(block_dict, k.modules);
  if (!subs) return false;
  py::object dicts[kOwners + 1];   // the owners' parameters
  for (int i = 0; i <= kOwners; ++i) {
    if (i && PyDict_GetItemWithError(subs, p.submodules[i - 1].ptr()) != p.owners[i - 1].ptr()) return false;
    const py::object d = i ? dict_of(p.owners[i - 1].ptr()) : py::reinterpret_borrow<py::object>(block_dict);
    dicts[i] = py::reinterpret_borrow<py::object>(d ? PyDict_GetItemWithError(d.ptr(), k.params) : nullptr);
    if (!dicts[i]) return false;
    if (i > 2 && (PyDict_Contains(d.ptr(), k.forward) != 0 || !empty(d.ptr(), k.hooks) || !empty(d.ptr(), k.pre_hooks))) return false;
  }
  for (size_t i = 0; i < p.params.size(); ++i) {
    PyObject* t = PyDict_GetItemWithError(dicts[p.names[i].first].ptr(), p.names[i].second.ptr());
    if (t != p.params[i].ptr() || !p.marks[i].holds(THPVariable_Unpack(t))) return false;
  }
  return true;
}

// block_step(block, x, incremental_state): the output, or None when the block has no plan for this call
PyObject* block_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    if (n != 3) throw py::type_error("block_step takes 3 arguments");
    if (!THPVariable_Check(a[1]) || !PyDict_Check(a[2]) || at::GradMode::is_enabled()) Py_RETURN_NONE;
    const Names& k = names();
    const py::object dict = dict_of(a[0]);
    PyObject* held = dict ? PyDict_GetItemWithError(dict.ptr(), k.block_plan) : nullptr;
    if (!held || held == Py_None) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const auto plans = py::cast<BlockPlans*>(py::handle(held))->plans;
    PyObject* ns = PyDict_GetItemWithError(a[2], py::cast<BlockPlans*>(py::handle(held))->nkey.ptr());
    PyObject* mean = ns && PyDict_Check(ns) ? PyDict_GetItemWithError(ns, k.mean) : nullptr;
    const auto found = plans->find(mean);
    if (found == plans->end()) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const std::shared_ptr<BlockPlan> keep_plan = found->second.plan;
    BlockPlan& p = *keep_plan;
    const Tensor& x = THPVariable_Unpack(a[1]);
    if (!block_matches(p, a[0], dict.ptr(), x, a[2])) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)p.device);
    void* stream = at::cuda::getCurrentCUDAStream((c10::DeviceIndex)p.device).stream();
    if ((uintptr_t)stream != p.stream) Py_RETURN_NONE;
    Tensor out(at::detail::empty_cuda(x.sizes(), x.scalar_type(), x.device(), std::nullopt));
    auto at = [](PyObject* t) { return THPVariable_Unpack(t).data_ptr(); };
    p.args.count = (int64_t*)at(p.count.ptr());
    p.args.count_next = (int64_t*)at(p.count_next.ptr());
    p.args.mean = (float*)at(p.mean);
    p.args.var = (float*)at(p.var.ptr());
    p.args.h = (float*)at(p.h.ptr());
    p.args.x = x.data_ptr();
    p.args.out = out.data_ptr();
    p.args.pos = p.pos;
    check(mega_block_step(&p.args, stream), "block_step");
    std::swap(p.count, p.count_next);   // the counts alternate between two arrays, the step wrote the second one
    if (PyDict_SetItem(PyDict_GetItemWithError(a[2], p.nkey.ptr()), k.count, p.count.ptr()) != 0) return nullptr;
    PyObject* as = PyDict_GetItemWithError(a[2], p.akey.ptr());
    if (!as || as == Py_None) {
      const auto fresh = py::dict();
      if (PyDict_SetItem(a[2], p.akey.ptr(), fresh.ptr()) != 0) return nullptr;
      as = PyDict_GetItemWithError(a[2], p.akey.ptr());
    }
    const int64_t pos = ++p.pos;
    if (p.chunk < 0 || pos % p.chunk != 0) {
      p.last_key = py::reinterpret_steal<py::object>(THPVariable_Wrap(p.keys.narrow(1, 0, pos)));
      p.last_value = py::reinterpret_steal<py::object>(THPVariable_Wrap(p.values.narrow(1, 0, pos)));
      if (PyDict_SetItem(as, k.key, p.last_key.ptr()) != 0 || PyDict_SetItem(as, k.value, p.last_value.ptr()) != 0 ||
          PyDict_SetItem(as, k.key_mask, Py_None) != 0)
        return nullptr;
    } else {   // the chunk is complete: the next token starts another one, in other buffers
      for (PyObject* key : {k.key, k.value, k.key_mask})
        if (PyDict_GetItemWithError(as, key) && PyDict_DelItem(as, key) != 0) return nullptr;
      plans->erase(p.mean);
    }
    return THPVariable_Wrap(std::move(out));
  } catch (py::error_already_set& e) {
    e.restore();
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

PyMethodDef g_raw[] = {{"norm_ema_step", (PyCFunction)(void (*)())norm_ema_step, METH_FASTCALL, nullptr},
                       {"block_step", (PyCFunction)(void (*)())block_step, METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(_mega_host, m) {
  py::class_<StepPlan>(m, "StepPlan")
      .def(py::init(&step_plan))
      .def("__deepcopy__", [](StepPlan&, py::object) { return py::none(); })   // (a copied or pickled layer builds its own)
      .def("__reduce__", [](StepPlan&) {
        return py::make_tuple(py::reinterpret_borrow<py::object>((PyObject*)Py_TYPE(Py_None)), py::tuple());
      });
  py::class_<BlockPlan, std::shared_ptr<BlockPlan>>(m, "BlockPlan").def(py::init(&block_plan));
  py::class_<BlockPlans>(m, "BlockPlans")
      .def(py::init<>())
      .def("add", &BlockPlans::add)
      .def("__len__", [](BlockPlans& b) { return b.plans->size(); })
      .def("__deepcopy__", [](BlockPlans&, py::object) { return py::none(); })
      .def("__reduce__", [](BlockPlans&) {
        return py::make_tuple(py::reinterpret_borrow<py::object>((PyObject*)Py_TYPE(Py_None)), py::tuple());
      });
  PyModule_AddFunctions(m.ptr(), g_raw);
  m.def("set_error", [](py::object e) { g_error = e.release().ptr(); });
  m.def("ema_forward", &ema_forward);
  m.def("ema_train", &ema_train);
  m.def("norm_prepare", &norm_prepare);
  m.def("timestep_norm_fwd", &timestep_norm_fwd);
  m.def("timestep_norm_train", &timestep_norm_train);
  m.def("sequence_norm_fwd", &sequence_norm_fwd);
  m.def("sequence_norm_train", &sequence_norm_train);
  m.def("tsn_ema_forward", &tsn_ema_forward);
  m.def("sqn_ema_forward", &sqn_ema_forward);
  m.def("gate_silu", &gate_silu);
  m.def("gate_mul_silu", &gate_mul_silu);
  m.def("gate_output", &gate_output);
  m.def("gate_qk", &gate_qk);
  m.def("attention_softmax_fwd", &softmax_fwd);
  m.def("block_train", &block_train);
  m.def("block_infer", &block_infer);
}
