// The operators' host side in one native call each: argument checks, output allocation and launches of `quantize`, `linear`,
// `linear_requant`, `attention` and `rope3d`.  Built by ac4k_kernel_b200/build.py (build_pybind) with the host compiler.
//
// Why: the Python wrappers cost 20 - 25 us per launch (argument checks, ctypes marshalling, the device guard), several
// times the kernels of a small call: a decode layer, quantisation and GEMM, took 78 us of which the GPU worked 12.
//
// Each function returns None instead of a result when anything about the call is not what it expects (a wrong shape, a
// tensor subclass, an option it does not know): the Python wrapper then takes its own path, which computes the same or
// raises its own error.  So nothing here decides what is accepted and what is refused.  The interpreter lock is given up for
// allocations and launches (a launch waits while the driver's queue is full).
#include <ATen/ATen.h>
#include <ATen/Context.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <cmath>
#include <optional>
#include <string>

#include "ac4k_b200.h"

namespace py = pybind11;

namespace {

int64_t align_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }
int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// A dense CUDA tensor whose memory may be handed to a kernel as it is: no mode tensor, no functorch wrapper.  (Python
// subclasses without a dispatch of their own look the same here; tensor_of declines them by their type.)
bool plain(const at::Tensor &t) {
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided) return false;
  const c10::DispatchKeySet odd({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::FuncTorchBatched,
                                 c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize, c10::DispatchKey::Negative,
                                 c10::DispatchKey::Conjugate, c10::DispatchKey::ZeroTensor});
  return !t.unsafeGetTensorImpl()->key_set().has_any(odd);
}

std::optional<at::Tensor> tensor_of(py::handle h, at::ScalarType dt, int64_t dim = -1, bool dense = true) {
  if (!THPVariable_CheckExact(h.ptr())) return std::nullopt;       // (a torch.Tensor or a Parameter, no subclass of them)
  const at::Tensor &t = THPVariable_Unpack(h.ptr());
  if (!plain(t) || t.scalar_type() != dt || (dim >= 0 && t.dim() != dim) || (dense && !t.is_contiguous())) return std::nullopt;
  return t;
}
bool scalar_of(py::handle h, at::Tensor *out) {
  auto t = tensor_of(h, at::kFloat, 0);
  if (!t) return false;
  *out = *t;
  return true;
}
bool same_shape(const at::Tensor &t, std::initializer_list<int64_t> want) { return t.sizes() == at::IntArrayRef(want.begin(), want.size()); }

// An uninitialised tensor.  Straight from the allocator's factory where nothing listens to operator calls (no dispatch mode, tracer
// or function transform, no deterministic filling, no profiler): through the dispatcher a tensor costs 0.2 us more, 0.6 us of the 6.3
// of a small quantize(), 0.9 us of the 17 of a small attention().
at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dt, const at::Tensor &like) {
  const c10::DispatchKeySet listeners({c10::DispatchKey::Tracer, c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::Functionalize,
                                       c10::DispatchKey::PythonDispatcher});
  if (c10::impl::dispatch_mode_enabled() || c10::impl::tls_local_dispatch_key_set().included_.has_any(listeners) ||
      at::globalContext().deterministicAlgorithms() || at::hasCallbacks())
    return at::empty(sizes, at::TensorOptions().dtype(dt).device(like.device()));
  return at::Tensor(at::detail::empty_cuda(sizes, dt, like.device(), std::nullopt));
}
at::Tensor scalar_like(const at::Tensor &like) { return empty({}, at::kFloat, like); }

void check(int rc, const char *what) {
  TORCH_CHECK(rc == 0, what, " failed (code ", rc, "): ", ac4k_last_error());
}
void *stream_of(const at::Tensor &t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

int dt_code(at::ScalarType t) { return t == at::kBFloat16 ? AC4K_DT_BF16 : (t == at::kHalf ? AC4K_DT_FP16 : (t == at::kFloat ? AC4K_DT_FP32 : -1)); }

// sizes and element strides ordered [outer0, outer1, cross, reduce], rank padded to 4 with leading 1s
struct View {
  int64_t shape[4], stride[4];
  at::DimVector lead;
  View(const at::Tensor &t, int64_t cross, int64_t reduce) {
    int o = 2 - ((int)t.dim() - 2);
    for (int i = 0; i < o; ++i) { shape[i] = 1; stride[i] = 0; }
    for (int64_t i = 0; i < t.dim(); ++i)
      if (i != cross && i != reduce) { shape[o] = t.size(i); stride[o] = t.stride(i); ++o; lead.push_back(t.size(i)); }
    shape[2] = t.size(cross);  stride[2] = t.stride(cross);
    shape[3] = t.size(reduce); stride[3] = t.stride(reduce);
  }
};

// `work` without the interpreter lock (taken again when it returns or throws)
template <typename F>
auto unlocked(F &&work) {
  py::gil_scoped_release release;
  return work();
}

struct Nvfp4 { at::Tensor q, sf, scale; };

Nvfp4 quantize_nvfp4_of(const at::Tensor &x, int64_t cross, int64_t reduce, float max_scale, bool swizzle, bool tiled) {
  const View v(x, cross, reduce);
  const int64_t m = v.shape[2], kp = align_up(v.shape[3], 64);
  at::DimVector so(v.lead), ss(v.lead);
  for (int64_t d : {m, kp / 2}) so.push_back(d);
  if (tiled) for (int64_t d : {ceil_div(m, 128), kp / 64, (int64_t)32, (int64_t)4, (int64_t)4}) ss.push_back(d);
  else for (int64_t d : {kp / 64, align_up(m, 16), (int64_t)4}) ss.push_back(d);
  Nvfp4 r{empty(so, at::kByte, x), empty(ss, at::kFloat8_e4m3fn, x), scalar_like(x)};
  // scratch for the per-CTA maxima; a tensor that one cluster takes needs none
  at::Tensor scratch;
  if (swizzle || v.stride[3] != 1 || v.shape[3] % 16 || v.shape[0] * v.shape[1] * m * (kp / 16) > AC4K_QUANTIZE_ONE_LAUNCH_BLOCKS) scratch = empty({AC4K_QUANTIZE_SCRATCH_BYTES / 4}, at::kInt, x);
  check(ac4k_quantize_nvfp4_dynamic(r.q.data_ptr(), r.sf.data_ptr(), static_cast<float *>(r.scale.data_ptr()),
                                    scratch.defined() ? scratch.data_ptr() : nullptr, x.data_ptr(), max_scale, v.shape, v.stride, swizzle ? 1 : 0,
                                    tiled ? AC4K_SF_TILE128X4 : AC4K_SF_AC4K, stream_of(x)),
        "quantize_nvfp4");
  return r;
}

struct Rowwise { at::Tensor q, sf; };

Rowwise quantize_rows_of(const at::Tensor &x, int64_t cross, int64_t reduce, bool fp8, double max_scale, bool swizzle) {
  const View v(x, cross, reduce);
  at::DimVector so(v.lead), ss(v.lead);
  for (int64_t d : {v.shape[2], align_up(v.shape[3], 16)}) so.push_back(d);
  ss.push_back(align_up(v.shape[2], 16));
  Rowwise r{empty(so, fp8 ? at::kFloat8_e4m3fn : at::kChar, x), empty(ss, at::kFloat, x)};
  float *sf = static_cast<float *>(r.sf.data_ptr());
  if (fp8)
    check(ac4k_quantize_fp8_max(r.q.data_ptr(), sf, x.data_ptr(), (float)max_scale, v.shape, v.stride, swizzle ? 1 : 0, stream_of(x)), "quantize_fp8");
  else
    check(ac4k_quantize_int8_max(r.q.data_ptr(), sf, x.data_ptr(), (int32_t)max_scale, v.shape, v.stride, stream_of(x)), "quantize_int8");
  return r;
}

// None, or a number that fp32 and int32 hold exactly enough for both Python paths to agree
std::optional<double> number_or(py::handle h, double fallback, bool whole) {
  if (h.is_none()) return fallback;
  if (!(PyLong_CheckExact(h.ptr()) || (!whole && PyFloat_CheckExact(h.ptr())))) return std::nullopt;
  const double v = PyFloat_CheckExact(h.ptr()) ? PyFloat_AS_DOUBLE(h.ptr()) : PyLong_AsDouble(h.ptr());
  if (PyErr_Occurred()) { PyErr_Clear(); return std::nullopt; }
  if (!(std::fabs(v) < 16777216.0)) return std::nullopt;
  return v;
}

// Options come as they are: pybind's own conversions would raise a TypeError for what a wrapper may accept or refuse otherwise.
std::optional<std::string> text_of(py::handle h) {
  if (!PyUnicode_CheckExact(h.ptr())) return std::nullopt;
  Py_ssize_t n = 0;
  const char *s = PyUnicode_AsUTF8AndSize(h.ptr(), &n);
  if (s == nullptr) { PyErr_Clear(); return std::nullopt; }
  return std::string(s, (size_t)n);
}
std::optional<int64_t> index_of(py::handle h) {
  if (!PyLong_CheckExact(h.ptr())) return std::nullopt;
  const int64_t v = PyLong_AsLongLong(h.ptr());
  if (PyErr_Occurred()) { PyErr_Clear(); return std::nullopt; }
  return v;
}

// precision, layouts: what the wrapper looks at for this precision, no more
py::object quantize(py::handle input, py::handle hcross, py::handle hreduce, py::handle max_scale, py::handle hprecision, py::handle hswizzle,
                    py::handle hlayout) {
  const auto x = tensor_of(input, at::kBFloat16);
  const auto icross = index_of(hcross), ireduce = index_of(hreduce);
  const auto iprecision = text_of(hprecision);
  if (!x || x->dim() < 2 || x->dim() > 4 || !icross || !ireduce || !iprecision || !PyBool_Check(hswizzle.ptr())) return py::none();
  int64_t cross = *icross, reduce = *ireduce;
  const std::string &precision = *iprecision;
  const bool swizzle = hswizzle.ptr() == Py_True;
  if (cross < 0) cross += x->dim();
  if (reduce < 0) reduce += x->dim();
  if (cross < 0 || reduce < 0 || cross >= x->dim() || reduce >= x->dim() || cross == reduce) return py::none();
  const c10::cuda::CUDAGuard guard(x->device());
  if (precision == "nvfp4") {
    const auto ms = number_or(max_scale, 6.0 * 448.0, false);
    const auto sf_layout = text_of(hlayout);
    if (!ms || !sf_layout || (*sf_layout != "ac4k" && *sf_layout != "128x4")) return py::none();
    const Nvfp4 r = unlocked([&] { return quantize_nvfp4_of(*x, cross, reduce, (float)*ms, swizzle, *sf_layout == "128x4"); });
    return py::make_tuple(r.q, r.sf, r.scale);
  }
  const bool fp8 = precision == "fp8e4m3";
  if (!fp8 && precision != "int8") return py::none();
  const auto ms = number_or(max_scale, fp8 ? 448.0 : 127.0, !fp8);
  if (!ms) return py::none();
  const Rowwise r = unlocked([&] { return quantize_rows_of(*x, cross, reduce, fp8, *ms, fp8 && swizzle); });
  return py::make_tuple(r.q, r.sf);
}

// The operands of a GEMM; ok stays false for a call the Python wrapper has to look at.
struct Gemm {
  at::Tensor a, a_sf, a_gs, b, b_sf, b_gs, bias;
  int64_t M = 0, N = 0, K = 0;
  int layout = 0;
  bool ok = false;
  Gemm(py::handle ha, py::handle hasf, py::handle hags, py::handle hb, py::handle hbsf, py::handle hbgs, py::handle hbias) {
    const auto ta = tensor_of(ha, at::kByte, 2), tb = tensor_of(hb, at::kByte, 2);
    const auto tas = tensor_of(hasf, at::kFloat8_e4m3fn), tbs = tensor_of(hbsf, at::kFloat8_e4m3fn);
    if (!ta || !tb || !tas || !tbs || !scalar_of(hags, &a_gs) || !scalar_of(hbgs, &b_gs)) return;
    a = *ta; b = *tb; a_sf = *tas; b_sf = *tbs;
    M = a.size(0); N = b.size(0); K = a.size(1) * 2;
    if (b.size(1) != a.size(1) || K % 16) return;
    const int64_t kt = ceil_div(K, 64);
    if (a_sf.dim() == 3) {
      layout = AC4K_SF_AC4K;
      if (!same_shape(a_sf, {kt, align_up(M, 16), 4}) || !same_shape(b_sf, {kt, align_up(N, 16), 4})) return;
    } else {
      layout = AC4K_SF_TILE128X4;
      if (!same_shape(a_sf, {ceil_div(M, 128), kt, 32, 4, 4}) || !same_shape(b_sf, {ceil_div(N, 128), kt, 32, 4, 4})) return;
    }
    if (!hbias.is_none()) {
      if (!THPVariable_CheckExact(hbias.ptr())) return;
      bias = THPVariable_Unpack(hbias.ptr());
      if (!plain(bias) || dt_code(bias.scalar_type()) < 0 || !bias.is_contiguous()) return;
      if (!(bias.dim() == 1 && bias.size(0) == N) && !(bias.dim() == 2 && bias.size(0) == 1 && bias.size(1) == N)) return;
    }
    ok = true;
  }
  const void *bias_ptr() const { return bias.defined() ? bias.data_ptr() : nullptr; }
  int bias_dt() const { return bias.defined() ? dt_code(bias.scalar_type()) : 0; }
  const float *ags() const { return static_cast<const float *>(a_gs.data_ptr()); }
  const float *bgs() const { return static_cast<const float *>(b_gs.data_ptr()); }
};

py::object linear(py::handle a, py::handle a_sf, py::handle a_gs, py::handle b, py::handle b_sf, py::handle b_gs, py::handle bias, py::handle out) {
  const Gemm g(a, a_sf, a_gs, b, b_sf, b_gs, bias);
  if (!g.ok) return py::none();
  at::Tensor d;
  if (!out.is_none()) {
    if (!THPVariable_CheckExact(out.ptr())) return py::none();
    d = THPVariable_Unpack(out.ptr());
    if (!plain(d) || !d.is_contiguous() || dt_code(d.scalar_type()) < 0 || !same_shape(d, {g.M, g.N})) return py::none();
  }
  const c10::cuda::CUDAGuard guard(d.defined() ? d.device() : g.a.device());
  unlocked([&] {
    if (!d.defined()) d = empty({g.M, g.N}, at::kBFloat16, g.a);
    check(ac4k_linear_nvfp4(d.data_ptr(), dt_code(d.scalar_type()), g.a.data_ptr(), g.a_sf.data_ptr(), g.ags(), g.b.data_ptr(), g.b_sf.data_ptr(),
                            g.bgs(), g.bias_ptr(), g.bias_dt(), g.M, g.N, g.K, g.layout, stream_of(d)),
          "linear_nvfp4");
  });
  return out.is_none() ? py::cast(d) : py::reinterpret_borrow<py::object>(out);
}

py::object linear_requant(py::handle a, py::handle a_sf, py::handle a_gs, py::handle b, py::handle b_sf, py::handle b_gs, py::handle out_gs,
                          py::handle bias, py::handle hlayout) {
  const Gemm g(a, a_sf, a_gs, b, b_sf, b_gs, bias);
  at::Tensor gs;
  const auto sf_layout = text_of(hlayout);
  if (!g.ok || !scalar_of(out_gs, &gs) || g.N % 64 || !sf_layout || (*sf_layout != "ac4k" && *sf_layout != "128x4")) return py::none();
  const bool tiled = *sf_layout == "128x4";
  const c10::cuda::CUDAGuard guard(g.a.device());
  at::Tensor o, sf;
  unlocked([&] {
    o = empty({g.M, g.N / 2}, at::kByte, g.a);
    sf = tiled ? empty({ceil_div(g.M, 128), g.N / 64, 32, 4, 4}, at::kFloat8_e4m3fn, g.a)
                          : empty({g.N / 64, align_up(g.M, 16), 4}, at::kFloat8_e4m3fn, g.a);
    check(ac4k_linear_nvfp4_requant(o.data_ptr(), sf.data_ptr(), static_cast<const float *>(gs.data_ptr()), tiled ? AC4K_SF_TILE128X4 : AC4K_SF_AC4K,
                                    g.a.data_ptr(), g.a_sf.data_ptr(), g.ags(), g.b.data_ptr(), g.b_sf.data_ptr(), g.bgs(), g.bias_ptr(),
                                    g.bias_dt(), g.M, g.N, g.K, g.layout, stream_of(o)),
          "linear_nvfp4_requant");
  });
  return py::make_tuple(o, sf, py::reinterpret_borrow<py::object>(out_gs));
}

py::object rope3d(py::handle hx, py::handle hgrid, py::handle hfreqs, py::handle hout) {
  const auto x = tensor_of(hx, at::kBFloat16, 4), freqs = tensor_of(hfreqs, at::kComplexDouble, 2), grid = tensor_of(hgrid, at::kInt, 2);
  if (!x || !freqs || !grid) return py::none();
  const int64_t B = x->size(0), S = x->size(1), N = x->size(2), D = x->size(3);
  if (!same_shape(*grid, {B, 3}) || D % 2 || freqs->size(1) != D / 2) return py::none();
  std::optional<at::Tensor> given;
  if (!hout.is_none()) {
    given = tensor_of(hout, at::kBFloat16, 4);
    if (!given || given->sizes() != x->sizes()) return py::none();
  }
  const c10::cuda::CUDAGuard guard(x->device());
  at::Tensor out = given ? *given : at::empty_like(*x);
  if (!out.is_contiguous()) return py::none();
  unlocked([&] {
    check(ac4k_rope3d(out.data_ptr(), x->data_ptr(), static_cast<const int32_t *>(grid->data_ptr()), freqs->data_ptr(), B, S, N, D, freqs->size(0),
                      stream_of(*x)),
          "rope3d");
  });
  return given ? py::reinterpret_borrow<py::object>(hout) : py::cast(out);
}

py::object attention(py::handle hq, py::handle hk, py::handle hv, py::handle hlayout, py::handle hprecision, py::handle hout) {
  const auto layout = text_of(hlayout), precision = text_of(hprecision);
  if (!layout || !precision) return py::none();
  const bool nvfp4 = *precision == "nvfp4", bnhd = *layout == "BNHD";
  if ((!nvfp4 && *precision != "int8+fp8e4m3") || (!bnhd && *layout != "BHND")) return py::none();
  const auto tq = tensor_of(hq, at::kBFloat16, 4, nvfp4), tk = tensor_of(hk, at::kBFloat16, 4, nvfp4), tv = tensor_of(hv, at::kBFloat16, 4);
  if (!tq || !tk || !tv) return py::none();
  const at::Tensor &q = *tq, &k = *tk, &v = *tv;
  const int64_t n_dim = bnhd ? 1 : 2, h_dim = bnhd ? 2 : 1;
  const int64_t B = q.size(0), H = q.size(h_dim), Nq = q.size(n_dim), D = q.size(3), Nkv = k.size(n_dim), Dv = v.size(3);
  for (const at::Tensor *t : {&k, &v})
    if (t->size(0) != B || t->size(h_dim) != H || t->size(n_dim) != Nkv) return py::none();
  if (k.size(3) != D || D < 1 || D > 128 || Dv < 1 || Dv > 128 || B < 1 || H < 1 || Nq < 1 || Nkv < 1) return py::none();
  if (k.device() != q.device() || v.device() != q.device()) return py::none();
  at::Tensor out;
  if (!hout.is_none()) {
    const auto t = tensor_of(hout, at::kBFloat16, 4, false);
    if (!t || t->device() != q.device()) return py::none();
    out = *t;
    if (out.size(0) != B || out.size(h_dim) != H || out.size(n_dim) != Nq || out.size(3) != Dv) return py::none();
  }
  const c10::cuda::CUDAGuard guard(q.device());
  const float sm_scale = (float)(1.0 / std::sqrt((double)D));
  auto out_strides = [&](int64_t (&s)[4]) {
    if (!out.defined()) out = bnhd ? empty({B, Nq, H, Dv}, at::kBFloat16, q) : empty({B, H, Nq, Dv}, at::kBFloat16, q);
    s[0] = out.stride(0); s[1] = out.stride(h_dim); s[2] = out.stride(n_dim); s[3] = out.stride(3);
  };
  int64_t os[4];
  const bool done = unlocked([&] {
    if (nvfp4) {
      const int64_t Dp = align_up(D, 64), Kp = align_up(Nkv, 64);
      auto operand = [&](int64_t m, int64_t kp) {
        return Nvfp4{empty({B, H, m, kp / 2}, at::kByte, q), empty({B, H, ceil_div(m, 128), kp / 64, 32, 4, 4}, at::kFloat8_e4m3fn, q), scalar_like(q)};
      };
      const Nvfp4 qq = operand(Nq, Dp), kk = operand(Nkv, Dp), vv = operand(Dv, Kp);
      const at::Tensor scratch = empty({AC4K_QUANTIZE_SCRATCH_BYTES / 4}, at::kInt, q);
      out_strides(os);
      void *const codes[3] = {qq.q.data_ptr(), kk.q.data_ptr(), vv.q.data_ptr()}, *const sfs[3] = {qq.sf.data_ptr(), kk.sf.data_ptr(), vv.sf.data_ptr()};
      auto gs = [](const Nvfp4 &t) { return static_cast<float *>(t.scale.data_ptr()); };
      float *const scales[3] = {gs(qq), gs(kk), gs(vv)};
      const void *const ins[3] = {q.data_ptr(), k.data_ptr(), v.data_ptr()};
      int64_t strides[3][4];
      for (int i = 0; i < 3; ++i) {
        const at::Tensor &t = i == 0 ? q : (i == 1 ? k : v);
        strides[i][0] = t.stride(0); strides[i][1] = t.stride(h_dim); strides[i][2] = t.stride(n_dim); strides[i][3] = t.stride(3);
      }
      check(ac4k_attention_quantize_nvfp4(codes, sfs, scales, scratch.data_ptr(), ins, strides, B, H, Nq, Nkv, D, Dv, stream_of(q)),
            "attention_quantize_nvfp4");
      check(ac4k_mha_nvfp4_fwd(out.data_ptr(), os, qq.q.data_ptr(), qq.sf.data_ptr(), gs(qq), kk.q.data_ptr(), kk.sf.data_ptr(), gs(kk),
                               vv.q.data_ptr(), vv.sf.data_ptr(), gs(vv), B, H, Nq, Nkv, qq.q.size(3) * 2, Dv, sm_scale, AC4K_SF_TILE128X4,
                               stream_of(q)),
            "mha_nvfp4_fwd");
    } else {
      // k - mean(k): the subtraction happens inside the K quantiser, the mean too where it takes that many keys
      at::Tensor mean;
      int64_t ms[2] = {0, 0};
      if (Nkv > AC4K_ATTENTION_MEAN_TOKENS) {
        mean = k.detach().mean(at::IntArrayRef{n_dim}, true);
        if (mean.stride(3) != 1) return false;
        ms[0] = mean.stride(0); ms[1] = mean.stride(h_dim);
      }
      const int64_t Dp = align_up(D, 16);
      const at::Tensor q8 = empty({B, H, Nq, Dp}, at::kChar, q), k8 = empty({B, H, Nkv, Dp}, at::kChar, q);
      const at::Tensor q_sf = empty({B, H, ceil_div(Nq, 64)}, at::kFloat, q), k_sf = empty({B, H, ceil_div(Nkv, 128)}, at::kFloat, q);
      const at::Tensor v8 = empty({B, H, Dv, align_up(Nkv, 16)}, at::kFloat8_e4m3fn, q), v_sf = empty({B, H, align_up(Dv, 16)}, at::kFloat, q);
      auto f = [](const at::Tensor &t) { return static_cast<float *>(t.data_ptr()); };
      auto order = [&](const at::Tensor &t) { return std::array<int64_t, 4>{t.stride(0), t.stride(h_dim), t.stride(n_dim), t.stride(3)}; };
      out_strides(os);          // (everything is allocated in front of the first launch: the quantisers run side by side)
      check(ac4k_attention_quantize_int8(q8.data_ptr(), f(q_sf), k8.data_ptr(), f(k_sf), v8.data_ptr(), f(v_sf), q.data_ptr(), order(q).data(),
                                         k.data_ptr(), order(k).data(), v.data_ptr(), order(v).data(), mean.defined() ? mean.data_ptr() : nullptr,
                                         ms, B, H, Nq, Nkv, D, Dv, stream_of(q)),
            "attention_quantize_int8");
      check(ac4k_mha_int8_x_fp8_fwd(out.data_ptr(), os, q8.data_ptr(), f(q_sf), 64, k8.data_ptr(), f(k_sf), 128, v8.data_ptr(), f(v_sf), B, H,
                                    Nq, Nkv, Dp, Dv, sm_scale, stream_of(q)),
            "mha_int8_x_fp8_fwd");
    }
    return true;
  });
  if (!done) return py::none();
  return hout.is_none() ? py::cast(out) : py::reinterpret_borrow<py::object>(hout);
}

}  // namespace

PYBIND11_MODULE(_host_calls, m) {
  m.doc() = "ac4k_kernel_b200 operators in one call each; None where the Python wrapper has to decide";
  m.def("quantize", &quantize);
  m.def("linear", &linear);
  m.def("linear_requant", &linear_requant);
  m.def("rope3d", &rope3d);
  m.def("attention", &attention);
}
