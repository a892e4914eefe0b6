// Native host path of the Python entry points: argument checks, output allocation, geometry structs and the library call of
// ssd.py / prepost.py in one C++ function each, called with positional arguments (METH_FASTCALL).
//
// A small call is bound by this code and not by its kernels: four streams of one decode step keep the GPU busy for 3 us,
// while the same checks, struct fields and ctypes conversions written in Python took 25 us per step, 75 us per prefill and
// 200 us per fp32 training step (forward + backward under autograd).  The autograd nodes live here as well, so a backward
// pass runs without taking the interpreter lock.
//
// The module links to nothing of libssd_b200: bind() hands it the addresses of the C ABI functions of the library that
// _lib.py loaded.  Argument errors are ValueError, library errors the SsdError class handed to bind(), with the texts a
// caller of the Python functions sees.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <sstream>
#include <string>

#include "../../include/ssd_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ---- the library's C ABI, bound at import ------------------------------------------------------------------------------
struct Api {
  decltype(&::ssd_workspace_bytes) workspace_bytes;
  decltype(&::ssd_forward_staged) forward_staged;
  decltype(&::ssd_backward_staged) backward_staged;
  decltype(&::ssd_state_update) state_update;
  decltype(&::ssd_state_update_host) state_update_host;
  decltype(&::ssd_last_error) last_error;
  decltype(&::ssd_conv1d_workspace_bytes) conv1d_workspace_bytes;
  decltype(&::ssd_conv1d_forward) conv1d_forward;
  decltype(&::ssd_conv1d_backward) conv1d_backward;
  decltype(&::ssd_rmsnorm_workspace_bytes) rmsnorm_workspace_bytes;
  decltype(&::ssd_rmsnorm_forward) rmsnorm_forward;
  decltype(&::ssd_rmsnorm_backward) rmsnorm_backward;
} api;
PyObject *ssd_error = nullptr, *oom_error = nullptr;   // _lib.SsdError, torch.OutOfMemoryError
constexpr int32_t kAllStages = SSD_STAGE_LOCAL | SSD_STAGE_FINISH;

// ---- errors ------------------------------------------------------------------------------------------------------------
struct ArgError : std::runtime_error { using std::runtime_error::runtime_error; };
struct LibError : std::runtime_error {
  int32_t code;
  LibError(int32_t c, const char* m) : std::runtime_error("ssd_b200 error " + std::to_string(c) + ": " + m), code(c), msg(m) {}
  std::string msg;
};
void check_rc(int32_t rc) { if (rc != SSD_OK) throw LibError(rc, api.last_error()); }

std::string str(at::ScalarType t) {
  return t == at::kBFloat16 ? "torch.bfloat16" : t == at::kFloat ? "torch.float32" : std::string("torch.") + c10::toString(t);
}
std::string str(at::IntArrayRef s) {
  std::ostringstream o;
  o << "(";
  for (size_t i = 0; i < s.size(); ++i) o << (i ? ", " : "") << s[i];
  o << (s.size() == 1 ? ",)" : ")");
  return o.str();
}
std::string str(const at::Device& d) { return d.str(); }
std::string str(const char* s) { return s; }
std::string str(const std::string& s) { return s; }
std::string str(int64_t v) { return std::to_string(v); }
template <class... A> [[noreturn]] void fail(const A&... a) { throw ArgError((str(a) + ...)); }

// Runs `f`, turning C++ exceptions into Python ones.
template <class F> PyObject* guarded(F f) {
  try {
    return f();
  } catch (const LibError& e) {
    PyObject* ex = PyObject_CallFunction(ssd_error, "is", (int)e.code, e.msg.c_str());
    if (ex) { PyErr_SetObject(ssd_error, ex); Py_DECREF(ex); }
  } catch (const ArgError& e) {
    PyErr_SetString(PyExc_ValueError, e.what());
  } catch (const c10::OutOfMemoryError& e) {
    PyErr_SetString(oom_error, e.what_without_backtrace());
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// ---- Python arguments --------------------------------------------------------------------------------------------------
struct Args {
  PyObject* const* a;
  Py_ssize_t n;
  Args(PyObject* const* args, Py_ssize_t got, Py_ssize_t want) : a(args), n(got) {
    if (got != want) fail("expected ", (int64_t)want, " arguments, got ", (int64_t)got);
  }
  const Tensor& tensor(int i, const char* name) const {
    if (!THPVariable_Check(a[i])) fail(name, ": expected a tensor, got ", Py_TYPE(a[i])->tp_name);
    return THPVariable_Unpack(a[i]);
  }
  const Tensor* opt(int i, const char* name) const { return a[i] == Py_None ? nullptr : &tensor(i, name); }
  int64_t integer(int i) const {
    const long long v = PyLong_AsLongLong(a[i]);
    if (v == -1 && PyErr_Occurred()) throw std::runtime_error("bad integer argument");
    return v;
  }
  double real(int i) const {
    const double v = PyFloat_AsDouble(a[i]);
    if (v == -1.0 && PyErr_Occurred()) throw std::runtime_error("bad float argument");
    return v;
  }
  bool flag(int i) const { return PyObject_IsTrue(a[i]) == 1; }
};
PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}

// ---- checks and geometry -----------------------------------------------------------------------------------------------
int32_t storage_type(const Tensor& x) {
  if (x.scalar_type() == at::kBFloat16) return SSD_BF16;
  if (x.scalar_type() != at::kFloat) fail("unsupported dtype ", x.scalar_type());
  return SSD_F32;
}
struct Shape {   // small fixed-size shape, no allocation
  int64_t v[4];
  int n;
  template <class... I> explicit Shape(I... i) : v{(int64_t)i...}, n((int)sizeof...(i)) {}
  operator at::IntArrayRef() const { return at::IntArrayRef(v, n); }
};
bool same(const Tensor& t, at::IntArrayRef s) { return t.sizes() == s; }

// The geometry structs take a stride of 0 as "dense", so rows that lie over one another cannot be described by them.
bool overlaid(const Tensor& t, int dims) {
  for (int i = 0; i < dims; ++i)
    if (t.size(i) > 1 && t.stride(i) == 0) return true;
  return false;
}
void check_seq(const char* name, const Tensor& t, const Shape& shape, at::ScalarType dtype, const at::Device& dev) {
  if (!same(t, shape)) {
    if (t.dim() != shape.n) fail(name, ": expected rank ", (int64_t)shape.n, ", got ", t.dim());
    fail(name, ": expected shape ", at::IntArrayRef(shape), ", got ", t.sizes());
  }
  if (t.scalar_type() != dtype) fail(name, ": expected dtype ", dtype, ", got ", t.scalar_type());
  if (t.device() != dev) fail(name, ": expected device ", dev, ", got ", t.device());
  if (t.stride(-1) != 1) fail(name, ": innermost stride must be 1");
  if (t.dim() == 4 && t.stride(2) != t.size(3)) fail(name, ": the last two dims must be dense");
  if (overlaid(t, 2)) fail(name, ": expanded over a dim (stride 0); make it contiguous");
}
void check_dense_f32(const char* name, const Tensor* t, const Shape& shape, const at::Device& dev) {
  if (!t) return;
  if (!same(*t, shape)) fail(name, ": expected shape ", at::IntArrayRef(shape), ", got ", t->sizes());
  if (t->scalar_type() != at::kFloat) fail(name, ": expected float32, got ", t->scalar_type());
  if (t->device() != dev || !t->is_contiguous()) fail(name, ": must be a contiguous tensor on ", dev);
}
void check_values_f32(const char* name, const Tensor* t, int64_t n, const at::Device& dev) {   // any shape
  if (t && (t->numel() != n || t->scalar_type() != at::kFloat || t->device() != dev || !t->is_contiguous()))
    fail(name, ": expected ", n, " contiguous fp32 values on ", dev, ", got ", t->sizes(), " ", t->scalar_type(), " on ", t->device());
}
Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const at::Device& dev) {
  return at::detail::empty_cuda(shape, dtype, dev, std::nullopt);
}
void* ptr(const Tensor* t) { return t && t->defined() ? t->data_ptr() : nullptr; }
float* fptr(const Tensor* t) { return (float*)ptr(t); }
void* stream_of(const at::Device& d) { return c10::cuda::getCurrentCUDAStream(d.index()).stream(); }

// The operands of one scan, as both passes take them.
struct Scan {
  const Tensor &x, &dt, &A, &Bm, &Cm;
  const Tensor *D, *z, *init, *bias;
  int64_t chunk, algo;
  bool softplus;
};

// Validates the sequence operands and fills the geometry struct.
SsdDims seq_dims(const Tensor& x, const Tensor& dt, const Tensor& Bm, const Tensor& Cm, const Tensor* z, const Tensor* y, int64_t chunk,
                 int64_t algo, bool softplus) {
  if (!x.is_cuda()) fail("x must be a CUDA tensor (there is no CPU path)");
  if (x.dim() != 4) fail("x must be [batch, seqlen, nheads, headdim]");
  const int32_t dtype = storage_type(x);
  if (Bm.dim() != 4) fail("B must be [batch, seqlen, ngroups, dstate]");
  const int64_t B = x.size(0), L = x.size(1), H = x.size(2), P = x.size(3), G = Bm.size(2), N = Bm.size(3);
  const at::Device dev = x.device();
  const at::ScalarType st = x.scalar_type();
  check_seq("x", x, Shape(B, L, H, P), st, dev);
  check_seq("dt", dt, Shape(B, L, H), st, dev);
  check_seq("B", Bm, Shape(B, L, G, N), st, dev);
  check_seq("C", Cm, Shape(B, L, G, N), st, dev);
  if (G <= 0 || H % G) fail("nheads (", H, ") must be a multiple of ngroups (", G, ")");
  if (chunk < 1 || chunk > 256) fail("chunk must be in [1, 256], got ", chunk);
  SsdDims d;
  std::memset(&d, 0, sizeof d);
  d.batch = (int32_t)B; d.seqlen = (int32_t)L; d.nheads = (int32_t)H; d.headdim = (int32_t)P;
  d.dstate = (int32_t)N; d.ngroups = (int32_t)G; d.chunk = (int32_t)chunk;
  d.dtype = dtype; d.algo = (int32_t)algo; d.device = dev.index(); d.has_z = z ? 1 : 0; d.dt_softplus = softplus ? 1 : 0;
  d.x_stride_b = x.stride(0); d.x_stride_l = x.stride(1);
  d.dt_stride_b = dt.stride(0); d.dt_stride_l = dt.stride(1);
  d.b_stride_b = Bm.stride(0); d.b_stride_l = Bm.stride(1);
  d.c_stride_b = Cm.stride(0); d.c_stride_l = Cm.stride(1);
  if (z) {
    check_seq("z", *z, Shape(B, L, H, P), st, dev);
    d.z_stride_b = z->stride(0); d.z_stride_l = z->stride(1);
  }
  if (y) {
    check_seq("y/dy", *y, Shape(B, L, H, P), st, dev);
    d.y_stride_b = y->stride(0); d.y_stride_l = y->stride(1);
  }
  return d;
}
SsdDims make_dims(const Scan& s, const Tensor* y) {
  const SsdDims d = seq_dims(s.x, s.dt, s.Bm, s.Cm, s.z, y, s.chunk, s.algo, s.softplus);
  const at::Device dev = s.x.device();
  const int64_t H = d.nheads;
  check_dense_f32("A", &s.A, Shape(H), dev);
  check_dense_f32("D", s.D, Shape(H), dev);
  check_dense_f32("dt_bias", s.bias, Shape(H), dev);
  check_dense_f32("init_state", s.init, Shape(d.batch, H, d.headdim, d.dstate), dev);
  return d;
}
Tensor workspace_for(const SsdDims& d, const at::Device& dev, bool backward) {
  const size_t n = api.workspace_bytes(&d, backward ? SSD_PASS_BWD : SSD_PASS_FWD);
  if (!n) throw LibError(-1, api.last_error());
  const int64_t size = (int64_t)n;
  return empty(at::IntArrayRef(&size, 1), at::kByte, dev);
}

void check_workspace(const Tensor& ws, const at::Device& dev) {
  if (ws.device() != dev || !ws.is_contiguous()) fail("workspace: must be a contiguous tensor on ", dev);
}

// y, final_state, workspace; undefined ones among the three are allocated here (final_state only when `want_final`).
void scan_forward(const Scan& s, Tensor& y, Tensor& fin, Tensor& ws, bool want_final, bool for_backward, int32_t stages) {
  const at::Device dev = s.x.device();
  if (!y.defined()) {
    if (!s.x.is_cuda()) fail("x must be a CUDA tensor (there is no CPU path)");
    y = empty(s.x.sizes(), s.x.scalar_type(), dev);
  }
  const SsdDims d = make_dims(s, &y);
  const Shape state(d.batch, d.nheads, d.headdim, d.dstate);
  if (fin.defined()) check_dense_f32("final_state", &fin, state, dev);
  else if (want_final) fin = empty(state, at::kFloat, dev);
  if (ws.defined()) check_workspace(ws, dev);
  else ws = workspace_for(d, dev, for_backward);
  SsdFwdPtrs p;
  std::memset(&p, 0, sizeof p);
  p.x = ptr(&s.x); p.dt = ptr(&s.dt); p.A = fptr(&s.A); p.Bm = ptr(&s.Bm); p.Cm = ptr(&s.Cm); p.D = fptr(s.D); p.z = ptr(s.z);
  p.init_state = fptr(s.init); p.y = ptr(&y); p.final_state = fptr(&fin); p.dt_bias = fptr(s.bias);
  const c10::cuda::CUDAGuard guard(dev);
  check_rc(api.forward_staged(&d, &p, ws.data_ptr(), (size_t)ws.numel(), stream_of(dev), stages));
}

struct Grads { Tensor dx, ddt, dA, dB, dC, dD, dz, dinit, dbias; };

// A caller-provided output must be dense, 16-byte aligned and of the right shape; a missing one is allocated.
void out_slot(const char* key, Tensor& t, const Shape& shape, at::ScalarType dtype, const at::Device& dev) {
  if (!t.defined()) { t = empty(shape, dtype, dev); return; }
  if (!same(t, shape) || t.scalar_type() != dtype || t.device() != dev)
    fail("out['", key, "']: expected ", at::IntArrayRef(shape), " ", dtype, " on ", dev, ", got ", t.sizes(), " ", t.scalar_type(),
         " on ", t.device());
  if (!t.is_contiguous() || (uintptr_t)t.data_ptr() % 16) fail("out['", key, "']: must be contiguous and 16-byte aligned");
}

void scan_backward(const Scan& s, const Tensor& dy, const Tensor* dfin, Tensor& ws, bool fwd_saved, bool want_dinit, int32_t stages,
                   Grads& o) {
  const SsdDims d = make_dims(s, &dy);
  const at::Device dev = s.x.device();
  const at::ScalarType st = s.x.scalar_type();
  const int64_t B = d.batch, L = d.seqlen, H = d.nheads, P = d.headdim, N = d.dstate, G = d.ngroups;
  check_dense_f32("dfinal_state", dfin, Shape(B, H, P, N), dev);
  out_slot("dx", o.dx, Shape(B, L, H, P), st, dev);
  out_slot("ddt", o.ddt, Shape(B, L, H), at::kFloat, dev);
  out_slot("dA", o.dA, Shape(H), at::kFloat, dev);
  out_slot("dB", o.dB, Shape(B, L, G, N), st, dev);
  out_slot("dC", o.dC, Shape(B, L, G, N), st, dev);
  if (s.D) out_slot("dD", o.dD, Shape(H), at::kFloat, dev);
  if (s.z) out_slot("dz", o.dz, Shape(B, L, H, P), st, dev);
  if (want_dinit || s.init) out_slot("dinit", o.dinit, Shape(B, H, P, N), at::kFloat, dev);
  if (s.bias) out_slot("ddt_bias", o.dbias, Shape(H), at::kFloat, dev);
  if (ws.defined()) {
    check_workspace(ws, dev);
  } else {
    if (fwd_saved) fail("fwd_saved=True needs the workspace the forward ran in");
    ws = workspace_for(d, dev, true);
  }
  SsdBwdPtrs p;
  std::memset(&p, 0, sizeof p);
  p.x = ptr(&s.x); p.dt = ptr(&s.dt); p.A = fptr(&s.A); p.Bm = ptr(&s.Bm); p.Cm = ptr(&s.Cm); p.D = fptr(s.D); p.z = ptr(s.z);
  p.init_state = fptr(s.init); p.dy = ptr(&dy); p.dfinal_state = fptr(dfin); p.dx = ptr(&o.dx); p.ddt = fptr(&o.ddt);
  p.dA = fptr(&o.dA); p.dB = ptr(&o.dB); p.dC = ptr(&o.dC); p.dD = fptr(&o.dD); p.dz = ptr(&o.dz); p.dinit_state = fptr(&o.dinit);
  p.fwd_saved = fwd_saved ? 1 : 0; p.dt_bias = fptr(s.bias); p.ddt_bias = fptr(&o.dbias);
  const c10::cuda::CUDAGuard guard(dev);
  check_rc(api.backward_staged(&d, &p, ws.data_ptr(), (size_t)ws.numel(), stream_of(dev), stages));
}

// ---- conv1d and RMS norm -----------------------------------------------------------------------------------------------
void check_conv_weights(const Tensor& in, const Tensor& weight, const Tensor* bias) {
  if (weight.scalar_type() != at::kFloat || !weight.is_contiguous() || weight.dim() != 2)
    fail("conv1d: weight must be contiguous fp32 [channels, width]");
  if (weight.device() != in.device()) fail("conv1d: weight: expected device ", in.device(), ", got ", weight.device());
  if (weight.size(0) != in.size(2)) fail("conv1d: weight rows must equal the channel count");
  check_values_f32("conv1d: bias", bias, weight.size(0), in.device());
}
SsdConvDims conv_dims(const Tensor& in, const Tensor& out, int64_t width, bool activation) {
  if (!in.is_cuda() || in.dim() != 3 || (in.scalar_type() != at::kBFloat16 && in.scalar_type() != at::kFloat))
    fail("conv1d: input must be a CUDA [batch, seqlen, channels] bf16/fp32 tensor");
  if (in.stride(2) != 1 || out.stride(2) != 1) fail("conv1d: the channel dim must be dense");
  SsdConvDims d;
  std::memset(&d, 0, sizeof d);
  d.batch = (int32_t)in.size(0); d.seqlen = (int32_t)in.size(1); d.channels = (int32_t)in.size(2);
  d.width = (int32_t)width; d.dtype = storage_type(in); d.device = in.device().index(); d.activation = activation ? 1 : 0;
  d.in_stride_b = in.stride(0); d.in_stride_l = in.stride(1); d.out_stride_b = out.stride(0); d.out_stride_l = out.stride(1);
  return d;
}
void conv_forward(const Tensor& in, const Tensor& weight, const Tensor* bias, bool activation, Tensor& out) {
  if (!in.is_cuda() || in.dim() != 3) fail("conv1d: input must be a CUDA [batch, seqlen, channels] bf16/fp32 tensor");
  check_conv_weights(in, weight, bias);
  if (!out.defined()) out = empty(in.sizes(), in.scalar_type(), in.device());
  if (!same(out, in.sizes()) || out.scalar_type() != in.scalar_type() || out.device() != in.device())
    fail("conv1d: out: expected ", in.sizes(), " ", in.scalar_type(), " on ", in.device(), ", got ", out.sizes(), " ", out.scalar_type(),
         " on ", out.device());
  const SsdConvDims d = conv_dims(in, out, weight.size(1), activation);
  const c10::cuda::CUDAGuard guard(in.device());
  check_rc(api.conv1d_forward(&d, ptr(&in), fptr(&weight), fptr(bias), ptr(&out), stream_of(in.device())));
}
struct ConvGrads { Tensor din, dweight, dbias; };
ConvGrads conv_backward(const Tensor& in, const Tensor& weight, const Tensor* bias, const Tensor* const* douts, int ndout, bool activation) {
  const at::Device dev = in.device();
  if (!in.is_cuda() || in.dim() != 3) fail("conv1d: input must be a CUDA [batch, seqlen, channels] bf16/fp32 tensor");
  check_conv_weights(in, weight, bias);
  ConvGrads g;
  g.din = empty(in.sizes(), in.scalar_type(), dev);
  const SsdConvDims d = conv_dims(in, g.din, weight.size(1), activation);
  SsdConvGrad segs[3];
  std::memset(segs, 0, sizeof segs);
  if (ndout > 3) fail("conv1d backward: 1 to 3 gradient segments, got ", (int64_t)ndout);
  for (int i = 0; i < ndout; ++i) {
    const Tensor& t = *douts[i];
    if (t.dim() != 3 || t.scalar_type() != in.scalar_type() || t.stride(2) != 1 || t.size(0) != in.size(0) || t.size(1) != in.size(1) || t.device() != dev)
      fail("conv1d backward: bad gradient segment");
    segs[i].ptr = ptr(&t); segs[i].channels = (int32_t)t.size(2); segs[i].stride_b = t.stride(0); segs[i].stride_l = t.stride(1);
  }
  g.dweight = empty(weight.sizes(), at::kFloat, dev);
  g.dbias = empty(Shape(weight.size(0)), at::kFloat, dev);
  const size_t nbytes = api.conv1d_workspace_bytes(&d);
  if (!nbytes) fail(api.last_error());
  Tensor ws = empty(Shape((int64_t)nbytes), at::kByte, dev);
  const c10::cuda::CUDAGuard guard(dev);
  check_rc(api.conv1d_backward(&d, ptr(&in), fptr(&weight), fptr(bias), segs, ndout, ptr(&g.din), g.din.stride(0), g.din.stride(1),
                               fptr(&g.dweight), fptr(&g.dbias), ws.data_ptr(), nbytes, stream_of(dev)));
  return g;
}

void check_norm(const Tensor& in, const Tensor* weight) {
  if (!in.is_cuda() || (in.scalar_type() != at::kBFloat16 && in.scalar_type() != at::kFloat) || !in.is_contiguous() || in.dim() < 1)
    fail("rmsnorm: input must be a contiguous CUDA bf16/fp32 tensor");
  check_values_f32("rmsnorm: weight", weight, in.size(-1), in.device());
}
SsdNormDims norm_dims(const Tensor& in, double eps) {   // `in` contiguous: every dim but the last is a row
  SsdNormDims d;
  std::memset(&d, 0, sizeof d);
  d.width = (int32_t)in.size(-1); d.rows = d.width ? in.numel() / d.width : 0;
  d.dtype = storage_type(in); d.device = in.device().index(); d.eps = (float)eps;
  d.in_stride_row = d.out_stride_row = d.width;
  return d;
}
void norm_forward(const Tensor& in, const Tensor* weight, double eps, Tensor& out, Tensor& rstd) {
  check_norm(in, weight);
  const SsdNormDims d = norm_dims(in, eps);
  out = empty(in.sizes(), in.scalar_type(), in.device());
  rstd = empty(Shape(d.rows), at::kFloat, in.device());
  const c10::cuda::CUDAGuard guard(in.device());
  check_rc(api.rmsnorm_forward(&d, ptr(&in), fptr(weight), ptr(&out), fptr(&rstd), stream_of(in.device())));
}
void norm_backward(const Tensor& in, const Tensor* weight, const Tensor& rstd, const Tensor& dout_, double eps, Tensor& din, Tensor& dweight) {
  check_norm(in, weight);
  if (dout_.numel() != in.numel() || dout_.scalar_type() != in.scalar_type() || dout_.device() != in.device())
    fail("rmsnorm: dout: expected ", in.sizes(), " ", in.scalar_type(), " on ", in.device(), ", got ", dout_.sizes(), " ", dout_.scalar_type(),
         " on ", dout_.device());
  const Tensor dout = dout_.contiguous();
  const SsdNormDims d = norm_dims(in, eps);
  check_values_f32("rmsnorm: rstd", &rstd, d.rows, in.device());
  const at::Device dev = in.device();
  din = empty(in.sizes(), in.scalar_type(), dev);
  Tensor ws;
  if (weight) {
    dweight = empty(weight->sizes(), at::kFloat, dev);
    const size_t n = api.rmsnorm_workspace_bytes(&d);
    ws = empty(Shape((int64_t)n), at::kByte, dev);
  }
  const c10::cuda::CUDAGuard guard(dev);
  check_rc(api.rmsnorm_backward(&d, ptr(&in), fptr(weight), fptr(&rstd), ptr(&dout), d.width, ptr(&din), d.width, fptr(&dweight), ptr(&ws),
                                ws.defined() ? (size_t)ws.numel() : 0, stream_of(dev)));
}

// ---- autograd nodes ----------------------------------------------------------------------------------------------------
bool any_requires_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts) if (t && t->requires_grad()) return true;
  return false;
}
using Opt = std::optional<Tensor>;   // an absent operand of a node: Function::apply takes no undefined tensors
Opt optional(const Tensor* t) { return t ? Opt(*t) : Opt(); }
const Tensor* or_null(const Opt& t) { return t.has_value() ? &*t : nullptr; }
Tensor or_undefined(const Opt& t) { return t.has_value() ? *t : Tensor(); }
Tensor or_undefined(const Tensor* t) { return t ? *t : Tensor(); }
const Tensor* or_null(const Tensor& t) { return t.defined() ? &t : nullptr; }
// An incoming gradient in the layout the kernels read: x's dtype, inner dims dense, rows apart (that of a sum or mean over the
// batch comes expanded).
Tensor usable_dy(const Tensor& g, const Tensor& x) {
  if (!g.defined()) return at::zeros(x.sizes(), x.options().requires_grad(false));
  Tensor dy = g.scalar_type() == x.scalar_type() ? g : g.to(x.scalar_type());
  if (dy.stride(-1) != 1 || dy.stride(2) != dy.size(3) || overlaid(dy, 2)) dy = dy.contiguous();
  return dy;
}
Tensor as_type(const Tensor& t, at::ScalarType st) { return t.scalar_type() == st ? t : t.to(st); }
int64_t pack(int64_t chunk, int64_t algo, bool softplus) { return chunk | (algo << 16) | ((int64_t)softplus << 24); }

struct ScanNode : public torch::autograd::Function<ScanNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& Bm, const Tensor& Cm,
                               const Opt& D, const Opt& z, const Opt& init, const Opt& bias, int64_t chunk, int64_t algo, bool softplus) {
    const Scan s{x, dt, A, Bm, Cm, or_null(D), or_null(z), or_null(init), or_null(bias), chunk, algo, softplus};
    Tensor y, fin, ws;
    scan_forward(s, y, fin, ws, true, true, kAllStages);
    ctx->set_materialize_grads(false);   // an unused final state has no gradient: no zeros to allocate, fill and read
    ctx->save_for_backward({x, dt, A, Bm, Cm, or_undefined(D), or_undefined(z), or_undefined(init), or_undefined(bias), ws});
    ctx->saved_data["how"] = pack(chunk, algo, softplus);
    return {y, fin};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list v = ctx->get_saved_variables();
    const int64_t how = ctx->saved_data["how"].toInt();
    const Scan s{v[0], v[1], v[2], v[3], v[4], or_null(v[5]), or_null(v[6]), or_null(v[7]), or_null(v[8]), how & 0xffff, (how >> 16) & 0xff,
                 ((how >> 24) & 1) != 0};
    const Tensor dy = usable_dy(grads[0], s.x);
    const Tensor dfin = grads[1].defined() ? grads[1].contiguous() : Tensor();
    Tensor ws = v[9];
    Grads g;
    scan_backward(s, dy, or_null(dfin), ws, true, false, kAllStages, g);
    return {g.dx, as_type(g.ddt, s.dt.scalar_type()), g.dA, g.dB, g.dC, g.dD, g.dz, g.dinit, g.dbias, Tensor(), Tensor(), Tensor()};
  }
};

// The whole mixer core as one node: conv + silu -> SSD (softplus step size and gate inside) -> RMS norm.
struct MixerNode : public torch::autograd::Function<MixerNode> {
  struct Parts { Tensor x, Bm, Cm; };
  static Parts parts(const Tensor& conv, int64_t H, int64_t P, int64_t G, int64_t N) {
    const int64_t B = conv.size(0), L = conv.size(1), c = conv.stride(1), b = conv.stride(0);
    return {conv.as_strided({B, L, H, P}, {b, c, P, 1}, 0), conv.as_strided({B, L, G, N}, {b, c, N, 1}, H * P),
            conv.as_strided({B, L, G, N}, {b, c, N, 1}, H * P + G * N)};
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& xBC, const Tensor& dt, const Opt& z, const Tensor& cw, const Opt& cb,
                               const Opt& bias, const Tensor& A, const Opt& D, const Opt& nw, const Opt& init, int64_t H, int64_t P,
                               int64_t N, int64_t G, int64_t chunk, double eps, int64_t algo, bool save) {
    if (xBC.dim() != 3 || xBC.size(2) != H * P + 2 * G * N) fail("xBC: expected [batch, seqlen, ", H * P + 2 * G * N, "], got ", xBC.sizes());
    Tensor conv, y, fin, ws, out, rstd;
    conv_forward(xBC, cw, or_null(cb), true, conv);
    const Parts q = parts(conv, H, P, G, N);
    const Scan s{q.x, dt, A, q.Bm, q.Cm, or_null(D), or_null(z), or_null(init), or_null(bias), chunk, algo, true};
    scan_forward(s, y, fin, ws, true, save, kAllStages);
    norm_forward(y.view({y.size(0), y.size(1), H * P}), or_null(nw), eps, out, rstd);
    if (save) {
      ctx->set_materialize_grads(false);
      ctx->save_for_backward({xBC, dt, or_undefined(z), cw, or_undefined(cb), or_undefined(bias), A, or_undefined(D), or_undefined(nw),
                              or_undefined(init), conv, y, rstd, ws});
      ctx->saved_data["how"] = pack(chunk, algo, true);
      ctx->saved_data["geo"] = (int64_t)N;
      ctx->saved_data["ngroups"] = (int64_t)G;
      ctx->saved_data["eps"] = eps;
    }
    return {out, fin};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list v = ctx->get_saved_variables();
    const Tensor &xBC = v[0], &dt = v[1], &cw = v[3], &A = v[6], &conv = v[10], &y = v[11], &rstd = v[12];
    const int64_t how = ctx->saved_data["how"].toInt(), N = ctx->saved_data["geo"].toInt(), G = ctx->saved_data["ngroups"].toInt();
    const double eps = ctx->saved_data["eps"].toDouble();
    const int64_t B = y.size(0), L = y.size(1), H = y.size(2), P = y.size(3);
    const Tensor yr = y.view({B, L, H * P});
    const Tensor dout = grads[0].defined() ? as_type(grads[0], y.scalar_type()) : at::zeros(yr.sizes(), yr.options());
    Tensor dy, dnw;
    norm_backward(yr, or_null(v[8]), rstd, dout, eps, dy, dnw);
    const Parts q = parts(conv, H, P, G, N);
    const Scan s{q.x, dt, A, q.Bm, q.Cm, or_null(v[7]), or_null(v[2]), or_null(v[9]), or_null(v[5]), how & 0xffff, (how >> 16) & 0xff, true};
    const Tensor dfin = grads[1].defined() ? grads[1].contiguous() : Tensor();
    Tensor ws = v[13];
    Grads g;
    scan_backward(s, dy.view({B, L, H, P}), or_null(dfin), ws, true, false, kAllStages, g);
    const Tensor segs[3] = {g.dx.view({B, L, H * P}), g.dB.view({B, L, G * N}), g.dC.view({B, L, G * N})};
    const Tensor* douts[3] = {&segs[0], &segs[1], &segs[2]};
    ConvGrads c = conv_backward(xBC, cw, or_null(v[4]), douts, 3, true);
    return {c.din, as_type(g.ddt, dt.scalar_type()), g.dz, c.dweight, v[4].defined() ? c.dbias : Tensor(), g.dbias, g.dA, g.dD, dnw, g.dinit,
            Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- Python functions --------------------------------------------------------------------------------------------------
PyObject* pair(const Tensor& a, const Tensor& b) {
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, wrap(a));
  PyTuple_SET_ITEM(r, 1, wrap(b));
  return r;
}
PyObject* triple(const Tensor& a, const Tensor& b, const Tensor& c) {
  PyObject* r = PyTuple_New(3);
  PyTuple_SET_ITEM(r, 0, wrap(a));
  PyTuple_SET_ITEM(r, 1, wrap(b));
  PyTuple_SET_ITEM(r, 2, wrap(c));
  return r;
}

// One step's operands: `where` is the device of the per-stream vectors (the state's, or the CPU).
struct Step {
  SsdStepDims d;
  SsdStepPtrs p;
  int64_t S, H, P;
};
Step step_of(const Tensor& state, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& Bm, const Tensor& Cm, const Tensor* D,
             const Tensor* z, const Tensor* bias, bool softplus, const at::Device& where) {
  const at::Device dev = state.device();
  if (state.dim() != 4 || state.scalar_type() != at::kFloat || !state.is_contiguous())
    fail("state must be a contiguous float32 [streams, nheads, headdim, dstate] tensor");
  const int64_t S = state.size(0), H = state.size(1), P = state.size(2), N = state.size(3);
  Step s;
  std::memset(&s, 0, sizeof s);
  SsdStepDims& d = s.d;
  d.dtype = storage_type(x);
  if (Bm.dim() != 3 || Bm.size(0) != S || Bm.size(2) != N) fail("B must be [streams, ngroups, dstate]");
  const int64_t G = Bm.size(1);
  if (G <= 0 || H % G) fail("nheads (", H, ") must be a multiple of ngroups (", G, ")");
  auto vec = [&](const char* name, const Tensor& t, const Shape& shape) {
    if (!same(t, shape) || t.scalar_type() != x.scalar_type() || t.device() != where)
      fail(name, ": expected ", at::IntArrayRef(shape), " ", x.scalar_type(), " on ", where);
    if (t.stride(-1) != 1 || (t.dim() >= 3 && t.stride(1) != t.size(2))) fail(name, ": inner dims must be dense");
    if (overlaid(t, 1)) fail(name, ": expanded over the streams (stride 0); make it contiguous");
  };
  vec("x", x, Shape(S, H, P)); vec("dt", dt, Shape(S, H)); vec("B", Bm, Shape(S, G, N)); vec("C", Cm, Shape(S, G, N));
  check_dense_f32("A", &A, Shape(H), dev);
  check_dense_f32("D", D, Shape(H), dev);
  check_dense_f32("dt_bias", bias, Shape(H), dev);
  if (z) vec("z", *z, Shape(S, H, P));
  d.streams = (int32_t)S; d.nheads = (int32_t)H; d.headdim = (int32_t)P; d.dstate = (int32_t)N; d.ngroups = (int32_t)G;
  d.device = dev.index(); d.dt_softplus = softplus ? 1 : 0;
  d.x_stride_s = x.stride(0); d.dt_stride_s = dt.stride(0); d.b_stride_s = Bm.stride(0); d.c_stride_s = Cm.stride(0);
  d.z_stride_s = z ? z->stride(0) : 0;
  SsdStepPtrs& p = s.p;
  p.state = fptr(&state); p.x = ptr(&x); p.dt = ptr(&dt); p.A = fptr(&A); p.Bm = ptr(&Bm); p.Cm = ptr(&Cm); p.D = fptr(D); p.z = ptr(z);
  p.dt_bias = fptr(bias);
  s.S = S; s.H = H; s.P = P;
  return s;
}

// state, x, dt, A, B, C, D, z, y, dt_bias, dt_softplus -> y
PyObject* py_state_update(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 11);
    const Tensor &state = a.tensor(0, "state"), &x = a.tensor(1, "x");
    if (!state.is_cuda()) fail("state must be a CUDA tensor (there is no CPU path)");
    const at::Device dev = state.device();
    Step s = step_of(state, x, a.tensor(2, "dt"), a.tensor(3, "A"), a.tensor(4, "B"), a.tensor(5, "C"), a.opt(6, "D"), a.opt(7, "z"),
                     a.opt(9, "dt_bias"), a.flag(10), dev);
    const Tensor* y_in = a.opt(8, "y");
    Tensor y = y_in ? *y_in : empty(Shape(s.S, s.H, s.P), x.scalar_type(), dev);
    if (y_in) {   // rows may lie apart, but not over one another
      const Shape shape(s.S, s.H, s.P);
      if (!same(y, shape) || y.scalar_type() != x.scalar_type() || y.device() != dev)
        fail("y: expected ", at::IntArrayRef(shape), " ", x.scalar_type(), " on ", dev, ", got ", y.sizes(), " ", y.scalar_type(), " on ", y.device());
      if ((s.P > 1 && y.stride(2) != 1) || (s.H > 1 && y.stride(1) != s.P) || (s.S > 1 && y.stride(0) < s.H * s.P)) fail("y: inner dims must be dense and rows apart");
    }
    s.d.y_stride_s = y.stride(0);
    s.p.y = ptr(&y);
    const c10::cuda::CUDAGuard guard(dev);
    check_rc(api.state_update(&s.d, &s.p, stream_of(dev)));
    return wrap(y);
  });
}

// state, x, dt, A, B, C, D, y, y_host: the vectors and y_host in pinned host memory -> None
PyObject* py_state_update_host(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 9);
    const Tensor &state = a.tensor(0, "state"), &y = a.tensor(7, "y"), &yh = a.tensor(8, "y_host");
    if (!state.is_cuda()) fail("state must be a CUDA tensor (there is no CPU path)");
    const at::Device dev = state.device();
    Step s = step_of(state, a.tensor(1, "x"), a.tensor(2, "dt"), a.tensor(3, "A"), a.tensor(4, "B"), a.tensor(5, "C"), a.opt(6, "D"), nullptr,
                     nullptr, false, at::Device(at::kCPU));
    for (const Tensor* t : {&y, &yh})
      if (!same(*t, Shape(s.S, s.H, s.P)) || t->scalar_type() != a.tensor(1, "x").scalar_type() || !t->is_contiguous())
        fail("y: expected a contiguous ", at::IntArrayRef(Shape(s.S, s.H, s.P)), " tensor");
    if (y.device() != dev) fail("y: expected device ", dev, ", got ", y.device());
    s.d.y_stride_s = s.H * s.P;
    s.p.y = ptr(&y);
    const c10::cuda::CUDAGuard guard(dev);
    check_rc(api.state_update_host(&s.d, &s.p, ptr(&yh), stream_of(dev)));
    Py_RETURN_NONE;
  });
}

Scan scan_of(const Args& a, int at, int chunk, int algo, int bias, int softplus) {
  return {a.tensor(at, "x"), a.tensor(at + 1, "dt"), a.tensor(at + 2, "A"), a.tensor(at + 3, "B"), a.tensor(at + 4, "C"), a.opt(at + 5, "D"),
          a.opt(at + 6, "z"), a.opt(at + 7, "init_state"), a.opt(bias, "dt_bias"), a.integer(chunk), a.integer(algo), a.flag(softplus)};
}

// x, dt, B, C, chunk, z, y, algo, dt_softplus -> the bytes of an SsdDims
PyObject* py_dims(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 9);
    const SsdDims d = seq_dims(a.tensor(0, "x"), a.tensor(1, "dt"), a.tensor(2, "B"), a.tensor(3, "C"), a.opt(5, "z"), a.opt(6, "y/dy"),
                               a.integer(4), a.integer(7), a.flag(8));
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&d), sizeof d);
  });
}

// x, dt, A, B, C, D, z, init_state, chunk, algo, workspace, y, final_state, want_final, for_backward, stages, dt_bias, dt_softplus
//   -> y, final_state, workspace
PyObject* py_forward(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 18);
    const Scan s = scan_of(a, 0, 8, 9, 16, 17);
    Tensor ws = or_undefined(a.opt(10, "workspace")), y = or_undefined(a.opt(11, "y")), fin = or_undefined(a.opt(12, "final_state"));
    scan_forward(s, y, fin, ws, a.flag(13), a.flag(14), a.a[15] == Py_None ? kAllStages : (int32_t)a.integer(15));
    return triple(y, fin, ws);
  });
}

// dy, x, dt, A, B, C, D, z, init_state, dfinal_state, chunk, algo, workspace, fwd_saved, want_dinit, stages, out (dict), dt_bias,
// dt_softplus -> out
PyObject* py_backward(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 19);
    const Scan s = scan_of(a, 1, 10, 11, 17, 18);
    PyObject* out = a.a[16];
    Tensor ws = or_undefined(a.opt(12, "workspace"));
    Grads g;
    struct Slot { const char* key; Tensor* t; };
    const Slot slots[] = {{"dx", &g.dx}, {"ddt", &g.ddt}, {"dA", &g.dA}, {"dB", &g.dB}, {"dC", &g.dC}, {"dD", &g.dD}, {"dz", &g.dz},
                          {"dinit", &g.dinit}, {"ddt_bias", &g.dbias}};
    bool given[9] = {};
    for (int i = 0; i < 9; ++i) {
      PyObject* t = PyDict_GetItemString(out, slots[i].key);   // borrowed
      if (!t || t == Py_None) continue;
      if (!THPVariable_Check(t)) fail("out['", slots[i].key, "']: expected a tensor");
      *slots[i].t = THPVariable_Unpack(t);
      given[i] = true;
    }
    scan_backward(s, a.tensor(0, "dy"), a.opt(9, "dfinal_state"), ws, a.flag(13), a.flag(14),
                  a.a[15] == Py_None ? kAllStages : (int32_t)a.integer(15), g);
    auto put = [&](const char* key, const Tensor& t) {
      PyObject* o = wrap(t);
      const int bad = !o || PyDict_SetItemString(out, key, o);
      Py_XDECREF(o);
      if (bad) throw std::runtime_error("out: cannot store a result");
    };
    for (int i = 0; i < 9; ++i)
      if (!given[i] && slots[i].t->defined()) put(slots[i].key, *slots[i].t);
    put("workspace", ws);
    Py_INCREF(out);
    return out;
  });
}

// x, dt, A, B, C, D, z, init_state, chunk, algo, dt_bias, dt_softplus -> y, final_state (differentiable)
PyObject* py_scan(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 12);
    const Scan s = scan_of(a, 0, 8, 9, 10, 11);
    if (!any_requires_grad({&s.x, &s.dt, &s.A, &s.Bm, &s.Cm, s.D, s.z, s.init, s.bias})) {
      Tensor y, fin, ws;
      scan_forward(s, y, fin, ws, true, false, kAllStages);
      return pair(y, fin);
    }
    const variable_list r = ScanNode::apply(s.x, s.dt, s.A, s.Bm, s.Cm, optional(s.D), optional(s.z), optional(s.init), optional(s.bias),
                                            s.chunk, s.algo, s.softplus);
    return pair(r[0], r[1]);
  });
}

// xBC, dt, z, conv_weight, conv_bias, dt_bias, A, D, norm_weight, init_state, nheads, headdim, dstate, ngroups, chunk, eps, algo
//   -> out, final_state (differentiable)
PyObject* py_mixer(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 17);
    const char* names[] = {"xBC", "dt", "z", "conv_weight", "conv_bias", "dt_bias", "A", "D", "norm_weight", "init_state"};
    const Tensor* t[10];
    bool save = false;
    for (int i = 0; i < 10; ++i) {
      t[i] = i == 0 || i == 1 || i == 3 || i == 6 ? &a.tensor(i, names[i]) : a.opt(i, names[i]);   // the rest may be None
      save |= t[i] && t[i]->requires_grad();
    }
    save = save && at::GradMode::is_enabled();
    const variable_list r = MixerNode::apply(*t[0], *t[1], optional(t[2]), *t[3], optional(t[4]), optional(t[5]), *t[6], optional(t[7]),
                                             optional(t[8]), optional(t[9]), a.integer(10), a.integer(11), a.integer(12), a.integer(13),
                                             a.integer(14), a.real(15), a.integer(16), save);
    return pair(r[0], r[1]);
  });
}

// in, weight, bias, activation, out -> out
PyObject* py_conv_forward(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 5);
    Tensor out = or_undefined(a.opt(4, "out"));
    conv_forward(a.tensor(0, "input"), a.tensor(1, "weight"), a.opt(2, "bias"), a.flag(3), out);
    return wrap(out);
  });
}
// in, weight, bias, activation, dout_0 [, dout_1 [, dout_2]] -> din, dweight, dbias
PyObject* py_conv_backward(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, argc);
    if (argc < 4 || argc > 7) fail("conv1d backward: 1 to 3 gradient segments, got ", (int64_t)argc - 4);
    const Tensor* douts[3];
    for (int i = 4; i < argc; ++i) douts[i - 4] = &a.tensor(i, "gradient segment");
    const ConvGrads g = conv_backward(a.tensor(0, "input"), a.tensor(1, "weight"), a.opt(2, "bias"), douts, (int)argc - 4, a.flag(3));
    return triple(g.din, g.dweight, g.dbias);
  });
}
// in, weight, eps -> out, rstd
PyObject* py_norm_forward(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 3);
    Tensor out, rstd;
    norm_forward(a.tensor(0, "input"), a.opt(1, "weight"), a.real(2), out, rstd);
    return pair(out, rstd);
  });
}
// in, weight, rstd, dout, eps -> din, dweight
PyObject* py_norm_backward(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 5);
    Tensor din, dweight;
    norm_backward(a.tensor(0, "input"), a.opt(1, "weight"), a.tensor(2, "rstd"), a.tensor(3, "dout"), a.real(4), din, dweight);
    return pair(din, dweight);
  });
}

// addresses (a tuple in Api's order), SsdError, torch.OutOfMemoryError
PyObject* py_bind(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  return guarded([&]() -> PyObject* {
    const Args a(argv, argc, 3);
    constexpr Py_ssize_t n = sizeof(Api) / sizeof(void*);
    if (!PyTuple_Check(argv[0]) || PyTuple_GET_SIZE(argv[0]) != n) fail("bind: expected ", (int64_t)n, " addresses");
    void** slot = reinterpret_cast<void**>(&api);
    for (Py_ssize_t i = 0; i < n; ++i) slot[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(argv[0], i));
    Py_INCREF(argv[1]);
    Py_INCREF(argv[2]);
    ssd_error = argv[1];   // the module is bound once and lives as long as the process
    oom_error = argv[2];
    Py_RETURN_NONE;
  });
}

#define FAST(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST("bind", py_bind), FAST("dims", py_dims), FAST("state_update", py_state_update), FAST("state_update_host", py_state_update_host), FAST("forward", py_forward),
                         FAST("backward", py_backward), FAST("scan", py_scan), FAST("mixer", py_mixer),
                         FAST("conv1d_forward", py_conv_forward), FAST("conv1d_backward", py_conv_backward),
                         FAST("rmsnorm_forward", py_norm_forward), FAST("rmsnorm_backward", py_norm_backward), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ssd_host", "native host path of the SSD entry points", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__ssd_host(void) { return PyModule_Create(&module); }
