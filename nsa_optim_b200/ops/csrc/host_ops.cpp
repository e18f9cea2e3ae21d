// Host side of the differentiable ops as a Python extension module (``_nsa_host``): one call prepares an op's inputs (contiguous, 16-byte
// aligned rows), allocates its outputs and launches its kernels.  ``ops/native.py`` keeps what autograd needs to see: the Function
// classes, what they save, and which calls they take.
//
// Why: a small op is bound by the host.  With the same steps in Python (views, allocations, addresses, a ctypes call with up to 35
// arguments) a norm of 64 rows took 16 us forward, 116 with its backward; now 7.4 and 77 (a recorded Python function that does nothing
// takes 40).  Evaluation attention 19 -> 13 us, a projection 13.6 -> 6.9, 100 tokens of the scan, forward and backward, 221 -> 141, an
// MLP 329 -> 201.
//
// The kernels' entry points are those of the library that ``native.load()`` opened (``bind``).  The GIL is given back while a call
// prepares and launches, as ctypes and PyTorch's operators do; with guard zones on (NSA_B200_DEBUG_CANARY) outputs come from
// ``native._guarded`` and it is kept.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cmath>
#include <limits>
#include <vector>

#include "nsa_b200.h"

namespace {
using at::Tensor;

// ------------------------------------------------------------------------------------- the library
#define NSA_ENTRIES(X)                                                                                                             \
  X(nsa_last_error) X(nsa_gemm_bf16) X(nsa_gemm_bf16_splitk) X(nsa_rmsnorm_fwd) X(nsa_rmsnorm_add_fwd) X(nsa_rmsnorm_fwd_ldg)        \
  X(nsa_rmsnorm_bwd) X(nsa_rmsnorm_bwd_res) X(nsa_rmsnorm_bwd_ldg) X(nsa_rmsnorm_bwd_parts) X(nsa_l2norm_fwd) X(nsa_l2norm_bwd)      \
  X(nsa_swiglu_fwd) X(nsa_swiglu_bwd) X(nsa_rope) X(nsa_conv1d_fwd) X(nsa_conv1d_bwd) X(nsa_conv1d_bwd_parts) X(nsa_embedding_fwd)  \
  X(nsa_cross_entropy) X(nsa_scale_bf16) X(nsa_attn_fwd) X(nsa_attn_bwd) X(nsa_attn_bwd_split) X(nsa_attn_bwd_walks)                 \
  X(nsa_attn_importance) X(nsa_union_blocks) X(nsa_inverse_chunks) X(nsa_inverse_blocks) X(nsa_select_blocks)                        \
  X(nsa_gate_combine_fwd_ex) X(nsa_gate_combine_bwd_ex) X(nsa_pool_fwd) X(nsa_pool_bwd) X(nsa_gdn_prep) X(nsa_gdn_seq_fwd)           \
  X(nsa_gdn_seq_bwd) X(nsa_gdn_post) X(nsa_ssd_states_form) X(nsa_ssd_states) X(nsa_ssd_chunk_state) X(nsa_ssd_state_fwd)         \
  X(nsa_ssd_state_bwd) X(nsa_ssd_chunk_out) X(nsa_ssd_chunk_grad) X(nsa_ssd_grad_slots) X(nsa_ssd_finish) X(nsa_adamw_multi)         \
  X(nsa_adamw8bit_multi) X(nsa_gates)

struct Lib {
#define X(f) decltype(&::f) f = nullptr;
  NSA_ENTRIES(X)
#undef X
} lib;
PyObject* g_native = nullptr;                    // the dictionary of ops/native.py
PyObject *g_canary = nullptr, *g_guarded = nullptr;   // its names
bool g_single_gemm = false;                      // see native.gemm_select
long g_splitk_max = 2;

cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// An entry point of the library; a partial build may lack some.
template <class F>
F* have(F* f) {
  TORCH_CHECK(f != nullptr, "nsa_optim_b200 native library lacks an entry point that this op needs");
  return f;
}
// Launches on the current stream.
template <class F, class... A>
void launch(F* f, A... a) {
  const int rc = have(f)(a..., stream());
  TORCH_CHECK(rc == 0, "nsa_optim_b200 native call failed (", rc, "): ", lib.nsa_last_error());
}

// ------------------------------------------------------------------------------------- calls and allocation
thread_local bool t_guarded = false;

// One call from Python: without the GIL, unless guard zones are on.
struct Call {
  PyThreadState* state = nullptr;
  bool outer = t_guarded;
  Call() {
    PyObject* on = g_native ? PyDict_GetItem(g_native, g_canary) : nullptr;
    t_guarded = on && PyObject_IsTrue(on) == 1;
    if (!t_guarded) state = PyEval_SaveThread();
  }
  ~Call() {
    if (state) PyEval_RestoreThread(state);
    t_guarded = outer;
  }
};

Tensor alloc(at::IntArrayRef shape, at::ScalarType dtype, const at::Device& dev, bool zero = false) {
  if (t_guarded && dev.is_cuda()) {
    THPObjectPtr size(PyTuple_New(shape.size()));
    for (size_t i = 0; i < shape.size(); ++i) PyTuple_SET_ITEM(size.get(), i, PyLong_FromLongLong(shape[i]));
    PyObject* guarded = PyDict_GetItem(g_native, g_guarded);
    THPObjectPtr device(THPDevice_New(dev));
    PyObject* type = reinterpret_cast<PyObject*>(torch::getTHPDtype(dtype));
    THPObjectPtr r(PyObject_CallFunctionObjArgs(guarded, size.get(), type, device.get(), zero ? Py_True : Py_False, nullptr));
    if (!r) throw python_error();
    return THPVariable_Unpack(r.get());
  }
  const auto options = at::TensorOptions().dtype(dtype).device(dev);
  return zero ? at::zeros(shape, options) : at::empty(shape, options);
}
constexpr auto BF = at::kBFloat16;
constexpr auto F32 = at::kFloat;
constexpr auto I32 = at::kInt;

void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* fp(const Tensor& t) { return static_cast<float*>(ptr(t)); }
int* ip(const Tensor& t) { return static_cast<int*>(ptr(t)); }
bool aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
Tensor to(const Tensor& t, at::ScalarType dtype) { return t.scalar_type() == dtype ? t : t.to(dtype); }
int dim(int64_t n) { return static_cast<int>(n); }
void want_dims(const Tensor& t, int64_t n) { TORCH_CHECK_VALUE(t.dim() == n, "expected a tensor of ", n, " dimensions, got ", t.dim()); }
int64_t rows_of(const Tensor& t) { return t.size(-1) ? t.numel() / t.size(-1) : 0; }

// ------------------------------------------------------------------------------------- arguments and results
struct Args {
  PyObject* const* a;
  Py_ssize_t n, i = 0;
  PyObject* next() {
    TORCH_CHECK_TYPE(i < n, "_nsa_host: an argument is missing");
    return a[i++];
  }
  const Tensor& t() {
    PyObject* o = next();
    TORCH_CHECK_TYPE(THPVariable_Check(o), "_nsa_host: argument ", i - 1, " has to be a tensor");
    return THPVariable_Unpack(o);
  }
  Tensor opt() {                                 // None: no tensor
    PyObject* o = next();
    if (o == Py_None) return Tensor();
    TORCH_CHECK_TYPE(THPVariable_Check(o), "_nsa_host: argument ", i - 1, " has to be a tensor or None");
    return THPVariable_Unpack(o);
  }
  std::vector<Tensor> ts() {                     // a tuple of tensors and None
    PyObject* o = next();
    TORCH_CHECK_TYPE(PyTuple_Check(o), "_nsa_host: argument ", i - 1, " has to be a tuple");
    std::vector<Tensor> v(PyTuple_GET_SIZE(o));
    for (size_t k = 0; k < v.size(); ++k) {
      PyObject* x = PyTuple_GET_ITEM(o, k);
      TORCH_CHECK_TYPE(x == Py_None || THPVariable_Check(x), "_nsa_host: argument ", i - 1, " has to be a tuple of tensors and None");
      if (x != Py_None) v[k] = THPVariable_Unpack(x);
    }
    return v;
  }
  long l() {                                     // numbers wider than 64 bits are cut, as ctypes does
    PyObject* o = next();
    if (o == Py_True) return 1;
    if (o == Py_False) return 0;
    const unsigned long v = PyLong_AsUnsignedLongMask(o);
    if (v == static_cast<unsigned long>(-1) && PyErr_Occurred()) throw python_error();
    return static_cast<long>(v);
  }
  long count() {                                 // as above, but wider numbers become the largest or the smallest
    PyObject* o = next();
    int over = 0;
    const long v = PyLong_AsLongAndOverflow(o, &over);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return over > 0 ? std::numeric_limits<long>::max() : over < 0 ? std::numeric_limits<long>::min() : v;
  }
  std::vector<bool> bools() {                    // a tuple of truth values
    PyObject* o = next();
    TORCH_CHECK_TYPE(PyTuple_Check(o), "_nsa_host: argument ", i - 1, " has to be a tuple");
    std::vector<bool> v(PyTuple_GET_SIZE(o));
    for (size_t k = 0; k < v.size(); ++k) v[k] = PyTuple_GET_ITEM(o, k) == Py_True;
    return v;
  }
  int w() { return static_cast<int>(l()); }
  bool b() { return l() != 0; }
  int flag() {                                   // as int() takes it: NumPy's truth values are not integers
    PyObject* o = next();
    if (o == Py_True) return 1;
    if (o == Py_False) return 0;
    THPObjectPtr n(PyNumber_Long(o));
    if (!n) throw python_error();
    return static_cast<int>(PyLong_AsUnsignedLongMask(n.get()));
  }
  float f() {
    const double v = PyFloat_AsDouble(next());
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return static_cast<float>(v);
  }
  at::ScalarType dtype() {
    PyObject* o = next();
    TORCH_CHECK_TYPE(THPDtype_Check(o), "_nsa_host: argument ", i - 1, " has to be a dtype");
    return reinterpret_cast<THPDtype*>(o)->scalar_type;
  }
};

PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* wrap(const std::vector<Tensor>& v) {
  PyObject* r = PyTuple_New(v.size());
  for (size_t i = 0; i < v.size(); ++i) PyTuple_SET_ITEM(r, i, wrap(v[i]));
  return r;
}

// A function of this module: reads its arguments with the GIL and returns the body, which runs as a Call; the result is
// a tensor, or several as a tuple.
template <class Body>
PyObject* entry(PyObject* const* a, Py_ssize_t n, Body make) {
  HANDLE_TH_ERRORS
  Args args{a, n};
  auto body = make(args);
  decltype(body()) r;
  {
    Call call;
    r = body();
  }
  return wrap(r);
  END_HANDLE_TH_ERRORS
}
#define OP(name) PyObject* name(PyObject*, PyObject* const* py, Py_ssize_t np)
using List = std::vector<Tensor>;

// ------------------------------------------------------------------------------------- norms
// (rows, d) contiguous without a copy where it can be
Tensor dense(const Tensor& t) { return t.contiguous(); }

OP(rms_fwd) {                                    // x, w, eps -> y, x dense, w bf16, rstd
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &w = a.t();
    const float eps = a.f();
    return [=]() -> List {
      const Tensor xc = dense(x), wb = to(w, BF);
      const long d = xc.size(-1), rows = rows_of(xc);
      const Tensor y = alloc(x.sizes(), x.scalar_type(), x.device()), rstd = alloc({rows}, F32, x.device());
      launch(lib.nsa_rmsnorm_fwd, ptr(xc), static_cast<const void*>(nullptr), ptr(wb), ptr(y), fp(rstd), rows, dim(d), eps, 0);
      return {y, xc, wb, rstd};
    };
  });
}

OP(add_rms_fwd) {                                // x, r, w, eps -> h, y, w bf16, rstd
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &r = a.t(), &w = a.t();
    const float eps = a.f();
    return [=]() -> List {
      const Tensor xc = dense(x), rc = dense(r), wb = to(w, BF);
      const long d = xc.size(-1), rows = rows_of(xc);
      const Tensor h = alloc(x.sizes(), x.scalar_type(), x.device()), y = alloc(x.sizes(), x.scalar_type(), x.device());
      const Tensor rstd = alloc({rows}, F32, x.device());
      launch(lib.nsa_rmsnorm_add_fwd, ptr(xc), ptr(rc), ptr(wb), ptr(h), ptr(y), fp(rstd), rows, dim(d), eps);
      return {h, y, wb, rstd};
    };
  });
}

OP(rms_bwd) {                                    // x, w, rstd, dy, gradient of the residual route or None, dtype of dw -> dx, dw
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &w = a.t(), &rstd = a.t(), &dy = a.t();
    const Tensor res = a.opt();
    const auto wtype = a.dtype();
    return [=]() -> List {
      const Tensor dyc = dense(dy), rc = res.defined() ? dense(res) : res;
      const long d = x.size(-1), rows = rows_of(x);
      const Tensor dx = alloc(dy.sizes(), x.scalar_type(), x.device()), dw = alloc({d}, BF, x.device());
      const Tensor part = alloc({have(lib.nsa_rmsnorm_bwd_parts)(rows, dim(d)) * d}, F32, x.device());
      float* none = nullptr;
      if (rc.defined())
        launch(lib.nsa_rmsnorm_bwd_res, ptr(x), ptr(w), ptr(dyc), fp(rstd), ptr(rc), ptr(dx), ptr(dw), none, fp(part), rows, dim(d));
      else
        launch(lib.nsa_rmsnorm_bwd, ptr(x), static_cast<const void*>(nullptr), ptr(w), ptr(dyc), fp(rstd), ptr(dx), static_cast<void*>(nullptr),
               ptr(dw), none, fp(part), rows, dim(d), 0);
      return {dx, to(dw, wtype)};
    };
  });
}

// Rows of a gate: a column slice of a wider row-major matrix is used in place when its rows are 16-byte aligned; anything else is
// made contiguous.
Tensor gate_rows(const Tensor& g) {
  const long d = g.size(-1);
  if (g.dim() >= 2 && d > 0 && g.stride(-1) == 1 && aligned(g)) {
    const long pitch = g.stride(-2);
    long expect = pitch;
    bool ok = pitch % 8 == 0 && pitch >= d;
    for (long k = g.dim() - 2; k >= 0; --k) {
      if (g.size(k) != 1 && g.stride(k) != expect) ok = false;
      expect *= g.size(k);
    }
    if (ok) return at::as_strided(g, {g.numel() / d, d}, {pitch, 1});
  }
  return g.reshape({-1, d}).contiguous();
}
// Elements from one row (last dimension) to the next; a single row of a dense tensor may have any stride.  Read from a saved tensor as it comes back: saved-tensor hooks (activations
// kept on the host) return a pitched view as a dense tensor.
long row_pitch(const Tensor& t) { return t.is_contiguous() ? t.size(-1) : t.stride(-2); }

OP(gated_rms_fwd) {                              // x, gate, w, eps, mode -> y, x dense, gate rows, w bf16, rstd
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &gate = a.t(), &w = a.t();
    const float eps = a.f();
    const int mode = a.w();
    return [=]() -> List {
      const Tensor xc = dense(x), g = gate_rows(gate), wb = to(w, BF);
      const long d = xc.size(-1), rows = rows_of(xc);
      const Tensor y = alloc(x.sizes(), x.scalar_type(), x.device()), rstd = alloc({rows}, F32, x.device());
      launch(lib.nsa_rmsnorm_fwd_ldg, ptr(xc), ptr(g), row_pitch(g), ptr(wb), ptr(y), fp(rstd), rows, dim(d), eps, mode);
      return {y, xc, g, wb, rstd};
    };
  });
}

OP(gated_rms_bwd) {                              // x, gate rows, w, rstd, dy, mode, dtype of dw -> dx, d gate (rows, d), dw
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &g = a.t(), &w = a.t(), &rstd = a.t(), &dy = a.t();
    const int mode = a.w();
    const auto wtype = a.dtype();
    return [=]() -> List {
      const Tensor dyc = dense(dy);
      const long d = x.size(-1), rows = rows_of(x);
      const Tensor dx = alloc(dy.sizes(), x.scalar_type(), x.device()), dg = alloc({rows, d}, x.scalar_type(), x.device());
      const Tensor dw = alloc({d}, BF, x.device()), part = alloc({have(lib.nsa_rmsnorm_bwd_parts)(rows, dim(d)) * d}, F32, x.device());
      float* none = nullptr;
      launch(lib.nsa_rmsnorm_bwd_ldg, ptr(x), ptr(g), row_pitch(g), ptr(w), ptr(dyc), fp(rstd), ptr(dx), ptr(dg), ptr(dw), none, fp(part),
             rows, dim(d), mode);
      return {dx, dg, to(dw, wtype)};
    };
  });
}

OP(l2_fwd) {                                     // x, eps -> y, 1 / norm
  return entry(py, np, [](Args& a) {
    const Tensor& x = a.t();
    const float eps = a.f();
    return [=]() -> List {
      const Tensor xc = dense(x);
      const long rows = rows_of(xc);
      const Tensor y = alloc(x.sizes(), x.scalar_type(), x.device()), rinv = alloc({rows}, F32, x.device());
      launch(lib.nsa_l2norm_fwd, ptr(xc), ptr(y), fp(rinv), rows, dim(xc.size(-1)), eps);
      return {y, rinv};
    };
  });
}

OP(l2_bwd) {                                     // y, 1 / norm, dy -> dx
  return entry(py, np, [](Args& a) {
    const Tensor &y = a.t(), &rinv = a.t(), &dy = a.t();
    return [=]() -> Tensor {
      const Tensor dyc = dense(dy), dx = alloc(dy.sizes(), y.scalar_type(), y.device());
      launch(lib.nsa_l2norm_bwd, ptr(y), ptr(dyc), fp(rinv), ptr(dx), rows_of(y), dim(y.size(-1)));
      return dx;
    };
  });
}

// ------------------------------------------------------------------------------------- SwiGLU, RoPE, convolution, embedding
// (rows, columns) with 16-byte aligned rows of any pitch
Tensor matrix(const Tensor& t) {
  Tensor m = t.dim() == 2 ? t : t.reshape({-1, t.size(-1)});
  return m.stride(1) != 1 || m.stride(0) % 8 || !aligned(m) ? m.contiguous() : m;
}

OP(swiglu_fwd) {                                 // gate, up -> y, gate rows, up rows
  return entry(py, np, [](Args& a) {
    const Tensor &gate = a.t(), &up = a.t();
    return [=]() -> List {
      const Tensor g = matrix(gate), u = matrix(up), y = alloc(gate.sizes(), gate.scalar_type(), gate.device());
      launch(lib.nsa_swiglu_fwd, ptr(g), ptr(u), ptr(y), g.size(0), dim(g.size(1)), g.stride(0), u.stride(0));
      return {y, g, u};
    };
  });
}

OP(swiglu_bwd) {                                 // gate rows, up rows, dy -> d gate, d up
  return entry(py, np, [](Args& a) {
    const Tensor &g = a.t(), &u = a.t(), &dy = a.t();
    return [=]() -> List {
      const Tensor dyc = dense(dy), dg = alloc(dy.sizes(), dy.scalar_type(), dy.device()), du = alloc(dy.sizes(), dy.scalar_type(), dy.device());
      const long rows = g.size(0), cols = g.size(1);
      launch(lib.nsa_swiglu_bwd, ptr(g), ptr(u), ptr(dyc), ptr(dg), ptr(du), rows, dim(cols), g.stride(0), u.stride(0), cols);
      return {dg, du};
    };
  });
}

OP(rope) {                                       // x, cos, sin (fp32, dense), backward -> y
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &c = a.t(), &s = a.t();
    const int back = a.w();
    return [=]() -> Tensor {
      want_dims(x, 4);
      const Tensor xc = dense(x), y = alloc(x.sizes(), x.scalar_type(), x.device());
      launch(lib.nsa_rope, ptr(xc), fp(c), fp(s), ptr(y), x.size(0), dim(x.size(1)), dim(x.size(2)), dim(x.size(3)), back);
      return y;
    };
  });
}

OP(conv_fwd) {                                   // x, w, bias or None, activation -> y, x rows, w bf16, bias bf16
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &w = a.t();
    const Tensor bias = a.opt();
    const int act = a.flag();
    return [=]() -> List {
      want_dims(x, 3);
      const long B = x.size(0), T = x.size(1), C = x.size(2);
      const Tensor xv = x.stride(2) == 1 && x.stride(1) % 8 == 0 && x.stride(0) == T * x.stride(1) && aligned(x) ? x : x.contiguous();
      const Tensor wb = to(w, BF).contiguous(), bb = bias.defined() ? to(bias, BF).contiguous() : bias;
      const Tensor y = alloc({B, T, C}, x.scalar_type(), x.device());
      launch(lib.nsa_conv1d_fwd, ptr(xv), ptr(wb), ptr(bb), ptr(y), dim(B), dim(T), dim(C), xv.stride(1), dim(w.size(-1)), act);
      return {y, xv, wb, bb};
    };
  });
}

OP(conv_bwd) {                                   // x rows, w, bias or None, dy, activation, dtype of dw -> dx, dw, db
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &w = a.t();
    const Tensor bias = a.opt();
    const Tensor& dy = a.t();
    const int act = a.flag();
    const auto wtype = a.dtype();
    return [=]() -> List {
      const long B = x.size(0), T = x.size(1), C = x.size(2), W = w.size(-1);
      const Tensor dyc = dense(dy), dx = alloc({B, T, C}, dy.scalar_type(), dy.device());
      const Tensor part = alloc({have(lib.nsa_conv1d_bwd_parts)(dim(B), dim(T), dim(C)) * (W + 1) * C}, F32, dy.device());
      const auto out = wtype == BF ? BF : F32;
      const Tensor dw = alloc({C, W}, out, dy.device()), db = bias.defined() ? alloc({C}, out, dy.device()) : Tensor();
      launch(lib.nsa_conv1d_bwd, ptr(x), ptr(w), ptr(bias), ptr(dyc), ptr(dx), fp(part), ptr(dw), ptr(db), static_cast<int>(out == F32),
             dim(B), dim(T), dim(C), x.stride(1), dim(W), act);
      return {dx, to(dw, wtype), db.defined() ? to(db, wtype) : db};
    };
  });
}

OP(embedding_fwd) {                              // ids, w -> y, flat ids
  return entry(py, np, [](Args& a) {
    const Tensor &ids = a.t(), &w = a.t();
    return [=]() -> List {
      const Tensor flat = ids.reshape(-1).contiguous();
      const long d = w.size(1);
      std::vector<int64_t> shape(ids.sizes().begin(), ids.sizes().end());
      shape.push_back(d);
      const Tensor y = alloc(shape, w.scalar_type(), w.device());
      launch(lib.nsa_embedding_fwd, static_cast<const long*>(ptr(flat)), ptr(w), ptr(y), flat.numel(), dim(d), w.size(0));
      return {y, flat};
    };
  });
}

// ------------------------------------------------------------------------------------- GEMM
// Parts to cut the reduction into: see native.split_k_choice
long split_k(long M, long N, long K, long clusters) {
  if (K < 8192 || M <= 128) return 1;
  const long tiles = (M + 255) / 256 * ((N + 255) / 256);
  if (tiles >= 6 * clusters) return 1;
  auto fill = [&](long S) {
    const double w = static_cast<double>(tiles * S) / clusters;
    return w / std::ceil(w);
  };
  long best = 1;
  for (long S = 2; S <= g_splitk_max; ++S)
    if (fill(S) - 0.01 * S > fill(best) - 0.01 * best) best = S;
  // Parts cost a pass that clears the fp32 sums and one that converts them, 1.6 ps an element; of the time that fuller waves save,
  // 1.25 fs a product, two fifths remain (sums pass through L2, and under the power cap idle SMs let the others clock higher).  5632 x
  // 2048: K = 8192 143 us in one part, 133 + 18 in two; K = 65536 saves 80.
  return fill(best) > fill(1) + 0.04 && K * (1 / fill(1) - 1 / fill(best)) > 3200 ? best : 1;
}

// C = op(A) op(B); a_mn: A is (K, M), b_mn: B is (K, N).  out undefined: allocated as (M, N).  parts 0: chosen.
Tensor gemm(const Tensor& a_, const Tensor& b_, bool a_mn, bool b_mn, Tensor out = Tensor(), at::ScalarType type = BF, bool accumulate = false,
            int max_ctas = 0, long parts = 0) {
  const Tensor a = matrix(a_), b = matrix(b_);
  const long M = a.size(a_mn ? 1 : 0), K = a.size(a_mn ? 0 : 1), N = b.size(b_mn ? 1 : 0), Kb = b.size(b_mn ? 0 : 1);
  TORCH_CHECK_VALUE(K == Kb, "gemm: reduction sizes differ (", K, " vs ", Kb, ")");
  if (!out.defined()) out = alloc({M, N}, type, a.device());
  if (parts == 0) parts = max_ctas == 0 && !g_single_gemm ? split_k(M, N, K, 74) : 1;
  if (parts > 1 && M > 128) {
    const bool direct = out.scalar_type() == F32 && out.stride(1) == 1 && out.stride(0) % 4 == 0 && aligned(out);
    Tensor ws;
    if (direct) {
      ws = out;
      if (!accumulate) ws.zero_();
    } else {
      ws = accumulate ? out.to(F32) : alloc({M, N}, F32, a.device(), true);
    }
    launch(lib.nsa_gemm_bf16_splitk, ptr(a), ptr(b), fp(ws), dim(M), dim(N), dim(K), dim(a.stride(0)), dim(b.stride(0)), dim(ws.stride(0)),
           static_cast<int>(a_mn), static_cast<int>(b_mn), dim(parts));
    if (!direct) out.copy_(ws);
    return out;
  }
  launch(lib.nsa_gemm_bf16, ptr(a), ptr(b), ptr(out), dim(M), dim(N), dim(K), dim(a.stride(0)), dim(b.stride(0)), dim(out.stride(0)),
         static_cast<int>(a_mn), static_cast<int>(b_mn), static_cast<int>(out.scalar_type() == F32), static_cast<int>(accumulate), max_ctas);
  return out;
}
// x w^T in the shape of x with its last dimension replaced
Tensor project(const Tensor& x2, const Tensor& w, const Tensor& x) {
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 1);
  shape.push_back(w.size(0));
  const Tensor y = alloc(shape, BF, x.device());
  gemm(x2, w, false, false, y.dim() == 2 ? y : y.view({-1, w.size(0)}));
  return y;
}
Tensor in_shape(const Tensor& g, std::vector<int64_t> shape, int64_t last) {
  shape.back() = last;
  return g.view(shape);
}

OP(matmul) {                                     // a, b, a_mn, b_mn, out or None, dtype, accumulate, max_ctas, parts -> C
  return entry(py, np, [](Args& g) {
    const Tensor &a = g.t(), &b = g.t();
    const bool a_mn = g.flag(), b_mn = g.flag();
    const Tensor out = g.opt();
    const auto type = g.dtype();
    const bool accumulate = g.flag();
    const int max_ctas = g.w();
    const long parts = g.l();
    return [=]() -> Tensor { return gemm(a, b, a_mn, b_mn, out, type, accumulate, max_ctas, parts); };
  });
}

OP(linear_fwd) {                                 // x, w -> y, x rows
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &w = a.t();
    return [=]() -> List {
      const Tensor x2 = matrix(x);
      return {project(x2, w, x), x2};
    };
  });
}

OP(multi_linear_fwd) {                           // x, weights -> outputs..., x rows
  return entry(py, np, [](Args& a) {
    const Tensor& x = a.t();
    const List ws = a.ts();
    return [=]() -> List {
      const Tensor x2 = matrix(x);
      List r;
      for (const Tensor& w : ws) r.push_back(project(x2, w, x));
      r.push_back(x2);
      return r;
    };
  });
}

OP(multi_linear_bwd) {                           // x rows, weights, gradients, want dx, want each dw -> dx, dw...
  return entry(py, np, [](Args& a) {
    const Tensor& x2 = a.t();
    const List ws = a.ts(), dys = a.ts();
    const bool want_x = a.b();
    const std::vector<bool> want_w = a.bools();
    TORCH_CHECK_VALUE(dys.size() == ws.size() && want_w.size() == ws.size(), "_nsa_host: as many gradients as weights");
    return [=]() -> List {
      List r(1 + ws.size());
      std::vector<int64_t> shape;
      for (size_t i = 0; i < ws.size(); ++i) {
        if (!dys[i].defined()) continue;
        const Tensor dy = matrix(dys[i]);
        if (want_x) {                            // the first product stores, the others add in the epilogue
          if (!r[0].defined()) { r[0] = gemm(dy, ws[i], false, true); shape = dys[i].sizes().vec(); }
          else gemm(dy, ws[i], false, true, r[0], BF, true, 0, 1);
        }
        if (want_w[i]) r[1 + i] = gemm(dy, x2, true, true);
      }
      if (r[0].defined()) r[0] = in_shape(r[0], shape, x2.size(1));
      return r;
    };
  });
}

OP(cross_entropy_fwd) {                          // hidden, w, labels, ignore, chunk, want dh, want dw -> loss, dh, dw (fp32)
  return entry(py, np, [](Args& a) {
    const Tensor &hidden = a.t(), &w = a.t(), &labels_ = a.t();
    const long ignore = a.l(), chunk = a.count();
    const bool need_h = a.b(), need_w = a.b();
    return [=]() -> List {
      want_dims(hidden, 2);
      TORCH_CHECK_VALUE(chunk > 0, "cross entropy: chunks of ", chunk, " tokens");
      const long N = hidden.size(0), d = hidden.size(1), V = w.size(0);
      const Tensor h = matrix(hidden), labels = labels_.contiguous();
      const Tensor inv = labels.ne(ignore).sum().clamp_min(1).to(F32).reciprocal().reshape(1);
      const Tensor loss = alloc({N}, F32, hidden.device());
      const Tensor dh = need_h ? alloc({N, d}, h.scalar_type(), h.device()) : Tensor();
      const Tensor dw = need_w ? alloc({V, d}, F32, h.device(), N == 0) : Tensor();   // the first chunk's product writes it whole
      const Tensor logits = alloc({std::min(chunk, N), V}, BF, h.device());
      for (long s0 = 0, n; s0 < N; s0 += n) {
        n = std::min(chunk, N - s0);
        const Tensor lg = logits.narrow(0, 0, n), hs = h.narrow(0, s0, n);
        gemm(hs, w, false, false, lg);
        launch(lib.nsa_cross_entropy, ptr(lg), static_cast<const long*>(ptr(labels.narrow(0, s0, n))), fp(loss.narrow(0, s0, n)), fp(inv), n,
               dim(V), lg.stride(0), ignore, static_cast<int>(need_h || need_w));
        if (need_h) gemm(lg, w, false, true, dh.narrow(0, s0, n));
        if (need_w) gemm(lg, hs, true, true, dw, F32, s0 > 0);
      }
      return {loss.sum().mul(inv.select(0, 0)), dh, dw};
    };
  });
}

OP(scale) {                                      // t, one-element tensor -> bf16 t * s, rounded once
  return entry(py, np, [](Args& a) {
    const Tensor &t = a.t(), &s = a.t();
    return [=]() -> Tensor {
      const Tensor out = alloc(t.sizes(), BF, t.device()), sf = s.reshape(1).to(F32);
      launch(lib.nsa_scale_bf16, ptr(t), ptr(out), fp(sf), t.numel(), static_cast<int>(t.scalar_type() == F32));
      return out;
    };
  });
}

// ------------------------------------------------------------------------------------- attention
struct Range {                                   // causal, window, scale, kp_stride, kp_off
  int causal, window;
  float scale;
  int kp_stride, kp_off;
  static Range of(Args& a) {
    const int causal = a.flag(), window = a.w();
    const float scale = a.f();
    const int kp_stride = a.w(), kp_off = a.w();
    return {causal, window, scale, kp_stride, kp_off};
  }
};
struct Tiles {                                   // union lists of selected blocks per query tile, and the selection they come from
  Tensor blocks, masks, counts, idx;
  int max_u = 0, nS = 0;
  bool any() const { return blocks.defined(); }
  const unsigned long long* mask() const { return static_cast<const unsigned long long*>(ptr(masks)); }
  static Tiles of(Args& a) {                     // None or (blocks, masks, counts, max_u, idx, nS)
    Tiles t;
    PyObject* o = a.next();
    if (o == Py_None) return t;
    TORCH_CHECK_TYPE(PyTuple_Check(o) && PyTuple_GET_SIZE(o) == 6, "_nsa_host: tiles have to be a tuple of six");
    PyObject* v[6];
    for (int i = 0; i < 6; ++i) v[i] = PyTuple_GET_ITEM(o, i);
    Args g{v, 6};
    t.blocks = g.t(); t.masks = g.t(); t.counts = g.t(); t.max_u = g.w(); t.idx = g.t(); t.nS = g.w();
    return t;
  }
};

std::pair<Tensor, Tensor> attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Range& r, const Tiles& t) {
  const Tensor o = alloc(q.sizes(), q.scalar_type(), q.device()), L = alloc(q.sizes().slice(0, 3), F32, q.device());
  launch(lib.nsa_attn_fwd, ptr(q), ptr(k), ptr(v), ptr(o), fp(L), dim(q.size(0)), dim(q.size(1)), dim(k.size(1)), dim(q.size(2)), dim(k.size(2)),
         dim(q.size(3)), r.scale, r.causal, r.window, r.kp_stride, r.kp_off, ip(t.blocks), t.mask(), ip(t.counts), t.max_u);
  return {o, L};
}

// (token lists, list starts, first CTA of a list, bound of the CTAs): see native.inverse_blocks
struct Inverse {
  Tensor tok, list_start, item_start;
  long bound = 0;
  static Inverse of(Args& a) {                   // None or (tok, list_start, item_start, nS, bound)
    Inverse v;
    PyObject* o = a.next();
    if (o == Py_None) return v;
    TORCH_CHECK_TYPE(PyTuple_Check(o) && PyTuple_GET_SIZE(o) == 5, "_nsa_host: inverse lists have to be a tuple of five");
    PyObject* p[5];
    for (int i = 0; i < 5; ++i) p[i] = PyTuple_GET_ITEM(o, i);
    Args g{p, 5};
    v.tok = g.t(); v.list_start = g.t(); v.item_start = g.t(); g.l(); v.bound = g.l();
    return v;
  }
};
Inverse inverse_lists(const Tensor& idx_, long nS, long R, long visits) {
  const Tensor idx = to(idx_, I32).contiguous();
  const long BH = idx.size(0) * idx.size(1), T = idx.size(2), n = idx.size(3), lists = BH * nS;
  const auto dev = idx.device();
  Inverse v;
  v.tok = alloc({BH * T * n}, I32, dev);
  v.list_start = alloc({lists + 1}, I32, dev);
  v.item_start = alloc({lists + 1}, I32, dev);
  const Tensor hist = alloc({BH * have(lib.nsa_inverse_chunks)(dim(BH), dim(T), dim(nS)) * nS}, I32, dev), count = alloc({lists}, I32, dev);
  launch(lib.nsa_inverse_blocks, ip(idx), ip(v.tok), ip(v.list_start), ip(v.item_start), ip(hist), ip(count), dim(BH), dim(T), dim(n), dim(nS),
         dim(R), dim(visits));
  v.bound = BH * T * n / (R * visits) + lists;
  return v;
}

// dQ from the query-tile kernel, dK and dV (fp32, added to; bf16, written) from the key-block kernel.  given: rowsum(dO * O) where the caller has it.
void attn_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& dO, const Tensor& L, const Tensor& dq,
                   const Tensor& dk, const Tensor& dv, const Range& r, const Tiles& t, const Inverse& inv, long visits, long walks,
                   const Tensor& given, bool add_dq) {
  const Tensor delta = given.defined() ? given : alloc(q.sizes().slice(0, 3), F32, q.device());
  const Tensor part = walks > 1 ? alloc({walks, 2, k.numel()}, F32, q.device()) : Tensor();
  launch(lib.nsa_attn_bwd_split, ptr(q), ptr(k), ptr(v), ptr(o), ptr(dO), fp(L), fp(delta), ptr(dq), ptr(dk), ptr(dv), dim(q.size(0)),
         dim(q.size(1)), dim(k.size(1)), dim(q.size(2)), dim(k.size(2)), dim(q.size(3)), r.scale, r.causal, r.window, r.kp_stride, r.kp_off,
         ip(t.blocks), t.mask(), ip(t.counts), t.max_u, ip(inv.tok), ip(inv.list_start), ip(inv.item_start), t.any() ? t.nS : 0,
         dim(inv.bound), dim(visits), fp(part), dim(walks), static_cast<int>(given.defined()), static_cast<int>(add_dq),
         static_cast<int>(dk.scalar_type() == BF));
}
// dK or dV: written whole by contiguous ranges of several walks, one, or 64 keys a CTA; else to be added to
Tensor key_grad(const Tensor& k, bool whole) { return alloc(k.sizes(), whole ? BF : F32, k.device(), !whole); }

OP(attn_fwd) {                                   // q, k, v, range, tiles -> o, L, q, k, v dense
  return entry(py, np, [](Args& a) {
    const Tensor &q_ = a.t(), &k_ = a.t(), &v_ = a.t();
    const Range r = Range::of(a);
    const Tiles t = Tiles::of(a);
    return [=]() -> List {
      want_dims(q_, 4);
      const Tensor q = dense(q_), k = dense(k_), v = dense(v_);
      auto [o, L] = attn_forward(q, k, v, r, t);
      return {o, L, q, k, v};
    };
  });
}

OP(attn_bwd) {                                   // q, k, v, o, dO, L, range, tiles, inverse lists or None, visits, walks, split -> dq, dk, dv
  return entry(py, np, [](Args& a) {
    const Tensor &q = a.t(), &k = a.t(), &v = a.t(), &o = a.t(), &dO_ = a.t(), &L = a.t();
    const Range r = Range::of(a);
    const Tiles t = Tiles::of(a);
    const Inverse inv = Inverse::of(a);
    const long visits = a.l(), walks = a.l();      // visits: query tiles per CTA of the dK / dV kernel, see native._range_visits
    const bool split = a.b();
    return [=]() -> List {
      const Tensor dO = dense(dO_), dq = alloc(q.sizes(), q.scalar_type(), q.device());
      const bool whole = split && !t.any() && walks != 0;
      const Tensor dk = key_grad(k, whole), dv = key_grad(v, whole);
      if (split) {
        attn_backward(q, k, v, o, dO, L, dq, dk, dv, r, t, inv, visits, walks, Tensor(), false);
      } else {
        const Tensor delta = alloc(q.sizes().slice(0, 3), F32, q.device());
        launch(lib.nsa_attn_bwd, ptr(q), ptr(k), ptr(v), ptr(o), ptr(dO), fp(L), fp(delta), ptr(dq), fp(dk), fp(dv), dim(q.size(0)), dim(q.size(1)),
               dim(k.size(1)), dim(q.size(2)), dim(k.size(2)), dim(q.size(3)), r.scale, r.causal, r.window, r.kp_stride, r.kp_off, ip(t.blocks),
               t.mask(), ip(t.counts), t.max_u);
      }
      return {dq, to(dk, k.scalar_type()), to(dv, v.scalar_type())};
    };
  });
}

// ------------------------------------------------------------------------------------- native sparse attention
Tiles union_lists(const Tensor& idx, long G, long nS) {
  TORCH_CHECK_VALUE(G > 0 && G <= 128, "union_blocks: groups of ", G, " query heads");
  const long B = idx.size(0), H = idx.size(1), T = idx.size(2), n = idx.size(3), R = 128 / G, tiles = (T + R - 1) / R;
  long most = std::min(R * n, nS);
  most += most & 1;
  Tiles t;
  t.max_u = dim(most);
  t.nS = dim(nS);
  t.idx = idx;
  t.blocks = alloc({B, H, tiles, most}, I32, idx.device());
  t.masks = alloc({B, H, tiles, most}, at::kLong, idx.device());
  t.counts = alloc({B, H, tiles}, I32, idx.device());
  launch(lib.nsa_union_blocks, ip(idx), ip(t.blocks), static_cast<unsigned long long*>(ptr(t.masks)), ip(t.counts), dim(B), dim(T), dim(H), dim(G),
         dim(n), dim(nS), t.max_u);
  return t;
}

OP(union_blocks) {                               // idx, G, nS -> blocks, masks, counts (their last dimension is max_u)
  return entry(py, np, [](Args& a) {
    const Tensor& idx = a.t();
    const long G = a.l(), nS = a.l();
    return [=]() -> List {
      want_dims(idx, 4);
      const Tiles t = union_lists(idx, G, nS);
      return {t.blocks, t.masks, t.counts};
    };
  });
}

OP(inverse_blocks) {                             // idx, nS, R, visits -> tok, list_start, item_start
  return entry(py, np, [](Args& a) {
    const Tensor& idx = a.t();
    const long nS = a.l(), R = a.l(), visits = a.l();
    return [=]() -> List {
      const Inverse v = inverse_lists(idx, nS, R, visits);
      return {v.tok, v.list_start, v.item_start};
    };
  });
}

OP(importance) {                                 // q, compressed keys, their L, nS, stride, block, scale -> importance
  return entry(py, np, [](Args& a) {
    const Tensor &q = a.t(), &kc = a.t(), &L = a.t();
    const int nS = a.w(), stride = a.w(), block = a.w();
    const float scale = a.f();
    return [=]() -> Tensor {
      want_dims(q, 4);
      const Tensor imp = alloc({q.size(0), kc.size(2), q.size(1), nS}, F32, q.device(), true);
      launch(lib.nsa_attn_importance, ptr(dense(q)), ptr(dense(kc)), fp(L), fp(imp), dim(q.size(0)), dim(q.size(1)), dim(kc.size(1)), dim(q.size(2)),
             dim(kc.size(2)), dim(q.size(3)), scale, stride, block - 1, nS);
      return imp;
    };
  });
}

OP(select) {                                     // importance, block, n -> idx
  return entry(py, np, [](Args& a) {
    const Tensor& imp_ = a.t();
    const int block = a.w(), n = a.w();
    return [=]() -> Tensor {
      const Tensor imp = dense(imp_);
      const long B = imp.size(0), H = imp.size(1), T = imp.size(2);
      const Tensor idx = alloc({B, H, T, n}, I32, imp.device());
      launch(lib.nsa_select_blocks, fp(imp), ip(idx), B * H * T, dim(T), dim(imp.size(3)), block, n);
      return idx;
    };
  });
}

OP(gates_fwd) {                                  // o1, o2, o3, logits -> o, bf16 logits
  return entry(py, np, [](Args& a) {
    const Tensor &o1 = a.t(), &o2 = a.t(), &o3 = a.t(), &gates = a.t();
    return [=]() -> List {
      const Tensor gl = to(gates, BF).contiguous(), o = alloc(o1.sizes(), o1.scalar_type(), o1.device());
      const long Hq = o1.size(-2), D = o1.size(-1), step = Hq * gl.element_size();
      const char* g = static_cast<const char*>(ptr(gl));
      launch(lib.nsa_gate_combine_fwd_ex, ptr(o1), ptr(o2), ptr(o3), g, g + step, g + 2 * step, gl.size(-1), dim(Hq), 1, ptr(o), o1.numel() / D, dim(D));
      return {o, gl};
    };
  });
}

OP(gates_bwd) {                                  // o1, o2, o3, logits, dO, row sums e1, e2, e3 or None -> dO1, dO2, dO3, d logits
  return entry(py, np, [](Args& a) {
    const Tensor &o1 = a.t(), &o2 = a.t(), &o3 = a.t(), &gl = a.t(), &dO_ = a.t();
    const Tensor e1 = a.opt(), e2 = a.opt(), e3 = a.opt();
    return [=]() -> List {
      const Tensor dO = dense(dO_);
      const long Hq = o1.size(-2), D = o1.size(-1), ldg = gl.size(-1), step = Hq * gl.element_size();
      List r;
      for (int i = 0; i < 3; ++i) r.push_back(alloc(o1.sizes(), o1.scalar_type(), o1.device()));
      r.push_back(alloc(gl.sizes(), gl.scalar_type(), gl.device(), ldg > 3 * Hq));
      const char* g = static_cast<const char*>(ptr(gl));
      char* dg = static_cast<char*>(ptr(r[3]));
      launch(lib.nsa_gate_combine_bwd_ex, ptr(o1), ptr(o2), ptr(o3), g, g + step, g + 2 * step, ldg, dim(Hq), 1, ptr(dO), ptr(r[0]), ptr(r[1]),
             ptr(r[2]), dg, dg + step, dg + 2 * step, fp(e1), fp(e2), fp(e3), o1.numel() / D, dim(D));
      return r;
    };
  });
}

OP(pool_fwd) {                                   // x, block, stride -> y
  return entry(py, np, [](Args& a) {
    const Tensor& x = a.t();
    const int block = a.w(), stride = a.w();
    return [=]() -> Tensor {
      want_dims(x, 4);
      TORCH_CHECK_VALUE(block > 0 && stride > 0, "nsa_compress: blocks of ", block, " tokens every ", stride);
      const long B = x.size(0), T = x.size(1), H = x.size(2), D = x.size(3);
      const bool ok = x.stride(3) == 1 && x.stride(2) == D && x.stride(1) % 8 == 0 && x.stride(0) == T * x.stride(1) && aligned(x);
      const Tensor xv = ok ? x : x.contiguous(), y = alloc({B, (T - block) / stride + 1, H, D}, x.scalar_type(), x.device());
      launch(lib.nsa_pool_fwd, ptr(xv), ptr(y), dim(B), dim(T), dim(H * D), xv.stride(1), block, stride);
      return y;
    };
  });
}

OP(pool_bwd) {                                   // dy, T, block, stride -> dx
  return entry(py, np, [](Args& a) {
    const Tensor& dy_ = a.t();
    const long T = a.l();
    const int block = a.w(), stride = a.w();
    return [=]() -> Tensor {
      const Tensor dy = dense(dy_);
      const long B = dy.size(0), H = dy.size(2), D = dy.size(3);
      const Tensor dx = alloc({B, T, H, D}, dy.scalar_type(), dy.device());
      launch(lib.nsa_pool_bwd, ptr(dy), ptr(dx), dim(B), dim(T), dim(H * D), block, stride);
      return dx;
    };
  });
}

OP(nsa_bwd) {                                    // q, k, v, kc, vc, o1, d1, L1, e1, ... of three branches, tiles, inverse lists, visits of ranges
  return entry(py, np, [](Args& a) {             // and lists, stride, block, window, scale -> dq, dk, dv, dkc, dvc
    const Tensor &q = a.t(), &k = a.t(), &v = a.t(), &kc = a.t(), &vc = a.t();
    Tensor o[3], d[3], L[3], e[3];
    for (int i = 0; i < 3; ++i) { o[i] = a.t(); d[i] = a.t(); L[i] = a.t(); e[i] = a.t(); }
    const Tiles t = Tiles::of(a);
    const Inverse lists = Inverse::of(a);
    const long visits = a.l(), per_list = a.l();
    const int stride = a.w(), block = a.w(), window = a.w();
    const float scale = a.f();
    return [=]() -> List {
      const auto dev = q.device();
      const int B = dim(q.size(0)), T = dim(q.size(1)), Hq = dim(q.size(2)), Hkv = dim(k.size(2));
      const Tensor dq = alloc(q.sizes(), q.scalar_type(), dev);
      Tensor dk = alloc(k.sizes(), F32, dev, true), dv = alloc(v.sizes(), F32, dev, true);
      auto walks = [&](const Tensor& keys, int win, int kp) { return have(lib.nsa_attn_bwd_walks)(B, T, dim(keys.size(1)), Hq, Hkv, 1, win, kp); };
      const int pooled = walks(kc, 0, stride);
      const Tensor dkc = key_grad(kc, pooled != 0), dvc = key_grad(vc, pooled != 0);
      attn_backward(q, kc, vc, o[0], d[0], L[0], dq, dkc, dvc, {1, 0, scale, stride, block - 1}, Tiles(), Inverse(), visits, pooled, e[0], false);
      attn_backward(q, k, v, o[1], d[1], L[1], dq, dk, dv, {1, 0, scale, 1, 0}, t, lists, per_list, 0, e[1], true);
      // The window branch shares dk / dv while a key block's gradients get one addition from it: one more to what is there gives
      // the same bits on every run, two in either order would not.
      const int own = walks(k, window, 1);
      Tensor dk3 = dk, dv3 = dv;
      if (own == 0) { dk3 = alloc(k.sizes(), F32, dev, true); dv3 = alloc(v.sizes(), F32, dev, true); }
      attn_backward(q, k, v, o[2], d[2], L[2], dq, dk3, dv3, {1, window, scale, 1, 0}, Tiles(), Inverse(), visits, own, e[2], true);
      if (own == 0) { dk = dk + dk3; dv = dv + dv3; }
      return {dq, to(dk, k.scalar_type()), to(dv, v.scalar_type()), to(dkc, kc.scalar_type()), to(dvc, vc.scalar_type())};
    };
  });
}

// ------------------------------------------------------------------------------------- gated delta rule
OP(gdn_fwd) {                                    // q, k, v, g, beta, scale, train -> o, w, qk, gc, X, v_new, S (the last three in training)
  return entry(py, np, [](Args& a) {
    const Tensor &q = a.t(), &k = a.t(), &v = a.t(), &g = a.t(), &beta = a.t();
    const float scale = a.f();
    const bool train = a.b();
    return [=]() -> List {
      const long B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(-1), BH = B * H, nc = (T + 63) / 64;
      const auto dev = q.device();
      const Tensor w = alloc({BH, nc, 64, K}, BF, dev), u = alloc({BH, nc, 64, V}, BF, dev);
      const Tensor qk = alloc({BH, nc, 64, 64}, BF, dev), gc = alloc({BH, nc, 64}, F32, dev);
      const Tensor X = train ? alloc({BH, nc, 64, 64}, F32, dev) : Tensor(), o = alloc({B, T, H, V}, BF, dev);
      const Tensor v_new = train ? alloc({BH, nc, 64, V}, BF, dev) : Tensor(), S = train ? alloc({BH, nc, K, V}, BF, dev) : Tensor();
      launch(lib.nsa_gdn_prep, ptr(q), ptr(k), ptr(v), fp(g), fp(beta), ptr(w), ptr(u), ptr(qk), fp(X), fp(gc), dim(B), dim(T), dim(H), dim(K),
             dim(V), scale);
      launch(lib.nsa_gdn_seq_fwd, ptr(q), ptr(k), ptr(w), ptr(u), ptr(qk), fp(gc), ptr(o), ptr(v_new), ptr(S), dim(B), dim(T), dim(H), dim(K),
             dim(V), scale);
      return {o, w, qk, gc, X, v_new, S};
    };
  });
}

OP(gdn_bwd) {                                    // q, k, v, beta, w, qk, gc, X, v_new, S, dO, scale -> dq, dk, dv, dg, dbeta
  return entry(py, np, [](Args& a) {
    const Tensor &q = a.t(), &k = a.t(), &v = a.t(), &beta = a.t(), &w = a.t(), &qk = a.t(), &gc = a.t(), &X = a.t(), &v_new = a.t(), &S = a.t(),
                 &dO_ = a.t();
    const float scale = a.f();
    return [=]() -> List {
      const long B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(-1), BH = B * H, nc = gc.size(1);
      const Tensor dO = to(dO_, BF).contiguous();
      auto like = [](const Tensor& t) { return alloc(t.sizes(), t.scalar_type(), t.device()); };
      const Tensor du = like(v_new), dS = like(S), dgamma = alloc({V / 64, BH, nc}, F32, q.device());
      const Tensor dq = like(q), dk = like(k), dv = like(v), dg = like(beta), dbeta = like(beta);
      launch(lib.nsa_gdn_seq_bwd, ptr(q), ptr(k), ptr(w), ptr(qk), ptr(S), ptr(dO), fp(gc), ptr(du), ptr(dS), fp(dgamma), dim(B), dim(T), dim(H),
             dim(K), dim(V), scale);
      launch(lib.nsa_gdn_post, ptr(q), ptr(k), ptr(v), ptr(dO), fp(beta), fp(gc), fp(X), ptr(v_new), ptr(du), ptr(S), ptr(dS), fp(dgamma), ptr(dq),
             ptr(dk), ptr(dv), fp(dg), fp(dbeta), dim(B), dim(T), dim(H), dim(K), dim(V), scale);
      return {dq, dk, dv, dg, dbeta};
    };
  });
}

// ------------------------------------------------------------------------------------- Mamba-2 scan
// (B, T, ..., inner-contiguous) view usable by a copy of rows = tokens; copied when it is not row-strided.
Tensor token_rows(const Tensor& t) {
  const bool ok = t.stride(-1) == 1 && t.stride(0) == t.size(1) * t.stride(1) && t.stride(1) % 8 == 0 && aligned(t) &&
                  t.select(0, 0).select(0, 0).is_contiguous();
  return ok ? t : t.contiguous();
}
// Elements from a token to the next, also of a saved tensor as it comes back.  Not the stride of a dense tensor: a single token may have any.
long token_pitch(const Tensor& t) { return t.is_contiguous() ? c10::multiply_integers(t.sizes().slice(2)) : t.stride(1); }

// bf16 states entering the chunks (back: gradients of those leaving them), and the chunks' decays where the two-kernel form needs them
std::pair<Tensor, Tensor> ssd_states(bool back, const Tensor& rows, long ld_rows, const Tensor& v, long ld_v, const Tensor& dt, const Tensor& A,
                                     Tensor gamma) {
  const long B = v.size(0), T = v.size(1), H = v.size(2), P = v.size(3), N = rows.size(-1), nc = (T + 127) / 128;
  const auto dev = v.device();
  const Tensor out = alloc({B, nc, H, N, P}, BF, dev);
  const int b = dim(B), t = dim(T), h = dim(H), n = dim(N), p = dim(P);
  if (have(lib.nsa_ssd_states_form)(b, t, h)) {
    launch(lib.nsa_ssd_states, static_cast<int>(back), ptr(rows), ld_rows, ptr(v), ld_v, fp(dt), fp(A), ptr(out), b, t, h, n, p);
    return {out, alloc({0}, F32, dev)};
  }
  if (!back) gamma = alloc({B, nc, H}, F32, dev);
  const Tensor local = alloc({B, nc, H, N, P}, F32, dev);
  launch(lib.nsa_ssd_chunk_state, static_cast<int>(back), ptr(rows), ld_rows, ptr(v), ld_v, fp(dt), fp(A), fp(local), back ? nullptr : fp(gamma),
         b, t, h, n, p);
  float* none = nullptr;
  if (back) launch(lib.nsa_ssd_state_bwd, fp(local), fp(gamma), none, ptr(out), b, dim(nc), h, N * P);
  else launch(lib.nsa_ssd_state_fwd, fp(local), fp(gamma), none, ptr(out), none, b, dim(nc), h, N * P);
  return {out, gamma};
}

OP(ssd_fwd) {                                    // x, dt, A, B, C, D or None -> y, x, dt, A, B, C, D as read, decays, states
  return entry(py, np, [](Args& a) {
    const Tensor &x_ = a.t(), &dt_ = a.t(), &A_ = a.t(), &B_ = a.t(), &C_ = a.t();
    const Tensor D_ = a.opt();
    return [=]() -> List {
      want_dims(x_, 4);
      const Tensor x = token_rows(x_), Bm = token_rows(B_), Cm = token_rows(C_);
      const Tensor dt = to(dt_, F32).contiguous(), A = to(A_, F32).contiguous(), D = D_.defined() ? to(D_, F32).contiguous() : D_;
      const long B = x.size(0), T = x.size(1), H = x.size(2), P = x.size(3), N = Bm.size(-1);
      const long ldx = token_pitch(x), ldb = token_pitch(Bm), ldc = token_pitch(Cm);
      auto [states, gamma] = ssd_states(false, Bm, ldb, x, ldx, dt, A, Tensor());
      const Tensor y = alloc({B, T, H, P}, BF, x.device());
      launch(lib.nsa_ssd_chunk_out, ptr(Cm), ldc, ptr(Bm), ldb, ptr(x), ldx, ptr(states), fp(dt), fp(A), fp(D), ptr(y),
             dim(B), dim(T), dim(H), dim(N), dim(P));
      return {y, x, dt, A, Bm, Cm, D.defined() ? D : alloc({0}, F32, x.device()), gamma, states};
    };
  });
}

OP(ssd_bwd) {                                    // x, dt, A, B, C, D, decays, states, dy, has D -> dx, ddt, dA, dB, dC, dD
  return entry(py, np, [](Args& a) {
    const Tensor &x = a.t(), &dt = a.t(), &A = a.t(), &Bm = a.t(), &Cm = a.t(), &D_ = a.t(), &gamma = a.t(), &states = a.t(), &dy_ = a.t();
    const bool has_D = a.b();
    return [=]() -> List {
      const long ldx = token_pitch(x), ldb = token_pitch(Bm), ldc = token_pitch(Cm);
      const Tensor D = has_D ? D_ : Tensor(), dy = dense(dy_);
      const long B = x.size(0), T = x.size(1), H = x.size(2), P = x.size(3), N = Bm.size(-1), nc = states.size(1);
      const int b = dim(B), t = dim(T), h = dim(H);
      const auto dev = x.device();
      const Tensor dHn = ssd_states(true, Cm, ldc, dy, H * P, dt, A, gamma).first;
      const Tensor dx = alloc({B, T, H, P}, BF, dev);
      // dB / dC: fp32 sums over the heads that one CTA has of a chunk, added up afterwards
      const long slots = have(lib.nsa_ssd_grad_slots)(b, t, h);
      const Tensor dB_part = alloc({B, T, slots, N}, F32, dev), dC_part = alloc({B, T, slots, N}, F32, dev);
      const Tensor q = alloc({B, T, H}, F32, dev), k = alloc({B, T, H}, F32, dev), rdx = has_D ? alloc({B, T, H}, F32, dev) : Tensor();
      launch(lib.nsa_ssd_chunk_grad, ptr(Cm), ldc, ptr(Bm), ldb, ptr(x), ldx, ptr(dy), ptr(states), ptr(dHn), fp(dt), fp(A), fp(D), ptr(dx),
             fp(dB_part), fp(dC_part), fp(q), fp(k), fp(rdx), b, t, h, dim(N), dim(P));
      // d(cum_t) = dy_t.(y_t - D x_t) - x_t.dx_t ;  a_k = dt_k A enters every cum_t with t >= k
      const Tensor dB = alloc({B, T, 1, N}, BF, dev), dC = alloc({B, T, 1, N}, BF, dev), ddt = alloc({B, T, H}, F32, dev);
      const Tensor dA = alloc({H}, F32, dev), dD = has_D ? alloc({H}, F32, dev) : Tensor(), scratch = alloc({3 * B * nc * H}, F32, dev);
      launch(lib.nsa_ssd_finish, fp(dB_part), fp(dC_part), fp(q), fp(k), fp(rdx), fp(dt), fp(A), fp(scratch), ptr(dB), ptr(dC), fp(ddt), fp(dA), fp(dD),
             b, t, h);
      return {dx, ddt, dA, dB, dC, dD};
    };
  });
}

// Rows of one pitch, the last dimension dense: used in place
Tensor pitched(const Tensor& t) {
  bool ok = t.stride(-1) == 1;
  for (long k = t.dim() - 2; k > 0; --k) ok = ok && t.stride(k - 1) == t.size(k) * t.stride(k);
  return ok ? t : t.contiguous();
}
OP(gates) {                                      // a, b or None, bias, A_log -> g and beta, or dt and A (fp32)
  return entry(py, np, [](Args& a) {
    const Tensor& x = a.t();
    const Tensor b = a.opt();
    const Tensor &bias = a.t(), &A_log = a.t();
    return [=]() -> List {
      const Tensor xp = pitched(x), bp = b.defined() ? pitched(b) : b, bc = dense(bias), Ac = dense(A_log);
      const long H = x.size(-1);
      const Tensor out0 = alloc(x.sizes(), F32, x.device()), out1 = b.defined() ? alloc(x.sizes(), F32, x.device()) : alloc({H}, F32, x.device());
      launch(lib.nsa_gates, ptr(xp), xp.stride(-2), ptr(bp), b.defined() ? bp.stride(-2) : 0l, ptr(bc), static_cast<int>(bc.scalar_type() == F32),
             ptr(Ac), static_cast<int>(Ac.scalar_type() == F32), fp(out0), fp(out1), rows_of(xp), dim(H));
      return {out0, out1};
    };
  });
}

// ------------------------------------------------------------------------------------- optimizer lists
void need(const char* what, PyObject* o, long n) {
  if (o == Py_None) return;
  const long have = THPVariable_Unpack(o).numel();
  TORCH_CHECK_VALUE(have == n, "optimizer state '", what, "' has ", have, " elements, the kernel needs ", n);
}

// A list or tuple (another sequence becomes a list), held while its items are read
struct Sequence {
  THPObjectPtr held;
  explicit Sequence(PyObject* o) {
    TORCH_CHECK_TYPE(PySequence_Check(o), "_nsa_host: the tensors to update have to be a sequence of sequences");
    held = PySequence_Fast(o, "_nsa_host: the tensors to update have to be a sequence of sequences");
    if (!held) throw python_error();
  }
  long size() const { return PySequence_Fast_GET_SIZE(held.get()); }
  PyObject* operator[](long i) const { return PySequence_Fast_GET_ITEM(held.get(), i); }
};

// Seven 64-bit words per tensor, (p, g, m, v, a, b, n).  Every state tensor is checked against n; with a block the last two are the
// scales of the quantised moments, else an fp32 master copy (or None) and nothing.
struct Updates {
  std::vector<long long> words;
  int count = 0, p_fp32 = 0, g_fp32 = 0;         // the types are those of the first
  Updates(PyObject* list, long block) {
    const Sequence items(list);
    count = dim(items.size());
    TORCH_CHECK_INDEX(count > 0, "_nsa_host: no tensors to update");
    words.reserve(7 * count);
    for (long i = 0; i < count; ++i) {
      const Sequence it(items[i]);
      TORCH_CHECK_VALUE(it.size() == 6, "_nsa_host: six tensors or None for each parameter");
      PyObject* o[6];
      for (int k = 0; k < 6; ++k) {
        o[k] = it[k];
        TORCH_CHECK_TYPE(THPVariable_Check(o[k]) || (k > 3 && o[k] == Py_None), "_nsa_host: six tensors or None for each parameter");
      }
      const long n = THPVariable_Unpack(o[0]).numel(), na = block ? n / block : n;
      TORCH_CHECK_VALUE(!block || n % block == 0, "8-bit AdamW needs a multiple of ", block, " elements, got ", n);
      need("grad", o[1], n);
      need("exp_avg", o[2], n);
      need("exp_avg_sq", o[3], n);
      need(block ? "exp_avg_absmax" : "master", o[4], na);
      need("exp_avg_sq_absmax", o[5], na);
      for (PyObject* x : o) words.push_back(x == Py_None ? 0 : reinterpret_cast<long long>(THPVariable_Unpack(x).data_ptr()));
      words.push_back(n);
      if (i == 0) {
        p_fp32 = THPVariable_Unpack(o[0]).scalar_type() == F32;
        g_fp32 = THPVariable_Unpack(o[1]).scalar_type() == F32;
      }
    }
  }
};

OP(adamw) {                                      // items, gradient scale or None, step, lr, b1, b2, eps, wd
  HANDLE_TH_ERRORS
  Args a{py, np};
  const Updates u(a.next(), 0);
  const Tensor s = a.opt();
  const int step = a.w();
  const float lr = a.f(), b1 = a.f(), b2 = a.f(), eps = a.f(), wd = a.f();
  {
    Call call;
    const Tensor sf = s.defined() ? s.reshape(1).to(F32) : s;
    launch(lib.nsa_adamw_multi, u.words.data(), u.count, fp(sf), u.p_fp32, u.g_fp32, step, lr, b1, b2, eps, wd);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

OP(adamw8bit) {                                  // items, code books, gradient scale or None, step, lr, b1, b2, eps, wd, block
  HANDLE_TH_ERRORS
  Args a{py, np};
  PyObject* items = a.next();
  const Tensor &cs = a.t(), &cu = a.t();
  const Tensor s = a.opt();
  const int step = a.w();
  const float lr = a.f(), b1 = a.f(), b2 = a.f(), eps = a.f(), wd = a.f();
  const Updates u(items, a.l());
  {
    Call call;
    const Tensor sf = s.defined() ? s.reshape(1).to(F32) : s;
    launch(lib.nsa_adamw8bit_multi, u.words.data(), u.count, fp(cs), fp(cu), fp(sf), u.p_fp32, u.g_fp32, step, lr, b1, b2, eps, wd);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------- the module
OP(bind) {                                       // path of the library, the dictionary of ops/native.py, most parts of a split reduction
  HANDLE_TH_ERRORS
  Args a{py, np};
  const char* path = PyUnicode_AsUTF8(a.next());
  if (!path) throw python_error();
  PyObject* native = a.next();
  TORCH_CHECK_TYPE(PyDict_Check(native), "_nsa_host: bind wants the module's dictionary");
  g_splitk_max = a.l();
  void* h = dlopen(path, RTLD_NOW);
  TORCH_CHECK(h != nullptr, "_nsa_host: ", dlerror());
#define X(f) lib.f = reinterpret_cast<decltype(lib.f)>(dlsym(h, #f));
  NSA_ENTRIES(X)
#undef X
  Py_INCREF(native);
  g_native = native;
  g_canary = PyUnicode_InternFromString("_CANARY");
  g_guarded = PyUnicode_InternFromString("_guarded");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

OP(gemm_single) {                                // whether plain GEMMs run on the single-CTA kernel
  HANDLE_TH_ERRORS
  Args a{py, np};
  g_single_gemm = a.b();
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

OP(split_k_choice) {                             // M, N, K, clusters
  HANDLE_TH_ERRORS
  Args a{py, np};
  const long M = a.l(), N = a.l(), K = a.l(), clusters = a.l();
  return PyLong_FromLong(split_k(M, N, K, clusters));
  END_HANDLE_TH_ERRORS
}

#define M(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    M(bind), M(gemm_single), M(split_k_choice), M(rms_fwd), M(add_rms_fwd), M(rms_bwd), M(gated_rms_fwd), M(gated_rms_bwd), M(l2_fwd), M(l2_bwd),
    M(swiglu_fwd), M(swiglu_bwd), M(rope), M(conv_fwd), M(conv_bwd), M(embedding_fwd), M(matmul), M(linear_fwd), M(multi_linear_fwd),
    M(multi_linear_bwd), M(cross_entropy_fwd), M(scale), M(attn_fwd), M(attn_bwd), M(union_blocks), M(inverse_blocks), M(importance), M(select),
    M(gates_fwd), M(gates_bwd), M(pool_fwd), M(pool_bwd), M(nsa_bwd), M(gdn_fwd), M(gdn_bwd), M(ssd_fwd), M(ssd_bwd), M(gates), M(adamw), M(adamw8bit),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_nsa_host", "Host side of the native ops.", -1, methods};
}  // namespace

PyMODINIT_FUNC PyInit__nsa_host() { return PyModule_Create(&module); }
