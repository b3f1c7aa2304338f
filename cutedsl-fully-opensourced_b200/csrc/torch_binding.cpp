// Host path of the hot operators: torch tensors in, one call of the C-ABI (include/b200fp4.h), torch tensors out.
//
// A decode step's norm or GEMM runs 3 to 15 us on the GPU.  The same checks, allocations and stream look-ups written
// in Python around a ctypes call took 20 to 30 us per call (60 to 80 us for the MoE operator), so the host, not the
// GPU, set the pace of every small call.  Here a call costs what its allocations and its launches cost.
//
// Every function takes positional arguments only: the Python wrappers of norm.py, gemm.py and moe.py own the
// signatures and the defaults.  Violated preconditions raise ValueError / NotImplementedError before anything is
// launched; a failing C call raises what its status code stands for.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdarg>
#include <cstdio>
#include <exception>
#include <optional>
#include <sstream>

#include "../../include/b200fp4.h"

namespace {

PyObject* g_error_class = nullptr;       // B200Fp4Error

// A Python exception of the given type; thrown through the C++ frames and set by the entry point's catch.
struct Raise {
  PyObject* type;
  std::string text;
};

[[noreturn]] void value_error(const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  throw Raise{PyExc_ValueError, buf};
}
[[noreturn]] void not_implemented(const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  throw Raise{PyExc_NotImplementedError, buf};
}

void check(int rc) {
  if (rc == B200FP4_OK) return;
  const char* msg = b200fp4_last_error();
  if (rc == B200FP4_INVALID_ARGUMENT) throw Raise{PyExc_ValueError, msg};
  if (rc == B200FP4_UNSUPPORTED) throw Raise{PyExc_NotImplementedError, msg};
  char buf[640];
  snprintf(buf, sizeof buf, "libb200fp4 status %d: %s", rc, msg);
  throw Raise{g_error_class != nullptr ? g_error_class : PyExc_RuntimeError, buf};
}

const at::Tensor& tensor(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) {
    std::ostringstream s;
    s << name << " must be a tensor (got " << Py_TYPE(o)->tp_name << ")";
    throw Raise{PyExc_TypeError, s.str()};
  }
  return THPVariable_Unpack(o);
}
// null: None was passed
const at::Tensor* maybe(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor(o, name); }

// Undefined: not a dtype
at::ScalarType dtype(PyObject* o) {
  return THPDtype_Check(o) ? reinterpret_cast<THPDtype*>(o)->scalar_type : at::ScalarType::Undefined;
}
// the type of a result that the call makes: None is torch's default type; nothing is asked of it where the caller gives
// the result's tensor
at::ScalarType result_dtype(PyObject* o, PyObject* out) {
  if (o == Py_None) return c10::get_default_dtype_as_scalartype();
  if (out == Py_None && !THPDtype_Check(o)) throw Raise{PyExc_TypeError, "out_dtype must be a torch.dtype"};
  return dtype(o);
}
int64_t integer(PyObject* o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw std::exception();
  return v;
}
// o == v in Python's sense (16.0 is 16)
bool equals(PyObject* o, long v) {
  if (PyLong_CheckExact(o)) return integer(o) == v;
  PyObject* want = PyLong_FromLong(v);
  const int eq = want == nullptr ? -1 : PyObject_RichCompareBool(o, want, Py_EQ);
  Py_XDECREF(want);
  if (eq < 0) throw std::exception();
  return eq != 0;
}
// int(o)
int64_t to_integer(PyObject* o) {
  if (PyLong_CheckExact(o)) return integer(o);
  PyObject* i = PyNumber_Long(o);
  if (i == nullptr) throw std::exception();
  const int64_t v = PyLong_AsLongLong(i);
  Py_DECREF(i);
  if (v == -1 && PyErr_Occurred()) throw std::exception();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw std::exception();
  return v != 0;
}

std::string shape_of(const at::Tensor& t) {
  std::ostringstream s;
  s << "(";
  for (int64_t i = 0; i < t.dim(); ++i) s << (i ? ", " : "") << t.size(i);
  s << ")";
  return s.str();
}
int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
int64_t tiled_bytes(int64_t rows, int64_t blocks) { return ceil_div(rows, 128) * ceil_div(blocks, 4) * 512; }

at::Tensor empty(at::IntArrayRef size, at::ScalarType type, at::Device dev) {
  return at::Tensor(at::detail::empty_cuda(size, type, dev, std::nullopt));
}
// the tensor itself when its elements are bytes, else a byte view of it
at::Tensor bytes(const at::Tensor& t) { return t.element_size() == 1 ? t : t.view(at::kByte); }
void* data(const at::Tensor& t) { return t.data_ptr(); }
void* data(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }

// a kernel of `dev` cannot read the address of a CPU tensor or of one on another GPU
void on_device(const at::Tensor* t, at::Device dev, const char* name) {
  if (t != nullptr && (!t->is_cuda() || t->device() != dev)) {
    std::ostringstream s;
    s << name << " must be a CUDA tensor on " << dev << " (got " << t->device() << ")";
    value_error("%s", s.str().c_str());
  }
}

// the GIL is given up for as long as this lives, and is held again when an exception passes through
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// `fn(stream)` with the tensor's device current and without the GIL (a launch blocks while the GPU's queue is full).
// `fn` takes the tensors' addresses, which throws for a tensor without storage (a vmap wrapper, a fake tensor).
template <typename Fn>
void launch(at::Device dev, Fn&& fn) {
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != dev.index()) guard.set_device(dev);
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int rc = [&] {
    WithoutGil released;
    return fn(stream);
  }();
  check(rc);
}

PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
// an argument handed back as it came, or a new tensor
PyObject* give(PyObject* arg, const at::Tensor& made) {
  if (arg != Py_None) {
    Py_INCREF(arg);
    return arg;
  }
  return wrap(made);
}

template <typename Fn>
PyObject* guarded(Py_ssize_t got, Py_ssize_t want, Fn&& fn) {
  try {
    if (got != want) throw Raise{PyExc_TypeError, "wrong number of arguments"};
    return fn();
  } catch (const Raise& r) {
    PyErr_SetString(r.type, r.text.c_str());
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// ---------------------------------------------------------------------------------------------------------------------
// norm(input, residual, weight, y_fp4, block_scale, block_scale_unswizzled, global_scale, eps, block_size, scale_format,
//      swizzled, both)
// ---------------------------------------------------------------------------------------------------------------------
PyObject* norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 12, [&]() -> PyObject* {
    const at::Tensor& x = tensor(a[0], "input");
    const bool add = a[1] != Py_None;
    const at::Tensor& w = tensor(a[2], "weight");
    if (!x.is_cuda()) value_error("input must be a CUDA tensor (there is no CPU implementation)");
    const at::ScalarType type = x.scalar_type();
    if (type != at::kHalf && type != at::kBFloat16) {
      std::ostringstream s;
      s << "input dtype " << type << " is not float16/bfloat16";
      value_error("%s", s.str().c_str());
    }
    if (w.scalar_type() != type || w.device() != x.device()) value_error("weight must have the dtype and device of input");
    if (!equals(a[8], 16)) not_implemented("only NVFP4 (block_size=16, e4m3 scale factors) is implemented");
    if (a[9] != Py_None && !(PyUnicode_Check(a[9]) && PyUnicode_CompareWithASCIIString(a[9], "e4m3") == 0))
      not_implemented("scale_format: only e4m3 is implemented");
    if (x.dim() != 2 && x.dim() != 3) value_error("input must be [B, H] or [B, S, H]");
    const int64_t hidden = x.size(-1);
    if (w.dim() != 1 || w.size(0) != hidden) value_error("weight must be [H]");
    if (hidden % 16 != 0 || hidden < 64) value_error("hidden size must be a multiple of 16 and at least 64");
    if (x.stride(-1) != 1) value_error("the last dimension of input must be contiguous");
    const at::Tensor* res = nullptr;
    if (add) {
      res = &tensor(a[1], "residual");
      if (res->sizes() != x.sizes() || res->scalar_type() != type || res->device() != x.device())
        value_error("residual must match input in shape, dtype and device");
      if (res->stride(-1) != 1) value_error("the last dimension of residual must be contiguous");
      if (res->dim() == 3 && !res->is_contiguous()) value_error("a 3-D residual must be contiguous: it is updated in place");
    }
    at::Tensor x3;                                  // a 3-D input as rows: without copying when its strides allow
    if (x.dim() == 3) x3 = x.reshape({-1, hidden});
    const at::Tensor& x2 = x.dim() == 3 ? x3 : x;
    const int64_t rows = x2.size(0), kb = hidden / 16;
    const int64_t x_stride = rows > 1 ? x2.stride(0) : hidden;
    const int64_t r_stride = add ? (rows > 1 && res->dim() == 2 ? res->stride(0) : hidden) : 0;
    const bool both = truth(a[11]), tiled = both || truth(a[10]);
    const at::Device dev = x.device();

    const bool flat = x.dim() == 2;
    at::Tensor y, sf, sfu;
    const at::Tensor* yp = maybe(a[3], "y_fp4");
    if (yp == nullptr) {
      y = flat ? empty({rows, hidden / 2}, at::kByte, dev) : empty({x.size(0), x.size(1), hidden / 2}, at::kByte, dev);
      yp = &y;
    } else if (yp->numel() * yp->element_size() != rows * hidden / 2 || !yp->is_contiguous()) {
      value_error("y_fp4 must be contiguous with hidden/2 bytes per row");
    }
    const at::Tensor* sfp = maybe(a[4], "block_scale");
    if (sfp == nullptr) {
      sf = tiled ? empty({ceil_div(rows, 128) * 128, ceil_div(kb, 4) * 4}, at::kByte, dev)
                 : (flat ? empty({rows, kb}, at::kByte, dev) : empty({x.size(0), x.size(1), kb}, at::kByte, dev));
      sfp = &sf;
    } else {
      const int64_t need = tiled ? tiled_bytes(rows, kb) : rows * kb;
      if (sfp->element_size() != 1 || sfp->numel() < need || !sfp->is_contiguous())
        value_error("block_scale must be a contiguous 1-byte tensor with at least %lld elements", static_cast<long long>(need));
    }
    const at::Tensor* sfup = nullptr;
    if (both) {
      sfup = maybe(a[5], "block_scale_unswizzled");
      if (sfup == nullptr) {
        sfu = flat ? empty({rows, kb}, at::kByte, dev) : empty({x.size(0), x.size(1), kb}, at::kByte, dev);
        sfup = &sfu;
      } else if (sfup->element_size() != 1 || sfup->numel() < rows * kb || !sfup->is_contiguous()) {
        value_error("block_scale_unswizzled must be a contiguous 1-byte tensor with at least %lld elements",
                    static_cast<long long>(rows * kb));
      }
    }
    for (const at::Tensor* t : {yp, sfp, sfup})
      if (t != nullptr && t->device() != dev) value_error("outputs must be on the input's device");
    const at::Tensor& gs = tensor(a[6], "global_scale");
    if (gs.scalar_type() != at::kFloat || gs.device() != dev)
      value_error("global_scale must be a float32 tensor on the input's device");
    const double eps = PyFloat_AsDouble(a[7]);
    if (eps == -1.0 && PyErr_Occurred()) throw std::exception();

    if (rows > 0) {
      at::Tensor wc;
      if (!w.is_contiguous()) wc = w.contiguous();
      const void* wp = data(w.is_contiguous() ? w : wc);
      const int dt = type == at::kHalf ? 0 : 1;
      launch(dev, [&](void* stream) {
        if (!add)
          return b200fp4_rmsnorm_fp4quant(data(x2), wp, data(yp), data(sfp), nullptr, static_cast<const float*>(data(gs)),
                                          static_cast<float>(eps), rows, static_cast<int>(hidden), x_stride, dt,
                                          tiled ? 1 : 0, stream);
        return b200fp4_add_rmsnorm_fp4quant(data(x2), data(res), wp, data(yp), data(sfp), data(sfup),
                                            static_cast<const float*>(data(gs)), static_cast<float>(eps), rows,
                                            static_cast<int>(hidden), x_stride, r_stride, dt, both ? 2 : (tiled ? 1 : 0),
                                            stream);
      });
    }
    PyObject* out = PyTuple_New(both ? 3 : 2);
    if (out == nullptr) return nullptr;
    PyTuple_SET_ITEM(out, 0, give(a[3], y));
    PyTuple_SET_ITEM(out, 1, give(a[4], sf));
    if (both) PyTuple_SET_ITEM(out, 2, give(a[5], sfu));
    return out;
  });
}

// ---------------------------------------------------------------------------------------------------------------------
// GEMM operands
// ---------------------------------------------------------------------------------------------------------------------
struct Matrix {
  int64_t l, rows, cols;
};
// [R, C], [L, R, C], or an (R, C, L) view of memory with L slowest; contiguous, never copied
Matrix matrix(const at::Tensor& t, const char* what) {
  if (t.dim() == 2 && t.is_contiguous()) return {1, t.size(0), t.size(1)};
  if (t.dim() == 3) {
    if (t.is_contiguous()) return {t.size(0), t.size(1), t.size(2)};
    if (t.permute({2, 0, 1}).is_contiguous()) return {t.size(2), t.size(0), t.size(1)};
  }
  value_error("%s must be contiguous [rows, cols], [L, rows, cols] or an (rows, cols, L) view of it", what);
}

int c_code(at::ScalarType t) {
  return t == at::kHalf ? 0 : (t == at::kBFloat16 ? 1 : (t == at::kFloat ? 2 : -1));
}

// The block-scaled product of two operands given as bytes.  fmt8 < 0: e2m1 pairs in a byte; else the float8 formats of
// a (bit 0) and b (bit 1), 1 = e5m2.
PyObject* product(const at::Tensor& a, const at::Tensor& b, const at::Tensor& sfa, const at::Tensor& sfb,
                  PyObject* alpha_arg, PyObject* out_arg, at::ScalarType out_type, int tile_n, PyObject* ws_arg,
                  int sf_vec, int fmt8) {
  if (!a.is_cuda() || !b.is_cuda() || !sfa.is_cuda() || !sfb.is_cuda())
    value_error("operands must be CUDA tensors (there is no CPU implementation)");
  const at::Device dev = a.device();
  on_device(&b, dev, "b");
  on_device(&sfa, dev, "sfa");
  on_device(&sfb, dev, "sfb");
  const Matrix am = matrix(a, "a"), bm = matrix(b, "b");
  if (am.l != bm.l || am.cols != bm.cols)
    value_error("a %s and b %s disagree on batch or K", shape_of(a).c_str(), shape_of(b).c_str());
  const int64_t m = am.rows, n = bm.rows, l = am.l, k = fmt8 >= 0 ? am.cols : am.cols * 2;
  if (k % (fmt8 >= 0 ? 16 : 32) != 0 || n % 8 != 0) value_error("Invalid tensor alignment");
  if (sf_vec != 16 && sf_vec != 32) not_implemented("sf_vec_size must be 16 (NVFP4) or 32 (MXFP4)");
  const int64_t need_a = l * tiled_bytes(m, ceil_div(k, sf_vec)), need_b = l * tiled_bytes(n, ceil_div(k, sf_vec));
  if (sfa.element_size() != 1 || sfb.element_size() != 1 || sfa.numel() < need_a || sfb.numel() < need_b)
    value_error("scale factors must be 1-byte tensors in the 128x4 tiled layout (%lld and %lld bytes)",
                static_cast<long long>(need_a), static_cast<long long>(need_b));
  // read as the run of bytes at their address: a view with gaps is not one (a permuted view of a run is)
  if (!sfa.is_non_overlapping_and_dense() || !sfb.is_non_overlapping_and_dense())
    value_error("scale factors must lie in one run of memory");
  at::Tensor made;
  if (out_arg == Py_None) {
    if (c_code(out_type) < 0)
      value_error("c must be [%lld, %lld] (x%lld) in float16, bfloat16 or float32", static_cast<long long>(m),
                  static_cast<long long>(n), static_cast<long long>(l));
    made = a.dim() == 2 ? empty({m, n}, out_type, dev) : empty({l, m, n}, out_type, dev);
  }
  const at::Tensor& c = out_arg == Py_None ? made : tensor(out_arg, "out");
  on_device(&c, dev, "c");
  const Matrix cm = matrix(c, "c");
  if (cm.l != l || cm.rows != m || cm.cols != n || c_code(c.scalar_type()) < 0)
    value_error("c must be [%lld, %lld] (x%lld) in float16, bfloat16 or float32", static_cast<long long>(m),
                static_cast<long long>(n), static_cast<long long>(l));
  const at::Tensor* alpha = maybe(alpha_arg, "alpha");
  if (alpha != nullptr && (alpha->scalar_type() != at::kFloat || !alpha->is_cuda()))
    value_error("alpha must be a float32 CUDA tensor");
  on_device(alpha, dev, "alpha");
  void* ws = nullptr;
  size_t ws_bytes = 0;
  if (ws_arg != Py_None && tile_n == 0 && sf_vec == 16 && fmt8 < 0) {
    const at::Tensor& w = tensor(ws_arg, "workspace");
    ws_bytes = b200fp4_nvfp4_gemm_workspace_bytes(static_cast<int>(m), static_cast<int>(n), static_cast<int>(k));
    if (ws_bytes != 0) {
      if (!w.is_cuda() || w.device() != dev || static_cast<size_t>(w.numel() * w.element_size()) < ws_bytes) {
        std::ostringstream s;
        s << "workspace must be a CUDA tensor on " << dev << " of at least " << ws_bytes << " bytes";
        value_error("%s", s.str().c_str());
      }
      ws = data(w);
    }
  }
  const int mi = static_cast<int>(m), ni = static_cast<int>(n), ki = static_cast<int>(k), li = static_cast<int>(l);
  launch(dev, [&](void* stream) {
    const float* al = static_cast<const float*>(data(alpha));
    const int cc = c_code(c.scalar_type());
    void *ap = data(a), *bp = data(b), *cp = data(c);
    if (fmt8 >= 0)
      return b200fp4_mxfp8_gemm(ap, bp, data(sfa), data(sfb), cp, al, mi, ni, ki, li, cc, tile_n, fmt8 & 1,
                                fmt8 >> 1, stream);
    if (sf_vec == 32)
      return b200fp4_mxfp4_gemm(ap, bp, data(sfa), data(sfb), cp, al, mi, ni, ki, li, cc, tile_n, stream);
    return b200fp4_nvfp4_gemm_ws(ap, bp, data(sfa), data(sfb), cp, al, mi, ni, ki, li, cc, tile_n, ws, ws_bytes,
                                 stream);
  });
  return give(out_arg, made);
}

// nvfp4_gemm(a, b, sfa, sfb, alpha, out, out_dtype, tile_n, workspace, sf_vec_size)
PyObject* nvfp4_gemm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 10, [&]() -> PyObject* {
    return product(bytes(tensor(v[0], "a")), bytes(tensor(v[1], "b")), tensor(v[2], "sfa"), tensor(v[3], "sfb"), v[4], v[5],
                   result_dtype(v[6], v[5]), static_cast<int>(integer(v[7])), v[8],
                   equals(v[9], 16) ? 16 : (equals(v[9], 32) ? 32 : 0), -1);
  });
}

// mxfp8_gemm(a, b, sfa, sfb, alpha, out, out_dtype, tile_n)
PyObject* mxfp8_gemm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 8, [&]() -> PyObject* {
    const at::Tensor &a = tensor(v[0], "a"), &b = tensor(v[1], "b");
    int fmt8 = 0;
    for (const at::Tensor* t : {&a, &b}) {
      if (t->scalar_type() == at::kFloat8_e5m2) fmt8 |= t == &a ? 1 : 2;
      else if (t->scalar_type() != at::kFloat8_e4m3fn) value_error("a and b must be float8_e4m3fn or float8_e5m2 tensors");
    }
    return product(a, b, tensor(v[2], "sfa"), tensor(v[3], "sfb"), v[4], v[5], result_dtype(v[6], v[5]),
                   static_cast<int>(integer(v[7])), Py_None, 32, fmt8);
  });
}

// mm_fp4(a, b, a_descale, b_descale, alpha, out, out_dtype): a weight (or its scales) that arrives as the transposed
// view of its row-major storage is taken as that storage
PyObject* mm_fp4(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 7, [&]() -> PyObject* {
    at::Tensor b = bytes(tensor(v[1], "b")), sfa = tensor(v[2], "a_descale"), sfb = tensor(v[3], "b_descale");
    const at::ScalarType out_type = dtype(v[6]);
    if (c_code(out_type) < 0) not_implemented("out_dtype must be torch.float16, torch.bfloat16 or torch.float32");
    auto storage = [](at::Tensor& t) {
      if (t.dim() != 2 || t.is_contiguous()) return;
      at::Tensor tt = t.t();
      if (tt.is_contiguous()) t = tt;
    };
    storage(b);
    storage(sfb);
    if (!sfa.is_contiguous()) sfa = sfa.contiguous();
    if (!sfb.is_contiguous()) sfb = sfb.contiguous();
    return product(bytes(tensor(v[0], "a")), b, bytes(sfa), bytes(sfb), v[4], v[5], out_type, 0, Py_None, 16, -1);
  });
}

// ---------------------------------------------------------------------------------------------------------------------
// topk_route(router_logits, top_k, renormalize)
// ---------------------------------------------------------------------------------------------------------------------
PyObject* topk_route(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 3, [&]() -> PyObject* {
    const at::Tensor& logits_arg = tensor(v[0], "router_logits");
    const int64_t top_k = integer(v[1]);
    if (!logits_arg.is_cuda() || logits_arg.scalar_type() != at::kFloat || logits_arg.dim() != 2)
      value_error("router_logits must be a float32 CUDA tensor [tokens, experts]");
    at::Tensor copy;
    if (!logits_arg.is_contiguous()) copy = logits_arg.contiguous();
    const at::Tensor& logits = copy.defined() ? copy : logits_arg;
    const int64_t t = logits.size(0), e = logits.size(1);
    const at::Device dev = logits.device();
    at::Tensor ids = empty({t, top_k}, at::kInt, dev), w = empty({t, top_k}, at::kFloat, dev);
    const int renorm = truth(v[2]) ? 1 : 0;
    launch(dev, [&](void* stream) {
      return b200fp4_topk_route(static_cast<const float*>(data(logits)), static_cast<int*>(data(ids)),
                                static_cast<float*>(data(w)), static_cast<int>(t), static_cast<int>(e),
                                static_cast<int>(top_k), renorm, stream);
    });
    PyObject* out = PyTuple_New(2);
    if (out == nullptr) return nullptr;
    PyTuple_SET_ITEM(out, 0, wrap(ids));
    PyTuple_SET_ITEM(out, 1, wrap(w));
    return out;
  });
}

// ---------------------------------------------------------------------------------------------------------------------
// moe(...): see moe.py for the meaning of the arguments
// ---------------------------------------------------------------------------------------------------------------------
// the six-mode view (32, 4, m_tiles, 4, k_tiles, E) of storage [E, m_tiles, k_tiles, 32, 4, 4], or that storage
at::Tensor scale_storage(const at::Tensor& sf, int64_t experts, int64_t rows, int64_t k, const char* name) {
  const int64_t need = tiled_bytes(rows, k / 16);
  at::Tensor st = sf;
  int64_t outer, inner;
  if (sf.dim() == 6) {
    if (sf.size(0) != 32 || sf.size(1) != 4 || sf.size(3) != 4)
      value_error("expected a (32,4,m_tiles,4,k_tiles,E) scale tensor, got %s", shape_of(sf).c_str());
    // strides of the view on contiguous storage; anything else is copied into that order
    const int64_t mt = sf.size(2), kt = sf.size(4);
    const int64_t want[6] = {16, 4, 512 * kt, 1, 512, 512 * kt * mt};
    bool as_is = true;
    for (int i = 0; i < 6; ++i) as_is = as_is && (sf.size(i) == 1 || sf.stride(i) == want[i]);
    if (!as_is) st = sf.permute({5, 2, 4, 0, 1, 3}).contiguous();
    outer = sf.size(5);
    inner = outer == 0 ? 0 : sf.numel() / outer * sf.element_size();
  } else {
    if (!st.is_contiguous()) st = st.contiguous();
    outer = experts;
    const int64_t total = st.numel() * st.element_size();
    if (experts <= 0 || total % experts != 0)
      value_error("%s: expected %lld x %lld scale bytes in 128x4 tiles, got %s", name, static_cast<long long>(experts),
                  static_cast<long long>(need), shape_of(sf).c_str());
    inner = total / experts;
  }
  if (outer != experts || inner != need)
    value_error("%s: expected %lld x %lld scale bytes in 128x4 tiles, got (%lld, %lld)", name,
                static_cast<long long>(experts), static_cast<long long>(need), static_cast<long long>(outer),
                static_cast<long long>(inner));
  return st;
}

enum MoeArg {
  kX, kW1, kW1Sf, kW2, kW2Sf, kIds, kScales, kExperts, kTopK, kW1Alpha, kW2Alpha, kFc2Scale, kLocal, kOffset, kOutput,
  kOutDtype, kAccumulate, kWorkspace, kSlotRows, kLogits, kRenorm, kMoeArgs
};

PyObject* moe(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, kMoeArgs, [&]() -> PyObject* {
    const at::Tensor& x = tensor(v[kX], "x");
    at::ScalarType out_type = dtype(v[kOutDtype]);
    if ((out_type != at::kBFloat16 && out_type != at::kFloat) || x.scalar_type() != at::kBFloat16)
      not_implemented("tokens must be bfloat16 and the output bfloat16 (or float32 partial sums)");
    if (!x.is_cuda()) value_error("x must be a CUDA tensor (there is no CPU implementation)");
    if (x.dim() != 2 || !x.is_contiguous()) value_error("x must be contiguous [tokens, hidden]");
    const int64_t tokens = x.size(0), hidden = x.size(1);
    const int64_t num_experts = integer(v[kExperts]), top_k = integer(v[kTopK]), offset = to_integer(v[kOffset]);
    const int64_t local = v[kLocal] == Py_None ? num_experts : integer(v[kLocal]);
    const bool accumulate = truth(v[kAccumulate]);
    const at::Device dev = x.device();
    const at::Tensor &w1_arg = tensor(v[kW1], "w1_weight"), &w1_sf = tensor(v[kW1Sf], "w1_weight_sf"),
                     &w2_arg = tensor(v[kW2], "w2_weight"), &w2_sf = tensor(v[kW2Sf], "w2_weight_sf");
    const at::Tensor *ids = maybe(v[kIds], "token_selected_experts"), *scales = maybe(v[kScales], "token_final_scales"),
                     *w1_alpha = maybe(v[kW1Alpha], "w1_alpha"), *w2_alpha = maybe(v[kW2Alpha], "w2_alpha"),
                     *fc2_scale = maybe(v[kFc2Scale], "fc2_input_scale"), *output = maybe(v[kOutput], "output"),
                     *workspace = maybe(v[kWorkspace], "workspace"), *logits = maybe(v[kLogits], "router_logits");
    on_device(&w1_arg, dev, "w1_weight");
    on_device(&w1_sf, dev, "w1_weight_sf");
    on_device(&w2_arg, dev, "w2_weight");
    on_device(&w2_sf, dev, "w2_weight_sf");
    on_device(ids, dev, "token_selected_experts");
    on_device(scales, dev, "token_final_scales");
    on_device(w1_alpha, dev, "w1_alpha");
    on_device(w2_alpha, dev, "w2_alpha");
    on_device(fc2_scale, dev, "fc2_input_scale");
    on_device(output, dev, "output");
    on_device(workspace, dev, "workspace");
    on_device(logits, dev, "router_logits");
    const at::Tensor w1 = bytes(w1_arg), w2 = bytes(w2_arg);
    if (w1.dim() != 3 || w1.size(0) != local || w1.size(2) * 2 != hidden || !w1.is_contiguous())
      value_error("w1_weight must be contiguous [%lld, 2*I, %lld]", static_cast<long long>(local),
                  static_cast<long long>(hidden / 2));
    const int64_t inter = w1.size(1) / 2;
    if (w2.dim() != 3 || w2.size(0) != local || w2.size(1) != hidden || w2.size(2) != inter / 2 || !w2.is_contiguous())
      value_error("w2_weight must be contiguous [%lld, %lld, %lld]", static_cast<long long>(local),
                  static_cast<long long>(hidden), static_cast<long long>(inter / 2));
    at::Tensor ids_made, scales_made;
    if (logits != nullptr) {
      if (logits->scalar_type() != at::kFloat || logits->dim() != 2 || logits->size(0) != tokens ||
          logits->size(1) != num_experts || !logits->is_contiguous())
        value_error("router_logits must be contiguous float32 [%lld, %lld]", static_cast<long long>(tokens),
                    static_cast<long long>(num_experts));
      if (ids == nullptr) {
        ids_made = empty({tokens, top_k}, at::kInt, dev);
        ids = &ids_made;
      }
      if (scales == nullptr) {
        scales_made = empty({tokens, top_k}, at::kFloat, dev);
        scales = &scales_made;
      }
    } else if (ids == nullptr || scales == nullptr) {
      value_error("token_selected_experts and token_final_scales are required without router_logits");
    }
    if (ids->scalar_type() != at::kInt || ids->dim() != 2 || ids->size(0) != tokens || ids->size(1) != top_k ||
        !ids->is_contiguous())
      value_error("token_selected_experts must be contiguous int32 [tokens, top_k]");
    if (scales->scalar_type() != at::kFloat || scales->dim() != 2 || scales->size(0) != tokens || scales->size(1) != top_k ||
        !scales->is_contiguous())
      value_error("token_final_scales must be contiguous float32 [tokens, top_k]");
    const at::Tensor s1 = scale_storage(w1_sf, local, 2 * inter, hidden, "w1_weight_sf");
    const at::Tensor s2 = scale_storage(w2_sf, local, hidden, inter, "w2_weight_sf");
    for (const auto& p : {std::make_pair("w1_alpha", w1_alpha), std::make_pair("w2_alpha", w2_alpha)})
      if (p.second != nullptr &&
          (p.second->scalar_type() != at::kFloat || p.second->numel() != local || !p.second->is_contiguous()))
        value_error("%s must be float32 [%lld]", p.first, static_cast<long long>(local));
    if (fc2_scale != nullptr && (fc2_scale->scalar_type() != at::kFloat || fc2_scale->numel() != 1))
      value_error("fc2_input_scale must be one float32");
    at::Tensor made;
    if (output == nullptr) {
      made = empty({tokens, hidden}, out_type, dev);
      if (accumulate) made.zero_();
      output = &made;
    } else if (output->dim() != 2 || output->size(0) != tokens || output->size(1) != hidden ||
               (output->scalar_type() != at::kBFloat16 && output->scalar_type() != at::kFloat) || !output->is_contiguous()) {
      value_error("output must be contiguous bfloat16 or float32 [tokens, hidden]");
    }
    out_type = output->scalar_type();
    at::ScalarType rows_type = out_type == at::kFloat ? at::kFloat : at::kBFloat16;
    if (v[kSlotRows] != Py_None) {
      rows_type = dtype(v[kSlotRows]);
      if (rows_type != at::kBFloat16 && rows_type != at::kFloat)
        value_error("slot_rows_dtype must be torch.bfloat16 or torch.float32");
    }
    if (out_type == at::kFloat && rows_type != at::kFloat)
      not_implemented("a float32 output keeps float32 per-slot rows");
    if (tokens == 0) return give(v[kOutput], made);
    const size_t need = b200fp4_moe_workspace_bytes(tokens, static_cast<int>(hidden), static_cast<int>(inter),
                                                    static_cast<int>(local), static_cast<int>(top_k));
    at::Tensor scratch;                // from the stream's pool: reused by the next call in stream order, safe with threads
    if (workspace == nullptr) {
      scratch = empty({static_cast<int64_t>(need)}, at::kByte, dev);
      workspace = &scratch;
    }
    const size_t have = static_cast<size_t>(workspace->numel() * workspace->element_size());
    if (have < need) value_error("workspace too small: %zu bytes needed", need);
    const int code = out_type == at::kFloat ? 2 : (rows_type == at::kBFloat16 ? 3 : 1);
    const int renorm = truth(v[kRenorm]) ? 1 : 0;
    launch(dev, [&](void* stream) {
      const float *a1 = static_cast<const float*>(data(w1_alpha)), *a2 = static_cast<const float*>(data(w2_alpha)),
                  *fs = static_cast<const float*>(data(fc2_scale));
      const int h = static_cast<int>(hidden), i = static_cast<int>(inter), e = static_cast<int>(local),
                k = static_cast<int>(top_k), lo = static_cast<int>(offset);
      int* idp = static_cast<int*>(data(ids));
      float* wp = static_cast<float*>(data(scales));
      if (logits == nullptr)
        return b200fp4_moe_fused(data(x), data(w1), data(s1), data(w2), data(s2), idp, wp, a1, a2, fs, data(output), tokens,
                                 h, i, e, k, lo, accumulate ? 1 : 0, code, data(workspace), have, stream);
      return b200fp4_moe_fused_routed(data(x), static_cast<const float*>(data(logits)), static_cast<int>(num_experts), renorm,
                                      data(w1), data(s1), data(w2), data(s2), idp, wp, a1, a2, fs, data(output), tokens, h, i,
                                      e, k, lo, accumulate ? 1 : 0, code, data(workspace), have, stream);
    });
    return give(v[kOutput], made);
  });
}

PyObject* set_error_class(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  Py_XDECREF(g_error_class);
  g_error_class = cls;
  Py_RETURN_NONE;
}

template <PyObject* (*fn)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn));
}

PyMethodDef g_methods[] = {
    {"norm", fast<norm>(), METH_FASTCALL, nullptr},
    {"nvfp4_gemm", fast<nvfp4_gemm>(), METH_FASTCALL, nullptr},
    {"mxfp8_gemm", fast<mxfp8_gemm>(), METH_FASTCALL, nullptr},
    {"mm_fp4", fast<mm_fp4>(), METH_FASTCALL, nullptr},
    {"topk_route", fast<topk_route>(), METH_FASTCALL, nullptr},
    {"moe", fast<moe>(), METH_FASTCALL, nullptr},
    {"set_error_class", set_error_class, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_b200fp4_torch", "host path of the b200fp4 operators", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200fp4_torch(void) { return PyModule_Create(&g_module); }
