// The torch side of the Python binding: tensor checks, result allocation, the current stream and the call into
// libcaifq.so for the entry points a program makes per layer and step.
//
// Why native: a few-token call keeps the GPU busy for 2.5 to 10 us, while the same steps in Python over ctypes took
// 13 us of host time per call (four ctypes conversions of pointers, torch.empty through the argument parser, the
// stream object) and 190 struct copies per grouped-expert call.  Here a call costs about 4 us, most of it the launch.
//
// Every function takes positional arguments only; native.py holds the documented signatures and the defaults.
// The GIL is released around the library call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include <cstdint>
#include <vector>

#include "caifq.h"

namespace
{

PyObject *g_error = nullptr;   // native.CaifqError

// entry points, looked up in the library that native.py loaded
#define CAIFQ_BOUND(X)                                                                                                \
  X(linear_fwd) X(linear_fwd_residual) X(linear_fwd_multi) X(linear_dx) X(linear_workspace_bytes) X(linear_fwd_ws) X(linear_dx_ws) X(linear_concat_workspace_bytes)              \
  X(linear_fwd_concat) X(linear_dx_concat) X(lora_fwd_workspace_bytes) X(lora_fwd_workspace_bytes_expanded)           \
  X(lora_bwd_workspace_bytes) X(lora_bwd_workspace_bytes_expanded) X(lora_linear_fwd) X(lora_linear_fwd_expanded)     \
  X(lora_linear_bwd) X(lora_linear_bwd_expanded) X(rmsnorm_fwd) X(rmsnorm_bwd) X(cast) X(quantize_int8_per_tensor)    \
  X(quantize_int8_per_channel) X(quantize_int4_per_group) X(moe_topk) X(moe_normalize_rows) X(moe_router_softmax)     \
  X(moe_build_dispatch) X(moe_dispatch) X(moe_combine) X(moe_combine_bwd_grad_expert)                                 \
  X(moe_combine_bwd_grad_weights) X(moe_dispatch_bwd) X(moe_router_bwd) X(grouped_expert_expand)                      \
  X(grouped_expert_fwd) X(grouped_expert_fwd_expanded) X(grouped_expert_bwd) X(grouped_expert_bwd_expanded)           \
  X(last_error)

struct Api
{
#define CAIFQ_FIELD(name) decltype(&caifq_##name) name;
  CAIFQ_BOUND(CAIFQ_FIELD)
#undef CAIFQ_FIELD
} api;

// A Python exception is set; unwinds to the wrapper below.
struct Raised
{
};

[[noreturn]] void raise(PyObject *type, const char *text)
{
  PyErr_SetString(type, text);
  throw Raised{};
}

void check(int rc, const char *what)
{
  if (rc != 0)
  {
    PyErr_Format(g_error, "%s failed (%d): %s", what, rc, api.last_error());
    throw Raised{};
  }
}

// Positional arguments of one call, taken in order.
class Args
{
public:
  Args(PyObject *const *args, Py_ssize_t n) : args_(args), n_(n) {}

  PyObject *next()
  {
    if (at_ >= n_)
    {
      raise(PyExc_TypeError, "missing argument");
    }
    return args_[at_++];
  }

  int64_t integer()
  {
    const long long v = PyLong_AsLongLong(next());
    if (v == -1 && PyErr_Occurred())
    {
      throw Raised{};
    }
    return v;
  }

  double real()
  {
    const double v = PyFloat_AsDouble(next());
    if (v == -1.0 && PyErr_Occurred())
    {
      throw Raised{};
    }
    return v;
  }

  bool truth()
  {
    const int v = PyObject_IsTrue(next());
    if (v < 0)
    {
      throw Raised{};
    }
    return v != 0;
  }

  // a contiguous CUDA tensor; null for None where `optional`
  const at::Tensor *tensor(bool optional = false)
  {
    const at::Tensor *t = buffer();
    if (t == nullptr)
    {
      if (optional)
      {
        return nullptr;
      }
      raise(PyExc_TypeError, "expected a torch.Tensor");
    }
    if (!t->is_cuda())
    {
      raise(g_error, "caifq works on CUDA tensors only (no CPU fallback)");
    }
    if (!t->is_contiguous())
    {
      raise(g_error, "caifq needs contiguous tensors");
    }
    return t;
  }

  // a tensor that the caller lays out (a result or scratch buffer), or null for None
  const at::Tensor *buffer()
  {
    PyObject *o = next();
    if (o == Py_None)
    {
      return nullptr;
    }
    if (!THPVariable_Check(o))
    {
      raise(PyExc_TypeError, "expected a torch.Tensor");
    }
    return &THPVariable_Unpack(o);
  }

  // None: torch's default, as in torch.empty
  at::ScalarType dtype()
  {
    PyObject *o = next();
    if (o == Py_None)
    {
      return c10::get_default_dtype_as_scalartype();
    }
    if (!THPDtype_Check(o))
    {
      raise(PyExc_TypeError, "expected a torch.dtype");
    }
    return reinterpret_cast<THPDtype *>(o)->scalar_type;
  }

  // the C struct inside a native.Weight or native.Lora
  template <typename T>
  const T *record()
  {
    return static_cast<const T *>(address(next()));
  }

  // a list of native.Weight as an array; false for None
  bool weights(std::vector<caifq_weight> &out)
  {
    PyObject *o = next();
    if (o == Py_None)
    {
      return false;
    }
    PyObject *seq = PySequence_Fast(o, "expected a list of weights");
    if (seq == nullptr)
    {
      throw Raised{};
    }
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    out.resize(static_cast<size_t>(n));
    try
    {
      for (Py_ssize_t i = 0; i < n; ++i)
      {
        out[static_cast<size_t>(i)] = *static_cast<const caifq_weight *>(address(PySequence_Fast_GET_ITEM(seq, i)));
      }
    }
    catch (...)
    {
      Py_DECREF(seq);
      throw;
    }
    Py_DECREF(seq);
    return true;
  }

  std::vector<int32_t> integers()
  {
    PyObject *seq = PySequence_Fast(next(), "expected a list of integers");
    if (seq == nullptr)
    {
      throw Raised{};
    }
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    std::vector<int32_t> out(static_cast<size_t>(n));
    for (Py_ssize_t i = 0; i < n; ++i)
    {
      PyObject *item = PySequence_Fast_GET_ITEM(seq, i);
      PyObject *whole = PyLong_Check(item) ? (Py_INCREF(item), item) : PyNumber_Long(item);
      out[static_cast<size_t>(i)] = whole != nullptr ? static_cast<int32_t>(PyLong_AsLong(whole)) : 0;
      Py_XDECREF(whole);
      if (PyErr_Occurred())
      {
        Py_DECREF(seq);
        throw Raised{};
      }
    }
    Py_DECREF(seq);
    return out;
  }

private:
  static void *address(PyObject *o)
  {
    static PyObject *name = PyUnicode_InternFromString("_addr");
    PyObject *v = PyObject_GetAttr(o, name);
    if (v == nullptr)
    {
      throw Raised{};
    }
    void *p = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    if (p == nullptr && PyErr_Occurred())
    {
      throw Raised{};
    }
    return p;
  }

  PyObject *const *args_;
  Py_ssize_t n_;
  Py_ssize_t at_ = 0;
};

int code_of(at::ScalarType t)
{
  switch (t)
  {
    case at::kFloat:
      return CAIFQ_F32;
    case at::kHalf:
      return CAIFQ_F16;
    case at::kBFloat16:
      return CAIFQ_BF16;
    case at::kChar:
      return CAIFQ_I8;
    default:
      PyErr_SetString(PyExc_KeyError, c10::toString(t));
      throw Raised{};
  }
}

int code_of(const at::Tensor &t) { return code_of(t.scalar_type()); }

void *ptr(const at::Tensor *t) { return t != nullptr ? t->data_ptr() : nullptr; }
void *ptr(const at::Tensor &t) { return t.data_ptr(); }

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, const at::Tensor &like)
{
  return at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt);
}

at::Tensor empty_like(const at::Tensor &t) { return empty(t.sizes(), t.scalar_type(), t); }

void *stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// x.shape with the last dimension replaced
std::vector<int64_t> shape_with_last(const at::Tensor &x, int64_t last)
{
  std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
  if (s.empty())
  {
    s.push_back(last);
  }
  s.back() = last;
  return s;
}

// an [rows, columns] operand: another rank would be read as one of the wrong width
void need_matrix(const at::Tensor &t, const char *who)
{
  if (t.dim() != 2)
  {
    PyErr_Format(PyExc_ValueError, "%s: a [rows, columns] tensor expected, got %lld dimensions", who,
                 static_cast<long long>(t.dim()));
    throw Raised{};
  }
}

// numel // width as Python has it: a width of zero is an exception there, and the end of the process in C
int64_t rows_of(const at::Tensor &t, int64_t width)
{
  if (width == 0)
  {
    raise(PyExc_ZeroDivisionError, "integer division or modulo by zero");
  }
  return t.numel() / width;
}

PyObject *wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

PyObject *wrap_or_none(const at::Tensor &t)
{
  if (!t.defined())
  {
    Py_RETURN_NONE;
  }
  return THPVariable_Wrap(t);
}

PyObject *pack(std::initializer_list<PyObject *> items)
{
  PyObject *t = PyTuple_New(static_cast<Py_ssize_t>(items.size()));
  Py_ssize_t i = 0;
  for (PyObject *o : items)
  {
    PyTuple_SET_ITEM(t, i++, o);
  }
  return t;
}

// the library call without the GIL
template <typename F>
int unlocked(F &&f)
{
  PyThreadState *save = PyEval_SaveThread();
  const int rc = f();
  PyEval_RestoreThread(save);
  return rc;
}

// Scratch that a call can do without: undefined when the device has no memory left for it.
at::Tensor scratch(size_t bytes, const at::Tensor &like)
{
  try
  {
    return empty({static_cast<int64_t>(bytes)}, at::kByte, like);
  }
  catch (const c10::OutOfMemoryError &)
  {
    return at::Tensor();
  }
}

// A call that is given its result allocates nothing while its stream is captured: the capture may be the caller's own, and
// scratch from the caching allocator would be somebody else's when that graph is replayed.  (With no result given the call
// takes that from the allocator too, so the capture must be one that torch knows of.)
bool may_take_scratch(const at::Tensor *out, void *s)
{
  if (out == nullptr)
  {
    return true;
  }
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(static_cast<cudaStream_t>(s), &status) == cudaSuccess && status == cudaStreamCaptureStatusNone;
}

// ---- frozen linear ------------------------------------------------------------------------------------------

// (weight, act, out_dtype, compute, out | None): forward or dX
PyObject *linear(Args &a, bool backward)
{
  const caifq_weight *w = a.record<caifq_weight>();
  const at::Tensor &x = *a.tensor();
  const at::ScalarType out_dtype = a.dtype();
  const int compute = static_cast<int>(a.integer());
  const at::Tensor *out = a.buffer();
  const int64_t m = rows_of(x, backward ? w->out_dim : w->in_dim);
  at::Tensor y = out != nullptr ? *out : empty(shape_with_last(x, backward ? w->in_dim : w->out_dim), out_dtype, x);
  const int xc = code_of(x), yc = code_of(y);
  void *s = stream();
  const size_t need = api.linear_workspace_bytes(w, backward ? 1 : 0, xc, m, compute);
  const at::Tensor work = need > 0 && may_take_scratch(out, s) ? scratch(need, x) : at::Tensor();
  void *scratch_ptr = work.defined() ? ptr(work) : nullptr;
  auto fn = backward ? api.linear_dx_ws : api.linear_fwd_ws;
  check(unlocked([&] { return fn(w, ptr(x), xc, m, ptr(y), yc, compute, scratch_ptr, scratch_ptr ? need : 0, s); }),
        backward ? "linear_dx" : "linear_fwd");
  return wrap(std::move(y));
}

PyObject *linear_fwd(Args &a) { return linear(a, false); }
PyObject *linear_dx(Args &a) { return linear(a, true); }

PyObject *linear_fwd_residual(Args &a)
{
  const caifq_weight *w = a.record<caifq_weight>();
  const at::Tensor &x = *a.tensor();
  const at::Tensor &res = *a.tensor();
  const int compute = static_cast<int>(a.integer());
  const int64_t m = rows_of(x, w->in_dim);
  const int xc = code_of(x), rc = code_of(res);
  void *s = stream();
  check(unlocked([&] { return api.linear_fwd_residual(w, ptr(x), xc, m, ptr(res), rc, compute, s); }),
        "caifq_linear_fwd_residual");
  return wrap(res);
}

PyObject *linear_fwd_multi(Args &a)
{
  std::vector<caifq_weight> ws;
  if (!a.weights(ws) || ws.empty())
  {
    raise(PyExc_IndexError, "linear_fwd_multi: no weights");
  }
  const at::Tensor &x = *a.tensor();
  const at::ScalarType out_dtype = a.dtype();
  const int compute = static_cast<int>(a.integer());
  const at::Tensor *out = a.buffer();
  const int64_t m = rows_of(x, ws[0].in_dim);
  int64_t total = 0;
  for (const caifq_weight &w : ws)
  {
    total += w.out_dim;
  }
  at::Tensor y = out != nullptr ? *out : empty({m, total}, out_dtype, x);
  const int xc = code_of(x), yc = code_of(y);
  void *s = stream();
  check(unlocked([&] {
          return api.linear_fwd_multi(ws.data(), static_cast<int32_t>(ws.size()), ptr(x), xc, m, ptr(y), yc, compute, s);
        }),
        "caifq_linear_fwd_multi");
  return wrap(std::move(y));
}

PyObject *linear_concat(Args &a)
{
  std::vector<caifq_weight> ws;
  if (!a.weights(ws) || ws.empty())
  {
    raise(PyExc_IndexError, "linear_concat: no weights");
  }
  const at::Tensor &act = *a.tensor();
  const bool backward = a.truth();
  const at::ScalarType out_dtype = a.dtype();
  const at::Tensor *given = a.tensor(true);
  const int32_t count = static_cast<int32_t>(ws.size());
  int64_t total = 0;
  for (const caifq_weight &w : ws)
  {
    total += w.out_dim;
  }
  at::Tensor work = given != nullptr ? *given
                                     : empty({static_cast<int64_t>(api.linear_concat_workspace_bytes(ws.data(), count))},
                                             at::kByte, act);
  const int64_t m = rows_of(act, backward ? total : ws[0].in_dim);
  at::Tensor out = empty({m, backward ? ws[0].in_dim : total}, out_dtype, act);
  const int ac = code_of(act), oc = code_of(out);
  void *s = stream();
  auto fn = backward ? api.linear_dx_concat : api.linear_fwd_concat;
  check(unlocked([&] {
          return fn(ws.data(), count, ptr(act), ac, m, ptr(out), oc, CAIFQ_BF16, ptr(work),
                    static_cast<size_t>(work.numel()), s);
        }),
        "caifq_linear_concat");
  return wrap(std::move(out));
}

// ---- LoRA ---------------------------------------------------------------------------------------------------

at::Tensor workspace_of(const at::Tensor *given, size_t need, const at::Tensor &like, const char *who)
{
  if (given == nullptr)
  {
    return empty({static_cast<int64_t>(need > 0 ? need : 1)}, at::kByte, like);
  }
  if (given->numel() < static_cast<int64_t>(need))
  {
    PyErr_Format(g_error, "%s: workspace of %lld bytes, %zu needed", who, static_cast<long long>(given->numel()), need);
    throw Raised{};
  }
  return *given;
}

PyObject *lora_linear_fwd(Args &a)
{
  const caifq_weight *w = a.record<caifq_weight>();
  const caifq_lora *l = a.record<caifq_lora>();
  const at::Tensor &x = *a.tensor();
  const int compute = static_cast<int>(a.integer());
  const at::Tensor *out = a.buffer();
  const at::Tensor *hid = a.buffer();
  const at::Tensor *given = a.buffer();
  const bool expanded = a.truth();
  const int64_t m = rows_of(x, w->in_dim);
  at::Tensor y = out != nullptr ? *out : empty(shape_with_last(x, w->out_dim), x.scalar_type(), x);
  at::Tensor hidden = hid != nullptr ? *hid : empty({m, l->rank}, x.scalar_type(), x);
  const size_t need =
      expanded ? api.lora_fwd_workspace_bytes_expanded(w, l, m, compute) : api.lora_fwd_workspace_bytes(w, l, m);
  at::Tensor work = workspace_of(given, need, x, "lora_linear_fwd");
  void *s = stream();
  auto fn = expanded ? api.lora_linear_fwd_expanded : api.lora_linear_fwd;
  check(unlocked([&] { return fn(w, l, ptr(x), m, ptr(y), ptr(hidden), ptr(work), compute, s); }), "lora_linear_fwd");
  return pack({wrap(std::move(y)), wrap(std::move(hidden))});
}

PyObject *lora_linear_bwd(Args &a)
{
  const caifq_weight *w = a.record<caifq_weight>();
  const caifq_lora *l = a.record<caifq_lora>();
  const at::Tensor *la = a.buffer();
  const at::Tensor *lb = a.buffer();
  const at::Tensor &dy = *a.tensor();
  const at::Tensor &x = *a.tensor();
  const at::Tensor &hidden = *a.tensor();
  const int compute = static_cast<int>(a.integer());
  const at::Tensor *dx_given = a.buffer();
  const at::Tensor *da_given = a.buffer();
  const at::Tensor *db_given = a.buffer();
  const at::Tensor *given = a.buffer();
  const bool expanded = a.truth();
  const int64_t m = rows_of(dy, w->out_dim);
  at::Tensor dx = dx_given != nullptr ? *dx_given : empty(shape_with_last(dy, w->in_dim), dy.scalar_type(), dy);
  at::Tensor da = da_given != nullptr ? *da_given : empty_like(*la);
  at::Tensor db = db_given != nullptr ? *db_given : empty_like(*lb);
  const size_t need =
      expanded ? api.lora_bwd_workspace_bytes_expanded(w, l, m, compute) : api.lora_bwd_workspace_bytes(w, l, m);
  at::Tensor work = workspace_of(given, need, dy, "lora_linear_bwd");
  void *s = stream();
  auto fn = expanded ? api.lora_linear_bwd_expanded : api.lora_linear_bwd;
  check(unlocked([&] {
          return fn(w, l, ptr(dy), ptr(x), ptr(hidden), m, ptr(dx), ptr(da), ptr(db), ptr(work), compute, s);
        }),
        "lora_linear_bwd");
  return pack({wrap(std::move(dx)), wrap(std::move(da)), wrap(std::move(db))});
}

// ---- norm, casts, quantizers --------------------------------------------------------------------------------

PyObject *rmsnorm_fwd(Args &a)
{
  const at::Tensor &x = *a.tensor();
  const at::Tensor &gamma = *a.tensor();
  const float eps = static_cast<float>(a.real());
  const int64_t dim = x.size(-1);
  const int64_t rows = rows_of(x, dim);
  at::Tensor y = empty_like(x);
  at::Tensor rms = empty({rows}, at::kFloat, x);
  const int xc = code_of(x);
  void *s = stream();
  check(unlocked([&] {
          return api.rmsnorm_fwd(ptr(x), static_cast<const float *>(ptr(gamma)), ptr(y), static_cast<float *>(ptr(rms)),
                                 eps, xc, static_cast<int32_t>(rows), static_cast<int32_t>(dim), s);
        }),
        "rmsnorm_fwd");
  return pack({wrap(std::move(y)), wrap(std::move(rms))});
}

PyObject *rmsnorm_bwd(Args &a)
{
  const at::Tensor &dy = *a.tensor();
  const at::Tensor &x = *a.tensor();
  const at::Tensor &gamma = *a.tensor();
  const at::Tensor &rms = *a.tensor();
  const at::Tensor *given = a.tensor(true);
  const int64_t dim = x.size(-1);
  const int64_t rows = rows_of(x, dim);
  at::Tensor dx = empty_like(x);
  at::Tensor dg = given != nullptr ? *given : empty({dim}, at::kFloat, x).zero_();
  const int xc = code_of(x);
  void *s = stream();
  check(unlocked([&] {
          return api.rmsnorm_bwd(ptr(dy), ptr(x), static_cast<const float *>(ptr(gamma)),
                                 static_cast<const float *>(ptr(rms)), ptr(dx), static_cast<float *>(ptr(dg)), xc,
                                 static_cast<int32_t>(rows), static_cast<int32_t>(dim), s);
        }),
        "rmsnorm_bwd");
  return pack({wrap(std::move(dx)), wrap(std::move(dg))});
}

PyObject *cast(Args &a)
{
  const at::Tensor &x = *a.tensor();
  const at::ScalarType dtype = a.dtype();
  at::Tensor out = empty(x.sizes(), dtype, x);
  const int xc = code_of(x), oc = code_of(out);
  void *s = stream();
  check(unlocked([&] { return api.cast(ptr(x), xc, ptr(out), oc, x.numel(), s); }), "cast");
  return wrap(std::move(out));
}

PyObject *quantize_int8_per_tensor(Args &a)
{
  const at::Tensor &x = *a.tensor();
  at::Tensor q = empty(x.sizes(), at::kChar, x);
  at::Tensor scale = empty({1}, at::kFloat, x);
  void *s = stream();
  check(unlocked([&] {
          return api.quantize_int8_per_tensor(static_cast<const float *>(ptr(x)), static_cast<int8_t *>(ptr(q)),
                                              static_cast<float *>(ptr(scale)), x.numel(), s);
        }),
        "quantize_int8_per_tensor");
  return pack({wrap(std::move(q)), wrap(std::move(scale))});
}

PyObject *quantize_int8_per_channel(Args &a)
{
  const at::Tensor &x = *a.tensor();
  need_matrix(x, "quantize_int8_per_channel");
  const int64_t rows = x.size(0), cols = x.size(1);
  at::Tensor q = empty(x.sizes(), at::kChar, x);
  at::Tensor scales = empty({cols}, at::kFloat, x);
  void *s = stream();
  check(unlocked([&] {
          return api.quantize_int8_per_channel(static_cast<const float *>(ptr(x)), static_cast<int8_t *>(ptr(q)),
                                               static_cast<float *>(ptr(scales)), static_cast<int32_t>(rows),
                                               static_cast<int32_t>(cols), s);
        }),
        "quantize_int8_per_channel");
  return pack({wrap(std::move(q)), wrap(std::move(scales))});
}

PyObject *quantize_int4(Args &a)
{
  const at::Tensor &x = *a.tensor();
  const int64_t group = a.integer();
  const int64_t n = x.numel();
  if (group <= 0)
  {
    raise(PyExc_ZeroDivisionError, "quantize_int4: group_size must be positive");
  }
  // every byte and scale is written by the kernel
  at::Tensor packed = empty({(n + 1) / 2}, at::kByte, x);
  at::Tensor scales = empty({(n + group - 1) / group}, at::kHalf, x);
  void *s = stream();
  check(unlocked([&] {
          return api.quantize_int4_per_group(static_cast<const float *>(ptr(x)), static_cast<uint8_t *>(ptr(packed)),
                                             static_cast<uint16_t *>(ptr(scales)), n, static_cast<int32_t>(group), s);
        }),
        "quantize_int4_per_group");
  return pack({wrap(std::move(packed)), wrap(std::move(scales))});
}

// ---- mixture of experts -------------------------------------------------------------------------------------

const int32_t *ints(const at::Tensor &t) { return static_cast<const int32_t *>(t.data_ptr()); }

PyObject *moe_topk(Args &a)
{
  const at::Tensor &probs = *a.tensor();
  const int64_t k = a.integer();
  need_matrix(probs, "moe_topk");
  const int64_t batch = probs.size(0), dim = probs.size(1);
  at::Tensor idx = empty({batch, k}, at::kInt, probs);
  at::Tensor val = empty({batch, k}, probs.scalar_type(), probs);
  const int pc = code_of(probs);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_topk(ptr(probs), pc, static_cast<int32_t *>(ptr(idx)), ptr(val), static_cast<int32_t>(batch),
                              static_cast<int32_t>(dim), static_cast<int32_t>(k), s);
        }),
        "moe_topk");
  return pack({wrap(std::move(idx)), wrap(std::move(val))});
}

PyObject *moe_normalize_rows(Args &a)
{
  const at::Tensor &x = *a.tensor();
  need_matrix(x, "moe_normalize_rows");
  at::Tensor out = empty_like(x);
  const int xc = code_of(x);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_normalize_rows(ptr(x), ptr(out), xc, static_cast<int32_t>(x.size(0)),
                                        static_cast<int32_t>(x.size(1)), s);
        }),
        "moe_normalize_rows");
  return wrap(std::move(out));
}

PyObject *moe_softmax(Args &a)
{
  const at::Tensor &x = *a.tensor();
  const at::Tensor *bias = a.tensor(true);
  need_matrix(x, "moe_softmax");
  at::Tensor out = empty_like(x);
  const int xc = code_of(x);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_router_softmax(ptr(x), ptr(bias), ptr(out), xc, static_cast<int32_t>(x.size(0)),
                                        static_cast<int32_t>(x.size(1)), s);
        }),
        "moe_router_softmax");
  return wrap(std::move(out));
}

PyObject *moe_build_dispatch(Args &a)
{
  const at::Tensor &idx = *a.tensor();
  const int64_t experts = a.integer();
  const int64_t capacity = a.integer();
  need_matrix(idx, "moe_build_dispatch");
  const int64_t tokens = idx.size(0), k = idx.size(1);
  at::Tensor map = empty({tokens, k}, at::kInt, idx);
  at::Tensor offsets = empty({experts + 1}, at::kInt, idx);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_build_dispatch(ints(idx), static_cast<int32_t>(tokens), static_cast<int32_t>(k),
                                        static_cast<int32_t>(experts), static_cast<int32_t>(capacity),
                                        static_cast<int32_t *>(ptr(map)), static_cast<int32_t *>(ptr(offsets)), s);
        }),
        "moe_build_dispatch");
  return pack({wrap(std::move(map)), wrap(std::move(offsets))});
}

// (rows, indices, map, offsets, total): a packed buffer that is not cleared first (every row below offsets[E] is
// written exactly once)
PyObject *moe_dispatch(Args &a)
{
  const at::Tensor &x = *a.tensor();
  const at::Tensor &idx = *a.tensor();
  const at::Tensor &map = *a.tensor();
  const at::Tensor &offs = *a.tensor();
  const int64_t total = a.integer();
  need_matrix(x, "moe_dispatch");
  at::Tensor buf = empty({total, x.size(1)}, x.scalar_type(), x);
  const int xc = code_of(x);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_dispatch(ptr(x), xc, ints(idx), ints(map), ints(offs), ptr(buf),
                                  static_cast<int32_t>(x.size(0)), static_cast<int32_t>(x.size(1)),
                                  static_cast<int32_t>(idx.size(1)), s);
        }),
        "moe_dispatch");
  return wrap(std::move(buf));
}

PyObject *moe_combine(Args &a)
{
  const at::Tensor &buf = *a.tensor();
  const at::Tensor &idx = *a.tensor();
  const at::Tensor &wts = *a.tensor();
  const at::Tensor &map = *a.tensor();
  const at::Tensor &offs = *a.tensor();
  const int64_t tokens = a.integer();
  at::Tensor out = empty({tokens, buf.size(1)}, buf.scalar_type(), buf);
  const int bc = code_of(buf);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_combine(ptr(buf), bc, ints(idx), ptr(wts), ints(map), ints(offs), ptr(out),
                                 static_cast<int32_t>(tokens), static_cast<int32_t>(buf.size(1)),
                                 static_cast<int32_t>(idx.size(1)), s);
        }),
        "moe_combine");
  return wrap(std::move(out));
}

PyObject *moe_combine_bwd_grad_expert(Args &a)
{
  const at::Tensor &g = *a.tensor();
  const at::Tensor &idx = *a.tensor();
  const at::Tensor &wts = *a.tensor();
  const at::Tensor &map = *a.tensor();
  const at::Tensor &offs = *a.tensor();
  const int64_t total = a.integer();
  need_matrix(g, "moe_combine_bwd_grad_expert");
  at::Tensor buf = empty({total, g.size(1)}, g.scalar_type(), g);
  const int gc = code_of(g);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_combine_bwd_grad_expert(ptr(g), gc, ints(idx), ptr(wts), ints(map), ints(offs), ptr(buf),
                                                 static_cast<int32_t>(g.size(0)), static_cast<int32_t>(g.size(1)),
                                                 static_cast<int32_t>(idx.size(1)), s);
        }),
        "moe_combine_bwd_grad_expert");
  return wrap(std::move(buf));
}

PyObject *moe_combine_bwd_grad_weights(Args &a)
{
  const at::Tensor &g = *a.tensor();
  const at::Tensor &buf = *a.tensor();
  const at::Tensor &idx = *a.tensor();
  const at::Tensor &map = *a.tensor();
  const at::Tensor &offs = *a.tensor();
  need_matrix(g, "moe_combine_bwd_grad_weights");
  at::Tensor out = empty({g.size(0), idx.size(1)}, g.scalar_type(), g);
  const int gc = code_of(g);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_combine_bwd_grad_weights(ptr(g), ptr(buf), gc, ints(idx), ints(map), ints(offs), ptr(out),
                                                  static_cast<int32_t>(g.size(0)), static_cast<int32_t>(g.size(1)),
                                                  static_cast<int32_t>(idx.size(1)), s);
        }),
        "moe_combine_bwd_grad_weights");
  return wrap(std::move(out));
}

PyObject *moe_dispatch_bwd(Args &a)
{
  const at::Tensor &g = *a.tensor();
  const at::Tensor &idx = *a.tensor();
  const at::Tensor &map = *a.tensor();
  const at::Tensor &offs = *a.tensor();
  const int64_t tokens = a.integer();
  at::Tensor out = empty({tokens, g.size(1)}, g.scalar_type(), g);
  const int gc = code_of(g);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_dispatch_bwd(ptr(g), gc, ints(idx), ints(map), ints(offs), ptr(out),
                                      static_cast<int32_t>(tokens), static_cast<int32_t>(g.size(1)),
                                      static_cast<int32_t>(idx.size(1)), s);
        }),
        "moe_dispatch_bwd");
  return wrap(std::move(out));
}

PyObject *moe_router_bwd(Args &a)
{
  const at::Tensor &gw = *a.tensor();
  const at::Tensor &probs = *a.tensor();
  const at::Tensor &idx = *a.tensor();
  const at::Tensor *bias = a.tensor(true);
  const at::Tensor *zls = a.tensor(true);
  const bool sigmoid = a.truth();
  const bool normalize = a.truth();
  const float scaling = static_cast<float>(a.real());
  const bool exact = a.truth();
  need_matrix(probs, "moe_router_bwd");
  at::Tensor gl = empty_like(probs);
  at::Tensor gt = empty_like(gw);
  const int pc = code_of(probs);
  void *s = stream();
  check(unlocked([&] {
          return api.moe_router_bwd(ptr(gw), ptr(probs), ints(idx), ptr(bias), ptr(zls), ptr(gt), ptr(gl), pc,
                                    static_cast<int32_t>(probs.size(0)), static_cast<int32_t>(probs.size(1)),
                                    static_cast<int32_t>(idx.size(1)), sigmoid ? 1 : 0, normalize ? 1 : 0, scaling,
                                    exact ? 1 : 0, s);
        }),
        "moe_router_bwd");
  return pack({wrap(std::move(gl)), wrap(std::move(gt))});
}

struct Experts
{
  std::vector<caifq_weight> gate, up, down;
  bool gated;
  int32_t count;

  explicit Experts(Args &a)
  {
    gated = a.weights(gate);
    if (!a.weights(up) || !a.weights(down) || up.empty())
    {
      raise(PyExc_TypeError, "grouped experts: up and down are lists of weights");
    }
    if (down.size() < up.size() || (gated && gate.size() < up.size()))
    {
      raise(PyExc_IndexError, "grouped experts: gate, up and down have one weight per expert");
    }
    count = static_cast<int32_t>(up.size());
  }

  const caifq_weight *gates() const { return gated ? gate.data() : nullptr; }
};

// the host copy of the offsets: [experts + 1]
std::vector<int32_t> offsets_of(Args &a, const Experts &e)
{
  std::vector<int32_t> offs = a.integers();
  if (offs.size() != static_cast<size_t>(e.count) + 1)
  {
    raise(PyExc_IndexError, "grouped experts: one offset per expert and the total");
  }
  return offs;
}

PyObject *grouped_expert_expand(Args &a)
{
  Experts e(a);
  const at::Tensor &expanded = *a.tensor();
  const int dtype = static_cast<int>(a.integer());
  const int compute = static_cast<int>(a.integer());
  void *s = stream();
  check(unlocked([&] {
          return api.grouped_expert_expand(e.gates(), e.up.data(), e.down.data(), e.count, ptr(expanded), dtype, compute,
                                           s);
        }),
        "grouped_expert_expand");
  return wrap(expanded);
}

PyObject *grouped_expert_fwd(Args &a)
{
  Experts e(a);
  const std::vector<int32_t> offs = offsets_of(a, e);
  const at::Tensor &x = *a.tensor();
  const int compute = static_cast<int>(a.integer());
  const at::Tensor *expanded = a.buffer();
  const int64_t total = offs.back(), hid = e.up[0].out_dim;
  const at::ScalarType dt = x.scalar_type();
  at::Tensor out = empty({total, e.up[0].in_dim}, dt, x);
  at::Tensor gate_out = e.gated ? empty({total, hid}, dt, x) : at::Tensor();
  at::Tensor up_out = empty({total, hid}, dt, x);
  at::Tensor hidden = empty({total, hid}, dt, x);
  const int xc = code_of(x);
  void *g = e.gated ? ptr(gate_out) : nullptr;
  void *s = stream();
  check(unlocked([&] {
          return expanded != nullptr
                     ? api.grouped_expert_fwd_expanded(e.gates(), e.up.data(), e.down.data(), e.count, offs.data(), ptr(x),
                                                       ptr(out), g, ptr(up_out), ptr(hidden), ptr(expanded), xc, compute,
                                                       s)
                     : api.grouped_expert_fwd(e.gates(), e.up.data(), e.down.data(), e.count, offs.data(), ptr(x),
                                              ptr(out), g, ptr(up_out), ptr(hidden), xc, compute, s);
        }),
        expanded != nullptr ? "grouped_expert_fwd_expanded" : "grouped_expert_fwd");
  return pack({wrap(std::move(out)), wrap_or_none(gate_out), wrap(std::move(up_out))});
}

PyObject *grouped_expert_bwd(Args &a)
{
  Experts e(a);
  const std::vector<int32_t> offs = offsets_of(a, e);
  const at::Tensor &dy = *a.tensor();
  const at::Tensor *gate_out = a.tensor(true);
  const at::Tensor *up_out = a.tensor(true);
  const int compute = static_cast<int>(a.integer());
  const at::Tensor *expanded = a.buffer();
  const int64_t total = offs.back(), hid = e.up[0].out_dim;
  at::Tensor dx = empty({total, e.up[0].in_dim}, dy.scalar_type(), dy);
  at::Tensor work = empty({3, total > 0 ? total : 1, hid}, dy.scalar_type(), dy);
  const int yc = code_of(dy);
  void *s = stream();
  check(unlocked([&] {
          return expanded != nullptr
                     ? api.grouped_expert_bwd_expanded(e.gates(), e.up.data(), e.down.data(), e.count, offs.data(),
                                                       ptr(dy), ptr(gate_out), ptr(up_out), ptr(dx), ptr(work),
                                                       ptr(expanded), yc, compute, s)
                     : api.grouped_expert_bwd(e.gates(), e.up.data(), e.down.data(), e.count, offs.data(), ptr(dy),
                                              ptr(gate_out), ptr(up_out), ptr(dx), ptr(work), yc, compute, s);
        }),
        expanded != nullptr ? "grouped_expert_bwd_expanded" : "grouped_expert_bwd");
  return wrap(std::move(dx));
}

// ---- module -------------------------------------------------------------------------------------------------

template <PyObject *(*F)(Args &)>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n)
{
  try
  {
    Args a(args, n);
    return F(a);
  }
  catch (const Raised &)
  {
    return nullptr;
  }
  catch (...)
  {
    // the Python types torch's own functions raise: torch.OutOfMemoryError, IndexError, ...
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

// load(path of libcaifq.so, exception class)
PyObject *load(PyObject *, PyObject *const *args, Py_ssize_t n)
{
  if (n != 2 || !PyUnicode_Check(args[0]) || !PyExceptionClass_Check(args[1]))
  {
    PyErr_SetString(PyExc_TypeError, "load(path, exception class)");
    return nullptr;
  }
  void *lib = dlopen(PyUnicode_AsUTF8(args[0]), RTLD_NOW | RTLD_LOCAL);
  if (lib == nullptr)
  {
    PyErr_SetString(args[1], dlerror());
    return nullptr;
  }
#define CAIFQ_LOOKUP(name)                                                                    \
  api.name = reinterpret_cast<decltype(&caifq_##name)>(dlsym(lib, "caifq_" #name));           \
  if (api.name == nullptr)                                                                    \
  {                                                                                           \
    PyErr_SetString(args[1], "libcaifq.so does not export caifq_" #name);                     \
    return nullptr;                                                                           \
  }
  CAIFQ_BOUND(CAIFQ_LOOKUP)
#undef CAIFQ_LOOKUP
  Py_INCREF(args[1]);
  Py_XSETREF(g_error, args[1]);
  Py_RETURN_NONE;
}

#define CAIFQ_METHOD(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name>)), METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    {"load", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&load)), METH_FASTCALL, nullptr},
    CAIFQ_METHOD(linear_fwd),
    CAIFQ_METHOD(linear_dx),
    CAIFQ_METHOD(linear_fwd_residual),
    CAIFQ_METHOD(linear_fwd_multi),
    CAIFQ_METHOD(linear_concat),
    CAIFQ_METHOD(lora_linear_fwd),
    CAIFQ_METHOD(lora_linear_bwd),
    CAIFQ_METHOD(rmsnorm_fwd),
    CAIFQ_METHOD(rmsnorm_bwd),
    CAIFQ_METHOD(cast),
    CAIFQ_METHOD(quantize_int8_per_tensor),
    CAIFQ_METHOD(quantize_int8_per_channel),
    CAIFQ_METHOD(quantize_int4),
    CAIFQ_METHOD(moe_topk),
    CAIFQ_METHOD(moe_normalize_rows),
    CAIFQ_METHOD(moe_softmax),
    CAIFQ_METHOD(moe_build_dispatch),
    CAIFQ_METHOD(moe_dispatch),
    CAIFQ_METHOD(moe_combine),
    CAIFQ_METHOD(moe_combine_bwd_grad_expert),
    CAIFQ_METHOD(moe_combine_bwd_grad_weights),
    CAIFQ_METHOD(moe_dispatch_bwd),
    CAIFQ_METHOD(moe_router_bwd),
    CAIFQ_METHOD(grouped_expert_expand),
    CAIFQ_METHOD(grouped_expert_fwd),
    CAIFQ_METHOD(grouped_expert_bwd),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding(void) { return PyModule_Create(&module); }
