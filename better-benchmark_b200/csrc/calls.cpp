// The host side of the most frequent calls in native code: argument checks, output tensors and the call of the C ABI's
// entry point in one step. kernels.py tries these functions first; a function that is handed anything but the usual form (a
// tensor subclass, a CPU tensor, another device, a dtype or layout that it does not handle, an empty tensor, an argument
// that is wrong) returns None without having done anything, and the Python code of that wrapper, which holds every rule and
// raises every error, takes the call.
//
// Why: a launch takes 2.5 us of host time, but a wrapper in Python took 7 us for a cast and 13 to 24 us for the calls with
// more operands, most of it in the shape arithmetic and in allocating outputs from Python, so that every tensor of less
// than some tens of MB waited for the host. us a call on tiny tensors, there and here: cast 7.1 / 4.5, row sum 11.4 / 4.0,
// LayerNorm forward 16.4 / 6.7, residual LayerNorm 24.1 / 6.4, norm backward 19.0 / 6.7, masked softmax 19.1 / 4.5, transpose 15.6 / 4.7,
// BatchNorm channels-last (three launches) forward 22.7 / 11.3, backward 24.0 / 10.8.
//
// Outputs come from at::empty / at::empty_strided through the dispatcher, as torch.empty_like's do: dispatch modes, deterministic
// filling and the allocator's rules for streams and captures apply to them unchanged. With a torch function mode active, which would
// have seen the Python calls, every function returns None. The interpreter lock is released while tensors are
// allocated and kernels launched. The library's entry points are handed over as addresses (bind), so that this module
// works with whichever build of the library the process has loaded.
#include <Python.h>

#include <ATen/Functions.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200_oracles.h"

namespace {

constexpr int kMaxDims = 8;

// ---- what bind() hands over ------------------------------------------------------------------------
struct Library {
  decltype(&b200_row_reduce) row_reduce = nullptr;
  decltype(&b200_softmax) softmax = nullptr;
  decltype(&b200_norm_fwd_residual) norm_fwd_residual = nullptr;
  decltype(&b200_norm_bwd) norm_bwd = nullptr;
  decltype(&b200_norm_bwd_scratch_bytes) norm_bwd_scratch_bytes = nullptr;
  decltype(&b200_batch_norm_fwd_ex) batch_norm_fwd = nullptr;
  decltype(&b200_batch_norm_scratch_bytes) batch_norm_scratch_bytes = nullptr;
  decltype(&b200_batch_norm_bwd_ex) batch_norm_bwd = nullptr;
  decltype(&b200_batch_norm_bwd_scratch_bytes) batch_norm_bwd_scratch_bytes = nullptr;
  decltype(&b200_transpose_copy) transpose_copy = nullptr;
  decltype(&b200_permute_copy) permute_copy = nullptr;
  decltype(&b200_cast_scale) cast_scale = nullptr;
};
Library lib;
PyObject* check_status = nullptr;        // native.check: raises what a status other than 0 stands for
PyObject* scratch_by_device = nullptr;   // kernels._scratch_by_device

struct NoLock {  // the interpreter lock is another thread's meanwhile
  PyThreadState* state = PyEval_SaveThread();
  ~NoLock() { PyEval_RestoreThread(state); }
};

// ---- arguments -------------------------------------------------------------------------------------
int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? 0 : t == at::kBFloat16 ? 1 : t == at::kHalf ? 2 : -1;
}

struct Args {
  bool fits = lib.cast_scale != nullptr && !at::impl::torch_function_mode_enabled();
  int device = -1;

  // A plain strided CUDA tensor on the device of the others; nullptr (and no longer fits) for anything else.
  const at::Tensor* tensor(PyObject* o) {
    if (!fits || !THPVariable_CheckExact(o)) return reject();
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_neg() ||
        t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::Functionalize})) ||
        dtype_code(t.scalar_type()) < 0 || t.dim() > kMaxDims)
      return reject();
    if (device < 0) device = t.get_device();
    return t.get_device() == device ? &t : reject();
  }
  const at::Tensor* optional(PyObject* o) { return o == Py_None ? nullptr : tensor(o); }
  // The scalar type of a torch.dtype, or `otherwise` for None.
  at::ScalarType dtype(PyObject* o, at::ScalarType otherwise) {
    if (o == Py_None) return otherwise;
    if (!THPDtype_Check(o)) {
      fits = false;
      return otherwise;
    }
    const at::ScalarType t = reinterpret_cast<THPDtype*>(o)->scalar_type;
    if (dtype_code(t) < 0) fits = false;
    return t;
  }
  double number(PyObject* o, double otherwise) {
    if (o == Py_None) return otherwise;
    if (PyFloat_Check(o)) return PyFloat_AS_DOUBLE(o);
    if (!PyLong_Check(o)) fits = false;
    const double v = fits ? PyLong_AsDouble(o) : 0.0;
    if (PyErr_Occurred()) {
      PyErr_Clear();
      fits = false;
    }
    return v;
  }
  int64_t integer(PyObject* o) {
    if (!PyLong_Check(o)) fits = false;
    const int64_t v = fits ? PyLong_AsLongLong(o) : 0;
    if (PyErr_Occurred()) {
      PyErr_Clear();
      fits = false;
    }
    return v;
  }
  bool flag(PyObject* o) {
    if (o != Py_True && o != Py_False) fits = false;
    return o == Py_True;
  }
  // A list or tuple of at most kMaxDims integers; with `numel` >= 0 one of them may be -1, and they multiply to it.
  int shape(PyObject* o, int64_t (&out)[kMaxDims], int64_t numel = -1) {
    if (!fits || !(PyList_Check(o) || PyTuple_Check(o))) return reject(), 0;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
    if (n > kMaxDims) return reject(), 0;
    int64_t known = 1;
    int open = -1;
    for (Py_ssize_t i = 0; i < n && fits; ++i) {
      out[i] = integer(PySequence_Fast_GET_ITEM(o, i));
      if (numel < 0) continue;
      if (out[i] == -1 && open < 0) open = (int)i;
      else if (out[i] < 1 || out[i] > numel / known) fits = false;
      else known *= out[i];
    }
    if (numel >= 0 && fits) {
      if (open >= 0) {
        if (numel % known != 0) fits = false;
        else out[open] = numel / known;
      } else if (known != numel) {
        fits = false;
      }
    }
    return (int)n;
  }
  // All tensors are on the current device.
  bool ready() { return fits && device >= 0 && c10::cuda::current_device() == device; }
  void* stream() const { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

 private:
  const at::Tensor* reject() {
    fits = false;
    return nullptr;
  }
};

void* address(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }
void* address(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* floats(const at::Tensor& t) { return static_cast<float*>(address(t)); }

at::Tensor make(const at::Tensor& like, at::IntArrayRef sizes, at::ScalarType type) {
  return at::empty(sizes, like.options().dtype(type));
}
// With the strides of `like`, which is dense.
at::Tensor make_alike(const at::Tensor& like, at::ScalarType type) {
  return at::empty_strided(like.sizes(), like.strides(), like.options().dtype(type));
}

bool channels_last(const at::Tensor& t) { return t.dim() == 4 && t.is_contiguous(at::MemoryFormat::ChannelsLast); }
bool plainly_dense(const at::Tensor& t) { return t.is_contiguous() || channels_last(t); }
bool vector_of(const at::Tensor* t, int64_t n) { return t->dim() == 1 && t->size(0) == n && t->is_contiguous(); }
bool fp32_values(const at::Tensor* t, int64_t n) {
  return t->scalar_type() == at::kFloat && t->numel() == n && t->is_contiguous();
}

// Dimensions that every operand steps through as one are one (collapse_outer and _collapse_all of kernels.py). Returns how many remain.
template <int OPERANDS>
int collapse(int count, const int64_t* sizes, const int64_t (&strides)[OPERANDS][kMaxDims], int64_t (&dims)[kMaxDims],
             int64_t (&steps)[OPERANDS][kMaxDims]) {
  int n = 0;
  for (int i = 0; i < count; ++i) {
    if (sizes[i] == 1) continue;
    bool joins = n > 0;
    for (int k = 0; k < OPERANDS; ++k) joins = joins && steps[k][n - 1] == strides[k][i] * sizes[i];
    if (joins) {
      dims[n - 1] *= sizes[i];
    } else {
      dims[n++] = sizes[i];
    }
    for (int k = 0; k < OPERANDS; ++k) steps[k][n - 1] = strides[k][i];
  }
  for (int i = n; i < kMaxDims; ++i) {
    dims[i] = 1;
    for (int k = 0; k < OPERANDS; ++k) steps[k][i] = 0;
  }
  return n;
}

// The shared scratch buffer of the device when it holds `bytes`; otherwise nothing (the Python code makes a larger one).
at::Tensor shared_scratch(int device, int64_t bytes) {
  static PyObject* keys[64] = {nullptr};
  if (device >= 64) return {};
  if (!keys[device]) keys[device] = Py_BuildValue("(si)", "cuda", device);
  PyObject* buffers = keys[device] ? PyDict_GetItemWithError(scratch_by_device, keys[device]) : nullptr;
  if (!buffers) {
    PyErr_Clear();
    return {};
  }
  if (!PyList_Check(buffers) || PyList_GET_SIZE(buffers) == 0) return {};
  PyObject* last = PyList_GET_ITEM(buffers, PyList_GET_SIZE(buffers) - 1);
  if (!THPVariable_Check(last)) return {};
  const at::Tensor& t = THPVariable_Unpack(last);
  return t.numel() >= bytes ? t : at::Tensor();
}
// A caller's own buffer, of any dtype.
at::Tensor own_scratch(Args& a, PyObject* o) {
  if (!THPVariable_CheckExact(o)) {
    a.fits = false;
    return {};
  }
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || !t.has_storage() || t.get_device() != a.device) {
    a.fits = false;
    return {};
  }
  return t;
}

// ---- results ---------------------------------------------------------------------------------------
bool failed(int status, const char* what) {
  if (status == 0) return false;
  PyObject* r = PyObject_CallFunction(check_status, "is", status, what);
  Py_XDECREF(r);  // check raises
  return true;
}
PyObject* wrapped(const at::Tensor& t) {
  if (t.defined()) return THPVariable_Wrap(t);
  Py_RETURN_NONE;
}
template <typename... Tensors>
PyObject* wrapped_tuple(const Tensors&... t) {
  PyObject* out = PyTuple_New(sizeof...(t));
  if (!out) return nullptr;
  Py_ssize_t i = 0;
  bool ok = true;
  auto put = [&](const at::Tensor& v) {
    PyObject* o = wrapped(v);
    ok = ok && o != nullptr;
    PyTuple_SET_ITEM(out, i++, o);
  };
  (put(t), ...);
  if (ok) return out;
  Py_DECREF(out);
  return nullptr;
}

// ---- the calls -------------------------------------------------------------------------------------
#define B200_CALL(name, arguments)                                      \
  PyObject* name(PyObject*, PyObject* const* v, Py_ssize_t count) {     \
    HANDLE_TH_ERRORS                                                    \
    if (count != (arguments)) {                                         \
      PyErr_SetString(PyExc_TypeError, #name ": wrong argument count"); \
      return nullptr;                                                   \
    }                                                                   \
    Args a;
#define B200_CALL_END   \
    END_HANDLE_TH_ERRORS \
  }

// row_reduce(x, op code, keepdim, out_dtype)
B200_CALL(row_reduce, 4)
  const at::Tensor* x = a.tensor(v[0]);
  const int64_t op = a.integer(v[1]);
  const bool keepdim = a.flag(v[2]);
  if (!a.fits || x->dim() < 1 || op < 0) Py_RETURN_NONE;
  const at::ScalarType type = a.dtype(v[3], x->scalar_type());
  const int outer = (int)x->dim() - 1;
  const int64_t n = x->size(outer);
  if (!a.ready() || x->numel() == 0 || (n > 1 && x->stride(outer) != 1)) Py_RETURN_NONE;
  int64_t strides[1][kMaxDims], dims[kMaxDims], steps[1][kMaxDims], shape[kMaxDims];
  for (int i = 0; i < outer; ++i) {
    strides[0][i] = x->stride(i);
    shape[i] = x->size(i);
  }
  shape[outer] = 1;
  if (collapse<1>(outer, shape, strides, dims, steps) > 3) Py_RETURN_NONE;
  at::Tensor out;
  int status;
  {
    NoLock no_lock;
    out = make(*x, at::IntArrayRef(shape, outer + (keepdim ? 1 : 0)), type);
    status = lib.row_reduce(address(x), address(out), x->numel() / n, n, dims[1], dims[2], steps[0], 1,
                            dtype_code(x->scalar_type()), dtype_code(type), (int)op, a.stream());
  }
  return failed(status, "b200_row_reduce") ? nullptr : wrapped(out);
B200_CALL_END

// softmax(x, mask, scale, log, out_dtype, round_intermediates)
B200_CALL(softmax, 6)
  const at::Tensor* x = a.tensor(v[0]);
  const at::Tensor* mask = a.optional(v[1]);
  const double scale = a.number(v[2], 1.0);
  const bool log = a.flag(v[3]), round = a.flag(v[5]);
  if (!a.fits || x->dim() < 1) Py_RETURN_NONE;
  const at::ScalarType type = a.dtype(v[4], x->scalar_type());
  const int outer = (int)x->dim() - 1;
  const int64_t n = x->size(outer);
  if (!a.ready() || x->numel() == 0 || (n > 1 && x->stride(outer) != 1)) Py_RETURN_NONE;
  const bool alike = plainly_dense(*x);  // the result has x's strides
  if (!alike && x->is_non_overlapping_and_dense()) Py_RETURN_NONE;
  int64_t sizes[kMaxDims], strides[3][kMaxDims], dims[kMaxDims], steps[3][kMaxDims];
  int64_t contiguous = n;
  for (int i = outer - 1; i >= 0; --i) {
    sizes[i] = x->size(i);
    strides[0][i] = x->stride(i);
    strides[1][i] = alike ? x->stride(i) : contiguous;
    strides[2][i] = 0;
    contiguous *= sizes[i];
  }
  if (mask) {
    if (mask->scalar_type() != x->scalar_type() || mask->dim() < 1 || mask->dim() > x->dim()) Py_RETURN_NONE;
    const int md = (int)mask->dim() - 1, shift = outer - md;
    if (mask->size(md) != n || (n > 1 && mask->stride(md) != 1)) Py_RETURN_NONE;
    for (int i = 0; i < md; ++i) {
      if (mask->size(i) == sizes[shift + i]) strides[2][shift + i] = mask->stride(i);
      else if (mask->size(i) != 1) Py_RETURN_NONE;
    }
  }
  int count_dims;
  if (mask) {
    count_dims = collapse<3>(outer, sizes, strides, dims, steps);
  } else {
    int64_t two[2][kMaxDims], two_steps[2][kMaxDims];
    for (int i = 0; i < outer; ++i) {
      two[0][i] = strides[0][i];
      two[1][i] = strides[1][i];
    }
    count_dims = collapse<2>(outer, sizes, two, dims, two_steps);
    for (int i = 0; i < 3; ++i) {
      steps[0][i] = two_steps[0][i];
      steps[1][i] = two_steps[1][i];
    }
  }
  if (count_dims > 3) Py_RETURN_NONE;
  const int flags = (log ? 1 : 0) | (v[2] != Py_None ? 2 : 0) | (round && x->scalar_type() != at::kFloat ? 4 : 0);
  at::Tensor out;
  int status;
  {
    NoLock no_lock;
    out = alike ? make_alike(*x, type) : make(*x, x->sizes(), type);
    status = lib.softmax(address(x), address(mask), address(out), x->numel() / n, n, dims[1], dims[2], steps[0],
                         mask ? steps[2] : nullptr, steps[1], dtype_code(x->scalar_type()), dtype_code(type), scale, flags,
                         a.stream());
  }
  return failed(status, "b200_softmax") ? nullptr : wrapped(out);
B200_CALL_END

// norm_fwd(x, weight, bias, eps, rms, out_dtype, want_y, want_mean, want_rstd, want_var, correction, keepdim, prologue code,
//          residual, want_sum, form of the sum, shapes, y in the second): the shapes are None, or two that x fits; it is (and with it the
//          residual, the sum and the statistics are) seen as the first, y as the first or the second.
B200_CALL(norm_fwd, 18)
  const at::Tensor* x = a.tensor(v[0]);
  const at::Tensor* weight = a.optional(v[1]);
  const at::Tensor* bias = a.optional(v[2]);
  const at::Tensor* residual = a.optional(v[13]);
  const double eps = a.number(v[3], 0.0), correction = a.number(v[10], 0.0);
  const bool rms = a.flag(v[4]), want_y = a.flag(v[6]), want_mean = a.flag(v[7]), want_rstd = a.flag(v[8]), want_var = a.flag(v[9]),
             keepdim = a.flag(v[11]), want_sum = a.flag(v[14]);
  const int64_t prologue = a.integer(v[12]), form = a.integer(v[15]);
  if (!a.fits || x->dim() < 1 || prologue < 0 || form < 0 || v[3] == Py_None || v[10] == Py_None) Py_RETURN_NONE;
  const at::ScalarType type = a.dtype(v[5], x->scalar_type());
  int xd = (int)x->dim(), second = 0;
  int64_t xs[kMaxDims], second_shape[kMaxDims];
  const int64_t numel = x->numel();
  const bool in_second = a.flag(v[17]);
  if (v[16] != Py_None) {
    if (!x->is_contiguous() || !PyTuple_Check(v[16]) || PyTuple_GET_SIZE(v[16]) != 2) Py_RETURN_NONE;
    xd = a.shape(PyTuple_GET_ITEM(v[16], 0), xs, numel);
    second = a.shape(PyTuple_GET_ITEM(v[16], 1), second_shape, numel);
  } else {
    for (int i = 0; i < xd; ++i) xs[i] = x->size(i);
  }
  if (!a.ready() || numel == 0 || xd < 1) Py_RETURN_NONE;
  const int64_t n = xs[xd - 1], rows = numel / n;
  int64_t stride = n;
  if (!x->is_contiguous()) {  // rows of a matrix at one distance
    if (x->dim() != 2 || residual || (n > 1 && x->stride(1) != 1)) Py_RETURN_NONE;
    if (rows > 1) stride = x->stride(0);
  }
  if (residual && (residual->scalar_type() != x->scalar_type() || !residual->is_contiguous() || residual->numel() != numel ||
                   type != x->scalar_type() ||
                   (v[16] == Py_None && (residual->sizes() != x->sizes() || residual->strides() != x->strides()))))
    Py_RETURN_NONE;
  if (want_sum && !residual) Py_RETURN_NONE;
  if ((weight && !vector_of(weight, n)) || (bias && !vector_of(bias, n))) Py_RETURN_NONE;
  if (weight && bias && weight->scalar_type() != bias->scalar_type()) Py_RETURN_NONE;
  const int w_code = bias ? dtype_code(bias->scalar_type()) : weight ? dtype_code(weight->scalar_type()) : 0;
  const int mode = (rms ? 1 : 0) | (int)prologue | (residual ? (int)form : 0);
  at::Tensor y, mean, rstd, var, sum;
  int status;
  {
    NoLock no_lock;
    int64_t ss[kMaxDims];
    for (int i = 0; i < xd; ++i) ss[i] = xs[i];
    ss[xd - 1] = 1;
    const at::IntArrayRef stat(ss, keepdim ? xd : xd - 1);
    if (want_y) y = make(*x, in_second ? at::IntArrayRef(second_shape, second) : at::IntArrayRef(xs, xd), type);
    if (want_mean && !rms) mean = make(*x, stat, at::kFloat);
    if (want_rstd) rstd = make(*x, stat, at::kFloat);
    if (want_var) var = make(*x, stat, at::kFloat);
    if (want_sum) sum = make(*x, at::IntArrayRef(xs, xd), x->scalar_type());
    status = lib.norm_fwd_residual(address(x), address(residual), address(sum), address(weight), address(bias), address(y),
                                   floats(mean), floats(rstd), floats(var), rows, n, stride, n, dtype_code(x->scalar_type()),
                                   w_code, dtype_code(type), eps, correction, mode, a.stream());
  }
  if (failed(status, residual ? "b200_norm_fwd_residual" : "b200_norm_fwd")) return nullptr;
  return want_sum ? wrapped_tuple(y, mean, rstd, var, sum) : wrapped_tuple(y, mean, rstd, var);
B200_CALL_END

// norm_bwd(x, dy, weight, rstd, mean, rms, heads, want_dweight, want_dbias, two_launch, scratch)
B200_CALL(norm_bwd, 11)
  const at::Tensor* x = a.tensor(v[0]);
  const at::Tensor* dy = a.tensor(v[1]);
  const at::Tensor* weight = a.optional(v[2]);
  const at::Tensor* rstd = a.tensor(v[3]);
  const at::Tensor* mean = a.optional(v[4]);
  const bool rms = a.flag(v[5]), want_dw = a.flag(v[7]), want_db = a.flag(v[8]) && !rms, two_launch = a.flag(v[9]);
  const int64_t heads = v[6] == Py_None ? 0 : a.integer(v[6]);
  // one element of dy may stand for all: left to the general code, as are rows that are not contiguous
  if (!a.ready() || x->dim() < 1 || x->numel() < 2 || x->scalar_type() != dy->scalar_type() || x->sizes() != dy->sizes() ||
      !x->is_contiguous() || !dy->is_contiguous())
    Py_RETURN_NONE;
  int64_t n = x->size(x->dim() - 1), seq = 1, head_dim = n, batch_step = n, seq_step = 0, head_step = n;
  int64_t shape[4];
  if (v[6] != Py_None) {
    if (x->dim() != 4 || heads < 1 || x->size(2) != heads) Py_RETURN_NONE;
    const int64_t b = x->size(0), s = x->size(1), d = n;
    n = heads * d;
    seq = s, head_dim = d, batch_step = n * s, seq_step = d, head_step = s * d;
    shape[0] = b, shape[1] = heads, shape[2] = s, shape[3] = d;
  }
  const int64_t rows = x->numel() / n;
  if (!fp32_values(rstd, rows) || (!rms && (!mean || !fp32_values(mean, rows))) || (weight && !vector_of(weight, n))) Py_RETURN_NONE;
  at::Tensor scratch;
  if (want_dw || want_db) {
    scratch = v[10] == Py_None ? shared_scratch(a.device, lib.norm_bwd_scratch_bytes(n)) : own_scratch(a, v[10]);
    if (!scratch.defined()) Py_RETURN_NONE;
  } else if (v[10] != Py_None && !own_scratch(a, v[10]).defined()) {
    Py_RETURN_NONE;
  }
  at::Tensor dx, dw, db;
  int status;
  {
    NoLock no_lock;
    dx = make(*x, heads ? at::IntArrayRef(shape, 4) : x->sizes(), x->scalar_type());
    if (want_dw) dw = make(*x, {n}, at::kFloat);
    if (want_db) db = make(*x, {n}, at::kFloat);
    status = lib.norm_bwd(address(x), address(dy), address(weight), static_cast<const float*>(address(mean)),
                          static_cast<const float*>(address(rstd)), address(dx), floats(dw), floats(db), rows, n, n, n,
                          dtype_code(x->scalar_type()), weight ? dtype_code(weight->scalar_type()) : 0, rms ? 1 : 0, seq, head_dim,
                          batch_step, seq_step, head_step, address(scratch),
                          scratch.defined() ? scratch.numel() * scratch.element_size() : 0, two_launch ? 1 : 0, a.stream());
  }
  return failed(status, "b200_norm_bwd") ? nullptr : wrapped_tuple(dx, dw, db);
B200_CALL_END

// The [N, C, H, W] geometry of a dense NCHW or channels-last tensor; false where H and W are not one strided dimension.
bool image(const at::Tensor& x, int64_t& spatial_stride) {
  if (x.dim() != 4 || x.numel() == 0 || !plainly_dense(x)) return false;
  const int64_t h = x.size(2), w = x.size(3), sh = x.stride(2), sw = x.stride(3);
  if (h > 1 && w > 1 && sh != w * sw) return false;
  spatial_stride = w > 1 ? sw : h > 1 ? sh : 1;
  return true;
}

// batch_norm_fwd(x, weight, bias, running_mean, running_var, eps, momentum, relu, unbiased_factor, scratch)
B200_CALL(batch_norm_fwd, 10)
  const at::Tensor* x = a.tensor(v[0]);
  const at::Tensor* weight = a.optional(v[1]);
  const at::Tensor* bias = a.optional(v[2]);
  const at::Tensor* running_mean = a.optional(v[3]);
  const at::Tensor* running_var = a.optional(v[4]);
  const double eps = a.number(v[5], 0.0), momentum = a.number(v[6], 0.0), factor = a.number(v[8], 0.0);
  const bool relu = a.flag(v[7]);
  int64_t ss;
  if (!a.ready() || v[5] == Py_None || v[6] == Py_None || !image(*x, ss)) Py_RETURN_NONE;
  const int64_t c = x->size(1);
  if ((weight && !vector_of(weight, c)) || (bias && !vector_of(bias, c))) Py_RETURN_NONE;
  if (weight && bias && weight->scalar_type() != bias->scalar_type()) Py_RETURN_NONE;
  for (const at::Tensor* t : {running_mean, running_var})
    if (t && !(t->dim() == 1 && fp32_values(t, c))) Py_RETURN_NONE;
  const at::Tensor scratch =
      v[9] == Py_None ? shared_scratch(a.device, lib.batch_norm_scratch_bytes(c)) : own_scratch(a, v[9]);
  if (!scratch.defined()) Py_RETURN_NONE;
  at::Tensor y, mean, invstd;
  int status;
  {
    NoLock no_lock;
    y = make_alike(*x, x->scalar_type());
    mean = make(*x, {c}, at::kFloat);
    invstd = make(*x, {c}, at::kFloat);
    status = lib.batch_norm_fwd(address(x), address(y), address(weight), address(bias), static_cast<float*>(address(running_mean)),
                                static_cast<float*>(address(running_var)), floats(mean), floats(invstd), x->size(0), c,
                                x->size(2) * x->size(3), x->stride(0), x->stride(1), ss, dtype_code(x->scalar_type()),
                                bias ? dtype_code(bias->scalar_type()) : weight ? dtype_code(weight->scalar_type()) : 0, eps,
                                momentum, factor, relu ? 1 : 0, address(scratch), scratch.numel() * scratch.element_size(),
                                a.stream());
  }
  return failed(status, "b200_batch_norm_fwd") ? nullptr : wrapped_tuple(y, mean, invstd);
B200_CALL_END

// batch_norm_bwd(dy, x, mean, invstd, weight, act, slope, want_dx, inv_count, scratch)
B200_CALL(batch_norm_bwd, 10)
  const at::Tensor* dy = a.tensor(v[0]);
  const at::Tensor* x = a.tensor(v[1]);
  const at::Tensor* mean = a.tensor(v[2]);
  const at::Tensor* invstd = a.tensor(v[3]);
  const at::Tensor* weight = a.optional(v[4]);
  const at::Tensor* act = a.optional(v[5]);
  const double slope = a.number(v[6], 0.0), inv_count = a.number(v[8], 0.0);
  const bool want_dx = a.flag(v[7]);
  int64_t ss;
  if (!a.ready() || v[6] == Py_None || !image(*x, ss)) Py_RETURN_NONE;
  for (const at::Tensor* t : {dy, act})
    if (t && (t->scalar_type() != x->scalar_type() || t->sizes() != x->sizes() || t->strides() != x->strides())) Py_RETURN_NONE;
  const int64_t c = x->size(1);
  if (!fp32_values(mean, c) || !fp32_values(invstd, c) || (weight && !vector_of(weight, c))) Py_RETURN_NONE;
  const at::Tensor scratch =
      v[9] == Py_None ? shared_scratch(a.device, lib.batch_norm_bwd_scratch_bytes(c) + 256) : own_scratch(a, v[9]);
  if (!scratch.defined()) Py_RETURN_NONE;
  // behind the 256 bytes that the norm backward keeps at zero
  const int64_t bytes = scratch.numel() * scratch.element_size() - 256;
  at::Tensor dx, dw, db;
  int status;
  {
    NoLock no_lock;
    if (want_dx) dx = make_alike(*x, x->scalar_type());
    dw = make(*x, {c}, at::kFloat);
    db = make(*x, {c}, at::kFloat);
    status = lib.batch_norm_bwd(address(dy), address(x), address(act), static_cast<const float*>(address(mean)),
                                static_cast<const float*>(address(invstd)), address(weight), address(dx), floats(dw), floats(db),
                                x->size(0), c, x->size(2) * x->size(3), x->stride(0), x->stride(1), ss,
                                dtype_code(x->scalar_type()), weight ? dtype_code(weight->scalar_type()) : 0, slope, inv_count,
                                static_cast<char*>(address(scratch)) + 256, bytes > 0 ? bytes : 0, a.stream());
  }
  return failed(status, "b200_batch_norm_bwd") ? nullptr : wrapped_tuple(dx, dw, db);
B200_CALL_END

// permute_copy(x, dims, scale, out_dtype, shape of the result): the shape is None, or what the result is to be seen as.
B200_CALL(permute_copy, 5)
  const at::Tensor* x = a.tensor(v[0]);
  const double scale = a.number(v[2], 1.0);
  if (!a.fits) Py_RETURN_NONE;
  const at::ScalarType type = a.dtype(v[3], x->scalar_type());
  int64_t order[kMaxDims], sizes[kMaxDims], strides[1][kMaxDims], dims[kMaxDims], steps[1][kMaxDims], shape[kMaxDims];
  const int nd = a.shape(v[1], order);
  if (!a.ready() || nd != x->dim() || nd < 1 || x->numel() == 0) Py_RETURN_NONE;
  unsigned seen = 0;
  for (int i = 0; i < nd; ++i) {
    if (order[i] < 0 || order[i] >= nd || (seen >> order[i] & 1u)) Py_RETURN_NONE;
    seen |= 1u << order[i];
    sizes[i] = x->size(order[i]);
    strides[0][i] = x->stride(order[i]);
  }
  int out_dims = nd;
  if (v[4] != Py_None) {
    out_dims = a.shape(v[4], shape, x->numel());
    if (!a.fits) Py_RETURN_NONE;
  } else {
    for (int i = 0; i < nd; ++i) shape[i] = sizes[i];
  }
  int m = collapse<1>(nd, sizes, strides, dims, steps);
  if (m == 0) {
    m = 1;
    steps[0][0] = 1;
  }
  if (m > 4) Py_RETURN_NONE;
  const int64_t* st = steps[0];
  const int in = dtype_code(x->scalar_type()), out_code = dtype_code(type), has_scale = v[2] != Py_None ? 1 : 0;
  const bool transpose = m >= 2 && m <= 3 && st[m - 2] == 1 && st[m - 1] != 1;
  at::Tensor out;
  int status;
  {
    NoLock no_lock;
    out = make(*x, at::IntArrayRef(shape, out_dims), type);
    if (transpose) {  // [..., P, C] -> [..., C, P]: output [batch, cols, rows], input [batch, rows, cols]
      status = lib.transpose_copy(address(x), address(out), m == 3 ? dims[0] : 1, dims[m - 1], dims[m - 2], m == 3 ? st[0] : 0,
                                  st[m - 1], in, out_code, scale, has_scale, a.stream());
    } else {
      int64_t shape4[4], strides4[4];
      for (int i = 0; i < 4; ++i) {
        const int from = i - (4 - m);
        shape4[i] = from < 0 ? 1 : dims[from];
        strides4[i] = from < 0 ? 0 : st[from];
      }
      status = lib.permute_copy(address(x), address(out), shape4, strides4, in, out_code, scale, has_scale, a.stream());
    }
  }
  return failed(status, transpose ? "b200_transpose_copy" : "b200_permute_copy") ? nullptr : wrapped(out);
B200_CALL_END

// cast_scale(x, out_dtype, scale, activation code)
B200_CALL(cast_scale, 4)
  const at::Tensor* x = a.tensor(v[0]);
  const double scale = a.number(v[2], 1.0);
  const int64_t activation = a.integer(v[3]);
  if (!a.fits || v[1] == Py_None || activation < 0) Py_RETURN_NONE;
  const at::ScalarType type = a.dtype(v[1], x->scalar_type());
  if (!a.ready() || x->numel() == 0 || !plainly_dense(*x)) Py_RETURN_NONE;
  at::Tensor out;
  int status;
  {
    NoLock no_lock;
    out = make_alike(*x, type);
    status = lib.cast_scale(address(x), address(out), x->numel(), dtype_code(x->scalar_type()), dtype_code(type), scale,
                            (v[2] != Py_None ? 1 : 0) | (int)activation, a.stream());
  }
  return failed(status, "b200_cast_scale") ? nullptr : wrapped(out);
B200_CALL_END

// bind({entry point: address}, check, scratch buffers by device)
PyObject* bind(PyObject*, PyObject* const* v, Py_ssize_t count) {
  if (count != 3 || !PyDict_Check(v[0]) || !PyDict_Check(v[2])) {
    PyErr_SetString(PyExc_TypeError, "bind: wrong arguments");
    return nullptr;
  }
  Library l;
  auto set = [&](const char* name, auto& slot) {
    PyObject* o = PyDict_GetItemString(v[0], name);
    void* p = o ? PyLong_AsVoidPtr(o) : nullptr;
    if (!p && !PyErr_Occurred()) PyErr_Format(PyExc_KeyError, "bind: no address of %s", name);
    slot = reinterpret_cast<std::decay_t<decltype(slot)>>(p);
    return p != nullptr;
  };
  if (!set("b200_row_reduce", l.row_reduce) || !set("b200_softmax", l.softmax) ||
      !set("b200_norm_fwd_residual", l.norm_fwd_residual) || !set("b200_norm_bwd", l.norm_bwd) ||
      !set("b200_norm_bwd_scratch_bytes", l.norm_bwd_scratch_bytes) || !set("b200_batch_norm_fwd_ex", l.batch_norm_fwd) ||
      !set("b200_batch_norm_scratch_bytes", l.batch_norm_scratch_bytes) || !set("b200_batch_norm_bwd_ex", l.batch_norm_bwd) ||
      !set("b200_batch_norm_bwd_scratch_bytes", l.batch_norm_bwd_scratch_bytes) || !set("b200_transpose_copy", l.transpose_copy) ||
      !set("b200_permute_copy", l.permute_copy) || !set("b200_cast_scale", l.cast_scale))
    return nullptr;
  Py_INCREF(v[1]);
  Py_INCREF(v[2]);
  Py_XDECREF(check_status);
  Py_XDECREF(scratch_by_device);
  check_status = v[1];
  scratch_by_device = v[2];
  lib = l;
  Py_RETURN_NONE;
}

#define B200_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {B200_METHOD(bind),           B200_METHOD(row_reduce),   B200_METHOD(softmax),
                         B200_METHOD(norm_fwd),       B200_METHOD(norm_bwd),     B200_METHOD(batch_norm_fwd),
                         B200_METHOD(batch_norm_bwd), B200_METHOD(permute_copy), B200_METHOD(cast_scale),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "b200_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b200_calls() { return PyModule_Create(&module); }
