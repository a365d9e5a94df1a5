// Python bindings of the C ABI (ss_conv/_host): what bounds a layer of a few thousand rows is the host that queues
// its kernels, and half of that was the conversion of arguments by ctypes (5 us for a call of twenty), the look at
// every tensor from Python and torch.empty (2 us).  A call through here converts its arguments by the C types
// of the header: pointers from CUDA tensors, integers, None or buffers (ctypes arrays); numbers from Python numbers.
// The interpreter lock is released during the call.
#include <torch/csrc/Device.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ops/empty.h>

#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/ssconv_b200.h"

namespace {

// Device pointer of a contiguous CUDA tensor; nullptr with a Python error otherwise.
bool tensor_pointer(const at::Tensor &t, void *&out) {
  if (!t.is_cuda()) {
    const std::string where = c10::DeviceTypeName(t.device().type(), true);
    PyErr_Format(PyExc_RuntimeError, "ssconv_b200 runs on CUDA tensors only (got a %s tensor)", where.c_str());
    return false;
  }
  if (!t.is_contiguous()) {
    PyErr_SetString(PyExc_ValueError, "tensor must be contiguous");
    return false;
  }
  out = t.data_ptr();
  return true;
}

template <typename T, typename = void>
struct Arg;

template <typename T>
struct Arg<T, std::enable_if_t<std::is_integral_v<T>>> {
  T value = 0;
  bool take(PyObject *o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) return false;
    value = (T)v;
    if ((long long)value != v) {
      PyErr_SetString(PyExc_OverflowError, "argument does not fit the C type");
      return false;
    }
    return true;
  }
};

template <typename T>
struct Arg<T, std::enable_if_t<std::is_floating_point_v<T>>> {
  T value = 0;
  bool take(PyObject *o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return false;
    value = (T)v;
    return true;
  }
};

template <typename T>
struct Arg<T, std::enable_if_t<std::is_pointer_v<T>>> {
  T value = nullptr;
  Py_buffer view{};
  bool held = false;
  bool take(PyObject *o) {
    void *p = nullptr;
    if (o == Py_None) {
    } else if (PyLong_Check(o)) {
      p = PyLong_AsVoidPtr(o);
      if (p == nullptr && PyErr_Occurred()) return false;
    } else if (THPVariable_Check(o)) {
      if (!tensor_pointer(THPVariable_Unpack(o), p)) return false;
    } else {
      if (PyObject_GetBuffer(o, &view, PyBUF_FORMAT | PyBUF_ND) != 0) return false;
      held = true;
      // a ctypes.c_void_p is the pointer, any other buffer (arrays, numbers to be written) is pointed to
      const char *format = view.format ? view.format : "";
      const bool pointer = view.ndim == 0 && format[0] != 0 && format[strlen(format) - 1] == 'P';
      p = pointer ? *(void **)view.buf : view.buf;
    }
    value = (T)p;
    return true;
  }
  ~Arg() {
    if (held) PyBuffer_Release(&view);
  }
};

PyObject *result(int v) { return PyLong_FromLong(v); }
PyObject *result(long long v) { return PyLong_FromLongLong(v); }
PyObject *result(unsigned long v) { return PyLong_FromUnsignedLong(v); }
PyObject *result(unsigned long long v) { return PyLong_FromUnsignedLongLong(v); }
PyObject *result(void *v) { return PyLong_FromVoidPtr(v); }
PyObject *result(int32_t *v) { return PyLong_FromVoidPtr(v); }
PyObject *result(const char *v) { return PyBytes_FromString(v ? v : ""); }

template <auto Fn, typename R, typename... A, size_t... I>
PyObject *call(PyObject *const *args, R (*)(A...), std::index_sequence<I...>) {
  std::tuple<Arg<A>...> in;
  if (!(std::get<I>(in).take(args[I]) && ...)) return nullptr;
  R r;
  Py_BEGIN_ALLOW_THREADS
  r = Fn(std::get<I>(in).value...);
  Py_END_ALLOW_THREADS
  return result(r);
}

template <typename F>
struct Arity;
template <typename R, typename... A>
struct Arity<R (*)(A...)> : std::integral_constant<size_t, sizeof...(A)> {};

template <auto Fn>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
  constexpr size_t want = Arity<decltype(Fn)>::value;
  if ((size_t)n != want) {
    PyErr_Format(PyExc_TypeError, "expected %zu arguments, got %zd", want, n);
    return nullptr;
  }
  return call<Fn>(args, Fn, std::make_index_sequence<want>());
}

// ptr(tensor or None, dtype=None): its device pointer, None for None.
PyObject *ptr(PyObject *, PyObject *const *args, Py_ssize_t n) {
  if (n < 1 || n > 2) {
    PyErr_SetString(PyExc_TypeError, "ptr(tensor, dtype=None)");
    return nullptr;
  }
  if (args[0] == Py_None) Py_RETURN_NONE;
  if (!THPVariable_Check(args[0])) {
    PyErr_SetString(PyExc_TypeError, "expected a tensor");
    return nullptr;
  }
  const at::Tensor &t = THPVariable_Unpack(args[0]);
  if (n == 2 && THPDtype_Check(args[1]) && t.is_cuda() && t.scalar_type() != ((THPDtype *)args[1])->scalar_type) {
    PyErr_Format(PyExc_TypeError, "expected dtype %S, got torch.%s", args[1], c10::toString(t.scalar_type()));
    return nullptr;
  }
  void *p = nullptr;
  return tensor_pointer(t, p) ? PyLong_FromVoidPtr(p) : nullptr;
}

// empty(shape, dtype, device): torch.empty.
PyObject *empty(PyObject *, PyObject *const *args, Py_ssize_t n) {
  if (n != 3 || !THPDtype_Check(args[1]) || !THPDevice_Check(args[2])) {
    PyErr_SetString(PyExc_TypeError, "empty(shape, torch.dtype, torch.device)");
    return nullptr;
  }
  int64_t sizes[8];
  size_t dims = 1;
  if (PyTuple_Check(args[0])) {
    dims = (size_t)PyTuple_GET_SIZE(args[0]);
    if (dims > 8) {
      PyErr_SetString(PyExc_ValueError, "empty: more than eight dimensions");
      return nullptr;
    }
    for (size_t i = 0; i < dims; ++i) sizes[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(args[0], i));
  } else {
    sizes[0] = PyLong_AsLongLong(args[0]);
  }
  if (PyErr_Occurred()) return nullptr;
  try {
    return THPVariable_Wrap(at::empty(at::IntArrayRef(sizes, dims), at::TensorOptions()
                                                                        .dtype(((THPDtype *)args[1])->scalar_type)
                                                                        .device(((THPDevice *)args[2])->device)));
  } catch (const c10::OutOfMemoryError &e) {
    PyObject *type = nullptr, *torch = PyImport_ImportModule("torch");
    if (torch) type = PyObject_GetAttrString(torch, "OutOfMemoryError");
    PyErr_SetString(type ? type : PyExc_MemoryError, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
    return nullptr;
  } catch (const std::exception &e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// head(tensor, n): its first n rows, tensor[:n].
PyObject *head(PyObject *, PyObject *const *args, Py_ssize_t n) {
  if (n != 2 || !THPVariable_Check(args[0])) {
    PyErr_SetString(PyExc_TypeError, "head(tensor, n)");
    return nullptr;
  }
  const long long rows = PyLong_AsLongLong(args[1]);
  if (rows == -1 && PyErr_Occurred()) return nullptr;
  try {
    return THPVariable_Wrap(THPVariable_Unpack(args[0]).narrow(0, 0, rows));
  } catch (const std::exception &e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

#define SSC_FUNCTIONS \
  X(ssc_version) X(ssc_last_error) X(ssc_has_tcgen05) X(ssc_kernel_launches) X(ssc_read_words) X(ssc_count_open) X(ssc_count_wait) X(ssc_count_close) X(ssc_count_post) X(ssc_alarm_open) \
  X(ssc_rulebook_scratch_bytes) X(ssc_rulebook_subm) X(ssc_rulebook_subm_static) X(ssc_rulebook_subm_ahead) \
  X(ssc_rulebook_conv_count) X(ssc_rulebook_conv_fill) X(ssc_rulebook_conv_ahead) X(ssc_pairs_to_nbr) X(ssc_pairs_from_nbr_scratch_bytes) \
  X(ssc_pairs_from_nbr) X(ssc_materialize) X(ssc_materialize_bwd) X(ssc_conv_packed_bytes) X(ssc_conv_pack_filters) \
  X(ssc_conv_scratch_bytes) X(ssc_conv_fwd) X(ssc_conv_pairs_list_bytes) X(ssc_conv_pairs_supported) \
  X(ssc_conv_pairs_build) X(ssc_conv_fwd_pairs) X(ssc_nbr_transpose) X(ssc_nbr_row_order_scratch_bytes) \
  X(ssc_nbr_row_order) X(ssc_nbr_row_order_planes_scratch_bytes) X(ssc_nbr_row_order_planes) X(ssc_conv_stage) \
  X(ssc_layer_struct_bytes) X(ssc_layer_ahead_bytes) X(ssc_layer_ahead) X(ssc_conv_gate_covered) \
  X(ssc_conv_fwd_gated) X(ssc_conv_fwd_ordered) X(ssc_conv_wgrad_scratch_bytes) X(ssc_conv_wgrad) \
  X(ssc_conv_wgrad_lists) X(ssc_maxpool_bwd) X(ssc_avgpool_bwd) X(ssc_global_avgpool_bwd) X(ssc_global_maxpool_bwd) \
  X(ssc_voxelize_bwd) X(ssc_three_interpolate_bwd) X(ssc_steer_matrices) X(ssc_steer_matrices64) X(ssc_steer_fwd) X(ssc_p2v_stats) \
  X(ssc_maxpool_fwd) X(ssc_avgpool_fwd) X(ssc_pool_fwd16) X(ssc_summary_rf) X(ssc_global_avgpool_fwd) \
  X(ssc_global_maxpool_fwd) X(ssc_batch_offsets) X(ssc_voxel2point_map) X(ssc_voxelize_fwd) X(ssc_p2v_scratch_bytes) \
  X(ssc_p2v_keep_scratch_bytes) X(ssc_p2v_keep) X(ssc_voxel_centres) X(ssc_point_rows) X(ssc_nn_weights) \
  X(ssc_p2v_count) X(ssc_p2v_fill) X(ssc_three_nn_scratch_bytes) X(ssc_three_nn) X(ssc_three_interpolate_fwd) \
  X(ssc_bn_fold) X(ssc_bn_gate_fwd) X(ssc_bn_gate_fwd16) X(ssc_bn_scratch_bytes) X(ssc_bn_stats) X(ssc_bn_train) \
  X(ssc_bn_gate_bwd) X(ssc_bn_bwd) X(ssc_gate_bwd) X(ssc_scatter_add_rate)

#define X(name) {#name, (PyCFunction)(void (*)())entry<&name>, METH_FASTCALL, nullptr},
PyMethodDef methods[] = {{"ptr", (PyCFunction)(void (*)())ptr, METH_FASTCALL, "device pointer of a contiguous CUDA tensor"},
                         {"empty", (PyCFunction)(void (*)())empty, METH_FASTCALL, "torch.empty(shape, dtype, device)"},
                         {"head", (PyCFunction)(void (*)())head, METH_FASTCALL, "tensor[:n]"},
                         SSC_FUNCTIONS{nullptr, nullptr, 0, nullptr}};
#undef X

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Python bindings of libssconv_b200.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
