// The host side of eager calls, natively: a projection, quantising and tiling a weight called from Python spend 10 to 15 us
// in argument checks, allocations and argument marshalling around kernels of 4 to 35 us.  Each function here
// does what fdk/models.py and fdk/native.py do for the ordinary case -- plain CUDA tensors on the current device, nothing
// that a dispatch mode, a tensor subclass or a transform would have to see -- and returns None for every other
// one (and for every error), whereupon the Python code runs as it would without it.  Nothing is kept between calls: the
// caches read here are the Python objects' own.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/fdk_b200.h"

namespace {

decltype(&fdk_linear_lut) g_linear_lut;
decltype(&fdk_quantise) g_quantise;
decltype(&fdk_repack) g_repack;
decltype(&fdk_tiled_size) g_tiled_size;
PyObject* g_workspaces;  // {(device, stream): scratch tensor}, native.py's own

PyObject *s_parameters, *s_buffers, *s_weight, *s_scale, *s_lut, *s_kernel, *s_tiled, *s_tiled_key, *s_lut_host, *s_lut_key,
    *s_in, *s_out;

// No key (nor backend: a difference of key sets keeps those) but the given ones.
bool within(c10::DispatchKeySet keys, c10::DispatchKeySet given) { return (keys.raw_repr() & ~given.raw_repr()) == 0; }

// Nobody is watching calls: no Python dispatch or function mode, no functorch level, no vmap, no tracing key.
bool plain_context() {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;
  if (at::impl::PythonTorchFunctionTLS::stack_len() != 0) return false;
  if (!within(c10::impl::tls_local_dispatch_key_set().included_, c10::default_included_set)) return false;
  return !(at::globalContext().deterministicAlgorithms() && at::globalContext().deterministicFillUninitializedMemory());
}

bool is_cuda(PyObject* o) { return THPVariable_CheckExact(o) && THPVariable_Unpack(o).is_cuda(); }

// A plain strided CUDA tensor on device `index`, or null.
const at::Tensor* plain(PyObject* o, c10::DeviceIndex index) {
  if (o == nullptr || !THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.device().index() != index) return nullptr;
  static const c10::DispatchKeySet ordinary = c10::DispatchKeySet(c10::DispatchKey::CUDA) |
                                              c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) |
                                              c10::getAutogradRelatedKeySetFromBackend(c10::BackendComponent::CUDABit) |
                                              c10::getAutocastRelatedKeySetFromBackend(c10::BackendComponent::CUDABit);
  if (!within(t.key_set(), ordinary)) return nullptr;
  return &t;
}

PyObject* item(PyObject* dict, PyObject* key) {  // borrowed, or null without an error
  return dict != nullptr && PyDict_Check(dict) ? PyDict_GetItemWithError(dict, key) : nullptr;
}

bool equals(PyObject* number, uint64_t value) {
  if (number == nullptr || !PyLong_Check(number)) return false;
  const unsigned long long v = PyLong_AsUnsignedLongLong(number);
  if (v == (unsigned long long)-1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return v == value;
}
bool positive_int(PyObject* number, int* out) {
  if (number == nullptr || !PyLong_Check(number)) return false;
  int overflow = 0;
  const long long v = PyLong_AsLongLongAndOverflow(number, &overflow);
  if (overflow != 0 || v <= 0 || v > 0x7FFFFFFF) return false;
  *out = (int)v;
  return true;
}

int dtype_code(const at::Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? FDK_DTYPE_BF16 : t.scalar_type() == at::kHalf ? FDK_DTYPE_F16 : -1;
}

PyObject* none() {
  PyErr_Clear();
  Py_RETURN_NONE;
}

// No C++ exception leaves an entry: whatever it was, the Python code runs into it again and reports it.
template <PyObject* (*Entry)(PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject*, PyObject* const* args, Py_ssize_t count) {
  try {
    return Entry(args, count);
  } catch (...) {
    return none();
  }
}

at::Tensor make(at::IntArrayRef sizes, at::ScalarType type, const at::Device& device) {
  return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}

// linear(the module's __dict__, x) -> x . W^T, or None
PyObject* linear(PyObject* const* args, Py_ssize_t count) {
  if (count != 2 || g_linear_lut == nullptr || !is_cuda(args[1]) || !plain_context()) return none();
  PyObject* const dict = args[0];
  const c10::DeviceIndex device = c10::cuda::current_device();
  const at::Tensor* x = plain(args[1], device);
  if (x == nullptr || x->dim() != 2 || x->size(0) < 1 || x->size(0) > 0x7FFFFFFF || !x->is_contiguous()) return none();
  PyObject* const kernel = item(dict, s_kernel);
  if (kernel == nullptr || !PyUnicode_Check(kernel) ||
      (PyUnicode_CompareWithASCIIString(kernel, "triton") != 0 && PyUnicode_CompareWithASCIIString(kernel, "marlin") != 0 &&
       PyUnicode_CompareWithASCIIString(kernel, "marlin-lut") != 0))
    return none();
  PyObject* const parameters = item(dict, s_parameters);
  const at::Tensor* weight = plain(item(parameters, s_weight), device);
  const at::Tensor* scale = plain(item(parameters, s_scale), device);
  const at::Tensor* lut = plain(item(item(dict, s_buffers), s_lut), device);
  const at::Tensor* tiled = plain(item(dict, s_tiled), device);
  if (!weight || !scale || !lut || !tiled || lut->dim() != 2 || lut->size(1) < 1) return none();
  const int dtype = dtype_code(*x);
  if (dtype < 0 || x->scalar_type() != lut->scalar_type() || x->scalar_type() != scale->scalar_type()) return none();
  int n = 0, k = 0;
  if (!positive_int(item(dict, s_out), &n) || !positive_int(item(dict, s_in), &k) || x->size(1) != k) return none();
  const int bits = lut->size(0) == 8 ? 3 : (int)(8 / lut->size(1));
  // the tiled copy and the host's copy of the table are those of these tensors (QuantisedLinear.tiled, lut_bytes)
  PyObject* const key = item(dict, s_tiled_key);
  if (key == nullptr || !PyTuple_Check(key) || PyTuple_GET_SIZE(key) != 5 || weight->is_inference() || scale->is_inference() ||
      lut->is_inference())
    return none();
  if (!equals(PyTuple_GET_ITEM(key, 0), (uint64_t)(uintptr_t)weight->data_ptr()) ||
      !equals(PyTuple_GET_ITEM(key, 1), (uint64_t)(uintptr_t)scale->data_ptr()) || !equals(PyTuple_GET_ITEM(key, 2), weight->_version()) ||
      !equals(PyTuple_GET_ITEM(key, 3), scale->_version()))
    return none();
  PyObject* const lut_key = item(dict, s_lut_key);
  PyObject* const lut_host = item(dict, s_lut_host);
  if (lut_key == nullptr || !PyTuple_Check(lut_key) || PyTuple_GET_SIZE(lut_key) != 2 || lut_host == nullptr || !PyBytes_Check(lut_host) ||
      (size_t)PyBytes_GET_SIZE(lut_host) != lut->nbytes() ||
      !equals(PyTuple_GET_ITEM(lut_key, 0), (uint64_t)(uintptr_t)lut->data_ptr()) || !equals(PyTuple_GET_ITEM(lut_key, 1), lut->_version()))
    return none();
  // the current stream's scratch
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
  PyObject* const stream_key = Py_BuildValue("(iK)", (int)device, (unsigned long long)(uintptr_t)stream);
  if (stream_key == nullptr) return none();
  const at::Tensor* workspace = plain(item(g_workspaces, stream_key), device);
  Py_DECREF(stream_key);
  if (workspace == nullptr) return none();
  // references of our own: another thread may replace the module's while this one is without the interpreter lock
  const at::Tensor x_ = *x, tiled_ = *tiled, lut_ = *lut, workspace_ = *workspace;
  Py_INCREF(lut_host);
  const char* const table = PyBytes_AS_STRING(lut_host);
  at::Tensor out;
  int status = FDK_ERR_CUDA;
  Py_BEGIN_ALLOW_THREADS;
  try {
    out = make({x_.size(0), n}, x_.scalar_type(), x_.device());
    status = g_linear_lut(x_.data_ptr(), tiled_.data_ptr(), lut_.data_ptr(), table, out.data_ptr(), (int)x_.size(0), n, k, bits, dtype,
                          workspace_.data_ptr(), (size_t)workspace_.nbytes(), FDK_FLAG_PDL, stream);
  } catch (...) {
    status = FDK_ERR_CUDA;
  }
  Py_END_ALLOW_THREADS;
  Py_DECREF(lut_host);
  return status == FDK_OK ? THPVariable_Wrap(out) : none();
}

// quantise(weight, bits, block_size, codebook, scale or None) -> (codes, scale, table), or None: native.can_quantise and
// native.quantise
PyObject* quantise(PyObject* const* args, Py_ssize_t count) {
  if (count != 5 || g_quantise == nullptr || !is_cuda(args[0]) || !plain_context()) return none();
  const c10::DeviceIndex device = c10::cuda::current_device();
  const at::Tensor *w = plain(args[0], device), *lut = plain(args[3], device);
  const at::Tensor* scale = args[4] == Py_None ? nullptr : plain(args[4], device);
  int bits = 0, block = 0;
  if (!w || !lut || (args[4] != Py_None && !scale) || !positive_int(args[1], &bits) || !positive_int(args[2], &block)) return none();
  const int dtype = dtype_code(*w);
  if (dtype < 0 || lut->scalar_type() != w->scalar_type() || w->dim() != 2 || w->numel() == 0 || !w->is_contiguous() || lut->dim() != 1 ||
      lut->numel() == 0 || !lut->is_contiguous() || (lut->requires_grad() && c10::GradMode::is_enabled()))
    return none();
  if (!(bits == 1 || bits == 2 || bits == 3 || bits == 4 || bits == 8) || lut->numel() > (1 << bits) || block < 8 || block > 256 ||
      (block & (block - 1)) != 0 || w->size(1) % block != 0 || w->size(0) > 0x7FFFFFFF || w->size(1) > 0x7FFFFFFF ||
      ((uintptr_t)w->data_ptr() & 15) != 0)
    return none();
  const int64_t n = w->size(0), k = w->size(1);
  if (scale != nullptr && (scale->scalar_type() != w->scalar_type() || !scale->is_contiguous() || scale->dim() != 2 || scale->size(0) != n ||
                           scale->size(1) != k / block))
    return none();
  const at::Tensor w_ = *w, lut_ = *lut;
  at::Tensor codes, table, out_scale;
  if (scale != nullptr) out_scale = *scale;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
  int status = FDK_ERR_CUDA;
  Py_BEGIN_ALLOW_THREADS;
  try {
    codes = make({n, k * bits / 8}, at::kByte, w_.device());
    table = bits == 3 ? make({8, 1}, w_.scalar_type(), w_.device()) : make({256, 8 / bits}, w_.scalar_type(), w_.device());
    const bool given = out_scale.defined();
    if (!given) out_scale = make({n, k / block}, w_.scalar_type(), w_.device());
    status = g_quantise(w_.data_ptr(), (int)n, (int)k, bits, block, dtype, lut_.data_ptr(), (int)lut_.numel(),
                        given ? out_scale.data_ptr() : nullptr, codes.data_ptr(), given ? nullptr : out_scale.data_ptr(), table.data_ptr(),
                        stream);
  } catch (...) {
    status = FDK_ERR_CUDA;
  }
  Py_END_ALLOW_THREADS;
  if (status != FDK_OK) return none();
  return Py_BuildValue("(NNN)", THPVariable_Wrap(codes), THPVariable_Wrap(out_scale), THPVariable_Wrap(table));
}

// repack(codes, scale, n, k, bits, block_size) -> tiled buffer, or None: native.repack
PyObject* repack(PyObject* const* args, Py_ssize_t count) {
  if (count != 6 || g_repack == nullptr || !is_cuda(args[0]) || !plain_context()) return none();
  const c10::DeviceIndex device = c10::cuda::current_device();
  const at::Tensor *codes = plain(args[0], device), *scale = plain(args[1], device);
  int n = 0, k = 0, bits = 0, block = 0;
  if (!codes || !scale || !positive_int(args[2], &n) || !positive_int(args[3], &k) || !positive_int(args[4], &bits) ||
      !positive_int(args[5], &block) || codes->scalar_type() != at::kByte || !codes->is_contiguous() || !scale->is_contiguous())
    return none();
  size_t bytes = 0;
  if (g_tiled_size(n, k, bits, &bytes) != FDK_OK) return none();
  const at::Tensor codes_ = *codes, scale_ = *scale;
  at::Tensor tiled;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
  int status = FDK_ERR_CUDA;
  Py_BEGIN_ALLOW_THREADS;
  try {
    tiled = make({(int64_t)bytes}, at::kByte, codes_.device());
    status = g_repack(codes_.data_ptr(), scale_.data_ptr(), n, k, bits, block, tiled.data_ptr(), stream);
  } catch (...) {
    status = FDK_ERR_CUDA;
  }
  Py_END_ALLOW_THREADS;
  return status == FDK_OK ? THPVariable_Wrap(tiled) : none();
}

// bind(addresses of fdk_linear_lut, fdk_quantise, fdk_repack, fdk_tiled_size; the dictionary of workspaces)
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long linear_lut, quantise, repack, tiled_size;
  PyObject* workspaces;
  if (!PyArg_ParseTuple(args, "KKKKO!", &linear_lut, &quantise, &repack, &tiled_size, &PyDict_Type, &workspaces)) return nullptr;
  Py_INCREF(workspaces);
  Py_XSETREF(g_workspaces, workspaces);
  g_quantise = reinterpret_cast<decltype(g_quantise)>((uintptr_t)quantise);
  g_repack = reinterpret_cast<decltype(g_repack)>((uintptr_t)repack);
  g_tiled_size = reinterpret_cast<decltype(g_tiled_size)>((uintptr_t)tiled_size);
  g_linear_lut = reinterpret_cast<decltype(g_linear_lut)>((uintptr_t)linear_lut);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"linear", (PyCFunction)(void (*)(void))guarded<linear>, METH_FASTCALL, nullptr},
    {"quantise", (PyCFunction)(void (*)(void))guarded<quantise>, METH_FASTCALL, nullptr},
    {"repack", (PyCFunction)(void (*)(void))guarded<repack>, METH_FASTCALL, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_eager", "Host side of eager calls (see fdk/native.py).", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__eager() {
  const struct { PyObject** to; const char* text; } names[] = {
      {&s_parameters, "_parameters"}, {&s_buffers, "_buffers"}, {&s_weight, "weight_data"}, {&s_scale, "scale"}, {&s_lut, "lut"},
      {&s_kernel, "kernel"}, {&s_tiled, "_tiled"}, {&s_tiled_key, "_tiled_key"}, {&s_lut_host, "_lut_host"},
      {&s_lut_key, "_lut_host_key"}, {&s_in, "in_features"}, {&s_out, "out_features"}};
  for (const auto& name : names)
    if ((*name.to = PyUnicode_InternFromString(name.text)) == nullptr) return nullptr;
  PyObject* const m = PyModule_Create(&module);
  // torch's inline code is compiled in, so native.py binds this only beside the same torch
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", FDK_TORCH_VERSION) != 0) return nullptr;
  return m;
}
