// Native form of the two linears that are called eagerly, one at a time: `W4A16Linear.forward` and `IntegerLinear.forward`
// (W8A8).  Such a call is bound by the host: through ctypes and tensor methods, the two launches of a 64 x 2048 x 2048 W8A8
// linear took 50 us around 6 us on the device, the one launch of a W4A16 row 26 us around 7 us.
//
// A call here takes the plain case only - exact CUDA tensors, contiguous rows, a workspace that exists, no dispatch mode - and
// answers None for everything else, errors included: the caller then goes its general way in Python, which repeats the
// checks and raises what it always raised.  Nothing is queued before all checks of arguments have passed (an error of the device
// itself can still come between the two launches), nothing is kept between calls.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/rk_b200.h"

namespace {

// entry points of librk_b200.so, handed over as addresses so that both bindings use the one loaded library
decltype(&rk_quant_rows) g_quant_rows = nullptr;
decltype(&rk_gemm_int) g_gemm_int = nullptr;
decltype(&rk_gemm_w4a16_g128) g_gemm_w4a16 = nullptr;
PyObject* g_workspaces = nullptr;  // {(device index, stream handle): [uint8 tensors, the newest last]}

PyObject* k_buffers = nullptr;
PyObject* k_packed_weight = nullptr;
PyObject* k_weight_scale = nullptr;
PyObject* k_bias = nullptr;
PyObject* k_in_features = nullptr;
PyObject* k_out_features = nullptr;
PyObject* k_bits = nullptr;
PyObject* k_tactic = nullptr;
PyObject* k_pack_input = nullptr;
PyObject* k_forward_packed = nullptr;

// borrowed tensor of an exact type with an ordinary CUDA storage, or null
const at::Tensor* plain_cuda(PyObject* obj) {
  if (obj == nullptr || !THPVariable_CheckExact(obj)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(obj);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage()) return nullptr;
  const c10::DispatchKeySet keys = t.key_set();
  if (keys.has_any(c10::functorch_transforms_ks) || keys.has(c10::DispatchKey::Python) || keys.has(c10::DispatchKey::Functionalize) ||
      keys.has(c10::DispatchKey::ZeroTensor))
    return nullptr;
  return &t;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

bool get_long(PyObject* dict, PyObject* key, int64_t* out) {
  PyObject* v = PyDict_GetItem(dict, key);
  if (v == nullptr || !PyLong_CheckExact(v)) return false;
  *out = PyLong_AsLongLong(v);
  if (*out == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// the stream's workspace (at least a header long), or null where none exists yet
void* workspace_of(int device, cudaStream_t stream, size_t* bytes) {
  PyObject* key = Py_BuildValue("(iK)", device, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)));
  if (key == nullptr) return nullptr;
  PyObject* list = PyDict_GetItem(g_workspaces, key);
  Py_DECREF(key);
  if (list == nullptr || !PyList_Check(list) || PyList_GET_SIZE(list) == 0) return nullptr;
  const at::Tensor* ws = plain_cuda(PyList_GET_ITEM(list, PyList_GET_SIZE(list) - 1));
  if (ws == nullptr) return nullptr;
  *bytes = static_cast<size_t>(ws->numel());
  return ws->data_ptr();
}

struct Layer {
  const at::Tensor *weight = nullptr, *scale = nullptr, *bias = nullptr;
  int64_t in_features = 0, out_features = 0, tactic = 0;
};

bool read_layer(PyObject* dict, Layer* layer) {
  if (dict == nullptr || !PyDict_CheckExact(dict)) return false;
  PyObject* buffers = PyDict_GetItem(dict, k_buffers);
  if (buffers == nullptr || !PyDict_Check(buffers)) return false;
  layer->weight = plain_cuda(PyDict_GetItem(buffers, k_packed_weight));
  layer->scale = plain_cuda(PyDict_GetItem(buffers, k_weight_scale));
  PyObject* bias = PyDict_GetItem(buffers, k_bias);
  if (bias == nullptr) return false;
  if (bias != Py_None && (layer->bias = plain_cuda(bias)) == nullptr) return false;
  if (layer->weight == nullptr || layer->scale == nullptr || layer->weight->dim() != 2 || !layer->weight->is_contiguous() ||
      !layer->scale->is_contiguous())
    return false;
  if (!get_long(dict, k_in_features, &layer->in_features) || !get_long(dict, k_out_features, &layer->out_features) ||
      !get_long(dict, k_tactic, &layer->tactic) || layer->tactic < 0 || layer->tactic > 63)
    return false;
  const int64_t n = layer->weight->size(0);
  if (layer->bias != nullptr && (layer->bias->scalar_type() != at::kBFloat16 || layer->bias->numel() != n || !layer->bias->is_contiguous()))
    return false;
  return layer->out_features == n && layer->in_features >= 1;
}

// rows of x for this layer, 0 if the call is not a plain one
int64_t plain_rows(const at::Tensor& x, const Layer& layer, int min_dim) {
  if (x.scalar_type() != at::kBFloat16 || x.dim() < min_dim || !x.is_contiguous() || x.size(-1) != layer.in_features) return 0;
  if (layer.weight->device() != x.device() || layer.scale->device() != x.device()) return 0;
  if (layer.bias != nullptr && layer.bias->device() != x.device()) return 0;
  return x.numel() / layer.in_features;
}

bool modes_active() {
  return g_workspaces == nullptr || c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled();
}

// W4A16Linear.forward(x) of the module whose __dict__ is given
PyObject* w4a16_linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2) Py_RETURN_NONE;
  try {
    Layer layer;
    const at::Tensor* x = plain_cuda(args[1]);
    if (x == nullptr || modes_active() || !read_layer(args[0], &layer)) Py_RETURN_NONE;
    const int64_t m = plain_rows(*x, layer, 1), n = layer.out_features, k = layer.in_features;
    if (m < 1 || k % 128 != 0 || layer.weight->scalar_type() != at::kByte || layer.weight->size(1) * 2 != k ||
        layer.scale->scalar_type() != at::kBFloat16 || layer.scale->dim() != 2 || layer.scale->size(0) != k / 128 || layer.scale->size(1) != n)
      Py_RETURN_NONE;
    const int device = x->device().index();
    const c10::cuda::OptionalCUDAGuard guard(x->device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
    size_t ws_bytes = 0;
    void* ws = workspace_of(device, stream, &ws_bytes);
    if (ws == nullptr) Py_RETURN_NONE;
    const void *px = x->data_ptr(), *pw = layer.weight->data_ptr(), *ps = layer.scale->data_ptr();
    const void* pb = layer.bias != nullptr ? layer.bias->data_ptr() : nullptr;
    // owned until the launch: another thread may replace the module's buffers while the interpreter lock is released
    const at::Tensor weight = *layer.weight, scale = *layer.scale, bias = layer.bias != nullptr ? *layer.bias : at::Tensor();
    c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = n;
    int code;
    at::Tensor out;
    Py_BEGIN_ALLOW_THREADS;
    try {
      out = at::empty(shape, x->options());
      code = g_gemm_w4a16(px, pw, ps, pb, out.data_ptr(), m, n, k, static_cast<int>(layer.tactic), ws, ws_bytes, stream);
    } catch (...) {
      code = RK_ECUDA;
    }
    Py_END_ALLOW_THREADS;
    if (code != RK_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
  } catch (...) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// IntegerLinear.forward(x) (8 bits, no residual) of the module whose __dict__ is given
PyObject* integer_linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2) Py_RETURN_NONE;
  try {
    Layer layer;
    const at::Tensor* x = plain_cuda(args[1]);
    int64_t bits = 0;
    if (x == nullptr || modes_active() || !read_layer(args[0], &layer) || !get_long(args[0], k_bits, &bits) || bits != 8) Py_RETURN_NONE;
    if (PyDict_GetItem(args[0], k_pack_input) != nullptr || PyDict_GetItem(args[0], k_forward_packed) != nullptr) Py_RETURN_NONE;
    const int64_t m = plain_rows(*x, layer, 2), n = layer.out_features, k = layer.in_features;
    const int64_t kpad = (k + 127) / 128 * 128;
    if (m < 1 || k > 65536 || layer.weight->scalar_type() != at::kChar || layer.weight->size(1) != kpad ||
        layer.scale->scalar_type() != at::kFloat || layer.scale->numel() != n)
      Py_RETURN_NONE;
    const int device = x->device().index();
    const c10::cuda::OptionalCUDAGuard guard(x->device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
    size_t ws_bytes = 0;
    void* ws = workspace_of(device, stream, &ws_bytes);
    if (ws == nullptr) Py_RETURN_NONE;
    const void *px = x->data_ptr(), *pw = layer.weight->data_ptr();
    const float* ps = layer.scale->const_data_ptr<float>();
    const void* pb = layer.bias != nullptr ? layer.bias->data_ptr() : nullptr;
    // what rk_gemm_int would refuse, so that no quantizer is queued for a call that the general path then repeats
    if (!aligned16(px) || !aligned16(pw) || !aligned16(ws) || ws_bytes < RK_WORKSPACE_HEADER || layer.tactic > 7 || n % 8 != 0 ||
        m > (1 << 24) || n > (1 << 24))
      Py_RETURN_NONE;
    // owned until the launch: another thread may replace the module's buffers while the interpreter lock is released
    const at::Tensor weight = *layer.weight, scale = *layer.scale, bias = layer.bias != nullptr ? *layer.bias : at::Tensor();
    c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = n;
    int code;
    at::Tensor out;
    Py_BEGIN_ALLOW_THREADS;
    try {
      // the row codes and their scales live for this call only: one block of the caching allocator, on the current stream
      const c10::DataPtr codes = c10::cuda::CUDACachingAllocator::get()->allocate(static_cast<size_t>(m) * kpad + static_cast<size_t>(m) * 4);
      float* const scales = reinterpret_cast<float*>(static_cast<uint8_t*>(codes.get()) + static_cast<size_t>(m) * kpad);
      out = at::empty(shape, x->options());
      code = g_quant_rows(px, m, k, k, nullptr, k, nullptr, 0, 8, codes.get(), scales, stream);
      if (code == RK_OK)
        code = g_gemm_int(codes.get(), scales, pw, ps, pb, out.data_ptr(), m, n, kpad, 8, static_cast<int>(layer.tactic), ws, ws_bytes,
                          stream);
    } catch (...) {
      code = RK_ECUDA;
    }
    Py_END_ALLOW_THREADS;
    if (code != RK_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
  } catch (...) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// bind({name: address}, workspaces): once, after the library has been loaded
PyObject* bind(PyObject*, PyObject* args) {
  PyObject *addresses = nullptr, *workspaces = nullptr;
  if (!PyArg_ParseTuple(args, "O!O!", &PyDict_Type, &addresses, &PyDict_Type, &workspaces)) return nullptr;
  auto address = [&](const char* name) -> void* {
    PyObject* v = PyDict_GetItemString(addresses, name);
    void* p = v != nullptr ? PyLong_AsVoidPtr(v) : nullptr;
    if (p == nullptr && !PyErr_Occurred()) PyErr_Format(PyExc_ValueError, "no address of %s", name);
    return p;
  };
  void* quant = address("rk_quant_rows");
  void* gemm = quant != nullptr ? address("rk_gemm_int") : nullptr;
  void* w4 = gemm != nullptr ? address("rk_gemm_w4a16_g128") : nullptr;
  if (w4 == nullptr) return nullptr;
  g_quant_rows = reinterpret_cast<decltype(g_quant_rows)>(quant);
  g_gemm_int = reinterpret_cast<decltype(g_gemm_int)>(gemm);
  g_gemm_w4a16 = reinterpret_cast<decltype(g_gemm_w4a16)>(w4);
  Py_INCREF(workspaces);
  Py_XSETREF(g_workspaces, workspaces);
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_VARARGS, "bind(addresses, workspaces): entry points of the loaded library, the workspaces by stream"},
    {"w4a16_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(w4a16_linear)), METH_FASTCALL,
     "w4a16_linear(module.__dict__, x) -> output, or None where the general path has to run"},
    {"integer_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(integer_linear)), METH_FASTCALL,
     "integer_linear(module.__dict__, x) -> output, or None where the general path has to run"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls() {
  const struct {
    PyObject** slot;
    const char* name;
  } names[] = {{&k_buffers, "_buffers"}, {&k_packed_weight, "packed_weight"}, {&k_weight_scale, "weight_scale"}, {&k_bias, "bias"},
               {&k_in_features, "in_features"}, {&k_out_features, "out_features"}, {&k_bits, "bits"}, {&k_tactic, "tactic"},
               {&k_pack_input, "pack_input"}, {&k_forward_packed, "forward_packed"}};
  for (const auto& n : names) {
    *n.slot = PyUnicode_InternFromString(n.name);
    if (*n.slot == nullptr) return nullptr;
  }
  return PyModule_Create(&kModule);
}
