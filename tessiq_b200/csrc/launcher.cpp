// The Python module `tessiq_b200._launcher`: repeated calls of the eager entry points, from the operands to the
// launch, in native code.
//
// The first call of a signature (an operation, and its operands' types, shapes, strides, devices and alignments)
// goes the long way through ops.py, which checks everything, picks the kernel and, once its launch has succeeded,
// leaves a plan here (`keep`). Later calls of that signature (`call`) find the plan, allocate the result, take
// torch's current stream and launch: 4 to 5 us an operation, of which the launch is about 3, where the same steps took 9 to 14 in
// Python, on kernels of 2 to 5. (The first call of a signature takes 1 to 4 us longer for it.)
// A plan holds numbers only (and the compiled kernel it names), never an address or a tensor of a call; the table's
// older half goes when it is full. Whatever is not a plain CUDA tensor, runs under a dispatch mode, or fails to launch
// is answered with None, and the caller takes the long way, which raises what there is to raise.
//
// torch's headers are used for tensors, the caching allocator and streams only; the kernels are reached through the
// C interface of libtessiq_b200.so, opened by its path as ctypes opens it. (Linked to this module it would resolve its own
// symbols among torch's libraries, and crashed there.) Tables are touched under the GIL, launches run without it (as they
// did through ctypes).
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/object_ptr.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/strides.h>

#include <dlfcn.h>

#include <cstring>
#include <memory>
#include <unordered_map>
#include <utility>
#include <vector>

#include "tessiq_b200.h"

namespace {

enum Family { kFused, kReduce, kPack, kSoftmax, kLayerNorm, kTransposed, kBatchNorm, kGemm, kAttention };

// The library's entry points.
struct Library {
  decltype(&tq_fused_launch) fused_launch = nullptr;
  decltype(&tq_reduce_launch) reduce_launch = nullptr;
  decltype(&tq_pack_launch) pack_launch = nullptr;
  decltype(&tq_softmax_launch) softmax_launch = nullptr;
  decltype(&tq_layer_norm_launch) layer_norm_launch = nullptr;
  decltype(&tq_softmax_transposed_launch) softmax_transposed_launch = nullptr;
  decltype(&tq_layer_norm_transposed_launch) layer_norm_transposed_launch = nullptr;
  decltype(&tq_batch_norm_eval_launch) batch_norm_eval_launch = nullptr;
  decltype(&tq_gemm_bias_act_residual_launch) gemm_bias_act_residual_launch = nullptr;
  decltype(&tq_attention_launch) attention_launch = nullptr;
} library;

template <typename Function>
bool find_entry(void* handle, const char* name, Function& entry) {
  entry = reinterpret_cast<Function>(dlsym(handle, name));
  return entry != nullptr;
}

struct Output {
  std::vector<int64_t> sizes, strides;
  at::ScalarType dtype;
  bool packed;      // the strides are those of `empty`
};

struct Plan {
  Family family;
  std::vector<int64_t> key;
  std::vector<Output> outputs;
  std::vector<int64_t> ints;
  std::vector<double> doubles;
  std::vector<tq_layout> layouts;
  PyObject* holder = nullptr;      // what the plan's handle belongs to
  ~Plan() {
    if (holder == nullptr) return;
    const PyGILState_STATE state = PyGILState_Ensure();
    Py_DECREF(holder);
    PyGILState_Release(state);
  }
};

constexpr size_t kMostPlans = 2048;       // of both generations
constexpr int kMostOperands = 16;

// Two generations: when the younger one is full the older one goes, and a plan found in the older one joins the younger. So a program of
// more signatures than the table holds loses those it has not used for kMostPlans / 2 others, and never all at once.
using PlanMap = std::unordered_multimap<uint64_t, std::shared_ptr<const Plan>>;
struct Plans {
  PlanMap young, old;
};
// (never destroyed: at exit there may be no interpreter left to give the holders back to)
Plans& plans() {
  static auto* table = new Plans;
  return *table;
}
PyObject* parameter_class = nullptr;     // torch.nn.Parameter
PyObject* workspace_function = nullptr;  // kernel.workspace(device, stream, nbytes) -> tensor

struct Call {
  std::vector<int64_t> key;
  const at::Tensor* tensors[kMostOperands];      // null: the operand is None
  int tensor_count = 0;
  double scalars[kMostOperands];                 // numbers of an elementwise call
  int scalar_count = 0;
  int device = -1;
};

bool add_number(Call& call, PyObject* value) {
  if (PyBool_Check(value)) {
    call.key.push_back(-3);
    call.key.push_back(value == Py_True);
  } else if (PyLong_CheckExact(value)) {
    const int64_t number = PyLong_AsLongLong(value);
    if (number == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    call.key.push_back(-4);
    call.key.push_back(number);
  } else if (PyFloat_CheckExact(value)) {
    const double number = PyFloat_AS_DOUBLE(value);
    int64_t bits;
    std::memcpy(&bits, &number, sizeof bits);
    call.key.push_back(-5);
    call.key.push_back(bits);
  } else {
    return false;
  }
  return true;
}

// The signature of a call. `by_type`: numbers are launch arguments, of which the signature has the type alone.
// False: something a plan cannot stand for.
bool read(Call& call, PyObject* const* values, Py_ssize_t count, bool by_type) {
  if (count > kMostOperands || c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;
  call.key.reserve(64);
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject* value = values[i];
    if (value == Py_None) {
      call.key.push_back(-1);
      call.tensors[call.tensor_count++] = nullptr;
    } else if (THPVariable_CheckExact(value) || reinterpret_cast<PyObject*>(Py_TYPE(value)) == parameter_class) {
      const at::Tensor& t = THPVariable_Unpack(value);
      const c10::TensorImpl* impl = t.unsafeGetTensorImpl();
      if (!t.is_cuda() || t.layout() != at::kStrided || impl->is_python_dispatch() || !impl->has_storage() ||
          impl->key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                                       c10::DispatchKey::Functionalize, c10::DispatchKey::Batched})))
        return false;
      const int device = t.get_device();
      if (call.device < 0) call.device = device;
      if (device != call.device) return false;
      const int64_t rank = t.dim();
      call.key.push_back(static_cast<int64_t>(t.scalar_type()) << 32 | rank << 8 | (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15));
      for (const int64_t n : t.sizes()) call.key.push_back(n);
      for (const int64_t n : t.strides()) call.key.push_back(n);
      call.tensors[call.tensor_count++] = &t;
    } else if (by_type) {
      if (PyBool_Check(value)) {
        call.key.push_back(-3);
        call.scalars[call.scalar_count++] = value == Py_True ? 1.0 : 0.0;
      } else if (PyLong_CheckExact(value) || PyFloat_CheckExact(value)) {
        const double number = PyFloat_AsDouble(value);
        if (number == -1.0 && PyErr_Occurred()) {
          PyErr_Clear();
          return false;
        }
        call.key.push_back(PyLong_CheckExact(value) ? -4 : -5);
        call.scalars[call.scalar_count++] = number;
      } else {
        return false;
      }
    } else if (PyTuple_Check(value) || PyList_Check(value)) {
      const Py_ssize_t length = PySequence_Fast_GET_SIZE(value);
      PyObject** items = PySequence_Fast_ITEMS(value);
      call.key.push_back(-6);
      call.key.push_back(length);
      for (Py_ssize_t k = 0; k < length; ++k)
        if (!add_number(call, items[k])) return false;
    } else if (!add_number(call, value)) {
      return false;
    }
  }
  if (call.device < 0) return false;
  call.key.push_back(call.device);
  return true;
}

uint64_t hash_of(const std::vector<int64_t>& key) {
  uint64_t h = 1469598103934665603ull;
  for (const int64_t word : key) {
    h ^= static_cast<uint64_t>(word);
    h *= 1099511628211ull;
    h ^= h >> 29;
  }
  return h;
}

// (a copy that shares ownership: the launch runs without the GIL, and the table may be emptied meanwhile)
void remember(uint64_t hash, std::shared_ptr<const Plan> plan) {
  PlanMap gone;      // (what the holders' destructors run finds the table whole)
  Plans& table = plans();
  if (table.young.size() >= kMostPlans / 2) {
    gone = std::exchange(table.old, std::exchange(table.young, PlanMap()));
  }
  table.young.emplace(hash, std::move(plan));
}

std::shared_ptr<const Plan> find(const std::vector<int64_t>& key) {
  const uint64_t hash = hash_of(key);
  Plans& table = plans();
  for (PlanMap* generation : {&table.young, &table.old}) {
    const auto range = generation->equal_range(hash);
    for (auto it = range.first; it != range.second; ++it) {
      if (it->second->key != key) continue;
      std::shared_ptr<const Plan> found = it->second;
      if (generation == &table.old) {
        table.old.erase(it);
        remember(hash, found);
      }
      return found;
    }
  }
  return nullptr;
}

tq_status launch(const Plan& p, const Call& call, const std::vector<at::Tensor>& out, void* scratch, size_t scratch_bytes, void* stream) {
  auto pointer = [&](int i) -> const void* {
    const at::Tensor* t = i < call.tensor_count ? call.tensors[i] : nullptr;
    return t == nullptr ? nullptr : t->const_data_ptr();
  };
  auto result = [&](size_t i) -> void* { return i < out.size() ? out[i].mutable_data_ptr() : nullptr; };
  const int64_t* n = p.ints.data();
  const int32_t device = call.device;
  auto small = [&](int i) { return static_cast<int32_t>(n[i]); };
  switch (p.family) {
    case kFused: {
      const void* inputs[kMostOperands];
      for (int i = 0; i < call.tensor_count; ++i) inputs[i] = pointer(i);
      return library.fused_launch(reinterpret_cast<const tq_fused*>(n[0]), inputs, result(0), n[1], n + 2, p.layouts.data(), call.scalars, device, stream);
    }
    case kReduce:
      return library.reduce_launch(small(0), small(1), pointer(0), result(0), n[2], n[3], n[4], scratch, scratch_bytes, device, stream);
    case kPack: {
      const int32_t rank = small(1);
      return library.pack_launch(small(0), rank, n + 2, n + 2 + rank, pointer(0), result(0), device, stream);
    }
    case kSoftmax:
      return library.softmax_launch(small(0), small(1), pointer(0), result(0), n[2], n[3], n[4], device, stream);
    case kLayerNorm:
      return library.layer_norm_launch(small(0), pointer(0), pointer(1), pointer(2), result(0), result(1), result(2), small(1), n[2], n[3], p.doubles[0],
                                  device, stream);
    case kTransposed:
      if (n[0] == 0) return library.softmax_transposed_launch(small(1), pointer(0), result(0), n[2], n[3], n[4], scratch, scratch_bytes, device, stream);
      return library.layer_norm_transposed_launch(small(1), pointer(0), pointer(1), pointer(2), result(0), n[2], n[3], n[4], p.doubles[0], scratch,
                                             scratch_bytes, device, stream);
    case kBatchNorm:
      return library.batch_norm_eval_launch(small(0), small(1), pointer(0), pointer(1), pointer(2), pointer(3), pointer(4), result(0), n[2], n[3], n[4],
                                       p.doubles[0], device, stream);
    case kGemm:
      return library.gemm_bias_act_residual_launch(small(0), small(1), pointer(0), n[2], small(3), pointer(1), n[4], small(5), pointer(2), pointer(3), n[7],
                                              n[6] * n[7], result(0), n[7], n[6], n[7], n[8], n[9], n[10], n[11], n[6] * n[7], device, stream);
    case kAttention:
      return library.attention_launch(small(0), pointer(0), pointer(1), pointer(2), result(0), n[1], n[2], n[3], n[4], n[5], n + 6, n + 9, n + 12, n + 15,
                                 p.doubles[0], small(18), device, stream);
  }
  return TQ_INTERNAL;
}

// A new reference: the scratch tensor a plan's launch needs, or None.
PyObject* needed(const Plan& plan, const Call& call, void* stream) {
  const int64_t bytes = plan.family == kReduce || plan.family == kTransposed ? plan.ints[5] : 0;
  if (bytes <= 0) Py_RETURN_NONE;
  return PyObject_CallFunction(workspace_function, "iKL", call.device, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)),
                               static_cast<long long>(bytes));
}

PyObject* run(PyObject* const* values, Py_ssize_t count, bool by_type) {
  if (count < 2 || !PyLong_CheckExact(values[0])) Py_RETURN_NONE;
  Call call;
  call.key.push_back(PyLong_AsLongLong(values[0]));
  if (!read(call, values + 1, count - 1, by_type)) Py_RETURN_NONE;
  const std::shared_ptr<const Plan> plan = find(call.key);
  if (plan == nullptr) Py_RETURN_NONE;
  void* const stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(call.device)).stream();
  void* scratch = nullptr;
  size_t scratch_bytes = 0;
  THPObjectPtr block(needed(*plan, call, stream));      // keeps the scratch until the launch has it, or an exception (no memory) leaves
  if (!block) return nullptr;
  if (THPVariable_Check(block.get())) {
    const at::Tensor& t = THPVariable_Unpack(block.get());
    scratch = t.mutable_data_ptr();
    scratch_bytes = static_cast<size_t>(t.numel());
  }
  std::vector<at::Tensor> out;
  tq_status status;
  {
    pybind11::gil_scoped_release unlocked;
    const c10::Device device(c10::kCUDA, static_cast<c10::DeviceIndex>(call.device));
    out.reserve(plan->outputs.size());
    for (const Output& o : plan->outputs)
      out.push_back(o.packed ? at::detail::empty_cuda(o.sizes, o.dtype, device, std::nullopt)
                             : at::detail::empty_strided_cuda(o.sizes, o.strides, o.dtype, device));
    status = launch(*plan, call, out, scratch, scratch_bytes, stream);
  }
  if (status != TQ_OK) Py_RETURN_NONE;
  if (out.size() == 1) return THPVariable_Wrap(std::move(out[0]));
  PyObject* tuple = PyTuple_New(static_cast<Py_ssize_t>(out.size()));
  if (tuple == nullptr) return nullptr;
  for (size_t i = 0; i < out.size(); ++i) PyTuple_SET_ITEM(tuple, static_cast<Py_ssize_t>(i), THPVariable_Wrap(std::move(out[i])));
  return tuple;
}

// call(code, *operands): numbers are part of the signature. elementwise(code, *operands): numbers are arguments of the launch.
PyObject* call_planned(PyObject*, PyObject* const* values, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  return run(values, count, false);
  END_HANDLE_TH_ERRORS
}
PyObject* call_elementwise(PyObject*, PyObject* const* values, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  return run(values, count, true);
  END_HANDLE_TH_ERRORS
}

bool int_list(PyObject* value, std::vector<int64_t>& to) {
  PyObject* fast = PySequence_Fast(value, "a sequence of integers");
  if (fast == nullptr) return false;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(fast); ++i) {
    const int64_t number = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(fast, i));
    if (number == -1 && PyErr_Occurred()) {
      Py_DECREF(fast);
      return false;
    }
    to.push_back(number);
  }
  Py_DECREF(fast);
  return true;
}

// keep(by_type, code, operands, family, outputs, ints, doubles, layouts, holder): outputs are tensors whose types, sizes and strides
// the results of later calls have; layouts the bytes of tq_layout structures. Whether the plan was kept.
PyObject* keep(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  int by_type = 0, family = 0;
  long long code = 0;
  PyObject *operands, *outputs, *ints, *doubles, *holder;
  Py_buffer layouts;
  if (!PyArg_ParseTuple(args, "pLO!iO!OO!y*O", &by_type, &code, &PyTuple_Type, &operands, &family, &PyTuple_Type, &outputs, &ints, &PyTuple_Type, &doubles,
                        &layouts, &holder))
    return nullptr;
  auto plan = std::make_shared<Plan>();
  plan->layouts.resize(layouts.len / sizeof(tq_layout));
  std::memcpy(plan->layouts.data(), layouts.buf, plan->layouts.size() * sizeof(tq_layout));
  PyBuffer_Release(&layouts);
  Call call;
  call.key.push_back(code);
  if (family < 0 || family > kAttention || !read(call, PySequence_Fast_ITEMS(operands), PyTuple_GET_SIZE(operands), by_type != 0)) Py_RETURN_FALSE;
  plan->family = static_cast<Family>(family);
  if (!int_list(ints, plan->ints)) return nullptr;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(doubles); ++i) plan->doubles.push_back(PyFloat_AsDouble(PyTuple_GET_ITEM(doubles, i)));
  if (PyErr_Occurred()) return nullptr;
  // Behind the operands that `launch` reads come numbers, whose values the key holds, unless a number came as a tensor: the long way
  // read its value, of which the key has nothing.
  const Py_ssize_t operands_of[] = {kMostOperands, 1, 1, 1, 3, plan->ints.size() > 0 && plan->ints[0] == 0 ? 1 : 3, 5, 4, 3};
  for (Py_ssize_t i = operands_of[family]; i < PyTuple_GET_SIZE(operands); ++i)
    if (THPVariable_Check(PyTuple_GET_ITEM(operands, i))) Py_RETURN_FALSE;
  // what `launch` reads of each family
  const size_t least[] = {2, 6, 2, 5, 4, 6, 5, 12, 19};
  const bool has_double = family == kLayerNorm || family == kTransposed || family == kBatchNorm || family == kAttention;
  if (plan->ints.size() < least[family] || (has_double && plan->doubles.empty()) ||
      (family == kPack && plan->ints.size() < 2 + 2 * static_cast<size_t>(plan->ints[1])))
    Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(outputs); ++i) {
    PyObject* o = PyTuple_GET_ITEM(outputs, i);
    if (!THPVariable_Check(o)) Py_RETURN_FALSE;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.get_device() != call.device) Py_RETURN_FALSE;
    // (contiguous tensors may have any stride along an axis of one element, and later results have the first one's)
    Output output{t.sizes().vec(), t.strides().vec(), t.scalar_type(), false};
    output.packed = c10::IntArrayRef(output.strides) == c10::IntArrayRef(c10::contiguous_strides(t.sizes()));
    plan->outputs.push_back(std::move(output));
  }
  if (plan->outputs.empty()) Py_RETURN_FALSE;
  if (family == kFused) plan->ints.push_back(1);      // (never without a divisor to point at)
  if (family == kFused && plan->layouts.empty()) plan->layouts.resize(1);
  plan->key = std::move(call.key);
  if (holder != Py_None) {
    Py_INCREF(holder);
    plan->holder = holder;
  }
  if (find(plan->key) == nullptr) {
    const uint64_t hash = hash_of(plan->key);
    remember(hash, std::move(plan));
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyObject* setup(PyObject*, PyObject* args) {
  PyObject *parameter, *workspace;
  const char* path;
  if (!PyArg_ParseTuple(args, "OOs", &parameter, &workspace, &path)) return nullptr;
  void* const handle = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (handle == nullptr || !(find_entry(handle, "tq_fused_launch", library.fused_launch) &&
        find_entry(handle, "tq_reduce_launch", library.reduce_launch) &&
        find_entry(handle, "tq_pack_launch", library.pack_launch) &&
        find_entry(handle, "tq_softmax_launch", library.softmax_launch) &&
        find_entry(handle, "tq_layer_norm_launch", library.layer_norm_launch) &&
        find_entry(handle, "tq_softmax_transposed_launch", library.softmax_transposed_launch) &&
        find_entry(handle, "tq_layer_norm_transposed_launch", library.layer_norm_transposed_launch) &&
        find_entry(handle, "tq_batch_norm_eval_launch", library.batch_norm_eval_launch) &&
        find_entry(handle, "tq_gemm_bias_act_residual_launch", library.gemm_bias_act_residual_launch) &&
        find_entry(handle, "tq_attention_launch", library.attention_launch))) {
    PyErr_Format(PyExc_ImportError, "%s: %s", path, dlerror());
    return nullptr;
  }
  Py_INCREF(parameter);
  Py_INCREF(workspace);
  Py_XSETREF(parameter_class, parameter);
  Py_XSETREF(workspace_function, workspace);
  Py_RETURN_NONE;
}

PyObject* size(PyObject*, PyObject*) { return PyLong_FromSize_t(plans().young.size() + plans().old.size()); }

PyMethodDef methods[] = {
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_planned)), METH_FASTCALL, nullptr},
    {"elementwise", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_elementwise)), METH_FASTCALL, nullptr},
    {"keep", keep, METH_VARARGS, nullptr},
    {"setup", setup, METH_VARARGS, nullptr},
    {"size", size, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_launcher", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__launcher() {
  PyObject* const made = PyModule_Create(&module);
  // the torch and the Python whose headers these are, for the importer to compare
  if (made != nullptr && PyModule_AddStringConstant(made, "BUILT_FOR", TQ_BUILT_FOR) != 0) {
    Py_DECREF(made);
    return nullptr;
  }
  return made;
}
