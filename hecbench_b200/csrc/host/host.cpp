// Python-side launch path of libhq: turns a call with torch tensors into the C-ABI
// call on the tensor's device and current stream.
//
// What bounds a small call is this path, not its kernel: argument checks, device
// switch and stream look-up in Python around ctypes cost 11-14 us per launch, the
// kernels of a decode step run in 3-10 us.  The same steps here cost well under a
// microsecond on top of the launch itself; the Python wrappers in api.py keep the
// signatures, the shape rules and the error texts.
//
// An Entry is one C-ABI function of one loaded library (the address comes from the
// ctypes handle, so another build of the library can stand in).  Its parameter list
// says how each Python argument becomes a C argument; a tensor is checked for
// device, type and contiguity.  The call releases the GIL around the launch, like
// ctypes does, and holds no state: threads and streams are the caller's.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <utility>

namespace {

constexpr int kMaxArgs = 20;

union Value {
  void* p;
  long long i;
  double f;
};

enum class Kind { kTensor, kOptionalTensor, kRaw, kInt, kFloat, kFourInts };
struct Param {
  Kind kind;
  const char* name;
  at::ScalarType type;
};

using Invoke = int (*)(void* fn, const Value* v, void* stream);

template <typename T>
inline T get(const Value& v) {
  if constexpr (std::is_pointer_v<T>) return static_cast<T>(v.p);
  else if constexpr (std::is_floating_point_v<T>) return static_cast<T>(v.f);
  else return static_cast<T>(v.i);
}
// C signature (P..., stream) -> int
template <typename... P>
struct Signature {
  template <size_t... I>
  static int run(void* fn, const Value* v, void* stream, std::index_sequence<I...>) {
    return reinterpret_cast<int (*)(P..., void*)>(fn)(get<P>(v[I])..., stream);
  }
  static int invoke(void* fn, const Value* v, void* stream) {
    return run(fn, v, stream, std::index_sequence_for<P...>{});
  }
};

struct Spec {
  const char* symbol;
  int device_arg;  // the argument whose device and current stream the launch uses
  Invoke invoke;
  int n;
  Param params[kMaxArgs];
};

using VP = void*;
constexpr Param T(const char* name, at::ScalarType t) { return {Kind::kTensor, name, t}; }
constexpr Param O(const char* name, at::ScalarType t) { return {Kind::kOptionalTensor, name, t}; }
// a CUDA tensor whose type and layout the wrapper has looked at
constexpr Param R(const char* name) { return {Kind::kRaw, name, at::kByte}; }
constexpr Param I() { return {Kind::kInt, nullptr, at::kByte}; }
constexpr Param F() { return {Kind::kFloat, nullptr, at::kByte}; }
// up to four numbers, zeros for the rest, passed as const int[4]
constexpr Param S(const char* name) { return {Kind::kFourInts, name, at::kByte}; }
constexpr auto f32 = at::kFloat;
constexpr auto f16 = at::kHalf;
constexpr auto i32 = at::kInt;
constexpr auto u8 = at::kByte;
constexpr auto i8 = at::kChar;

template <typename... P, typename... Q>
constexpr Spec spec(const char* symbol, int device_arg, Signature<P...>, Q... q) {
  static_assert(sizeof...(P) == sizeof...(Q), "one parameter per C argument");
  return {symbol, device_arg, &Signature<P...>::invoke, (int)sizeof...(Q), {q...}};
}

const Spec kSpecs[] = {
    spec("hq_q3_gemv_f32", 1, Signature<VP, VP, VP, VP, VP, int, int>{}, T("vec", f32),
         T("mat", i32), T("mul", f32), T("scales", f32), T("zeros", f32), I(), I()),
    spec("hq_q3_gemv_f16in", 1, Signature<VP, VP, VP, VP, VP, int, int>{}, T("vec", f16),
         T("mat", i32), T("mul", f32), T("scales", f32), T("zeros", f32), I(), I()),
    spec("hq_q3_dequant_f32", 0, Signature<VP, VP, VP, VP, int, int>{}, T("mat", i32),
         T("scales", f32), T("zeros", f32), T("W", f32), I(), I()),
    spec("hq_q3_dequant_f16", 0, Signature<VP, VP, VP, VP, int, int>{}, T("mat", i32),
         T("scales", f32), T("zeros", f32), T("W", f16), I(), I()),
    spec("hq_bnb_quantize_u8", 1, Signature<VP, VP, VP, size_t>{}, T("code", f32), T("A", f32),
         T("out", u8), I()),
    spec("hq_nf4_dequant_f16", 0, Signature<VP, VP, VP, VP, size_t, int, int>{}, T("B", u8),
         T("absmax", f32), T("lut16", f32), T("out", f16), I(), I(), I()),
    spec("hq_nf4_gemv_f16", 1, Signature<VP, VP, VP, VP, VP, int, int, int, int>{}, T("A", f16),
         T("B", u8), T("absmax", f32), T("lut16", f32), T("out", f16), I(), I(), I(), I()),
    spec("hq_vllm_static_scaled_int8_quant", 1, Signature<VP, VP, int, int, int, float, int>{},
         T("output", i8), R("input"), I(), I(), I(), F(), I()),
    spec("hq_vllm_dynamic_scaled_int8_quant", 1, Signature<VP, VP, int, int, int, VP, VP>{},
         T("output", i8), R("input"), I(), I(), I(), T("scales", f32), O("azp", i32)),
    spec("hq_gemv_f16", 0, Signature<VP, VP, VP, int, int>{}, T("mat", f16), T("vec", f16),
         T("out", f16), I(), I()),
    spec("hq_gemv_int8_f16", 0, Signature<VP, VP, VP, int, int, float, float>{}, T("mat", i8),
         T("vec", f16), T("out", f16), I(), I(), F(), F()),
    spec("hq_gemv_int4_f16", 0, Signature<VP, VP, VP, int, int, float, float>{}, T("mat", u8),
         T("vec", f16), T("out", f16), I(), I(), F(), F()),
    spec("hq_zero_point", 0, Signature<VP, VP, int, int, int, int, VP, VP>{}, T("x_min", f32),
         T("x_max", f32), I(), I(), I(), I(), T("scale", f32), T("zero_point", i32)),
    spec("hq_q3_quantize", 0, Signature<VP, int, int, int, VP, VP, VP, VP, size_t>{}, R("W"), I(),
         I(), I(), T("mat", i32), T("scales", f32), T("zeros", f32), T("workspace", u8), I()),
    spec("hq_lutgemm_quantize", 0, Signature<VP, int, int, int, int, int, VP, VP, VP>{}, R("W"),
         I(), I(), I(), I(), I(), T("bW", i32), T("alpha", f16), O("q_bias", f16)),
    spec("hq_nf4_quantize", 0, Signature<VP, int, size_t, int, VP, int, VP, VP>{}, R("W"), I(),
         I(), I(), T("lut16", f32), I(), T("B", u8), T("absmax", f32)),
    spec("hq_mxfp4_qdq", 0, Signature<VP, VP, size_t, int>{}, R("a"), R("y"), I(), I()),
    spec("hq_mxfp4_quantize", 0, Signature<VP, VP, VP, size_t, int>{}, R("a"), T("codes", u8),
         T("scales", u8), I(), I()),
    spec("hq_mxfp4_dequantize", 0, Signature<VP, VP, VP, size_t, int>{}, T("codes", u8),
         T("scales", u8), R("out"), I(), I()),
    spec("hq_gemv_fused_f16", 0, Signature<VP, VP, float, VP, VP, int, int, int>{}, T("x", f16),
         O("gamma", f16), F(), T("mat", f16), T("out", f16), I(), I(), I()),
    spec("hq_gemv_fused_int8_f16", 0,
         Signature<VP, VP, float, VP, VP, int, int, float, float, int>{}, T("x", f16),
         O("gamma", f16), F(), T("mat", i8), T("out", f16), I(), I(), F(), F(), I()),
    spec("hq_gemv_fused_int4_f16", 0,
         Signature<VP, VP, float, VP, VP, int, int, float, float, int>{}, T("x", f16),
         O("gamma", f16), F(), T("mat", u8), T("out", f16), I(), I(), F(), F(), I()),
    spec("hq_gemv_fused_nf4_f16", 0,
         Signature<VP, VP, float, VP, VP, VP, VP, int, int, int, int, int>{}, T("x", f16),
         O("gamma", f16), F(), T("mat", u8), T("absmax", f32), T("lut16", f32), T("out", f16), I(),
         I(), I(), I(), I()),
    spec("hq_lutgemm_nqmv", 2, Signature<VP, VP, VP, VP, VP, int, int, int, int, VP, size_t>{},
         T("output", f16), T("input", f16), T("bWeight", i32), T("alpha", f16), O("q_bias", f16),
         I(), I(), I(), I(), T("workspace", u8), I()),
    spec("hq_aqlm_1x16_matvec", 0, Signature<VP, VP, VP, VP, int, int, VP, int, VP>{}, R("A"),
         T("B", f16), T("C", f16), T("codebook", f16), I(), I(), S("codebook_a_sizes"), I(),
         O("scales", f16)),
    spec("hq_aqlm_2x8_matvec", 0, Signature<VP, VP, VP, VP, int, int, VP>{}, T("A", u8),
         T("B", f16), T("C", f16), T("codebooks", f16), I(), I(), O("scales", f16)),
    spec("hq_qgemm_q3_f16", 0,
         Signature<VP, VP, VP, VP, VP, int, int, int, int, VP, size_t, VP>{}, T("X", f16),
         T("mat", i32), T("scales", f16), T("zeros", f16), T("out", f16), I(), I(), I(), I(),
         O("workspace", u8), I(), O("status", i32)),
    spec("hq_qgemm_nf4_f16", 0,
         Signature<VP, VP, VP, VP, VP, int, int, int, int, int, VP, size_t, VP>{}, T("X", f16),
         T("B", u8), T("absmax", f32), T("lut16", f32), T("out", f16), I(), I(), I(), I(), I(),
         O("workspace", u8), I(), O("status", i32)),
    spec("hq_qgemm_q3_f16_peers", 0,
         Signature<VP, VP, VP, VP, VP, long long, int, int, int, int, int, VP, size_t, VP>{},
         T("X", f16), T("mat", i32), T("scales", f16), T("zeros", f16), I(), I(), I(), I(), I(),
         I(), I(), O("workspace", u8), I(), O("status", i32)),
    spec("hq_qgemm_nf4_f16_peers", 0,
         Signature<VP, VP, VP, VP, VP, long long, int, int, int, int, int, int, VP, size_t, VP>{},
         T("X", f16), T("B", u8), T("absmax", f32), T("lut16", f32), I(), I(), I(), I(), I(), I(),
         I(), I(), O("workspace", u8), I(), O("status", i32)),
};

struct Entry {
  PyObject_HEAD
  vectorcallfunc call;
  const Spec* spec;
  void* fn;
  PyObject* on_error;  // called with (symbol, status) for a status that is not 0; raises
};

// An error text that shows an attribute of the tensor, e.g. its dtype.
void set_type_error(PyObject* tensor, const Param& q) {
  PyObject* got = PyObject_GetAttrString(tensor, "dtype");
  PyObject* want = THPVariable_Check(tensor)
                       ? reinterpret_cast<PyObject*>(torch::getTHPDtype(q.type))
                       : nullptr;
  if (got && want) PyErr_Format(PyExc_TypeError, "%s: expected dtype %S, got %S", q.name, want, got);
  Py_XDECREF(got);
}

// The tensor behind `o`, or nullptr with a Python error set.
const at::Tensor* checked_tensor(PyObject* o, const Param& q) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s: expected a torch.Tensor", q.name);
    return nullptr;
  }
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda()) {
    PyErr_Format(PyExc_TypeError, "%s: must be a CUDA tensor (there is no CPU path)", q.name);
    return nullptr;
  }
  if (q.kind != Kind::kRaw && t.scalar_type() != q.type) {
    set_type_error(o, q);
    return nullptr;
  }
  if (!t.is_contiguous()) {
    PyErr_Format(PyExc_TypeError, "%s: must be contiguous", q.name);
    return nullptr;
  }
  return &t;
}

PyObject* entry_call(PyObject* self_, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  HANDLE_TH_ERRORS
  Entry* self = reinterpret_cast<Entry*>(self_);
  const Spec& s = *self->spec;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != s.n || (kwnames && PyTuple_GET_SIZE(kwnames))) {
    PyErr_Format(PyExc_TypeError, "%s takes %d positional arguments", s.symbol, s.n);
    return nullptr;
  }
  Value v[kMaxArgs];
  int four[4];
  c10::DeviceIndex device = -1;
  for (int k = 0; k < s.n; k++) {
    const Param& q = s.params[k];
    switch (q.kind) {
      case Kind::kOptionalTensor:
        if (args[k] == Py_None) {
          v[k].p = nullptr;
          break;
        }
        [[fallthrough]];
      case Kind::kTensor:
      case Kind::kRaw: {
        const at::Tensor* t = checked_tensor(args[k], q);
        if (!t) return nullptr;
        v[k].p = t->data_ptr();
        if (k == s.device_arg) device = t->device().index();
        break;
      }
      case Kind::kInt:
        v[k].i = PyLong_AsLongLong(args[k]);
        if (v[k].i == -1 && PyErr_Occurred()) return nullptr;
        break;
      case Kind::kFloat:
        v[k].f = PyFloat_AsDouble(args[k]);
        if (v[k].f == -1.0 && PyErr_Occurred()) return nullptr;
        break;
      case Kind::kFourInts: {
        PyObject* seq = PySequence_Fast(args[k], q.name);
        if (!seq) return nullptr;
        const Py_ssize_t given = PySequence_Fast_GET_SIZE(seq);
        if (given > 4) {
          Py_DECREF(seq);
          PyErr_Format(PyExc_ValueError, "%s: expected at most four numbers", q.name);
          return nullptr;
        }
        for (int i = 0; i < 4; i++) four[i] = 0;
        for (Py_ssize_t i = 0; i < given; i++) {  // what int() takes
          PyObject* whole = PyNumber_Long(PySequence_Fast_GET_ITEM(seq, i));
          if (!whole) break;
          four[i] = (int)PyLong_AsUnsignedLongLongMask(whole);
          Py_DECREF(whole);
        }
        Py_DECREF(seq);
        if (PyErr_Occurred()) return nullptr;
        v[k].p = four;
        break;
      }
    }
  }
  int status;
  {
    c10::cuda::CUDAGuard guard(device);
    void* stream = c10::cuda::getCurrentCUDAStream(device).stream();
    Py_BEGIN_ALLOW_THREADS
    status = s.invoke(self->fn, v, stream);
    Py_END_ALLOW_THREADS
  }
  if (status != 0) return PyObject_CallFunction(self->on_error, "si", s.symbol, status);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* entry_new(PyTypeObject* type, PyObject* args, PyObject*) {
  const char* symbol;
  unsigned long long address;
  PyObject* on_error;
  if (!PyArg_ParseTuple(args, "sKO", &symbol, &address, &on_error)) return nullptr;
  for (const Spec& s : kSpecs) {
    if (std::strcmp(s.symbol, symbol) != 0) continue;
    Entry* e = reinterpret_cast<Entry*>(type->tp_alloc(type, 0));
    if (!e) return nullptr;
    e->call = entry_call;
    e->spec = &s;
    e->fn = reinterpret_cast<void*>(address);
    e->on_error = Py_NewRef(on_error);
    return reinterpret_cast<PyObject*>(e);
  }
  return PyErr_Format(PyExc_KeyError, "no entry %s", symbol);
}

void entry_dealloc(PyObject* self) {
  Py_XDECREF(reinterpret_cast<Entry*>(self)->on_error);
  Py_TYPE(self)->tp_free(self);
}

PyTypeObject EntryType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// empty(like, dtype, *sizes): an uninitialised tensor on the device of `like`.
PyObject* host_empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 3 || n > 6 || !THPVariable_Check(args[0]) || !THPDtype_Check(args[1])) {
    PyErr_SetString(PyExc_TypeError, "empty(like, dtype, *sizes)");
    return nullptr;
  }
  const at::Tensor& like = THPVariable_Unpack(args[0]);
  if (!like.is_cuda()) {
    PyErr_SetString(PyExc_TypeError, "expected a CUDA tensor (there is no CPU path)");
    return nullptr;
  }
  int64_t sizes[4];
  for (Py_ssize_t k = 2; k < n; k++) {
    sizes[k - 2] = PyLong_AsLongLong(args[k]);
    if (sizes[k - 2] == -1 && PyErr_Occurred()) return nullptr;
  }
  return THPVariable_Wrap(at::Tensor(at::detail::empty_cuda(
      at::IntArrayRef(sizes, (size_t)(n - 2)),
      reinterpret_cast<THPDtype*>(args[1])->scalar_type, like.device(), std::nullopt)));
  END_HANDLE_TH_ERRORS
}

// place(t): a number for the device of t and the current stream there.
PyObject* host_place(PyObject*, PyObject* t) {
  HANDLE_TH_ERRORS
  if (!THPVariable_Check(t) || !THPVariable_Unpack(t).is_cuda()) {
    PyErr_SetString(PyExc_TypeError, "expected a CUDA tensor (there is no CPU path)");
    return nullptr;
  }
  const c10::DeviceIndex d = THPVariable_Unpack(t).device().index();
  const auto s = reinterpret_cast<unsigned long long>(c10::cuda::getCurrentCUDAStream(d).stream());
  return Py_BuildValue("(iK)", (int)d, s);
  END_HANDLE_TH_ERRORS
}

// capturing(t): whether the current stream on the device of t is being captured.
PyObject* host_capturing(PyObject*, PyObject* t) {
  HANDLE_TH_ERRORS
  if (!THPVariable_Check(t) || !THPVariable_Unpack(t).is_cuda()) {
    PyErr_SetString(PyExc_TypeError, "expected a CUDA tensor (there is no CPU path)");
    return nullptr;
  }
  c10::cuda::CUDAGuard guard(THPVariable_Unpack(t).device().index());
  return PyBool_FromLong(c10::cuda::currentStreamCaptureStatusMayInitCtx() !=
                         c10::cuda::CaptureStatus::None);
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"empty", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&host_empty)), METH_FASTCALL,
     nullptr},
    {"place", &host_place, METH_O, nullptr},
    {"capturing", &host_capturing, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  EntryType.tp_name = "hecbench_b200._host.Entry";
  EntryType.tp_basicsize = sizeof(Entry);
  EntryType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  EntryType.tp_vectorcall_offset = offsetof(Entry, call);
  EntryType.tp_call = PyVectorcall_Call;
  EntryType.tp_new = entry_new;
  EntryType.tp_dealloc = entry_dealloc;
  if (PyType_Ready(&EntryType) < 0) return nullptr;
  PyObject* m = PyModule_Create(&kModule);
  if (!m) return nullptr;
  PyObject* symbols = PyList_New(0);
  for (const Spec& s : kSpecs) {
    PyObject* name = PyUnicode_FromString(s.symbol);
    PyList_Append(symbols, name);
    Py_DECREF(name);
  }
  if (PyModule_AddObject(m, "symbols", symbols) < 0 ||
      PyModule_AddObjectRef(m, "Entry", reinterpret_cast<PyObject*>(&EntryType)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
