// The launchers of the C ABI as CPython functions.  A call is a dozen pointers and one or two small structs, and through
// ctypes their conversion cost more than the launch behind it (attention prologue 5.9 us, prefill 4.9, norm + RoPE 3.1,
// split 2.6 on the host, without the library's own work): prompts in short calls and eager serving steps were bound by
// it.  Here an argument is one type check and, for a tensor, one data_ptr() call; the interpreter lock is released
// around the library as ctypes does.
//
// Nothing of the library is linked in: kernels.py hands over the addresses of the entry points it has loaded and the
// exception types that carry a failing status.  Read here are the plain kinds of arguments: tensors, addresses, streams, the
// shapes, integers (whatever has __index__; they wrap to their field, as in ctypes) and floats.  A call with any argument
// that does not read as such goes to `through_ctypes` of kernels.py, so that what ctypes accepts is accepted and what it
// refuses is refused with its own exceptions.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../../include/rib200.h"

#include <cstddef>
#include <cstdint>
#include <tuple>
#include <type_traits>
#include <utility>

namespace {

PyObject *g_through_ctypes = nullptr; // (name, arguments ...)
PyObject *g_errors[2] = {nullptr, nullptr}; // attention, gated delta
PyObject *g_data_ptr = nullptr;
PyObject *g_cuda_stream = nullptr;

// The readers return false for what they do not take, with or without an exception set.
bool read_integer(PyObject *o, unsigned long long &value) {
  value = PyLong_AsUnsignedLongLongMask(o); // calls __index__ of what is no int
  return !(value == static_cast<unsigned long long>(-1) && PyErr_Occurred());
}
bool read_float(PyObject *o, float &value) {
  const double v = PyFloat_AsDouble(o);
  value = static_cast<float>(v);
  return !(v == -1.0 && PyErr_Occurred());
}
template <class T> bool read_field(PyObject *o, const char *name, T &field) {
  PyObject *attribute = PyObject_GetAttrString(o, name);
  if (attribute == nullptr) {
    return false;
  }
  bool ok;
  if constexpr (std::is_same_v<T, float>) {
    ok = read_float(attribute, field);
  } else {
    unsigned long long value = 0;
    ok = read_integer(attribute, value);
    field = static_cast<T>(value);
  }
  Py_DECREF(attribute);
  return ok;
}

// ---- one converter per kind of argument: read() from Python, get() for the call ----
template <class T> struct Integer {
  T value{};
  bool read(PyObject *o) {
    unsigned long long v = 0;
    if (!read_integer(o, v)) {
      return false;
    }
    value = static_cast<T>(v);
    return true;
  }
  T get() const { return value; }
};
struct Float {
  float value = 0.0F;
  bool read(PyObject *o) { return read_float(o, value); }
  float get() const { return value; }
};
// None, an address, or an object with data_ptr(); converts to whatever pointer the parameter is
struct Address {
  void *value;
  template <class T> operator T *() const { return static_cast<T *>(value); }
};
bool read_address(PyObject *owned, void *&value) {
  if (owned == nullptr) {
    return false;
  }
  unsigned long long v = 0;
  const bool ok = PyLong_Check(owned) && read_integer(owned, v);
  Py_DECREF(owned);
  value = reinterpret_cast<void *>(static_cast<std::uintptr_t>(v));
  return ok;
}
struct Pointer {
  void *value = nullptr;
  bool read(PyObject *o) {
    if (o == Py_None) {
      return true;
    }
    return read_address(PyLong_Check(o) ? Py_NewRef(o) : PyObject_CallMethodNoArgs(o, g_data_ptr), value);
  }
  Address get() const { return Address{value}; }
};
// None, a handle, or an object with cuda_stream
struct Stream {
  void *value = nullptr;
  bool read(PyObject *o) {
    if (o == Py_None) {
      return true;
    }
    return read_address(PyLong_Check(o) ? Py_NewRef(o) : PyObject_GetAttr(o, g_cuda_stream), value);
  }
  void *get() const { return value; }
};
struct AttentionShape {
  Rib200AttentionShape value{};
  bool read(PyObject *o) {
    return read_field(o, "tokens", value.tokens) && read_field(o, "query_heads", value.query_heads) &&
           read_field(o, "kv_heads", value.kv_heads) && read_field(o, "head_dim", value.head_dim) &&
           read_field(o, "max_context_tokens", value.max_context_tokens) &&
           read_field(o, "past_tokens", value.past_tokens);
  }
  const Rib200AttentionShape *get() const { return &value; }
};
struct RopeShape {
  Rib200QkNormRopeShape value{};
  bool read(PyObject *o) {
    return read_field(o, "tokens", value.tokens) && read_field(o, "heads", value.heads) &&
           read_field(o, "head_dim", value.head_dim) && read_field(o, "rotary_dim", value.rotary_dim) &&
           read_field(o, "position_offset", value.position_offset) && read_field(o, "rope_base", value.rope_base);
  }
  const Rib200QkNormRopeShape *get() const { return &value; }
};
struct AttentionPolicy {
  Rib200AttentionLaunchPolicy value{};
  bool read(PyObject *o) {
    return read_field(o, "implementation", value.implementation) &&
           read_field(o, "kv_cache_dtype", value.kv_cache_dtype) &&
           read_field(o, "kv_cache_layout", value.kv_cache_layout);
  }
  Rib200AttentionLaunchPolicy get() const { return value; }
};
struct DecodePlan {
  Rib200OnlineDecodePlan value{};
  bool read(PyObject *o) {
    return read_field(o, "resolved_mode", value.resolved_mode) &&
           read_field(o, "partition_tokens", value.partition_tokens) &&
           read_field(o, "split_k_threshold_tokens", value.split_k_threshold_tokens) &&
           read_field(o, "context_bucket_tokens", value.context_bucket_tokens) &&
           read_field(o, "active_partition_capacity", value.active_partition_capacity);
  }
  const Rib200OnlineDecodePlan *get() const { return &value; }
};
struct DeltaShape {
  Rib200GatedDeltaShape value{};
  bool read(PyObject *o) {
    return read_field(o, "tokens", value.tokens) && read_field(o, "hidden_size", value.hidden_size) &&
           read_field(o, "key_heads", value.key_heads) && read_field(o, "value_heads", value.value_heads) &&
           read_field(o, "key_dim", value.key_dim) && read_field(o, "value_dim", value.value_dim) &&
           read_field(o, "conv_width", value.conv_width) && read_field(o, "epsilon", value.epsilon);
  }
  const Rib200GatedDeltaShape *get() const { return &value; }
};
struct DeltaPolicy {
  Rib200GatedDeltaLaunchPolicy value{};
  bool read(PyObject *o) {
    if (!read_field(o, "schedule", value.schedule) || !read_field(o, "warps_per_block", value.warps_per_block)) {
      return false;
    }
    PyObject *transposed = PyObject_GetAttrString(o, "transposed_boundary_state");
    if (transposed == nullptr) {
      return false;
    }
    const int truth = PyObject_IsTrue(transposed);
    Py_DECREF(transposed);
    value.transposed_boundary_state = truth > 0 ? 1 : 0;
    return truth >= 0;
  }
  Rib200GatedDeltaLaunchPolicy get() const { return value; }
};

using Size = Integer<std::size_t>;
using Code = Integer<std::int32_t>;
using Byte = Integer<std::uint8_t>;
using P = Pointer;

// An entry point: its address in the loaded library, the kinds of its arguments and whose errors it raises.
template <auto Declared, int Errors, class... Kinds> struct Entry {
  static inline decltype(Declared) function = nullptr;
  static inline PyObject *name = nullptr;
  static PyObject *call(PyObject *, PyObject *const *args, Py_ssize_t count) {
    if (count != static_cast<Py_ssize_t>(sizeof...(Kinds))) {
      PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", static_cast<Py_ssize_t>(sizeof...(Kinds)), count);
      return nullptr;
    }
    return run(args, std::index_sequence_for<Kinds...>{});
  }
  template <std::size_t... I> static PyObject *run(PyObject *const *args, std::index_sequence<I...>) {
    std::tuple<Kinds...> kinds;
    if (!(std::get<I>(kinds).read(args[I]) && ...)) {
      PyErr_Clear();
      if (g_through_ctypes == nullptr) {
        PyErr_SetString(PyExc_RuntimeError, "entry point is not bound");
        return nullptr;
      }
      return PyObject_CallFunctionObjArgs(g_through_ctypes, name, args[I]..., nullptr);
    }
    if (function == nullptr) {
      PyErr_SetString(PyExc_RuntimeError, "entry point is not bound");
      return nullptr;
    }
    Rib200Status status;
    Py_BEGIN_ALLOW_THREADS;
    status = function(std::get<I>(kinds).get()...);
    Py_END_ALLOW_THREADS;
    if (status.code != RIB200_STATUS_OK) {
      PyObject *error = PyObject_CallFunction(g_errors[Errors], "is", static_cast<int>(status.code),
                                              status.message != nullptr ? status.message : "");
      if (error != nullptr) {
        PyErr_SetObject(reinterpret_cast<PyObject *>(Py_TYPE(error)), error);
        Py_DECREF(error);
      }
      return nullptr;
    }
    Py_RETURN_NONE;
  }
  static void bind(void *address, PyObject *bound_name) {
    function = reinterpret_cast<decltype(Declared)>(address);
    Py_XSETREF(name, Py_NewRef(bound_name));
  }
};

constexpr int kAttention = 0;
constexpr int kDelta = 1;

// Arguments in the order of the declarations in rib200.h.
using CausalAttention = Entry<rib200_causal_attention, kAttention, P, P, P, P, P, P, Size, P, Size, AttentionShape, Code,
                              AttentionPolicy, Stream>;
using Prefill = Entry<rib200_online_attention_prefill, kAttention, P, P, P, P, P, P, Size, AttentionShape, Code, Byte, Byte,
                      Stream>;
using Decode = Entry<rib200_online_attention_decode, kAttention, P, P, P, P, P, P, Size, P, Size, AttentionShape, Code, Byte,
                     Byte, DecodePlan, P, Stream>;
using DecodeEarly = Entry<rib200_online_attention_decode_early_kv_fetch, kAttention, P, P, P, P, P, P, Size, P, Size,
                          AttentionShape, Code, Byte, Byte, DecodePlan, Stream>;
using BatchedDecode = Entry<rib200_batched_decode_attention, kAttention, P, P, P, P, P, P, P, P, Size, Size, P, Size, Stream>;
using PagedDecode = Entry<rib200_paged_decode_attention, kAttention, P, P, P, P, P, P, Size, P, Size, P, Size, P, Size, Stream>;
using NormRope = Entry<rib200_qk_norm_rope, kAttention, P, P, P, RopeShape, Float, Code, Code, Stream, P>;
using SplitGate = Entry<rib200_split_full_query_gate, kAttention, P, P, P, Size, Size, Size, Code, Stream>;
using Prologue = Entry<rib200_attention_prologue, kAttention, P, P, P, P, P, P, P, P, P, AttentionShape, Size, Float, Float,
                       Code, Code, Code, P, Stream>;
using GatedDelta = Entry<rib200_gated_delta, kDelta, P, P, P, P, P, P, P, P, P, Size, DeltaShape, DeltaPolicy, Code, Code,
                         Stream>;
using DeltaCore = Entry<rib200_gdn_core, kDelta, P, P, P, P, P, P, P, P, Size, Size, Size, Size, Size, Size, Code, Stream>;
using BatchedDelta = Entry<rib200_batched_gdn_decode, kDelta, P, P, P, P, P, P, P, Size, Size, Size, Stream>;

using FastCall = PyObject *(*)(PyObject *, PyObject *const *, Py_ssize_t);
struct Row {
  const char *name;
  FastCall call;
  void (*bind)(void *, PyObject *);
};
template <class E> constexpr Row row(const char *name) { return Row{name, &E::call, &E::bind}; }
const Row kRows[] = {
    row<CausalAttention>("rib200_causal_attention"),
    row<Prefill>("rib200_online_attention_prefill"),
    row<Decode>("rib200_online_attention_decode"),
    row<DecodeEarly>("rib200_online_attention_decode_early_kv_fetch"),
    row<BatchedDecode>("rib200_batched_decode_attention"),
    row<PagedDecode>("rib200_paged_decode_attention"),
    row<NormRope>("rib200_qk_norm_rope"),
    row<SplitGate>("rib200_split_full_query_gate"),
    row<Prologue>("rib200_attention_prologue"),
    row<GatedDelta>("rib200_gated_delta"),
    row<DeltaCore>("rib200_gdn_core"),
    row<BatchedDelta>("rib200_batched_gdn_decode"),
};
constexpr std::size_t kRowCount = sizeof(kRows) / sizeof(kRows[0]);

// bind(address of a name, through_ctypes, attention error, gated-delta error)
PyObject *bind(PyObject *, PyObject *const *args, Py_ssize_t count) {
  if (count != 4) {
    PyErr_SetString(PyExc_TypeError, "bind takes two functions and two exception types");
    return nullptr;
  }
  for (const Row &row : kRows) {
    PyObject *name = PyUnicode_FromString(row.name);
    PyObject *address = name != nullptr ? PyObject_CallOneArg(args[0], name) : nullptr;
    if (address == nullptr) {
      Py_XDECREF(name);
      return nullptr;
    }
    void *value = PyLong_AsVoidPtr(address);
    Py_DECREF(address);
    if (value == nullptr) {
      if (!PyErr_Occurred()) {
        PyErr_Format(PyExc_ImportError, "%s has no address", row.name);
      }
      Py_DECREF(name);
      return nullptr;
    }
    row.bind(value, name);
    Py_DECREF(name);
  }
  Py_XSETREF(g_through_ctypes, Py_NewRef(args[1]));
  Py_XSETREF(g_errors[kAttention], Py_NewRef(args[2]));
  Py_XSETREF(g_errors[kDelta], Py_NewRef(args[3]));
  Py_RETURN_NONE;
}

PyMethodDef g_methods[kRowCount + 2];
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_call", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__call() {
  g_methods[0] = {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr};
  for (std::size_t i = 0; i < kRowCount; ++i) {
    g_methods[i + 1] = {kRows[i].name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(kRows[i].call)),
                        METH_FASTCALL, nullptr};
  }
  g_data_ptr = PyUnicode_InternFromString("data_ptr");
  g_cuda_stream = PyUnicode_InternFromString("cuda_stream");
  if (g_data_ptr == nullptr || g_cuda_stream == nullptr) {
    return nullptr;
  }
  return PyModule_Create(&g_module);
}
