// How Python calls the C entry points of the kernel libraries: torch tensors go in as they are.
//
// A prompt of a length that does not come again is launched call by call (nine launches a layer), and small models wait
// for the host then.  ctypes took 4 us for twenty arguments (an object an argument, a lock round every call) beside 1 to 2
// for the checks of the tensors and 2 for an output tensor made through Python; here a call is a loop over its arguments.
//
// entry(address) gives a callable whose arguments say by their type what they are:
//   a tensor, None, a ctypes structure or array     a pointer (to the tensor's data, null, to the object's memory)
//   an int (a bool, an address)                     an integer of up to 64 bits
//   a float                                         a 32-bit float
// The entry points take these three kinds alone, return an int, and take at most MAX_INTS of the first two and MAX_FLOATS of
// the third.  Under both calling conventions that a B200 host has (System V x86-64, AAPCS64) integers and floats are counted
// apart: each kind fills its own registers in order, what integers do not fit follows on the stack in slots of eight bytes,
// and what a callee does not ask for it does not look at.  So one call through one type with all of them reaches every such
// function; the order between ints and floats of a signature does not matter, their order among themselves does.
//
// record() ... finish(slots): the calls that this thread makes in between are kept beside being made, and replay(values) makes them
// again with other tensors in the places of `slots` (a layer's weights and cache, its input and its output).  A step's layers
// that are alike make the same calls on the same sizes: one goes through Python, the others are issued by one loop here (a
// layer of a prompt took the host 108 us, nine launches of 5).  A recording lives as long as its step.  It is of use only where every
// place that another layer's memory could stand in is known: an argument that leads into a slot's memory behind its start, a plain
// address of it, a block of parameters or a descriptor that is no slot (addresses may stand in it), or a product of another view
// than the slot's make replay() leave the layers to Python.
#include <torch/csrc/Device.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/torch.h>
#include <ATen/EmptyTensor.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#if !defined(__x86_64__) && !defined(__aarch64__)
#error "the calling convention of this host is not known to pass integers and floats apart"
#endif
#if defined(_WIN32) || defined(__APPLE__)
#error "System V x86-64 or AAPCS64 with eight-byte stack slots"
#endif

namespace {

constexpr int MAX_INTS = 48, FEW_INTS = 16, MAX_FLOATS = 8;
using I = std::int64_t;

#define I8(a, n) a[n], a[n + 1], a[n + 2], a[n + 3], a[n + 4], a[n + 5], a[n + 6], a[n + 7]
#define F8(f) f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]
#define T8 I, I, I, I, I, I, I, I
#define TF float, float, float, float, float, float, float, float
using FewFn = int (*)(T8, T8, TF);
using MostFn = int (*)(T8, T8, T8, T8, T8, T8, TF);

struct Entry {
  PyObject_HEAD
  vectorcallfunc call;
  void* fn;
};

PyObject *structure_type, *array_type;      // of ctypes

// What an integer argument was.
enum : unsigned char { NUMBER, TENSOR, OBJECT };      // (OBJECT: a ctypes structure or array)

// A call as it was made: an entry point with its arguments (and, behind finish(), which of them are a slot's), or a product of
// the library.
struct Call {
  void* fn = nullptr;                       // null: out = x . w^T
  int ni = 0, nf = 0;
  I ints[MAX_INTS];
  float floats[MAX_FLOATS];
  unsigned char kind[MAX_INTS];
  int slot[MAX_INTS];
  at::Tensor x, w, out;
  int x_slot = -1, w_slot = -1, out_slot = -1;
};
struct Recording {
  std::vector<Call> calls;
  std::vector<PyObject*> held;              // whose memory the calls' pointers lead to
  struct Slot { at::Tensor tensor; bool aligned; };
  std::vector<Slot> slots;                  // as they were recorded (no tensor: a ctypes object)
  ~Recording() { for (PyObject* o : held) Py_DECREF(o); }
};
thread_local Recording* recording = nullptr;

int invoke(void* fn, const I* ints, int ni, const float* floats) {
  if (ni <= FEW_INTS) return reinterpret_cast<FewFn>(fn)(I8(ints, 0), I8(ints, 8), F8(floats));
  return reinterpret_cast<MostFn>(fn)(I8(ints, 0), I8(ints, 8), I8(ints, 16), I8(ints, 24), I8(ints, 32), I8(ints, 40), F8(floats));
}

PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  HANDLE_TH_ERRORS
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (kwnames != nullptr && PyTuple_GET_SIZE(kwnames) != 0) {
    PyErr_SetString(PyExc_TypeError, "an entry point takes no keyword arguments");
    return nullptr;
  }
  I ints[MAX_INTS] = {};
  float floats[MAX_FLOATS] = {};
  unsigned char kind[MAX_INTS] = {};
  int ni = 0, nf = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* a = args[i];
    if (PyFloat_CheckExact(a)) {
      if (nf == MAX_FLOATS) { PyErr_SetString(PyExc_TypeError, "too many floats for an entry point"); return nullptr; }
      floats[nf++] = static_cast<float>(PyFloat_AS_DOUBLE(a));
      continue;
    }
    I v = 0;
    unsigned char is = NUMBER;
    if (a == Py_None) {
    } else if (PyLong_Check(a)) {
      v = PyLong_AsLongLong(a);
      if (v == -1 && PyErr_Occurred()) return nullptr;
    } else if (THPVariable_Check(a)) {
      is = TENSOR;
      v = reinterpret_cast<I>(THPVariable_Unpack(a).mutable_data_ptr());
    } else if (PyObject_IsInstance(a, structure_type) == 1 || PyObject_IsInstance(a, array_type) == 1) {
      // (the caller's argument holds the object, and with it its memory, until the call has returned)
      Py_buffer view;
      if (PyObject_GetBuffer(a, &view, PyBUF_SIMPLE) != 0) return nullptr;
      is = OBJECT;
      v = reinterpret_cast<I>(view.buf);
      PyBuffer_Release(&view);
    } else {
      PyErr_Format(PyExc_TypeError, "argument %zd of an entry point is a %s", i, Py_TYPE(a)->tp_name);
      return nullptr;
    }
    if (ni == MAX_INTS) { PyErr_SetString(PyExc_TypeError, "too many arguments for an entry point"); return nullptr; }
    kind[ni] = is;
    if (recording != nullptr && is != NUMBER) {
      Py_INCREF(a);
      recording->held.push_back(a);
    }
    ints[ni++] = v;
  }
  void* fn = reinterpret_cast<Entry*>(self)->fn;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = invoke(fn, ints, ni, floats);
  Py_END_ALLOW_THREADS
  if (recording != nullptr && rc == 0) {      // (another result is a question's answer, which the wrapper has gone by, or an error)
    Call& c = recording->calls.emplace_back();
    c.fn = fn;
    c.ni = ni;
    c.nf = nf;
    std::copy(ints, ints + MAX_INTS, c.ints);
    std::copy(floats, floats + MAX_FLOATS, c.floats);
    std::copy(kind, kind + MAX_INTS, c.kind);
  }
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

PyTypeObject entry_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* make_entry(PyObject*, PyObject* address) {
  void* fn = PyLong_AsVoidPtr(address);
  if (fn == nullptr) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "an entry point has an address");
    return nullptr;
  }
  Entry* e = PyObject_New(Entry, &entry_type);
  if (e == nullptr) return nullptr;
  e->call = entry_call;
  e->fn = fn;
  return reinterpret_cast<PyObject*>(e);
}

// Whether every argument is None or a tensor for which `holds` is true.
template <typename Holds>
PyObject* all_of(PyObject* const* args, Py_ssize_t n, Holds holds) {
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (args[i] == Py_None) continue;
    if (!THPVariable_Check(args[i])) {
      PyErr_Format(PyExc_TypeError, "a tensor was expected, not a %s", Py_TYPE(args[i])->tp_name);
      return nullptr;
    }
    if (!holds(THPVariable_Unpack(args[i]))) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
}
PyObject* all_cuda(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return all_of(args, n, [](const at::Tensor& t) { return t.is_cuda(); });
  END_HANDLE_TH_ERRORS
}
PyObject* all_contiguous(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return all_of(args, n, [](const at::Tensor& t) { return t.is_contiguous(); });
  END_HANDLE_TH_ERRORS
}

// empty(shape, dtype, device)
PyObject* empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || !PyTuple_Check(args[0]) || !THPDtype_Check(args[1]) || !THPDevice_Check(args[2])) {
    PyErr_SetString(PyExc_TypeError, "empty(shape, dtype, device)");
    return nullptr;
  }
  c10::SmallVector<int64_t, 6> shape;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[0]); ++i) {
    shape.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(args[0], i)));
    if (shape.back() == -1 && PyErr_Occurred()) return nullptr;
  }
  const auto options = at::TensorOptions().dtype(reinterpret_cast<THPDtype*>(args[1])->scalar_type).device(reinterpret_cast<THPDevice*>(args[2])->device);
  at::Tensor out;
  {
    pybind11::gil_scoped_release free;
    out = at::empty(shape, options);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// mm_t(x, w): x . w^T by the library
PyObject* mm_t(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) {
    PyErr_SetString(PyExc_TypeError, "mm_t(x, w)");
    return nullptr;
  }
  const at::Tensor x = THPVariable_Unpack(args[0]), w = THPVariable_Unpack(args[1]);
  at::Tensor out;
  {
    pybind11::gil_scoped_release free;
    out = at::mm(x, w.t());
  }
  if (recording != nullptr) {
    Call& c = recording->calls.emplace_back();
    c.x = x;
    c.w = w;
    c.out = out;
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// ---- recordings
struct RecordingObject {
  PyObject_HEAD
  Recording* r;
};
PyTypeObject recording_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// The address of a tensor's data or a ctypes object's memory; -1 (with an error set) for anything else.
I address_of(PyObject* o) {
  if (THPVariable_Check(o)) return reinterpret_cast<I>(THPVariable_Unpack(o).mutable_data_ptr());
  if (PyObject_IsInstance(o, structure_type) == 1 || PyObject_IsInstance(o, array_type) == 1) {
    Py_buffer view;
    if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) return -1;
    const I at = reinterpret_cast<I>(view.buf);
    PyBuffer_Release(&view);
    return at;
  }
  PyErr_Format(PyExc_TypeError, "a recording's slots are tensors and ctypes objects, not a %s", Py_TYPE(o)->tp_name);
  return -1;
}

PyObject* record(PyObject*, PyObject*) {
  if (recording != nullptr) {
    PyErr_SetString(PyExc_RuntimeError, "this thread records already");
    return nullptr;
  }
  recording = new Recording;
  Py_RETURN_NONE;
}
PyObject* discard(PyObject*, PyObject*) {
  delete recording;
  recording = nullptr;
  Py_RETURN_NONE;
}
// finish(slots) -> the recording.  An argument that leads to the start of a slot's memory is the slot's; a tensor of a product
// likewise.  Where an argument might lead to a slot's memory in another way the recording keeps no slots and replay() does nothing.
PyObject* finish(PyObject*, PyObject* slots) {
  HANDLE_TH_ERRORS
  if (recording == nullptr || !PyTuple_Check(slots)) {
    PyErr_SetString(PyExc_RuntimeError, "finish(slots), a tuple, behind record()");
    return nullptr;
  }
  const int n = static_cast<int>(PyTuple_GET_SIZE(slots));
  std::vector<I> at(n), bytes(n, 1);
  recording->slots.clear();
  for (int i = 0; i < n; ++i) {
    PyObject* o = PyTuple_GET_ITEM(slots, i);
    at[i] = address_of(o);
    if (PyErr_Occurred()) return nullptr;
    recording->slots.push_back({THPVariable_Check(o) ? THPVariable_Unpack(o) : at::Tensor(), at[i] % 16 == 0});
    const at::Tensor& t = recording->slots.back().tensor;
    if (t.defined()) bytes[i] = static_cast<I>(at::detail::computeStorageNbytes(t.sizes(), t.strides(), t.element_size()));
  }
  // (two slots of one address: an argument does not say whose it is, and no other layer is like this one)
  bool known = true;
  for (int i = 0; i < n; ++i) known = known && std::count(at.begin(), at.end(), at[i]) == 1;
  auto slot_of = [&](I address) {
    for (int i = 0; i < n; ++i)
      if (at[i] == address) return i;
    return -1;
  };
  auto inside = [&](I address) {
    for (int i = 0; i < n; ++i)
      if (address >= at[i] && address - at[i] < bytes[i]) return true;
    return false;
  };
  // a tensor of a product: the slot's own view of its memory, or none of it
  auto product_slot = [&](const at::Tensor& t) {
    const I address = reinterpret_cast<I>(t.mutable_data_ptr());
    const int s = slot_of(address);
    if (s < 0) known = known && !inside(address);
    else known = known && recording->slots[s].tensor.defined() && t.sizes() == recording->slots[s].tensor.sizes() &&
                 t.strides() == recording->slots[s].tensor.strides();
    return s;
  };
  for (Call& c : recording->calls) {
    for (int i = 0; i < c.ni; ++i) {
      c.slot[i] = c.kind[i] == NUMBER ? -1 : slot_of(c.ints[i]);
      if (c.slot[i] >= 0) known = known && (c.kind[i] == TENSOR) == recording->slots[c.slot[i]].tensor.defined();
      else known = known && c.kind[i] != OBJECT && !inside(c.ints[i]);
    }
    if (c.fn == nullptr) {
      c.x_slot = product_slot(c.x);
      c.w_slot = product_slot(c.w);
      c.out_slot = product_slot(c.out);
    }
  }
  if (!known) recording->slots.clear();
  RecordingObject* o = PyObject_New(RecordingObject, &recording_type);
  if (o == nullptr) return nullptr;
  o->r = recording;
  recording = nullptr;
  return reinterpret_cast<PyObject*>(o);
  END_HANDLE_TH_ERRORS
}
// replay(recording, values) -> 0, or the first code that is not; None, and nothing done, where a value is not like its slot (an
// entry point chooses its kernel by sizes, types and alignment, the wrappers choose entry points by them).
PyObject* replay(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2 || Py_TYPE(args[0]) != &recording_type || !PyTuple_Check(args[1])) {
    PyErr_SetString(PyExc_TypeError, "replay(recording, values)");
    return nullptr;
  }
  const Recording& r = *reinterpret_cast<RecordingObject*>(args[0])->r;
  const int n = static_cast<int>(PyTuple_GET_SIZE(args[1]));
  if (n != static_cast<int>(r.slots.size())) Py_RETURN_NONE;
  std::vector<I> at(n);
  std::vector<at::Tensor> tensors(n);
  for (int i = 0; i < n; ++i) {
    PyObject* o = PyTuple_GET_ITEM(args[1], i);
    at[i] = address_of(o);
    if (PyErr_Occurred()) return nullptr;
    const at::Tensor& was = r.slots[i].tensor;
    if (THPVariable_Check(o) != was.defined() || (at[i] % 16 == 0) != r.slots[i].aligned) Py_RETURN_NONE;
    if (!was.defined()) continue;
    tensors[i] = THPVariable_Unpack(o);
    if (tensors[i].scalar_type() != was.scalar_type() || tensors[i].device() != was.device() || tensors[i].sizes() != was.sizes() ||
        tensors[i].strides() != was.strides())
      Py_RETURN_NONE;
  }
  int rc = 0;
  {
    pybind11::gil_scoped_release free;
    at::NoGradGuard no_grad;
    for (const Call& c : r.calls) {
      if (c.fn != nullptr) {
        I ints[MAX_INTS];
        std::copy(c.ints, c.ints + MAX_INTS, ints);
        for (int i = 0; i < c.ni; ++i)
          if (c.slot[i] >= 0) ints[i] = at[c.slot[i]];
        rc = invoke(c.fn, ints, c.ni, c.floats);
        if (rc != 0) break;
      } else {
        at::Tensor out = c.out_slot >= 0 ? tensors[c.out_slot] : c.out;
        at::mm_out(out, c.x_slot >= 0 ? tensors[c.x_slot] : c.x, (c.w_slot >= 0 ? tensors[c.w_slot] : c.w).t());
      }
    }
  }
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"record", record, METH_NOARGS, "keep the calls that this thread makes from now on"},
    {"discard", discard, METH_NOARGS, "forget what record() has kept"},
    {"finish", finish, METH_O, "finish(slots): the recording since record()"},
    {"replay", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(replay)), METH_FASTCALL, "replay(recording, values): its calls with values in the slots' places"},
    {"entry", make_entry, METH_O, "entry(address): the C entry point at an address as a callable"},
    {"all_cuda", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(all_cuda)), METH_FASTCALL, "whether every tensor (None counts as one) is on a GPU"},
    {"all_contiguous", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(all_contiguous)), METH_FASTCALL, "whether every tensor (None counts as one) is contiguous"},
    {"empty", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(empty)), METH_FASTCALL, "empty(shape, dtype, device)"},
    {"mm_t", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(mm_t)), METH_FASTCALL, "mm_t(x, w): x . w^T"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  PyObject* ctypes = PyImport_ImportModule("ctypes");
  if (ctypes == nullptr) return nullptr;
  structure_type = PyObject_GetAttrString(ctypes, "Structure");
  array_type = PyObject_GetAttrString(ctypes, "Array");
  Py_DECREF(ctypes);
  if (structure_type == nullptr || array_type == nullptr) return nullptr;
  entry_type.tp_name = "_calls.Entry";
  entry_type.tp_basicsize = sizeof(Entry);
  entry_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  entry_type.tp_vectorcall_offset = offsetof(Entry, call);
  entry_type.tp_call = PyVectorcall_Call;
  entry_type.tp_dealloc = [](PyObject* o) { PyObject_Free(o); };
  recording_type.tp_name = "_calls.Recording";
  recording_type.tp_basicsize = sizeof(RecordingObject);
  recording_type.tp_flags = Py_TPFLAGS_DEFAULT;
  recording_type.tp_dealloc = [](PyObject* o) {
    delete reinterpret_cast<RecordingObject*>(o)->r;
    PyObject_Free(o);
  };
  if (PyType_Ready(&entry_type) < 0 || PyType_Ready(&recording_type) < 0) return nullptr;
  return PyModule_Create(&module);
}
