// The Python side's per-call work as a CPython extension (module _native): the
// addresses behind tensors, parts lists and per-sequence dicts are gathered here
// and handed to the C ABI in one call.
//
// A decode batch hands over dozens of tensors per call, and through ctypes each
// of them cost an attribute lookup, a method call and a wrapped integer: 100 us
// of Python for a mixer step of 32 sequences whose kernels take 44 us, 19 us for
// an 8-sequence DeltaNet update of 4 us; here both are hidden behind the kernels.
// Only the calls of the per-token path come through this file; set-up stays with
// ctypes.
// Every function returns the C ABI's status, which the caller turns into an
// exception, and runs the call itself without the interpreter lock, as ctypes
// does. bind() takes the handle of the already loaded library, so nothing here
// links against it.
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include <memory>
#include <vector>

#include "gufo_cuda.h"

namespace {

struct Api {
  decltype(&gufo_cuda_matmul) matmul;
  decltype(&gufo_cuda_matmul_device) matmul_device;
  decltype(&gufo_cuda_delta_rule_device) delta_rule;
  decltype(&gufo_cuda_deltanet_linear_device) deltanet_linear;
  decltype(&gufo_cuda_deltanet_step_device) deltanet_step;
  decltype(&gufo_cuda_route_device) route;
  decltype(&gufo_cuda_moe_ffn_device) moe_ffn;
  decltype(&gufo_cuda_moe_layer_device) moe_layer;
  decltype(&gufo_cuda_decoder_step) decoder_step;
  decltype(&gufo_cuda_decoder_step_tokens) decoder_step_tokens;
  decltype(&gufo_cuda_host_take) host_take;
  decltype(&gufo_cuda_host_give) host_give;
} api;

// Raised to the interpreter as whatever exception is already set.
struct Failed {};

PyObject* Must(PyObject* o) {
  if (o == nullptr) {
    throw Failed();
  }
  return o;
}

long long Int(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    throw Failed();
  }
  return v;
}

int SmallInt(PyObject* o) {
  const long long v = Int(o);
  if (v < INT32_MIN || v > INT32_MAX) {
    PyErr_SetString(PyExc_OverflowError, "gufo_cuda: integer out of range");
    throw Failed();
  }
  return static_cast<int>(v);
}

float Float(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    throw Failed();
  }
  return static_cast<float>(v);
}

struct Ref {
  explicit Ref(PyObject* o) : o(Must(o)) {}
  ~Ref() { Py_DECREF(o); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  PyObject* o;
};

// Device or host address of a torch tensor, numpy array or raw integer; None is null.
template <typename T>
T* Ptr(PyObject* o) {
  if (o == Py_None) {
    return nullptr;
  }
  if (THPVariable_Check(o)) {
    return static_cast<T*>(THPVariable_Unpack(o).data_ptr());
  }
  if (PyLong_Check(o)) {
    void* p = PyLong_AsVoidPtr(o);
    if (p == nullptr && PyErr_Occurred()) {
      throw Failed();
    }
    return static_cast<T*>(p);
  }
  if (PyObject_HasAttrString(o, "__array_interface__")) {   // numpy
    Py_buffer view;
    if (PyObject_GetBuffer(o, &view, PyBUF_STRIDED_RO) == 0) {
      void* p = view.buf;
      PyBuffer_Release(&view);   // the array outlives the call: the caller holds it
      return static_cast<T*>(p);
    }
    PyErr_Clear();   // an element type that the buffer protocol has no name for
    Ref ctypes(PyObject_GetAttrString(o, "ctypes"));
    Ref data(PyObject_GetAttrString(ctypes.o, "data"));
    return static_cast<T*>(PyLong_AsVoidPtr(data.o));
  }
  Ref data(PyObject_CallMethod(o, "data_ptr", nullptr));
  return static_cast<T*>(PyLong_AsVoidPtr(data.o));
}

int64_t RowStride(PyObject* o) {
  if (THPVariable_Check(o) && THPVariable_Unpack(o).dim() > 0) {
    return THPVariable_Unpack(o).stride(0);
  }
  Ref s(PyObject_CallMethod(o, "stride", "i", 0));
  return Int(s.o);
}

// The keys of the per-sequence dicts, interned once.
struct Keys {
  PyObject *state, *state_out, *q, *k, *v, *decay, *beta, *y, *in, *h, *conv_in, *conv_out, *conv_saved, *ssm,
      *ssm_out, *ssm_spec, *n_tokens, *get;
} keys;

// One sequence's description: a dict, which keeps its values alive, or any other
// mapping, whose values are held here.
struct Entries {
  explicit Entries(PyObject* o) : o(o), plain(PyDict_CheckExact(o)) {}
  ~Entries() {
    for (PyObject* v : held) {
      Py_DECREF(v);
    }
  }
  Entries(const Entries&) = delete;
  Entries& operator=(const Entries&) = delete;
  PyObject* Hold(PyObject* v) {
    held.push_back(Must(v));
    return v;
  }
  // A required entry (KeyError as from `seq[key]`).
  PyObject* Item(PyObject* key) {
    if (!plain) {
      return Hold(PyObject_GetItem(o, key));
    }
    PyObject* v = PyDict_GetItemWithError(o, key);
    if (v == nullptr) {
      if (!PyErr_Occurred()) {
        PyErr_SetObject(PyExc_KeyError, key);
      }
      throw Failed();
    }
    return v;
  }
  PyObject* Optional(PyObject* key) {
    if (!plain) {
      return Hold(PyObject_CallMethodObjArgs(o, keys.get, key, nullptr));
    }
    PyObject* v = PyDict_GetItemWithError(o, key);
    if (v == nullptr && PyErr_Occurred()) {
      throw Failed();
    }
    return v == nullptr ? Py_None : v;
  }
  PyObject* o;
  bool plain;
  std::vector<PyObject*> held;
};

gufo_cuda_ctx* Context(PyObject* o) { return static_cast<gufo_cuda_ctx*>(PyLong_AsVoidPtr(o)); }

// parts: a ctypes array of gufo_cuda_rows (used in place), or a sequence of
// (matrix, first, rows).
struct Parts {
  explicit Parts(PyObject* o) {
    if (PyObject_CheckBuffer(o)) {
      if (PyObject_GetBuffer(o, &view, PyBUF_ND) == 0) {
        if (view.itemsize == sizeof(gufo_cuda_rows)) {
          held = true;
          data = static_cast<const gufo_cuda_rows*>(view.buf);
          count = static_cast<int>(view.len / sizeof(gufo_cuda_rows));
          return;
        }
        PyBuffer_Release(&view);
      }
      PyErr_Clear();   // an array of numbers: a sequence like any other
    }
    Ref list(PySequence_Fast(o, "gufo_cuda: parts must be a sequence"));
    count = static_cast<int>(PySequence_Fast_GET_SIZE(list.o));
    own.resize(count > 0 ? count : 1);
    for (int i = 0; i < count; ++i) {
      Ref part(PySequence_Fast(PySequence_Fast_GET_ITEM(list.o, i), "gufo_cuda: a part is (matrix, first, rows)"));
      if (PySequence_Fast_GET_SIZE(part.o) != 3) {
        PyErr_SetString(PyExc_ValueError, "gufo_cuda: a part is (matrix, first, rows)");
        throw Failed();
      }
      own[i].w = Int(PySequence_Fast_GET_ITEM(part.o, 0));
      own[i].first = Int(PySequence_Fast_GET_ITEM(part.o, 1));
      own[i].rows = Int(PySequence_Fast_GET_ITEM(part.o, 2));
    }
    data = own.data();
  }
  ~Parts() {
    if (held) {
      PyBuffer_Release(&view);
    }
  }
  Parts(const Parts&) = delete;
  Parts& operator=(const Parts&) = delete;
  Py_buffer view;
  bool held = false;
  std::vector<gufo_cuda_rows> own;
  const gufo_cuda_rows* data = nullptr;
  int count = 0;
};

// One C array element per dict of a sequence of dicts.
template <typename Seq>
struct Gathered {
  template <typename Fill>
  Gathered(PyObject* seqs, Fill fill) : list(PySequence_Fast(seqs, "gufo_cuda: a sequence of dicts is needed")) {
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(list.o);
    all.reserve(n > 0 ? n : 1);
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* d = PySequence_Fast_GET_ITEM(list.o, i);
      all.emplace_back();
      if (PyDict_CheckExact(d)) {
        Entries plain(d);
        fill(plain, &all.back());
      } else {
        mappings.emplace_back(std::make_unique<Entries>(d));
        fill(*mappings.back(), &all.back());
      }
    }
  }
  const Seq* data() const { return all.data(); }
  int count() const { return static_cast<int>(all.size()); }
  Ref list;
  std::vector<Seq> all;
  std::vector<std::unique_ptr<Entries>> mappings;
};

template <typename Call>
PyObject* Unlocked(Call call) {
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = call();
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(status);
}

// Runs `body` with the arguments; C++ exceptions become Python ones.
template <typename Body>
PyObject* Guarded(Py_ssize_t got, Py_ssize_t want, Body body) {
  if (got != want) {
    PyErr_Format(PyExc_TypeError, "_native: %zd arguments expected, got %zd", want, got);
    return nullptr;
  }
  try {
    return body();
  } catch (const Failed&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// matmul(ctx, parts, x address, tokens, y address): host buffers.
PyObject* Matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 5, [&] {
    Parts parts(a[1]);
    gufo_cuda_ctx* ctx = Context(a[0]);
    const float* x = Ptr<const float>(a[2]);
    const int tokens = SmallInt(a[3]);
    float* y = Ptr<float>(a[4]);
    return Unlocked([&] { return api.matmul(ctx, parts.data, parts.count, x, tokens, y); });
  });
}

// matmul_device(ctx, parts, count or None for all, x, tokens, y)
PyObject* MatmulDevice(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 6, [&] {
    Parts parts(a[1]);
    gufo_cuda_ctx* ctx = Context(a[0]);
    const int count = a[2] == Py_None ? parts.count : SmallInt(a[2]);
    if (count > parts.count) {
      PyErr_SetString(PyExc_ValueError, "gufo_cuda: more parts than the array holds");
      throw Failed();
    }
    const float* x = Ptr<const float>(a[3]);
    const int tokens = SmallInt(a[4]);
    float* y = Ptr<float>(a[5]);
    return Unlocked([&] { return api.matmul_device(ctx, parts.data, count, x, tokens, y); });
  });
}

// delta_rule(ctx, seqs, key_heads, value_heads, head_dim)
PyObject* DeltaRule(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 5, [&] {
    gufo_cuda_ctx* ctx = Context(a[0]);
    const Gathered<gufo_cuda_delta_seq> seqs(a[1], [](Entries& d, gufo_cuda_delta_seq* s) {
      s->state = Ptr<float>(d.Item(keys.state));
      s->state_out = Ptr<float>(d.Optional(keys.state_out));
      s->q = Ptr<const float>(d.Item(keys.q));
      s->k = Ptr<const float>(d.Item(keys.k));
      s->v = Ptr<const float>(d.Item(keys.v));
      s->decay = Ptr<const float>(d.Item(keys.decay));
      s->beta = Ptr<const float>(d.Item(keys.beta));
      s->y = Ptr<float>(d.Item(keys.y));
    });
    const int hk = SmallInt(a[2]), hv = SmallInt(a[3]), dk = SmallInt(a[4]);
    const int count = seqs.count();
    return Unlocked([&] { return api.delta_rule(ctx, seqs.data(), count, hk, hv, dk); });
  });
}

// deltanet_linear(ctx, layer, seqs)
PyObject* DeltaNetLinear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 3, [&] {
    gufo_cuda_ctx* ctx = Context(a[0]);
    const long long layer = Int(a[1]);
    const Gathered<gufo_cuda_linear_seq> seqs(a[2], [](Entries& d, gufo_cuda_linear_seq* s) {
      s->in = Ptr<const float>(d.Item(keys.in));
      s->conv_in = Ptr<const float>(d.Item(keys.conv_in));
      s->conv_out = Ptr<float>(d.Item(keys.conv_out));
      s->ssm = Ptr<float>(d.Item(keys.ssm));
      s->ssm_out = Ptr<float>(d.Optional(keys.ssm_out));
      s->y = Ptr<float>(d.Item(keys.y));
    });
    const int count = seqs.count();
    return Unlocked([&] { return api.deltanet_linear(ctx, layer, seqs.data(), count); });
  });
}

// deltanet_step(ctx, layer, alpha, beta, norm, eps, seqs)
PyObject* DeltaNetStep(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 7, [&] {
    gufo_cuda_ctx* ctx = Context(a[0]);
    const long long layer = Int(a[1]), alpha = Int(a[2]), beta = Int(a[3]);
    const float* norm = Ptr<const float>(a[4]);
    const float eps = Float(a[5]);
    const Gathered<gufo_cuda_deltanet_step_seq> seqs(a[6], [](Entries& d, gufo_cuda_deltanet_step_seq* s) {
      PyObject *in = d.Item(keys.in), *h = d.Item(keys.h), *y = d.Item(keys.y);
      s->n_tokens = SmallInt(d.Item(keys.n_tokens));
      s->in = Ptr<const float>(in);
      s->in_stride = RowStride(in);
      s->h = Ptr<const float>(h);
      s->h_stride = RowStride(h);
      s->conv_in = Ptr<const float>(d.Item(keys.conv_in));
      s->conv_out = Ptr<float>(d.Item(keys.conv_out));
      s->conv_saved = Ptr<float>(d.Optional(keys.conv_saved));
      s->ssm = Ptr<float>(d.Item(keys.ssm));
      s->ssm_spec = Ptr<float>(d.Optional(keys.ssm_spec));
      s->y = Ptr<float>(y);
      s->y_stride = RowStride(y);
    });
    const int count = seqs.count();
    return Unlocked([&] { return api.deltanet_step(ctx, layer, alpha, beta, norm, eps, seqs.data(), count); });
  });
}

// route(ctx, router, stride, tokens, experts, k, chosen, weights, shared_scale)
PyObject* Route(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 9, [&] {
    gufo_cuda_ctx* ctx = Context(a[0]);
    const float* router = Ptr<const float>(a[1]);
    const int stride = SmallInt(a[2]), tokens = SmallInt(a[3]), experts = SmallInt(a[4]), k = SmallInt(a[5]);
    int* chosen = Ptr<int>(a[6]);
    float *weights = Ptr<float>(a[7]), *scale = Ptr<float>(a[8]);
    return Unlocked([&] { return api.route(ctx, router, stride, tokens, experts, k, chosen, weights, scale); });
  });
}

gufo_cuda_expert_bank Bank(PyObject* o) {
  gufo_cuda_expert_bank bank;
  Py_buffer view;
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) {
    throw Failed();
  }
  const bool fits = view.len == static_cast<Py_ssize_t>(sizeof(bank));
  if (fits) {
    bank = *static_cast<const gufo_cuda_expert_bank*>(view.buf);
  }
  PyBuffer_Release(&view);
  if (!fits) {
    PyErr_SetString(PyExc_TypeError, "gufo_cuda: an ExpertBank is needed");
    throw Failed();
  }
  return bank;
}

// moe_ffn(ctx, bank, ids, weights, scale, tokens, k, x, x_stride, shared, ffn, act, expert_out, out)
PyObject* MoeFfn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 14, [&] {
    gufo_cuda_ctx* ctx = Context(a[0]);
    const gufo_cuda_expert_bank bank = Bank(a[1]);
    const int* ids = Ptr<const int>(a[2]);
    const float *weights = Ptr<const float>(a[3]), *scale = Ptr<const float>(a[4]);
    const int tokens = SmallInt(a[5]), k = SmallInt(a[6]);
    const float* x = Ptr<const float>(a[7]);
    const long long x_stride = Int(a[8]);
    const float* shared = Ptr<const float>(a[9]);
    float *ffn = Ptr<float>(a[10]), *act = Ptr<float>(a[11]), *expert_out = Ptr<float>(a[12]), *out = Ptr<float>(a[13]);
    return Unlocked([&] {
      return api.moe_ffn(ctx, &bank, ids, weights, scale, tokens, k, x, x_stride, shared, ffn, act, expert_out, out);
    });
  });
}

// moe_layer(ctx, bank, router, stride, tokens, k, chosen, weights, scale, x, x_stride, shared, ffn, act, expert_out, out)
PyObject* MoeLayer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 16, [&] {
    gufo_cuda_ctx* ctx = Context(a[0]);
    const gufo_cuda_expert_bank bank = Bank(a[1]);
    const float* router = Ptr<const float>(a[2]);
    const int stride = SmallInt(a[3]), tokens = SmallInt(a[4]), k = SmallInt(a[5]);
    int* chosen = Ptr<int>(a[6]);
    float *weights = Ptr<float>(a[7]), *scale = Ptr<float>(a[8]);
    const float* x = Ptr<const float>(a[9]);
    const long long x_stride = Int(a[10]);
    const float* shared = Ptr<const float>(a[11]);
    float *ffn = Ptr<float>(a[12]), *act = Ptr<float>(a[13]), *expert_out = Ptr<float>(a[14]), *out = Ptr<float>(a[15]);
    return Unlocked([&] {
      return api.moe_layer(ctx, &bank, router, stride, tokens, k, chosen, weights, scale, x, x_stride, shared, ffn, act,
                           expert_out, out);
    });
  });
}

// decoder_step(decoder address, token, logits)
PyObject* DecoderStep(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 3, [&] {
    auto* decoder = static_cast<gufo_cuda_decoder*>(PyLong_AsVoidPtr(a[0]));
    const int token = SmallInt(a[1]);
    float* logits = Ptr<float>(a[2]);
    return Unlocked([&] { return api.decoder_step(decoder, token, logits); });
  });
}

// decoder_step_tokens(decoder address, tokens, want_logits, logits)
PyObject* DecoderStepTokens(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 4, [&] {
    auto* decoder = static_cast<gufo_cuda_decoder*>(PyLong_AsVoidPtr(a[0]));
    Ref list(PySequence_Fast(a[1], "gufo_cuda: tokens must be a sequence"));
    const int count = static_cast<int>(PySequence_Fast_GET_SIZE(list.o));
    std::vector<int> tokens(count > 0 ? count : 1);
    for (int i = 0; i < count; ++i) {
      tokens[i] = SmallInt(PySequence_Fast_GET_ITEM(list.o, i));
    }
    const int want = SmallInt(a[2]);
    float* logits = Ptr<float>(a[3]);
    return Unlocked([&] { return api.decoder_step_tokens(decoder, tokens.data(), count, want, logits); });
  });
}

// A block of the library's pinned memory, exposed through the buffer protocol and
// given back when the last array over it has gone.
struct HostBuffer {
  PyObject_HEAD
  void* data;
  Py_ssize_t bytes;
};

void HostBufferDealloc(PyObject* self) {
  api.host_give(reinterpret_cast<HostBuffer*>(self)->data);
  Py_TYPE(self)->tp_free(self);
}

int HostBufferGet(PyObject* self, Py_buffer* view, int flags) {
  auto* b = reinterpret_cast<HostBuffer*>(self);
  return PyBuffer_FillInfo(view, self, b->data, b->bytes, 0, flags);
}

PyBufferProcs host_buffer_procs = {HostBufferGet, nullptr};
PyTypeObject host_buffer_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// host_buffer(ctx, bytes): a HostBuffer, or None where the pool is at its bound.
PyObject* NewHostBuffer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return Guarded(n, 2, [&]() -> PyObject* {
    gufo_cuda_ctx* ctx = Context(a[0]);
    const long long bytes = Int(a[1]);
    void* data = nullptr;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = api.host_take(ctx, static_cast<size_t>(bytes), &data);
    Py_END_ALLOW_THREADS
    if (status != GUFO_CUDA_OK || data == nullptr) {
      Py_RETURN_NONE;
    }
    auto* b = PyObject_New(HostBuffer, &host_buffer_type);
    if (b == nullptr) {
      api.host_give(data);
      throw Failed();
    }
    b->data = data;
    b->bytes = bytes;
    return reinterpret_cast<PyObject*>(b);
  });
}

// bind(library handle): looks the entry points up in the loaded library.
PyObject* Bind(PyObject*, PyObject* handle) {
  void* lib = PyLong_AsVoidPtr(handle);
  if (lib == nullptr) {
    return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "_native.bind: null library handle");
  }
  const char* missing = nullptr;
  auto find = [&](auto* fn, const char* name) {
    void* at = dlsym(lib, name);
    if (at == nullptr) {
      missing = name;
    }
    *fn = reinterpret_cast<std::remove_reference_t<decltype(*fn)>>(at);
  };
  find(&api.matmul, "gufo_cuda_matmul");
  find(&api.matmul_device, "gufo_cuda_matmul_device");
  find(&api.delta_rule, "gufo_cuda_delta_rule_device");
  find(&api.deltanet_linear, "gufo_cuda_deltanet_linear_device");
  find(&api.deltanet_step, "gufo_cuda_deltanet_step_device");
  find(&api.route, "gufo_cuda_route_device");
  find(&api.moe_ffn, "gufo_cuda_moe_ffn_device");
  find(&api.moe_layer, "gufo_cuda_moe_layer_device");
  find(&api.decoder_step, "gufo_cuda_decoder_step");
  find(&api.decoder_step_tokens, "gufo_cuda_decoder_step_tokens");
  find(&api.host_take, "gufo_cuda_host_take");
  find(&api.host_give, "gufo_cuda_host_give");
  if (missing != nullptr) {
    return PyErr_Format(PyExc_ImportError, "libgufo_cuda.so has no %s", missing);
  }
  Py_RETURN_NONE;
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", Bind, METH_O, nullptr},
    FAST("matmul", Matmul),
    FAST("matmul_device", MatmulDevice),
    FAST("delta_rule", DeltaRule),
    FAST("deltanet_linear", DeltaNetLinear),
    FAST("deltanet_step", DeltaNetStep),
    FAST("route", Route),
    FAST("moe_ffn", MoeFfn),
    FAST("moe_layer", MoeLayer),
    FAST("decoder_step", DecoderStep),
    FAST("decoder_step_tokens", DecoderStepTokens),
    FAST("host_buffer", NewHostBuffer),
    {nullptr, nullptr, 0, nullptr},
};
#undef FAST

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Per-call host path of the C ABI.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  struct {
    PyObject** key;
    const char* name;
  } const names[] = {{&keys.state, "state"}, {&keys.state_out, "state_out"}, {&keys.q, "q"}, {&keys.k, "k"},
                     {&keys.v, "v"}, {&keys.decay, "decay"}, {&keys.beta, "beta"}, {&keys.y, "y"}, {&keys.in, "in"},
                     {&keys.h, "h"}, {&keys.conv_in, "conv_in"}, {&keys.conv_out, "conv_out"},
                     {&keys.conv_saved, "conv_saved"}, {&keys.ssm, "ssm"}, {&keys.ssm_out, "ssm_out"},
                     {&keys.ssm_spec, "ssm_spec"}, {&keys.n_tokens, "n_tokens"},
                     {&keys.get, "get"}};
  for (const auto& n : names) {
    if ((*n.key = PyUnicode_InternFromString(n.name)) == nullptr) {
      return nullptr;
    }
  }
  host_buffer_type.tp_name = "gufo_npu_b200._native.HostBuffer";
  host_buffer_type.tp_basicsize = sizeof(HostBuffer);
  host_buffer_type.tp_dealloc = HostBufferDealloc;
  host_buffer_type.tp_as_buffer = &host_buffer_procs;
  host_buffer_type.tp_flags = Py_TPFLAGS_DEFAULT;
  if (PyType_Ready(&host_buffer_type) != 0) {
    return nullptr;
  }
  PyObject* m = PyModule_Create(&module);
  // torch's C++ classes differ from release to release: load_native compares.
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", GUFO_TORCH_VERSION) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
