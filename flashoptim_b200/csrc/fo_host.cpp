// Host path of the fused optimizer steps: a CPython extension that walks a parameter group and
// launches the multi-tensor kernels.
//
// What bounds a step of a small or many-tensor model is not the kernel but the walk over the
// parameters: gradient, state and correction look-ups, extent checks and address packing cost
// 6-7 us per tensor in Python (1.9 ms for the 292 tensors of GPT-2-medium, whose kernel takes
// 0.75 ms).  The same walk here reads the tensors through their C++ objects.  Nothing is cached
// between steps except device copies of address tables, which are compared in full before every
// use, so states may be replaced, emptied or loaded at any time.
//
// A group that this walk does not serve (CPU or non-contiguous tensors, a gradient of another
// dtype, an optimizer with methods of its own in the walk's place, ...) is left untouched and
// reported to the caller, whose Python walk updates it or says what is wrong with it.  It takes the place of the per-tensor launch wrappers of the reference
// (flashoptim/optimizers.py:1535-1583, :2203-2252).
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <ATen/record_function.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <nvtx3/nvToolsExt.h>

#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "fo_api.h"

namespace {

// ---------------------------------------------------------------- library entry points
struct Api {
  decltype(&fo_adam_step) adam_step = nullptr;
  decltype(&fo_momentum_step) momentum_step = nullptr;
  int chunk = 0;
} g_api;

PyObject* g_ensure_status = nullptr;  // ops.step._ensure_status
PyObject* g_native_error = nullptr;   // ops.native.NativeError
bool g_nvtx = false;
uint64_t g_status_ready = 0;  // bit per device whose kernels know their status word
long long g_launches = 0;

PyObject *s_step, *s_error_bits, *s_local_tensor, *s_ensure, *s_check, *s_walked_natively;

// Slots of MaybeQuantizedTensor, read at their offsets: an attribute look-up per slot would be a
// quarter of the whole walk.
PyTypeObject* g_state_type = nullptr;
Py_ssize_t g_off_data = 0, g_off_codes = 0, g_off_scales = 0;

Py_ssize_t slot_offset(PyTypeObject* type, const char* name) {
  PyObject* d = PyObject_GetAttrString(reinterpret_cast<PyObject*>(type), name);
  if (!d) return -1;
  Py_ssize_t off = -1;
  if (Py_TYPE(d) == &PyMemberDescr_Type) off = reinterpret_cast<PyMemberDescrObject*>(d)->d_member->offset;
  else PyErr_Format(PyExc_TypeError, "%s is not a slot", name);
  Py_DECREF(d);
  return off;
}
PyObject* slot(PyObject* o, Py_ssize_t off) {  // borrowed; null for None or never assigned
  PyObject* v = *reinterpret_cast<PyObject**>(reinterpret_cast<char*>(o) + off);
  return v == Py_None ? nullptr : v;
}

// The methods whose place the walk takes, by name.  A class that describes its rule to the walk
// keeps those that it describes in `_walked_natively` (optim/base.py).
PyObject* g_walked = nullptr;

// A class as it was looked at last: the interpreter gives a class another version whenever it, or a
// class above it, is changed.
struct Looked {
  PyTypeObject* type = nullptr;
  unsigned int version = 0;
};

// Whether the class of `opt`, or `opt` itself, has other methods than those; -1 with an exception.
// Every call asks, so a class that is as it was is not looked through again.
int overrides(PyObject* opt, Looked& last) {
  PyTypeObject* type = Py_TYPE(opt);
  const Py_ssize_t n = PyTuple_GET_SIZE(g_walked);
  if (last.type != type || !PyType_HasFeature(type, Py_TPFLAGS_VALID_VERSION_TAG) || type->tp_version_tag == 0 ||
      type->tp_version_tag != last.version) {
    last.type = nullptr;
    PyObject* cls = reinterpret_cast<PyObject*>(type);
    PyObject* known = PyObject_GetAttr(cls, s_walked_natively);
    if (!known) return -1;
    int other = !PyTuple_Check(known) || PyTuple_GET_SIZE(known) != n;
    for (Py_ssize_t i = 0; !other && i < n; ++i) {
      PyObject* now = PyObject_GetAttr(cls, PyTuple_GET_ITEM(g_walked, i));
      other = now ? now != PyTuple_GET_ITEM(known, i) : -1;
      Py_XDECREF(now);
    }
    Py_DECREF(known);
    if (other) return other;
    last.type = type;
    last.version = type->tp_version_tag;
  }
  PyObject* own = PyObject_GenericGetDict(opt, nullptr);
  int other = own ? 0 : -1;
  for (Py_ssize_t i = 0; !other && i < n; ++i) other = PyDict_Contains(own, PyTuple_GET_ITEM(g_walked, i));
  Py_XDECREF(own);
  return other;
}

// ---------------------------------------------------------------- one launch
// Device copy of a table that does not fit the kernel parameters.  It is written and read on one
// stream, the one it was allocated on, and is not freed while its optimizer lives.
struct Table {
  c10::DeviceIndex device;
  c10::StreamId stream;
  int dtype, err, mode;
  std::vector<FoSeg> sent;  // what `dev` holds; empty when that is not known
  size_t n;                 // rows that it has room for, exactly
  at::Tensor dev;
  at::Tensor staged;        // of a captured step: its replays copy from here again
  long long call = 0;       // last call that used it
};

struct Bucket {
  c10::DeviceIndex device;
  int dtype, err, mode;
  long long step;  // Adam only: bias corrections are per step count
  std::vector<FoSeg> rows;
  std::vector<int32_t> chunks;
  Table* table;
};

struct Group {
  std::vector<std::unique_ptr<Bucket>> buckets;
  size_t used = 0;
  std::vector<std::unique_ptr<Table>> tables;
  long long calls = 0;
};

struct Counter {
  float* at;
  float was;
};

struct Walker {
  PyObject_HEAD
  std::vector<Group>* groups;
  std::vector<Counter>* steps;      // Adam step counters to advance
  std::vector<PyObject*>* updated;  // parameters of this call that the launches update (borrowed)
  std::vector<PyObject*>* skipped;  // those that a collective-fused update has done already (borrowed)
  // kept until the call is launched, whatever Python code runs meanwhile lets go of
  std::vector<at::Tensor>* held;        // parameters and gradients
  std::vector<PyObject*>* held_states;  // and the dictionaries of their states
  Looked* looked;
  bool busy;
};

enum Verdict { kOk, kFallback, kError };

// The plain tensor behind `o`: itself, or the local shard of a DTensor.  False: not served.
bool local_tensor(PyObject* o, at::Tensor& out) {
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.unsafeGetTensorImpl()->key_set().has(c10::DispatchKey::Python)) {
    out = t;
    return true;
  }
  PyObject* lt = PyObject_GetAttr(o, s_local_tensor);
  if (!lt) {
    PyErr_Clear();
    return false;
  }
  const bool ok = THPVariable_Check(lt) &&
                  !THPVariable_Unpack(lt).unsafeGetTensorImpl()->key_set().has(c10::DispatchKey::Python);
  if (ok) out = THPVariable_Unpack(lt);
  Py_DECREF(lt);
  return ok;
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return FO_BF16;
    case at::kHalf: return FO_FP16;
    case at::kFloat: return FO_FP32;
    default: return -1;
  }
}

struct Call {
  PyObject *opt, *params, *state, *ready, *skip, *group;
  Py_ssize_t group_index;
  PyObject* keys;  // names of the moments, in kernel order
  bool adam, check, listeners;
  PyObject *lr, *width;  // arguments of the numerics check
};

Bucket& bucket_for(Group& g, c10::DeviceIndex device, int dtype, int err, int mode, long long step) {
  for (size_t i = 0; i < g.used; ++i) {
    Bucket& b = *g.buckets[i];
    if (b.device == device && b.dtype == dtype && b.err == err && b.mode == mode && b.step == step) return b;
  }
  if (g.used == g.buckets.size()) g.buckets.push_back(std::make_unique<Bucket>());
  Bucket& b = *g.buckets[g.used++];
  b.device = device;
  b.dtype = dtype;
  b.err = err;
  b.mode = mode;
  b.step = step;
  b.rows.clear();
  return b;
}

// Looks one parameter over and appends its row.  No side effects besides state creation.
Verdict visit(Walker* w, Group& g, const Call& c, PyObject* p) {
  if (!THPVariable_Check(p)) return kFallback;
  PyObject* id = PyLong_FromVoidPtr(p);
  if (!id) return kError;
  PyObject* st = _PyDict_GetItem_KnownHash(c.state, p, PyObject_Hash(id));
  if (!st && PyErr_Occurred()) {
    Py_DECREF(id);
    return kError;
  }
  int ready = PySet_Contains(c.ready, id);
  const int skip = PySet_GET_SIZE(c.skip) ? PySet_Contains(c.skip, id) : 0;
  Py_DECREF(id);
  if (ready < 0 || skip < 0) return kError;
  if (!st || !ready || !PyDict_Check(st) || PyDict_GET_SIZE(st) == 0 || c.check) {
    at::NoGradGuard no_grad;
    PyObject* r = PyObject_CallMethodObjArgs(c.opt, s_ensure, p, c.group, nullptr);
    if (!r) return kError;
    Py_DECREF(r);
    st = PyDict_GetItemWithError(c.state, p);
    if (!st) return PyErr_Occurred() ? kError : kFallback;
    if (!PyDict_Check(st)) return kFallback;
  }
  if (skip) {
    w->skipped->push_back(p);
    return kOk;
  }
  const at::Tensor& full = THPVariable_Unpack(p);
  if (!full.requires_grad() || full.numel() < 1) return kOk;
  const at::Tensor& full_grad = full.grad();
  if (!full_grad.defined()) return kOk;
  at::Tensor t, grad;
  if (!local_tensor(p, t)) return kFallback;
  if (full_grad.unsafeGetTensorImpl()->key_set().has(c10::DispatchKey::Python)) {
    PyObject* go = THPVariable_Wrap(full_grad);
    if (!go) return kError;
    const bool ok = local_tensor(go, grad);
    Py_DECREF(go);
    if (!ok) return kFallback;
  } else {
    grad = full_grad;
  }
  const int64_t n = t.numel();
  if (n < 1) return kOk;
  const int dtype = dtype_code(t.scalar_type());
  if (!t.is_cuda() || dtype < 0 || !t.is_contiguous() || !grad.is_cuda() || grad.device() != t.device() ||
      !grad.is_contiguous() || grad.scalar_type() != t.scalar_type() || grad.numel() != n)
    return kFallback;
  if (c.check) {
    at::NoGradGuard no_grad;
    PyObject* r = PyObject_CallMethodObjArgs(c.opt, s_check, p, c.lr, c.width, nullptr);
    if (!r) return kError;
    Py_DECREF(r);
  }

  FoSeg row;
  std::memset(&row, 0, sizeof(row));
  row.p = t.data_ptr();
  row.g = grad.data_ptr();
  row.n = n;
  int err = 0;
  PyObject* e = PyDict_GetItemWithError(st, s_error_bits);
  if (!e && PyErr_Occurred()) return kError;
  if (e && e != Py_None) {
    if (!THPVariable_Check(e)) return kFallback;
    const at::Tensor& et = THPVariable_Unpack(e);
    if (et.device() != t.device() || et.numel() != n || !et.is_contiguous()) return kFallback;
    err = (int)et.element_size();
    row.ecc = et.data_ptr();
  }
  const Py_ssize_t n_keys = PyTuple_GET_SIZE(c.keys);
  int mode = n_keys ? -1 : FO_STATE_NONE;
  for (Py_ssize_t k = 0; k < n_keys; ++k) {
    PyObject* m = PyDict_GetItemWithError(st, PyTuple_GET_ITEM(c.keys, k));
    if (!m) return PyErr_Occurred() ? kError : kFallback;
    if (Py_TYPE(m) != g_state_type) return kFallback;
    PyObject* data = slot(m, g_off_data);
    void *codes = nullptr, *scales = nullptr;
    int this_mode;
    if (!data) {
      PyObject *q = slot(m, g_off_codes), *sc = slot(m, g_off_scales);
      if (!q || !sc || !THPVariable_Check(q) || !THPVariable_Check(sc)) return kFallback;
      const at::Tensor &qt = THPVariable_Unpack(q), &sct = THPVariable_Unpack(sc);
      if (qt.device() != t.device() || sct.device() != t.device() || qt.numel() != n || qt.element_size() != 1 ||
          sct.numel() != (n + 31) / 32 || sct.scalar_type() != at::kHalf || !qt.is_contiguous() ||
          !sct.is_contiguous())
        return kFallback;
      codes = qt.data_ptr();
      scales = sct.data_ptr();
      this_mode = FO_STATE_Q8;
    } else {
      if (!THPVariable_Check(data)) return kFallback;
      const at::Tensor& d = THPVariable_Unpack(data);
      if (d.device() != t.device() || d.numel() != n || d.scalar_type() != t.scalar_type() || !d.is_contiguous())
        return kFallback;
      codes = d.data_ptr();
      this_mode = FO_STATE_FULL;
    }
    if (mode >= 0 && mode != this_mode) return kFallback;  // one moment quantised, the other not
    mode = this_mode;
    if (k == 0) {
      row.s0 = codes;
      row.s0s = scales;
    } else {
      row.s1 = codes;
      row.s1s = scales;
    }
  }
  long long step = 0;
  if (c.adam) {
    PyObject* so = PyDict_GetItemWithError(st, s_step);
    if (!so) return PyErr_Occurred() ? kError : kFallback;
    if (!THPVariable_Check(so)) return kFallback;
    const at::Tensor& sten = THPVariable_Unpack(so);
    if (!sten.is_cpu() || sten.scalar_type() != at::kFloat || sten.numel() != 1) return kFallback;
    float* counter = static_cast<float*>(sten.data_ptr());
    if (!(*counter >= 0.0f && *counter < 1e9f)) return kFallback;
    step = (long long)(*counter + 1.0f);
    w->steps->push_back({counter, *counter});
  }
  Bucket& b = bucket_for(g, t.device().index(), dtype, err, mode, step);
  b.rows.push_back(row);
  w->updated->push_back(p);
  w->held->push_back(std::move(t));
  w->held->push_back(std::move(grad));
  w->held_states->push_back(Py_NewRef(st));
  return kOk;
}

// Adam's scalars, or those of the momentum family, as the C ABI wants them.  All complements are
// evaluated in double precision like ops/step.py does.
struct Hyper {
  double v[6];
  int flag[3];
};

// 1 / (1 - beta^step); false outside the range where that is at least 1: the Python walk then
// says what is wrong (a division by zero, a root of a negative number, an overflow).
bool bias_correction(double beta, long long step, double& out) {
  if (!(beta >= 0.0 && beta < 1.0) || step < 1) return false;
  out = 1.0 / (1.0 - std::pow(beta, (double)step));
  return true;
}

bool adam_hyper(const Hyper& h, long long step, FoAdamHyper& o) {
  const double lr = h.v[0], b1 = h.v[1], b2 = h.v[2], eps = h.v[3], wd = h.v[4];
  double rbc1, rbc2;
  if (!bias_correction(b1, step, rbc1) || !bias_correction(b2, step, rbc2)) return false;
  o.lr = (float)lr;
  o.beta1 = (float)b1;
  o.beta2 = (float)b2;
  o.eps = (float)eps;
  o.one_minus_beta1 = (float)(1.0 - b1);
  o.one_minus_beta2 = (float)(1.0 - b2);
  o.weight_decay = (float)wd;
  o.decay = (float)(h.flag[0] ? 1.0 - wd : 1.0);
  o.rbc1 = (float)rbc1;
  o.sqrt_rbc2 = (float)std::sqrt(rbc2);
  o.grad_scale = 1.0f;
  o.decoupled = h.flag[0];
  return true;
}

void momentum_hyper(const Hyper& h, FoMomentumHyper& o) {
  const double lr = h.v[0], mom = h.v[1], upd = h.v[2], wd = h.v[3];
  o.lr = (float)lr;
  o.mom_coef = (float)mom;
  o.update_coef = (float)upd;
  o.one_minus_mom_coef = (float)(1.0 - mom);
  o.one_minus_update_coef = (float)(1.0 - upd);
  o.weight_decay = (float)wd;
  o.decay = (float)(h.flag[0] || h.flag[1] ? 1.0 - wd : 1.0);
  o.grad_scale = 1.0f;
  o.lion = h.flag[1];
  o.nesterov = h.flag[2];
  o.decoupled = h.flag[0];
}

// Chunk prefix of a bucket; false when the list is too long for one launch.
bool prefix(Bucket& b) {
  b.chunks.resize(b.rows.size() + 1);
  int64_t at = 0;
  b.chunks[0] = 0;
  for (size_t i = 0; i < b.rows.size(); ++i) {
    at += (b.rows[i].n + g_api.chunk - 1) / g_api.chunk;
    if (at >= (int64_t(1) << 31)) return false;
    b.chunks[i + 1] = (int32_t)at;
  }
  return true;
}

// The device copy of a long table, re-sent only when a row changed (in steady state the caching
// allocator returns gradients at the same addresses step after step).  Each stream and number of
// rows has a copy of its own, so that none is replaced when parameters come and go or written while
// a launch on another stream reads it; two buckets of one call share none.  A captured step gets
// one that no other step shares: the copy runs when the graph is replayed, so that the host does
// not know what the buffer holds, and what it copies from has to stay as long as the graph may.
void upload(Group& g, Bucket& b) {
  const size_t n = b.rows.size(), seg_bytes = n * sizeof(FoSeg), bytes = seg_bytes + (n + 1) * sizeof(int32_t);
  const c10::StreamId stream = c10::cuda::getCurrentCUDAStream(b.device).id();
  const bool capturing = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
  Table* t = nullptr;
  for (auto& have : g.tables)
    if (!capturing && !have->staged.defined() && have->n == n && have->call != g.calls && have->device == b.device && have->stream == stream &&
        have->dtype == b.dtype && have->err == b.err && have->mode == b.mode) {
      t = have.get();
      break;
    }
  if (!t) {
    auto fresh = std::make_unique<Table>();
    fresh->device = b.device;
    fresh->stream = stream;
    fresh->dtype = b.dtype;
    fresh->err = b.err;
    fresh->mode = b.mode;
    fresh->n = n;
    fresh->dev = at::empty({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).device(
                                                 c10::Device(c10::DeviceType::CUDA, b.device)));
    t = fresh.get();
    g.tables.push_back(std::move(fresh));
  }
  t->call = g.calls;
  b.table = t;
  if (t->sent.size() == n && std::memcmp(t->sent.data(), b.rows.data(), seg_bytes) == 0) return;
  t->sent.clear();  // any line below may throw; what the buffer holds is known again once all have passed
  at::Tensor staged = at::empty({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).pinned_memory(true));
  std::memcpy(staged.data_ptr(), b.rows.data(), seg_bytes);
  std::memcpy(static_cast<char*>(staged.data_ptr()) + seg_bytes, b.chunks.data(), (n + 1) * sizeof(int32_t));
  if (capturing) t->staged = staged;
  t->dev.copy_(staged, /*non_blocking=*/true);  // the host allocator keeps `staged` until the copy is done
  t->sent = b.rows;
}

bool on_device(const Bucket& b) { return b.rows.size() > FO_MAX_INLINE_SEGS; }

// Launches one bucket, whose table is in place; 0 or a cudaError_t.
int launch(Bucket& b, bool adam, const FoAdamHyper& ah, const FoMomentumHyper& mh) {
  c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::DeviceType::CUDA, b.device));
  const int n = (int)b.rows.size();
  const FoSeg* segs = b.rows.data();
  const int32_t* chunks = b.chunks.data();
  if (on_device(b)) {
    segs = static_cast<const FoSeg*>(b.table->dev.data_ptr());
    chunks = reinterpret_cast<const int32_t*>(segs + n);
  }
  void* stream = c10::cuda::getCurrentCUDAStream(b.device).stream();
  const int total = b.chunks[n];
  if (g_nvtx) nvtxRangePushA(adam ? "fo_adam_step" : "fo_momentum_step");
  const int rc = adam ? g_api.adam_step(segs, chunks, n, total, on_device(b), b.dtype, b.err, b.mode == FO_STATE_Q8,
                                        &ah, stream)
                      : g_api.momentum_step(segs, chunks, n, total, on_device(b), b.dtype, b.err, b.mode, &mh, stream);
  if (g_nvtx) nvtxRangePop();
  return rc;
}

bool ensure_status(c10::DeviceIndex device) {
  if (device < 64 && (g_status_ready >> device) & 1) return true;
  PyObject* d = PyLong_FromLong(device);
  if (!d) return false;
  PyObject* r = PyObject_CallOneArg(g_ensure_status, d);
  Py_DECREF(d);
  if (!r) return false;
  Py_DECREF(r);
  if (device < 64) g_status_ready |= uint64_t(1) << device;
  return true;
}

// Gives the GIL away for a scope.  What throws inside takes it back on its way out, before a
// handler touches the interpreter.
struct GilReleased {
  PyThreadState* state = PyEval_SaveThread();
  ~GilReleased() { PyEval_RestoreThread(state); }
};

// One call of a walker.  What it holds is let go under the GIL, which its owner has at the end.
struct Busy {
  Walker* w;
  explicit Busy(Walker* walker) : w(walker) { w->busy = true; }
  ~Busy() {
    w->held->clear();
    for (PyObject* st : *w->held_states) Py_DECREF(st);
    w->held_states->clear();
    w->busy = false;
  }
};

// Nothing is done for an optimizer with methods of its own in the walk's place.
// Walker.step(opt, params, state, ready, skip, group, group_index, keys, adam, check, listeners,
//             hyper) -> False (nothing done, not served), True, or the list of updated parameters.
PyObject* walker_step(Walker* w, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 12) {
    PyErr_SetString(PyExc_TypeError, "Walker.step takes 12 arguments");
    return nullptr;
  }
  if (w->busy) Py_RETURN_FALSE;  // another thread is inside a launch of this optimizer
  if (const int other = overrides(args[0], *w->looked)) {
    if (other < 0) return nullptr;
    Py_RETURN_FALSE;
  }
  Call c;
  c.opt = args[0];
  c.params = args[1];
  c.state = args[2];
  c.ready = args[3];
  c.skip = args[4];
  c.group = args[5];
  c.group_index = PyLong_AsSsize_t(args[6]);
  c.keys = args[7];
  c.adam = args[8] == Py_True;
  c.check = args[9] != Py_None;
  c.listeners = args[10] == Py_True;
  c.lr = c.check ? PyTuple_GET_ITEM(args[9], 0) : nullptr;
  c.width = c.check ? PyTuple_GET_ITEM(args[9], 1) : nullptr;
  if (c.group_index == -1 && PyErr_Occurred()) return nullptr;
  if (!PyList_Check(c.params) || !PyDict_Check(c.state) || !PySet_Check(c.ready) || !PySet_Check(c.skip) ||
      !PyTuple_Check(c.keys) || PyTuple_GET_SIZE(c.keys) > 2 || !PyTuple_Check(args[11]))
    Py_RETURN_FALSE;
  // scalars: floats first, then flags
  Hyper h;
  const Py_ssize_t n_flags = c.adam ? 1 : 3, n_vals = PyTuple_GET_SIZE(args[11]) - n_flags;
  if (n_vals != (c.adam ? 5 : 4)) {
    PyErr_SetString(PyExc_TypeError, "Walker.step: wrong number of scalars");
    return nullptr;
  }
  for (Py_ssize_t i = 0; i < n_vals; ++i) {
    PyObject* v = PyTuple_GET_ITEM(args[11], i);
    // anything else (a tensor as learning rate) is folded by the Python walk in its own arithmetic
    if (!PyFloat_CheckExact(v) && !PyLong_CheckExact(v)) Py_RETURN_FALSE;
    h.v[i] = PyFloat_AsDouble(v);
    if (h.v[i] == -1.0 && PyErr_Occurred()) return nullptr;
  }
  for (Py_ssize_t i = 0; i < n_flags; ++i) {
    h.flag[i] = PyObject_IsTrue(PyTuple_GET_ITEM(args[11], n_vals + i));
    if (h.flag[i] < 0) return nullptr;
  }

  Busy busy(w);
  try {
    // groups are numbered from -1 (a group dict that the optimizer does not own)
    const size_t slot_index = (size_t)(c.group_index + 1);
    if (w->groups->size() <= slot_index) w->groups->resize(slot_index + 1);
    Group& g = (*w->groups)[slot_index];
    g.used = 0;
    ++g.calls;
    w->steps->clear();
    w->updated->clear();
    w->skipped->clear();
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(c.params); ++i) {
      const Verdict v = visit(w, g, c, PyList_GET_ITEM(c.params, i));
      if (v == kFallback) Py_RETURN_FALSE;
      if (v == kError) return nullptr;
    }
    std::vector<FoAdamHyper> ah(c.adam ? g.used : 0);
    FoMomentumHyper mh;
    for (size_t i = 0; i < g.used; ++i) {
      if (!prefix(*g.buckets[i])) Py_RETURN_FALSE;
      if (c.adam && !adam_hyper(h, g.buckets[i]->step, ah[i])) Py_RETURN_FALSE;
    }
    if (!c.adam) momentum_hyper(h, mh);
    // taken down before the GIL is given away, after which the group's list is no longer ours
    THPObjectPtr list(c.listeners ? PyList_New((Py_ssize_t)w->updated->size()) : nullptr);
    if (c.listeners && !list) return nullptr;
    for (size_t i = 0; c.listeners && i < w->updated->size(); ++i)
      PyList_SET_ITEM(list.get(), (Py_ssize_t)i, Py_NewRef((*w->updated)[i]));
    for (size_t i = 0; i < g.used; ++i)
      if (!ensure_status(g.buckets[i]->device)) return nullptr;
    for (size_t i = 0; i < g.used; ++i) {
      Bucket& b = *g.buckets[i];
      if (!on_device(b)) continue;
      GilReleased released;  // allocates and copies; whatever fails here leaves the step undone
      c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::DeviceType::CUDA, b.device));
      upload(g, b);
    }

    // a counter that several parameters share advances once for each before any of them is read
    bool shared = false;
    for (const Counter& s : *w->steps) *s.at += 1.0f;
    for (const Counter& s : *w->steps) shared = shared || *s.at != s.was + 1.0f;
    if (shared) {
      for (const Counter& s : *w->steps) *s.at = s.was;
      Py_RETURN_FALSE;
    }
    // from here on the call is committed
    for (PyObject* p : *w->skipped) {
      PyObject* id = PyLong_FromVoidPtr(p);
      if (!id || PySet_Discard(c.skip, id) < 0) {
        Py_XDECREF(id);
        return nullptr;
      }
      Py_DECREF(id);
    }
    for (size_t i = 0; i < g.used; ++i) {
      static const FoAdamHyper none = {};
      int rc;
      {
        GilReleased released;
        rc = launch(*g.buckets[i], c.adam, c.adam ? ah[i] : none, mh);
      }
      if (rc) {
        PyErr_Format(g_native_error, "%s failed with CUDA error %d", c.adam ? "fo_adam_step" : "fo_momentum_step", rc);
        return nullptr;
      }
      ++g_launches;
    }
    if (!c.listeners) Py_RETURN_TRUE;
    return list.release();
  } catch (...) {  // as the Python exception that torch makes of it, OutOfMemoryError among them
    if (!PyErr_Occurred()) torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

PyObject* walker_new(PyTypeObject* type, PyObject*, PyObject*) {
  Walker* w = reinterpret_cast<Walker*>(type->tp_alloc(type, 0));
  if (!w) return nullptr;
  w->groups = new std::vector<Group>();
  w->steps = new std::vector<Counter>();
  w->updated = new std::vector<PyObject*>();
  w->skipped = new std::vector<PyObject*>();
  w->held = new std::vector<at::Tensor>();
  w->held_states = new std::vector<PyObject*>();
  w->looked = new Looked();
  w->busy = false;
  return reinterpret_cast<PyObject*>(w);
}
// The device tables: a list of (rows, address, host address that replays copy from or 0).
PyObject* walker_tables(Walker* w, PyObject*) {
  PyObject* list = PyList_New(0);
  if (w->busy) return list;  // another thread is writing them
  for (size_t i = 0; list && i < w->groups->size(); ++i)
    for (auto& t : (*w->groups)[i].tables) {
      PyObject* item = Py_BuildValue("nnn", (Py_ssize_t)t->n, (Py_ssize_t)t->dev.data_ptr(),
                                     t->staged.defined() ? (Py_ssize_t)t->staged.data_ptr() : (Py_ssize_t)0);
      if (!item || PyList_Append(list, item) < 0) Py_CLEAR(list);
      Py_XDECREF(item);
      if (!list) break;
    }
  return list;
}
void walker_dealloc(Walker* w) {
  delete w->groups;
  delete w->steps;
  delete w->updated;
  delete w->skipped;
  delete w->held;
  delete w->held_states;
  delete w->looked;
  Py_TYPE(w)->tp_free(reinterpret_cast<PyObject*>(w));
}

PyMethodDef walker_methods[] = {
    {"step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(walker_step)), METH_FASTCALL, nullptr},
    {"tables", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(walker_tables)), METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyTypeObject walker_type = [] {
  PyTypeObject t = {PyVarObject_HEAD_INIT(nullptr, 0)};
  t.tp_name = "flashoptim_b200.Walker";
  t.tp_basicsize = sizeof(Walker);
  t.tp_flags = Py_TPFLAGS_DEFAULT;
  t.tp_new = walker_new;
  t.tp_dealloc = reinterpret_cast<destructor>(walker_dealloc);
  t.tp_methods = walker_methods;
  return t;
}();

// ---------------------------------------------------------------- module
// setup(adam_step, momentum_step, chunk, state_type, ensure_status, native_error, nvtx, walked)
PyObject* host_setup(PyObject*, PyObject* args) {
  unsigned long long adam, mom;
  int chunk, nvtx;
  PyObject *type, *ensure, *error, *walked;
  if (!PyArg_ParseTuple(args, "KKiO!OOpO!", &adam, &mom, &chunk, &PyType_Type, &type, &ensure, &error, &nvtx,
                        &PyTuple_Type, &walked))
    return nullptr;
  PyTypeObject* t = reinterpret_cast<PyTypeObject*>(type);
  g_off_data = slot_offset(t, "_data");
  g_off_codes = slot_offset(t, "_quantized");
  g_off_scales = slot_offset(t, "_scales");
  if (PyErr_Occurred()) return nullptr;
  g_api.adam_step = reinterpret_cast<decltype(&fo_adam_step)>(adam);
  g_api.momentum_step = reinterpret_cast<decltype(&fo_momentum_step)>(mom);
  g_api.chunk = chunk;
  g_nvtx = nvtx != 0;
  Py_XSETREF(g_ensure_status, Py_NewRef(ensure));
  Py_XSETREF(g_native_error, Py_NewRef(error));
  Py_XSETREF(g_walked, Py_NewRef(walked));
  PyTypeObject* old = g_state_type;
  g_state_type = reinterpret_cast<PyTypeObject*>(Py_NewRef(type));
  Py_XDECREF(old);
  Py_RETURN_NONE;
}

PyObject* host_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches); }

PyObject* host_overrides(PyObject*, PyObject* opt) {
  Looked nothing_yet;
  const int other = overrides(opt, nothing_yet);
  return other < 0 ? nullptr : PyBool_FromLong(other);
}

// Whether somebody (a profiler, an execution trace) observes operator calls right now.
PyObject* host_observed(PyObject*, PyObject*) {
  return PyBool_FromLong(at::hasThreadLocalCallbacks() || at::hasGlobalCallbacks());
}

PyMethodDef host_methods[] = {
    {"setup", host_setup, METH_VARARGS, nullptr},
    {"launches", host_launches, METH_NOARGS, nullptr},
    {"overrides", host_overrides, METH_O, nullptr},
    {"observed", host_observed, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef host_module = {PyModuleDef_HEAD_INIT, "_fo_host", nullptr, -1, host_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fo_host() {
  s_step = PyUnicode_InternFromString("step");
  s_error_bits = PyUnicode_InternFromString("error_bits");
  s_local_tensor = PyUnicode_InternFromString("_local_tensor");
  s_ensure = PyUnicode_InternFromString("_ensure_state_initialized");
  s_check = PyUnicode_InternFromString("_check_param_numerics");
  s_walked_natively = PyUnicode_InternFromString("_walked_natively");
  if (!s_walked_natively || !s_step || !s_error_bits || !s_local_tensor || !s_ensure || !s_check) return nullptr;
  if (PyType_Ready(&walker_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&host_module);
  if (!m) return nullptr;
  if (PyModule_AddObjectRef(m, "Walker", reinterpret_cast<PyObject*>(&walker_type)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
