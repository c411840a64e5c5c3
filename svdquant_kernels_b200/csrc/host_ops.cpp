// Host path of the operators: contract checks, output allocation, lookup of the layout twins and the
// launch, in one native call per operator, for the Python operators (ops.py) and for the dispatcher
// (torch.ops.svdq_b200.*).
//
// A layer of a few hundred rows keeps the GPU busy for some 15-20 us, so the host's part decides how fast
// such layers can follow each other.  In Python it took 20 us per operator (about 60 interpreter-level
// calls: assertions, tensor attributes, five torch.empty, ctypes conversions) and the registered ops
// another 20 us in torch.library's Python wrappers; here an operator takes a few microseconds.
//
// Only calls that need nothing but a launch are taken: plain contiguous CUDA tensors on the current
// device that meet every condition of the contract and whose twins exist.  For anything else (first use
// of a weight, strided inputs, a shape that breaks the contract, tensor subclasses) the functions return
// None and the Python operator, which owns the checks and their messages, does the call.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/Storage.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <functional>
#include <typeinfo>
#include <unordered_map>

#include "../../include/svdq_b200.h"

namespace {

using at::ScalarType;
using at::Tensor;

PyObject* g_twins_name = nullptr;     // interned "_svdq_twins": attribute of a storage object, see ops._attach
PyObject* g_split_ws = nullptr;       // ops._SPLIT_WS: {(device, stream): workspace}
PyObject* g_py_quantize = nullptr;    // the Python operators behind the dispatcher, for calls not taken here
PyObject* g_py_gemm = nullptr;

int dtype_code(ScalarType t) {
  return t == at::kHalf ? SVDQ_DTYPE_F16 : t == at::kBFloat16 ? SVDQ_DTYPE_BF16 : t == at::kFloat ? SVDQ_DTYPE_F32 : -1;
}

struct GilAcquire {
  PyGILState_STATE st = PyGILState_Ensure();
  ~GilAcquire() { PyGILState_Release(st); }
};
struct GilRelease {
  PyThreadState* st = PyEval_SaveThread();
  ~GilRelease() { PyEval_RestoreThread(st); }
};
struct Ref {                            // owned reference
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) {}
  Ref(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
};

// A twin as the launches need it; `hold` or `hold_storage` keeps it alive.
struct Twin {
  void* ptr = nullptr;
  ScalarType type = at::kByte;
  int64_t numel = 0;
  Tensor hold;
  c10::intrusive_ptr<c10::StorageImpl> hold_storage = {};
  bool found() const { return ptr != nullptr || hold.defined(); }
  void* data() const { return numel > 0 ? ptr : nullptr; }
};

// The storage of an output that has a twin: the twin hangs on it directly and goes when it goes, with no Python object
// in between (a record on a storage's Python object costs a call some 1.5 us).  It stands for the whole output,
// (offset 0, numel); twins of other views of it are recorded on the Python object like everything else's.  All access
// with the GIL held.
struct OutputStorage final : c10::StorageImpl {
  OutputStorage(size_t nbytes, c10::Allocator* allocator, int64_t numel)
      : c10::StorageImpl(use_byte_size_t(), nbytes, allocator, /*resizable=*/true), numel(numel) {}
  void release_resources() override {
    c10::StorageImpl::release_resources();
    twin = Twin();
  }
  const int64_t numel;
  Twin twin;
  uint32_t version = 0;                 // of the owner that the twin was made from
};
OutputStorage* output_storage(const Tensor& owner) {
  c10::StorageImpl* const st = owner.storage().unsafeGetStorageImpl();
  if (st == nullptr || typeid(*st) != typeid(OutputStorage)) return nullptr;             // (a final class)
  auto* const out = static_cast<OutputStorage*>(st);
  return owner.storage_offset() == 0 && owner.numel() == out->numel ? out : nullptr;
}

// What `attached` found on the storage objects of weights and smoothing factors, which a layer looks up on every call: a
// hash lookup instead of half a dozen Python calls (0.25 us each, three a layer).  One entry per owner - the views of a
// flat buffer are owners each - good for one version of it.  It holds nothing alive: its weak references keep the
// StorageImpls' addresses from being used again, not their memory.  Entries of storages that are gone are swept out every
// kSweep insertions.
constexpr size_t kSweep = 256;
struct Owner {
  const c10::StorageImpl* storage;
  int64_t offset, numel;
  explicit Owner(const Tensor& t) : storage(t.storage().unsafeGetStorageImpl()), offset(t.storage_offset()), numel(t.numel()) {}
  bool operator==(const Owner& o) const { return storage == o.storage && offset == o.offset && numel == o.numel; }
};
struct OwnerHash {
  size_t operator()(const Owner& o) const {
    return std::hash<const void*>()(o.storage) ^ (static_cast<size_t>(o.offset) * 0x9E3779B97F4A7C15ull + static_cast<size_t>(o.numel));
  }
};
struct KnownTwin {
  c10::weak_intrusive_ptr<c10::StorageImpl> owner, twin;
  uint32_t version;
  void* ptr;
  ScalarType type;
  int64_t twin_numel;
};
std::unordered_map<Owner, KnownTwin, OwnerHash>& known_twins() {
  static auto* table = new std::unordered_map<Owner, KnownTwin, OwnerHash>();             // outlives every tensor
  return *table;
}
c10::weak_intrusive_ptr<c10::StorageImpl> weak(const Tensor& t) {
  return c10::weak_intrusive_ptr<c10::StorageImpl>(
      c10::intrusive_ptr<c10::StorageImpl>::unsafe_reclaim_from_nonowning(t.storage().unsafeGetStorageImpl()));
}

// The twin recorded for `owner`: on its storage, or on the storage's Python object (the records ops._attach keeps:
// {(offset, numel): (twin, version)}); not found if there is none or it is out of date.  GIL held.
Twin attached(const Tensor& owner, bool any_version = false) {
  if (const OutputStorage* st = output_storage(owner))
    return any_version || st->version == owner._version() ? st->twin : Twin();
  auto& known = known_twins();
  const Owner me(owner);
  if (!any_version) {
    const auto it = known.find(me);
    if (it != known.end() && it->second.version == owner._version()) {
      auto alive = it->second.twin.lock();
      if (alive) return Twin{it->second.ptr, it->second.type, it->second.twin_numel, Tensor(), std::move(alive)};
    }
  }
  Ref st(THPStorage_Wrap(owner.storage()));
  if (st.p == nullptr) { PyErr_Clear(); return Twin(); }
  Ref recs(PyObject_GetAttr(st.p, g_twins_name));
  if (recs.p == nullptr) { PyErr_Clear(); return Twin(); }
  if (!PyDict_Check(recs.p)) return Twin();
  Ref key(Py_BuildValue("(LL)", static_cast<long long>(owner.storage_offset()), static_cast<long long>(owner.numel())));
  PyObject* rec = key.p != nullptr ? PyDict_GetItemWithError(recs.p, key.p) : nullptr;     // borrowed
  if (rec == nullptr || !PyTuple_Check(rec) || PyTuple_GET_SIZE(rec) != 2) { PyErr_Clear(); return Twin(); }
  if (!any_version && PyLong_AsLong(PyTuple_GET_ITEM(rec, 1)) != static_cast<long>(owner._version())) return Twin();
  PyObject* twin = PyTuple_GET_ITEM(rec, 0);
  if (!THPVariable_Check(twin)) return Twin();
  const Tensor& t = THPVariable_Unpack(twin);
  void* const ptr = t.numel() > 0 ? t.data_ptr() : nullptr;
  if (!any_version && ptr != nullptr) {
    static size_t inserted = 0;
    if (++inserted % kSweep == 0)
      for (auto it = known.begin(); it != known.end();)
        it = it->second.owner.expired() || it->second.twin.expired() ? known.erase(it) : std::next(it);
    known.insert_or_assign(me, KnownTwin{weak(owner), weak(t), static_cast<uint32_t>(owner._version()), ptr, t.scalar_type(), t.numel()});
  }
  return Twin{ptr, t.scalar_type(), t.numel(), t, {}};
}

// A tensor on a storage of its own, without the checks and guards of at::empty: every caller has seen a tensor on the
// current device `dev` already.  Four of these are most of a small quantizer call's host time.
Tensor on_storage(c10::intrusive_ptr<c10::StorageImpl> st, at::IntArrayRef sizes, ScalarType t) {
  Tensor r = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(std::move(st)), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                      c10::scalarTypeToTypeMeta(t));
  r.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
  return r;
}
c10::intrusive_ptr<c10::StorageImpl> new_storage(int64_t numel, ScalarType t) {
  return c10::make_intrusive<c10::StorageImpl>(c10::StorageImpl::use_byte_size_t(), static_cast<size_t>(numel) * c10::elementSize(t),
                                               c10::cuda::CUDACachingAllocator::get(), /*resizable=*/true);
}
Tensor empty(at::IntArrayRef sizes, ScalarType t) { return on_storage(new_storage(c10::multiply_integers(sizes), t), sizes, t); }
// An output that gets a twin, on a storage that the twin can hang on
Tensor empty_output(int64_t rows, int64_t cols, ScalarType t) {
  const int64_t numel = rows * cols;
  return on_storage(c10::make_intrusive<OutputStorage>(static_cast<size_t>(numel) * c10::elementSize(t), c10::cuda::CUDACachingAllocator::get(), numel),
                    {rows, cols}, t);
}
Twin empty_twin(int64_t numel, ScalarType t) {
  auto st = new_storage(numel, t);
  void* const ptr = st->mutable_data();
  return Twin{ptr, t, numel, Tensor(), std::move(st)};
}
Tensor tensor_of(const Twin& twin) { return twin.hold.defined() ? twin.hold : on_storage(twin.hold_storage, {twin.numel}, twin.type); }

// Record `twin` as the derived form of `owner`'s current contents.  GIL held; false with a Python error set.
bool attach(const Tensor& owner, const Twin& twin) {
  if (OutputStorage* st = output_storage(owner)) {
    st->twin = twin;
    st->version = static_cast<uint32_t>(owner._version());
    return true;
  }
  Ref st(THPStorage_Wrap(owner.storage()));
  if (st.p == nullptr) return false;
  PyObject* recs = PyObject_GetAttr(st.p, g_twins_name);
  if (recs == nullptr) {
    PyErr_Clear();
    recs = PyDict_New();
    if (recs == nullptr || PyObject_SetAttr(st.p, g_twins_name, recs) != 0) { Py_XDECREF(recs); return false; }
  }
  Ref hold(recs);
  Ref key(Py_BuildValue("(LL)", static_cast<long long>(owner.storage_offset()), static_cast<long long>(owner.numel())));
  Ref wrapped(THPVariable_Wrap(tensor_of(twin)));
  if (key.p == nullptr || wrapped.p == nullptr) return false;
  Ref rec(Py_BuildValue("(Ol)", wrapped.p, static_cast<long>(owner._version())));
  return rec.p != nullptr && PyDict_SetItem(recs, key.p, rec.p) == 0;
}

// A tensor the kernels can take as it is: on the current device, contiguous, no subclass behaviour, and
// with a version counter (inference tensors have none, so no twin can be tied to their contents).
bool plain(const Tensor& t, c10::DeviceIndex dev) {
  return t.defined() && t.is_cuda() && t.device().index() == dev && t.is_contiguous() && !t.is_inference() &&
         t.layout() == at::kStrided && !t.is_conj() && !t.is_neg();
}

void throw_status(const char* what, int rc) {
  throw std::runtime_error(std::string(what) + ": svdq status " + std::to_string(rc) + " (" + svdq_status_string(rc) + ")");
}

bool int_sized(int64_t v) { return v >= 0 && v <= INT32_MAX; }

struct Quantized {
  Tensor act, ascales, lora_act;
};

// GIL held.  False: not taken.
bool quantize(const Tensor& x, const Tensor& ld, const Tensor& smooth, int64_t pad, const Quantized* into, Quantized& out) {
  if (!x.is_cuda()) return false;
  const c10::DeviceIndex dev = c10::cuda::current_device();
  if (!plain(x, dev) || !plain(ld, dev) || x.dim() != 2 || ld.dim() != 2) return false;
  const ScalarType t = x.scalar_type();
  if ((t != at::kHalf && t != at::kBFloat16) || ld.scalar_type() != t) return false;
  const int64_t M = x.size(0), K = x.size(1), R = ld.size(1);
  if (ld.size(0) != K || K % 16 != 0 || K == 0 || M == 0 || pad < 1) return false;
  const int64_t Mp = (M + pad - 1) / pad * pad;
  if (!int_sized(Mp) || !int_sized(K) || !int_sized(R)) return false;
  Twin table;
  if (smooth.defined()) {
    if (!plain(smooth, dev) || smooth.dim() != 1 || smooth.size(0) != K || smooth.scalar_type() != t) return false;
    table = attached(smooth);
    if (!table.found()) return false;
  }
  const bool want_swz = Mp % 128 == 0 && K % 64 == 0;
  Twin swz, la16;
  if (into != nullptr) {
    out = *into;
    if (!plain(out.act, dev) || !plain(out.ascales, dev) || !plain(out.lora_act, dev)) return false;
    if (out.act.scalar_type() != at::kByte || out.act.dim() != 2 || out.act.size(0) != Mp || out.act.size(1) != K / 2) return false;
    if (out.ascales.scalar_type() != at::kFloat8_e4m3fn || out.ascales.dim() != 2 || out.ascales.size(0) != K / 16 ||
        out.ascales.size(1) != Mp)
      return false;
    if (out.lora_act.scalar_type() != at::kFloat || out.lora_act.dim() != 2 || out.lora_act.size(0) != Mp || out.lora_act.size(1) != R)
      return false;
    swz = attached(out.ascales, true);
    la16 = attached(out.lora_act, true);
    if (la16.found() && la16.type != t) la16 = Twin();
  } else {
    out.act = empty({Mp, K / 2}, at::kByte);
    out.ascales = empty_output(K / 16, Mp, at::kFloat8_e4m3fn);
    out.lora_act = R > 0 ? empty_output(Mp, R, at::kFloat) : empty({Mp, R}, at::kFloat);
  }
  // (a storage each: one kept by the scales would keep lora_act's planes too)
  if (want_swz && !swz.found()) swz = empty_twin(Mp * (K / 16), at::kByte);
  if (R > 0 && !la16.found()) la16 = empty_twin(svdq_lora_act16_elems(static_cast<int>(Mp), static_cast<int>(R), dtype_code(t)), t);
  void* const stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  auto ptr = [](const Tensor& v) -> void* { return v.defined() && v.numel() > 0 ? v.data_ptr() : nullptr; };
  int rc;
  {
    GilRelease nogil;
    rc = svdq_quantize_w4a4_act_fuse_lora(ptr(x), ptr(ld), ptr(smooth), table.data(), ptr(out.act), ptr(out.ascales),
                                          static_cast<float*>(ptr(out.lora_act)), swz.data(), la16.data(), static_cast<int>(M),
                                          static_cast<int>(K), static_cast<int>(R), static_cast<int>(Mp), dtype_code(t), 0, stream);
  }
  if (rc != SVDQ_OK) throw_status("quantize_w4a4_act_fuse_lora", rc);
  if (swz.found() && !attach(out.ascales, swz)) throw python_error();
  if (la16.found() && !attach(out.lora_act, la16)) throw python_error();
  return true;
}

struct GemmArgs {
  Tensor act, wgt, ascales, wscales, lora_act, lora_up, wcscales, bias, smooth_next, out;   // the last six may be undefined
};
struct GemmResult {
  Tensor y, qout, oscales;                                                                  // the last two with smooth_next
};

// GIL held.  False: not taken.
bool gemm(const GemmArgs& a, ScalarType out_t, GemmResult& r) {
  if (!a.act.is_cuda()) return false;
  const c10::DeviceIndex dev = c10::cuda::current_device();
  if (out_t != at::kHalf && out_t != at::kBFloat16) return false;
  if (!plain(a.act, dev) || !plain(a.wgt, dev) || !plain(a.ascales, dev) || !plain(a.wscales, dev)) return false;
  if (a.act.scalar_type() != at::kByte || a.wgt.scalar_type() != at::kByte || a.act.dim() != 2 || a.wgt.dim() != 2) return false;
  if (a.ascales.scalar_type() != at::kFloat8_e4m3fn || a.wscales.scalar_type() != at::kFloat8_e4m3fn) return false;
  const int64_t M = a.act.size(0), K = a.act.size(1) * 2, N = a.wgt.size(0), G = K / 16;
  if (a.wgt.size(1) * 2 != K || M == 0 || N == 0 || K == 0 || M % 128 != 0 || N % 128 != 0 || K % 64 != 0) return false;
  if (!int_sized(M) || !int_sized(N) || !int_sized(K)) return false;
  if (a.ascales.dim() != 2 || a.ascales.size(0) != G || a.ascales.size(1) != M) return false;
  if (a.wscales.dim() != 2 || a.wscales.size(0) != G || a.wscales.size(1) != N) return false;
  if (a.lora_act.defined() != a.lora_up.defined()) return false;
  int64_t R = 0;
  Twin la, lu16;
  Tensor lu;
  if (a.lora_act.defined()) {
    if (!plain(a.lora_act, dev) || !plain(a.lora_up, dev) || a.lora_act.dim() != 2 || a.lora_up.dim() != 2) return false;
    R = a.lora_up.size(1);
    if (a.lora_act.size(0) != M || a.lora_up.size(0) != N || a.lora_act.size(1) != R || R % 16 != 0 || !int_sized(R)) return false;
    if (a.lora_up.scalar_type() != out_t) return false;
    if (R > 0) {
      la = attached(a.lora_act);
      if (!la.found() || la.type != out_t) return false;
      lu = a.lora_up;
      if (out_t == at::kBFloat16) {
        lu16 = attached(a.lora_up);
        if (!lu16.found()) return false;                     // recorded empty if a value does not fit fp16
      }
    }
  }
  for (const Tensor* v : {&a.wcscales, &a.bias, &a.smooth_next})
    if (v->defined() && (!plain(*v, dev) || v->dim() != 1 || v->size(0) != N || v->scalar_type() != out_t)) return false;
  const Twin sa = attached(a.ascales), sw = attached(a.wscales);
  if (!sa.found() || !sw.found()) return false;
  if (a.out.defined()) {
    if (!plain(a.out, dev) || a.out.dim() != 2 || a.out.size(0) != M || a.out.size(1) != N || a.out.scalar_type() != out_t) return false;
    r.y = a.out;
  }
  void* const stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  const int m = static_cast<int>(M), n = static_cast<int>(N), k = static_cast<int>(K), rr = static_cast<int>(R), dt = dtype_code(out_t);
  auto ptr = [](const Tensor& v) -> void* { return v.defined() && v.numel() > 0 ? v.data_ptr() : nullptr; };
  if (a.smooth_next.defined()) {
    if (!r.y.defined()) r.y = empty({M, N}, out_t);
    r.qout = empty({M, N / 2}, at::kByte);
    r.oscales = empty_output(N / 16, M, at::kFloat8_e4m3fn);
    const Twin oswz = empty_twin(M * (N / 16), at::kByte);
    int rc;
    {
      GilRelease nogil;
      rc = svdq_gemm_w4a4_next(ptr(a.act), ptr(a.wgt), sa.data(), sw.data(), la.data(), ptr(lu), lu16.data(), ptr(a.wcscales), ptr(a.bias),
                               ptr(r.y), ptr(a.smooth_next), ptr(r.qout), ptr(r.oscales), oswz.data(), m, n, k, rr, dt, 0, stream);
    }
    if (rc != SVDQ_OK) throw_status("gemm_w4a4_next", rc);
    if (!attach(r.oscales, oswz)) throw python_error();
    return true;
  }
  Tensor ws;                                                  // split-K: the workspace of this device and stream
  const unsigned long long need = m % 256 != 0 ? svdq_gemm_w4a4_workspace_bytes(m, n, k, rr) : 0;
  if (need > 0) {
    Ref key(Py_BuildValue("(iK)", static_cast<int>(dev), static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream))));
    PyObject* w = key.p != nullptr ? PyDict_GetItemWithError(g_split_ws, key.p) : nullptr;
    if (w == nullptr || !THPVariable_Check(w)) { PyErr_Clear(); return false; }            // made on the first call
    ws = THPVariable_Unpack(w);
    if (static_cast<unsigned long long>(ws.numel()) < need) return false;
  }
  if (!r.y.defined()) r.y = empty({M, N}, out_t);
  int rc;
  {
    GilRelease nogil;
    rc = svdq_gemm_w4a4_ws(ptr(a.act), ptr(a.wgt), sa.data(), sw.data(), la.data(), ptr(lu), lu16.data(), ptr(a.wcscales), ptr(a.bias),
                           ptr(r.y), m, n, k, rr, dt, 0, ptr(ws), ws.defined() ? static_cast<unsigned long long>(ws.numel()) : 0, stream);
  }
  if (rc != SVDQ_OK) throw_status("gemm_w4a4", rc);
  return true;
}

// ---------------------------------------------------------------------------
// Python entry points
// ---------------------------------------------------------------------------
// None -> undefined tensor; a tensor subclass or anything else -> false
bool unpack(PyObject* o, Tensor& t, bool optional) {
  if (o == Py_None) { t = Tensor(); return optional; }
  if (!THPVariable_CheckExact(o)) return false;
  t = THPVariable_Unpack(o);
  return true;
}

PyObject* py_quantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5) { PyErr_SetString(PyExc_TypeError, "quantize(input, lora_down, smooth, pad_size, out)"); return nullptr; }
  Tensor x, ld, smooth;
  if (!unpack(args[0], x, false) || !unpack(args[1], ld, false) || !unpack(args[2], smooth, true) || !PyLong_CheckExact(args[3]))
    Py_RETURN_NONE;
  int overflow = 0;
  const long long pad = PyLong_AsLongLongAndOverflow(args[3], &overflow);
  if (overflow != 0) Py_RETURN_NONE;
  Quantized into, out;
  const bool reuse = args[4] != Py_None;
  if (reuse) {
    if (!PyTuple_Check(args[4]) || PyTuple_GET_SIZE(args[4]) != 3 || !unpack(PyTuple_GET_ITEM(args[4], 0), into.act, false) ||
        !unpack(PyTuple_GET_ITEM(args[4], 1), into.ascales, false) || !unpack(PyTuple_GET_ITEM(args[4], 2), into.lora_act, false))
      Py_RETURN_NONE;
  }
  if (!quantize(x, ld, smooth, pad, reuse ? &into : nullptr, out)) Py_RETURN_NONE;
  if (reuse) return Py_NewRef(args[4]);
  Ref a(THPVariable_Wrap(std::move(out.act))), s(THPVariable_Wrap(std::move(out.ascales))), l(THPVariable_Wrap(std::move(out.lora_act)));
  if (a.p == nullptr || s.p == nullptr || l.p == nullptr) return nullptr;
  return PyTuple_Pack(3, a.p, s.p, l.p);
  END_HANDLE_TH_ERRORS
}

PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 11) {
    PyErr_SetString(PyExc_TypeError, "gemm(act, wgt, ascales, wscales, lora_act, lora_up, wcscales, bias, out_dtype, smooth_next, out)");
    return nullptr;
  }
  GemmArgs a;
  if (!unpack(args[0], a.act, false) || !unpack(args[1], a.wgt, false) || !unpack(args[2], a.ascales, false) ||
      !unpack(args[3], a.wscales, false) || !unpack(args[4], a.lora_act, true) || !unpack(args[5], a.lora_up, true) ||
      !unpack(args[6], a.wcscales, true) || !unpack(args[7], a.bias, true) || !unpack(args[9], a.smooth_next, true) ||
      !unpack(args[10], a.out, true))
    Py_RETURN_NONE;
  ScalarType t = a.lora_up.defined() ? a.lora_up.scalar_type() : at::kHalf;
  if (args[8] != Py_None) {
    if (!THPDtype_Check(args[8])) Py_RETURN_NONE;
    t = reinterpret_cast<THPDtype*>(args[8])->scalar_type;
  }
  GemmResult r;
  if (!gemm(a, t, r)) Py_RETURN_NONE;
  PyObject* y = args[10] != Py_None ? Py_NewRef(args[10]) : THPVariable_Wrap(std::move(r.y));
  if (!a.smooth_next.defined() || y == nullptr) return y;
  Ref hold(y), q(THPVariable_Wrap(std::move(r.qout))), s(THPVariable_Wrap(std::move(r.oscales)));
  if (q.p == nullptr || s.p == nullptr) return nullptr;
  return PyTuple_Pack(3, y, q.p, s.p);
  END_HANDLE_TH_ERRORS
}

PyObject* py_pack(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "pack(x, pad_size)"); return nullptr; }
  Tensor x;
  if (!unpack(args[0], x, false) || !PyLong_CheckExact(args[1])) Py_RETURN_NONE;
  int overflow = 0;
  const long long pad = PyLong_AsLongLongAndOverflow(args[1], &overflow);
  if (!x.is_cuda()) Py_RETURN_NONE;
  const c10::DeviceIndex dev = c10::cuda::current_device();
  if (overflow != 0 || pad < 1 || !plain(x, dev) || x.dim() != 2 || dtype_code(x.scalar_type()) < 0) Py_RETURN_NONE;
  const int64_t rows = x.size(0), K = x.size(1);
  if (rows == 0 || K == 0 || K % 16 != 0) Py_RETURN_NONE;
  const int64_t rp = (rows + pad - 1) / pad * pad;
  if (!int_sized(rp) || !int_sized(K)) Py_RETURN_NONE;
  Tensor packed = empty({rp, K / 2}, at::kByte), scales = empty({K / 16, rp}, at::kFloat8_e4m3fn);
  Twin swz;
  if (rp % 128 == 0 && K % 64 == 0) swz = empty_twin(rp * (K / 16), at::kByte);
  void* const stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  {
    GilRelease nogil;
    rc = svdq_quantize_nvfp4_rows(x.data_ptr(), packed.data_ptr(), scales.data_ptr(), swz.data(),
                                  static_cast<int>(rows), static_cast<int>(rp), static_cast<int>(K), dtype_code(x.scalar_type()), stream);
  }
  if (rc != SVDQ_OK) throw_status("quantize_nvfp4_rows", rc);
  if (swz.found() && !attach(scales, swz)) throw python_error();
  Ref p(THPVariable_Wrap(std::move(packed))), s(THPVariable_Wrap(std::move(scales)));
  if (p.p == nullptr || s.p == nullptr) return nullptr;
  return PyTuple_Pack(2, p.p, s.p);
  END_HANDLE_TH_ERRORS
}

// output_twin(owner, any_version): what `attached` finds on the owner's storage itself, or None
PyObject* py_output_twin(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2 || !THPVariable_Check(args[0])) { PyErr_SetString(PyExc_TypeError, "output_twin(owner, any_version)"); return nullptr; }
  const Tensor& owner = THPVariable_Unpack(args[0]);
  if (output_storage(owner) == nullptr) Py_RETURN_NONE;
  const Twin twin = attached(owner, PyObject_IsTrue(args[1]) == 1);
  if (!twin.found()) Py_RETURN_NONE;
  return THPVariable_Wrap(tensor_of(twin));
  END_HANDLE_TH_ERRORS
}

// attach_output(owner, twin): record the twin if it belongs on the owner's storage itself; whether it does
PyObject* py_attach_output(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) {
    PyErr_SetString(PyExc_TypeError, "attach_output(owner, twin)");
    return nullptr;
  }
  const Tensor& owner = THPVariable_Unpack(args[0]);
  if (output_storage(owner) == nullptr) Py_RETURN_FALSE;
  const Tensor& t = THPVariable_Unpack(args[1]);
  attach(owner, Twin{t.numel() > 0 ? t.data_ptr() : nullptr, t.scalar_type(), t.numel(), t, {}});
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// bind(split_workspaces, quantize, gemm): the workspace table and the Python operators of ops.py
PyObject* py_bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3 || !PyDict_Check(args[0])) { PyErr_SetString(PyExc_TypeError, "bind(split_workspaces, quantize, gemm)"); return nullptr; }
  Py_XSETREF(g_split_ws, Py_NewRef(args[0]));
  Py_XSETREF(g_py_quantize, Py_NewRef(args[1]));
  Py_XSETREF(g_py_gemm, Py_NewRef(args[2]));
  Py_RETURN_NONE;
}

// ---------------------------------------------------------------------------
// dispatcher (torch.ops.svdq_b200.*)
// ---------------------------------------------------------------------------
using OptTensor = std::optional<Tensor>;

Tensor value(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
PyObject* wrap(const Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None); }
Tensor take(PyObject* o) {
  TORCH_CHECK(o != nullptr && THPVariable_Check(o), "svdq_b200: the Python operator returned something else than tensors");
  return THPVariable_Unpack(o);
}

std::tuple<Tensor, Tensor, Tensor> op_quantize(const Tensor& x, const Tensor& ld, const OptTensor& smooth, int64_t pad) {
  GilAcquire gil;
  TORCH_CHECK(g_py_quantize != nullptr, "svdq_b200: import svdquant_kernels_b200.torch_ops first");
  Quantized q;
  if (quantize(x, ld, value(smooth), pad, nullptr, q)) return {q.act, q.ascales, q.lora_act};
  Ref args(Py_BuildValue("(NNN)", wrap(x), wrap(ld), wrap(value(smooth))));
  Ref kw(Py_BuildValue("{s:L}", "pad_size", static_cast<long long>(pad)));
  if (args.p == nullptr || kw.p == nullptr) throw python_error();
  Ref res(PyObject_Call(g_py_quantize, args.p, kw.p));
  if (res.p == nullptr) throw python_error();
  TORCH_CHECK(PyTuple_Check(res.p) && PyTuple_GET_SIZE(res.p) == 3);
  return {take(PyTuple_GET_ITEM(res.p, 0)), take(PyTuple_GET_ITEM(res.p, 1)), take(PyTuple_GET_ITEM(res.p, 2))};
}

Tensor op_gemm(const Tensor& act, const Tensor& wgt, const Tensor& ascales, const Tensor& wscales, const OptTensor& lora_act,
               const OptTensor& lora_up, const OptTensor& wcscales, const OptTensor& bias, std::optional<ScalarType> out_dtype) {
  GilAcquire gil;
  TORCH_CHECK(g_py_gemm != nullptr, "svdq_b200: import svdquant_kernels_b200.torch_ops first");
  GemmArgs a{act, wgt, ascales, wscales, value(lora_act), value(lora_up), value(wcscales), value(bias), Tensor(), Tensor()};
  const ScalarType t = out_dtype.has_value() ? *out_dtype : a.lora_up.defined() ? a.lora_up.scalar_type() : at::kHalf;
  GemmResult r;
  if (gemm(a, t, r)) return r.y;
  PyObject* dt = Py_None;
  if (out_dtype.has_value()) dt = reinterpret_cast<PyObject*>(torch::getTHPDtype(*out_dtype));
  Ref args(Py_BuildValue("(NNNNNNNNO)", wrap(act), wrap(wgt), wrap(ascales), wrap(wscales), wrap(a.lora_act), wrap(a.lora_up),
                         wrap(a.wcscales), wrap(a.bias), dt));
  if (args.p == nullptr) throw python_error();
  Ref res(PyObject_Call(g_py_gemm, args.p, nullptr));
  if (res.p == nullptr) throw python_error();
  return take(res.p);
}

// The operators have no backward pass: results of inputs that require a gradient carry a node that says so
// when it is reached.
template <typename... In>
std::shared_ptr<torch::autograd::Node> no_backward(const char* name, const In&... in) {
  if (!torch::autograd::compute_requires_grad(in...)) return nullptr;
  auto node = std::make_shared<torch::autograd::NotImplemented>(name);
  node->set_next_edges(torch::autograd::collect_next_edges(in...));
  return node;
}

// (Called through the dispatcher again, so that tracing and fake tensors, which sit below autograd, are seen.)
using QuantizeSig = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const OptTensor&, c10::SymInt);
using GemmSig = Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const OptTensor&,
                       const OptTensor&, const OptTensor&, std::optional<ScalarType>);

std::tuple<Tensor, Tensor, Tensor> op_quantize_autograd(const Tensor& x, const Tensor& ld, const OptTensor& smooth, c10::SymInt pad) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("svdq_b200::quantize_w4a4_act_fuse_lora", "").typed<QuantizeSig>();
  const auto node = no_backward("svdq_b200::quantize_w4a4_act_fuse_lora", x, ld, value(smooth));
  at::AutoDispatchBelowADInplaceOrView below;
  auto r = op.call(x, ld, smooth, std::move(pad));
  if (node) {                                                 // the integer codes are not differentiable
    torch::autograd::set_history(std::get<1>(r), node);
    torch::autograd::set_history(std::get<2>(r), node);
  }
  return r;
}

Tensor op_gemm_autograd(const Tensor& act, const Tensor& wgt, const Tensor& ascales, const Tensor& wscales, const OptTensor& lora_act,
                        const OptTensor& lora_up, const OptTensor& wcscales, const OptTensor& bias, std::optional<ScalarType> out_dtype) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("svdq_b200::gemm_w4a4", "").typed<GemmSig>();
  const auto node = no_backward("svdq_b200::gemm_w4a4", act, wgt, ascales, wscales, value(lora_act), value(lora_up), value(wcscales), value(bias));
  at::AutoDispatchBelowADInplaceOrView below;
  Tensor y = op.call(act, wgt, ascales, wscales, lora_act, lora_up, wcscales, bias, out_dtype);
  if (node) torch::autograd::set_history(y, node);
  return y;
}

TORCH_LIBRARY(svdq_b200, m) {
  m.def("quantize_w4a4_act_fuse_lora(Tensor input, Tensor lora_down, Tensor? smooth=None, SymInt pad_size=256) -> (Tensor, Tensor, Tensor)");
  m.def("gemm_w4a4(Tensor act, Tensor wgt, Tensor ascales, Tensor wscales, Tensor? lora_act_in=None, Tensor? lora_up=None, "
        "Tensor? wcscales=None, Tensor? bias=None, ScalarType? out_dtype=None) -> Tensor");
}
TORCH_LIBRARY_IMPL(svdq_b200, CUDA, m) {
  m.impl("quantize_w4a4_act_fuse_lora", op_quantize);
  m.impl("gemm_w4a4", op_gemm);
}
TORCH_LIBRARY_IMPL(svdq_b200, AutogradCUDA, m) {
  m.impl("quantize_w4a4_act_fuse_lora", op_quantize_autograd);
  m.impl("gemm_w4a4", op_gemm_autograd);
}

PyMethodDef g_methods[] = {
    {"quantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_quantize)), METH_FASTCALL, nullptr},
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_gemm)), METH_FASTCALL, nullptr},
    {"pack", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_pack)), METH_FASTCALL, nullptr},
    {"output_twin", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_output_twin)), METH_FASTCALL, nullptr},
    {"attach_output", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attach_output)), METH_FASTCALL, nullptr},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_bind)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the operators.", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  g_twins_name = PyUnicode_InternFromString("_svdq_twins");
  return g_twins_name != nullptr ? PyModule_Create(&g_module) : nullptr;
}
