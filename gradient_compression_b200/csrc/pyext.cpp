// The reducers' way from Python into the kernels: a CPython extension module.
//
// A reduce of a whole model hands over some hundred tensors, and what it computes takes a few dozen microseconds; looking at
// the tensors through the Python interpreter (dtype, layout, address, adjacency) takes ten times that.  This module reads
// them natively, merges neighbours, and calls the C ABI of the kernel library, whose entry points it is given as addresses
// (`bind`), so that the regular and the bounds-checking build are served by the same module.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <unordered_map>
#include <vector>

namespace {

struct SegDesc {            // csrc/gc_segs.cuh
  const float* in;
  float* out;
  int64_t start;
};

// Entry points of the kernel library.
struct Api {
  int (*solo_max_segs)();
  int (*comm_device)(void*);
  int (*solo_maxnorm)(void*, const void*, int, int64_t, int, int, uint64_t, uint32_t, int, int, void*);
  int (*solo_copy)(void*, const void*, int, int64_t, void*);
  int64_t (*solo_randk_limit)(void*, int);
  int (*solo_randk)(void*, const void*, int, int64_t, uint64_t, uint32_t, int64_t, int64_t, int64_t*, int, int, int, uint32_t, int, int, void*);
  int (*topk_run)(const void*, int, int64_t, const int64_t*, int, float*, void*, void*, int32_t*, float*, void*);
  int (*psgd_solo)(int, const void*, int, float*, const int64_t*, int, int64_t, int64_t, int, const int64_t*, int, float*, float*, float*, int64_t, uint64_t,
                   uint32_t, uint32_t*, void*);
  int64_t (*absmax_scratch_bytes)();
  int (*absmax)(const float*, int64_t, void*, float*, void*);
  int (*quantize)(const float*, int64_t, const float*, int, int, uint64_t, uint32_t, uint32_t, void*, int, void*);
  int (*quantize_fit)(const float*, int64_t, const float*, int, int, uint64_t, uint32_t, uint32_t, void*, int, int8_t*, void*);
  int (*dequantize)(const void*, int, int64_t, const float*, int, int, float*, void*);
  int64_t (*conv_bn_eval_scratch)(int, int, int, int, int, int, int, int);
  int (*conv_bn_eval)(const float*, const float*, float*, const float*, int, int, int, int, int, int, int, int, const float*, const float*, const float*,
                      const float*, float, const float*, int, float*, int*, void*);
  int (*head_eval)(const float*, int, int, int, const float*, const float*, int, float*, void*);
  int (*logit_metrics)(const float*, const int64_t*, int, int, float*, void*);
  int (*max_pool2)(const float*, int, int, int, int, float*, void*);
  int (*bn_supported)(int64_t, int);
  int (*bn_eval_apply)(const float*, int64_t, int, const float*, const float*, float, const float*, const float*, const float*, int, float*, void*);
  int (*dequantize_two)(const void*, int, const int8_t*, int64_t, const float*, int, int, int, float*, void*);
} api;
int max_segs = 0;

struct Entry { const char* name; void** slot; };
const Entry entries[] = {
    {"gc_solo_max_segs", (void**)&api.solo_max_segs},
    {"gc_comm_device", (void**)&api.comm_device},
    {"gc_solo_maxnorm", (void**)&api.solo_maxnorm},
    {"gc_solo_copy", (void**)&api.solo_copy},
    {"gc_solo_randk_limit", (void**)&api.solo_randk_limit},
    {"gc_solo_randk", (void**)&api.solo_randk},
    {"gc_cuda_topk_run", (void**)&api.topk_run},
    {"gc_cuda_psgd_solo", (void**)&api.psgd_solo},
    {"gc_cuda_absmax_scratch_bytes", (void**)&api.absmax_scratch_bytes},
    {"gc_cuda_absmax", (void**)&api.absmax},
    {"gc_cuda_quantize_levels", (void**)&api.quantize},
    {"gc_cuda_quantize_fit", (void**)&api.quantize_fit},
    {"gc_cuda_dequantize_levels", (void**)&api.dequantize},
    {"gc_cuda_conv_bn_eval_scratch", (void**)&api.conv_bn_eval_scratch},
    {"gc_cuda_conv_bn_eval", (void**)&api.conv_bn_eval},
    {"gc_cuda_head_eval", (void**)&api.head_eval},
    {"gc_cuda_logit_metrics", (void**)&api.logit_metrics},
    {"gc_cuda_max_pool2", (void**)&api.max_pool2},
    {"gc_cuda_bn_supported", (void**)&api.bn_supported},
    {"gc_cuda_bn_eval_apply", (void**)&api.bn_eval_apply},
    {"gc_cuda_dequantize_two", (void**)&api.dequantize_two},
};

// What one reducer saw last: its segment table, and the fact that its inputs and outputs do not overlap in an unsafe way
// (checked once per set of addresses).
struct Plan {
  std::vector<SegDesc> segs, checked;
  std::vector<int64_t> shape, shape_seen;     // dimensions, first extent and elements of every tensor
  int64_t n = 0;
  int64_t generation = 0;          // counts changes of the tensors' shapes
  int device = -1;
};

void plan_free(PyObject* cap) { delete (Plan*)PyCapsule_GetPointer(cap, "gcb200.plan"); }
Plan* plan_of(PyObject* o) { return (Plan*)PyCapsule_GetPointer(o, "gcb200.plan"); }

PyObject* plan_new(PyObject*, PyObject*) { return PyCapsule_New(new Plan(), "gcb200.plan", plan_free); }

// Address of a dense fp32 CUDA tensor in one of the two memory orders reducers take (contiguous, or channels-last for four
// dimensions); nullptr for anything else.  `order`: 0 contiguous, 1 channels-last.
float* dense_ptr(PyObject* o, int64_t* n, int* device, int* order) {
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.scalar_type() != at::kFloat || t.layout() != at::kStrided) return nullptr;
  if (t.is_contiguous()) *order = 0;
  else if (t.dim() == 4 && t.is_contiguous(at::MemoryFormat::ChannelsLast)) *order = 1;
  else return nullptr;
  *n = t.numel();
  *device = t.device().index();
  return (float*)t.data_ptr();
}

// Inputs are read again after outputs have been written: an output may be its own input, but must not touch another one.
bool overlap_free(const std::vector<SegDesc>& segs, int64_t n) {
  struct Range { uintptr_t lo, hi; int seg; bool out; };
  std::vector<Range> r;
  r.reserve(segs.size() * 2);
  for (size_t i = 0; i < segs.size(); ++i) {
    const int64_t len = (i + 1 < segs.size() ? segs[i + 1].start : n) - segs[i].start;
    if (len <= 0) continue;
    const uintptr_t a = (uintptr_t)segs[i].in, b = (uintptr_t)segs[i].out;
    r.push_back({a, a + (uintptr_t)len * 4, (int)i, false});
    r.push_back({b, b + (uintptr_t)len * 4, (int)i, true});
  }
  std::sort(r.begin(), r.end(), [](const Range& x, const Range& y) { return x.lo < y.lo || (x.lo == y.lo && x.seg < y.seg); });
  // sweep: the furthest end of any input / output seen so far, and whose it is
  uintptr_t in_hi = 0, out_hi = 0;
  int in_seg = -1, out_seg = -1;
  for (const Range& x : r) {
    const bool same_in = in_seg == x.seg && segs[x.seg].in == segs[x.seg].out, same_out = out_seg == x.seg && segs[x.seg].in == segs[x.seg].out;
    if (x.lo < out_hi && !same_out) return false;
    if (x.out && x.lo < in_hi && !same_in) return false;
    if (x.out) { if (x.hi > out_hi) { out_hi = x.hi; out_seg = x.seg; } }
    else if (x.hi > in_hi) { in_hi = x.hi; in_seg = x.seg; }
  }
  return true;
}

// Fills the plan from two lists of tensors.  False: not a case for the segment kernels (the caller takes the general path).
// `merge`: neighbours in memory become one segment (otherwise a segment per non-empty tensor).  The kernels run where the tensors
// are and synchronise on words of the arena `ctx`: both have to be on one device.
bool collect(Plan& p, void* ctx, PyObject* ins, PyObject* outs, bool merge = true) {
  const THPObjectPtr fa(PySequence_Fast(ins, "reduce() takes lists of tensors"));
  if (!fa) return false;
  const THPObjectPtr fb(ins == outs ? Py_NewRef(fa.get()) : PySequence_Fast(outs, "reduce() takes lists of tensors"));
  if (!fb) return false;
  const Py_ssize_t k = PySequence_Fast_GET_SIZE(fa.get());
  bool ok = k > 0 && PySequence_Fast_GET_SIZE(fb.get()) == k;
  p.segs.clear();
  p.shape.clear();
  p.n = 0;
  p.device = -1;
  for (Py_ssize_t i = 0; ok && i < k; ++i) {
    int64_t na = 0, nb = 0;
    int da = 0, db = 0, oa = 0, ob = 0;
    PyObject *pa = PySequence_Fast_GET_ITEM(fa.get(), i), *pb = PySequence_Fast_GET_ITEM(fb.get(), i);
    float* a = dense_ptr(pa, &na, &da, &oa);
    float* b = a;
    if (pa == pb) { nb = na; db = da; ob = oa; }
    else b = dense_ptr(pb, &nb, &db, &ob);
    if (a != nullptr || na == 0) {
      if (THPVariable_Check(pa)) {
        const at::Tensor& t = THPVariable_Unpack(pa);
        p.shape.push_back(t.dim());
        p.shape.push_back(t.dim() > 0 ? t.size(0) : 1);
        p.shape.push_back(na);
      }
    }
    if (na == 0 && nb == 0 && THPVariable_Check(pa) && THPVariable_Check(pb)) continue;
    if (a == nullptr || b == nullptr || na != nb || da != db || oa != ob || (p.device >= 0 && da != p.device)) { ok = false; break; }
    if (oa == 1 && pa != pb && THPVariable_Unpack(pa).sizes() != THPVariable_Unpack(pb).sizes()) { ok = false; break; }
    p.device = da;
    if (merge && !p.segs.empty()) {
      const SegDesc& last = p.segs.back();
      const int64_t len = p.n - last.start;
      if (a == last.in + len && b == last.out + len) { p.n += na; continue; }
    }
    p.segs.push_back({a, b, p.n});
    p.n += na;
  }
  if (PyErr_Occurred()) return false;
  if (!ok || p.segs.empty() || (int)p.segs.size() > max_segs || p.device != api.comm_device(ctx)) return false;
  const bool known = p.checked.size() == p.segs.size() + 1 && p.checked.back().start == p.n &&
                     memcmp(p.checked.data(), p.segs.data(), p.segs.size() * sizeof(SegDesc)) == 0;
  if (!known) {
    p.checked.clear();
    if (!overlap_free(p.segs, p.n)) return false;
    p.checked = p.segs;
    p.checked.push_back({nullptr, nullptr, p.n});
  }
  return true;
}

void* stream_on(int device) { return (void*)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

// A call's entry from Python: what libtorch throws (out of memory, a tensor without storage) becomes a Python exception instead of
// leaving through the interpreter's C frames, which ends the process.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* entry(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, a, n);
  END_HANDLE_TH_ERRORS
}
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction method() { return (PyCFunction)(void (*)(void))entry<F>; }

// Allocations and launches run without the interpreter lock: either may wait for the GPU (a full launch queue, an allocator that
// synchronises), and what the GPU waits for may be another thread's next launch.
struct NoGil {
  PyThreadState* const state = PyEval_SaveThread();
  NoGil() = default;
  NoGil(const NoGil&) = delete;
  ~NoGil() { PyEval_RestoreThread(state); }
};
template <class F>
auto unlocked(F f) {
  const NoGil released;
  return f();
}

PyObject* cuda_error(const char* what, int err) {
  PyErr_Format(PyExc_RuntimeError, "%s: CUDA error %d", what, err);
  return nullptr;
}

// A launch's own copy of a plan's tensors: the plan may be filled again while the lock is released.
struct Tensors {
  const std::vector<SegDesc> segs;
  const int64_t n;
  const int device;
  explicit Tensors(const Plan& p) : segs(p.segs), n(p.n), device(p.device) {}
  const void* data() const { return segs.data(); }
  int count() const { return (int)segs.size(); }
  void* stream() const { return stream_on(device); }
};

// Counts and scales come as any number, as int() takes them.
int64_t as_int(PyObject* o) {
  if (PyLong_Check(o)) return PyLong_AsLongLong(o);
  THPObjectPtr i(PyNumber_Long(o));
  return i ? PyLong_AsLongLong(i.get()) : -1;
}
uint64_t as_bits(PyObject* o) {            // modulo 2^64
  if (PyLong_Check(o)) return PyLong_AsUnsignedLongLongMask(o);
  THPObjectPtr i(PyNumber_Long(o));
  return i ? PyLong_AsUnsignedLongLongMask(i.get()) : 0;
}

bool want(Py_ssize_t nargs, Py_ssize_t n, const char* name) {
  if (nargs == n) return true;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given)", name, n, nargs);
  return false;
}

// solo_maxnorm(plan, ctx, grad_in, grad_out, bits_lo, bits_hi, seed, step, timeout_ms, max_blocks) -> elements, or None
PyObject* solo_maxnorm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 10, "solo_maxnorm")) return nullptr;
  Plan* p = plan_of(a[0]);
  if (!p) return nullptr;
  void* ctx = (void*)PyLong_AsUnsignedLongLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  if (!collect(*p, ctx, a[2], a[3])) { if (PyErr_Occurred()) return nullptr; Py_RETURN_NONE; }
  const int lo = (int)as_int(a[4]), hi = (int)as_int(a[5]), timeout = (int)as_int(a[8]), blocks = (int)as_int(a[9]);
  const uint64_t seed = PyLong_AsUnsignedLongLongMask(a[6]);
  const uint32_t step = (uint32_t)PyLong_AsUnsignedLongLongMask(a[7]);
  if (PyErr_Occurred()) return nullptr;
  c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, (c10::DeviceIndex)p->device));
  const Tensors t(*p);
  const int err = unlocked([&] { return api.solo_maxnorm(ctx, t.data(), t.count(), t.n, lo, hi, seed, step, timeout, blocks, t.stream()); });
  if (err) return cuda_error("solo_maxnorm", err);
  return PyLong_FromLongLong(t.n);
}

// solo_copy(plan, ctx, grad_in, grad_out) -> elements, or None
PyObject* solo_copy(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 4, "solo_copy")) return nullptr;
  Plan* p = plan_of(a[0]);
  if (!p) return nullptr;
  void* ctx = (void*)PyLong_AsUnsignedLongLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  if (!collect(*p, ctx, a[2], a[3])) { if (PyErr_Occurred()) return nullptr; Py_RETURN_NONE; }
  bool moves = false;
  for (const SegDesc& s : p->segs) moves = moves || s.in != s.out;
  if (moves) {
    c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, (c10::DeviceIndex)p->device));
    const Tensors t(*p);
    const int err = unlocked([&] { return api.solo_copy(ctx, t.data(), t.count(), t.n, t.stream()); });
    if (err) return cuda_error("solo_copy", err);
    return PyLong_FromLongLong(t.n);
  }
  return PyLong_FromLongLong(p->n);
}

// collect(plan, ctx, grad_in, grad_out, merge) -> (elements, generation of the tensors' shapes, segments), or None.
// merge: 1 neighbours become one segment, 0 a segment per tensor, 2 one segment if all of them are neighbours, else one per tensor
PyObject* collect_py(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 5, "collect")) return nullptr;
  Plan* p = plan_of(a[0]);
  if (!p) return nullptr;
  void* ctx = (void*)PyLong_AsUnsignedLongLong(a[1]);
  const int merge = (int)as_int(a[4]);
  if (PyErr_Occurred()) return nullptr;
  bool ok = collect(*p, ctx, a[2], a[3], merge != 0);
  if (ok && merge == 2 && p->segs.size() > 1) ok = collect(*p, ctx, a[2], a[3], false);
  if (!ok) { if (PyErr_Occurred()) return nullptr; Py_RETURN_NONE; }
  if (p->shape != p->shape_seen) {
    p->shape_seen = p->shape;
    ++p->generation;
  }
  return Py_BuildValue("LLn", (long long)p->n, (long long)p->generation, (Py_ssize_t)p->segs.size());
}

// solo_randk(plan, ctx, seed, npass, start, k, window or 0, bits_lo, bits_hi, zero, step, timeout_ms, max_blocks): on what collect() found
PyObject* solo_randk(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 13, "solo_randk")) return nullptr;
  Plan* p = plan_of(a[0]);
  if (!p) return nullptr;
  void* ctx = (void*)PyLong_AsUnsignedLongLong(a[1]);
  const uint64_t seed = PyLong_AsUnsignedLongLongMask(a[2]);
  const uint32_t npass = (uint32_t)PyLong_AsUnsignedLongLongMask(a[3]), step = (uint32_t)PyLong_AsUnsignedLongLongMask(a[10]);
  const int64_t start = as_int(a[4]), k = as_int(a[5]);
  int64_t* window = (int64_t*)PyLong_AsUnsignedLongLong(a[6]);
  const int lo = (int)as_int(a[7]), hi = (int)as_int(a[8]), zero = (int)as_int(a[9]), timeout = (int)as_int(a[11]), blocks = (int)as_int(a[12]);
  if (PyErr_Occurred()) return nullptr;
  c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, (c10::DeviceIndex)p->device));
  const Tensors t(*p);
  const int err = unlocked([&] {
    return api.solo_randk(ctx, t.data(), t.count(), t.n, seed, npass, start, k, window, lo, hi, zero, step, timeout, blocks, t.stream());
  });
  if (err) return cuda_error("solo_randk", err);
  Py_RETURN_NONE;
}

// solo_randk_limit(ctx, max_blocks) -> most coordinates solo_randk takes
PyObject* solo_randk_limit(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 2, "solo_randk_limit")) return nullptr;
  void* ctx = (void*)PyLong_AsUnsignedLongLong(a[0]);
  const int blocks = (int)as_int(a[1]);
  if (PyErr_Occurred()) return nullptr;
  return PyLong_FromLongLong(api.solo_randk_limit(ctx, blocks));
}

// solo_psgd(plan, rank, memory, tab, n_mats, rows, tiles, max_rows, vtab, n_vecs, q, p, q_parts, q_total, seed, stream, step or 0)
PyObject* solo_psgd(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 17, "solo_psgd")) return nullptr;
  Plan* p = plan_of(a[0]);
  if (!p) return nullptr;
  const int rank = (int)as_int(a[1]);
  uint64_t v[16] = {};
  for (int i = 1; i < 16; ++i) v[i] = i == 13 ? PyLong_AsUnsignedLongLongMask(a[i + 1]) : PyLong_AsUnsignedLongLong(a[i + 1]);
  if (PyErr_Occurred()) return nullptr;
  c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, (c10::DeviceIndex)p->device));
  const Tensors t(*p);
  const int err = unlocked([&] {
    return api.psgd_solo(rank, t.data(), t.count(), (float*)v[1], (const int64_t*)v[2], (int)v[3], (int64_t)v[4], (int64_t)v[5], (int)v[6], (const int64_t*)v[7],
                         (int)v[8], (float*)v[9], (float*)v[10], (float*)v[11], (int64_t)v[12], v[13], (uint32_t)v[14], (uint32_t*)v[15], t.stream());
  });
  if (err) return cuda_error("solo_psgd", err);
  Py_RETURN_NONE;
}

// solo_topk(plan, counts (address of int64 per group), per_tensor, memory, state, lists: addresses): on what collect() found
PyObject* solo_topk(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 6, "solo_topk")) return nullptr;
  Plan* p = plan_of(a[0]);
  if (!p) return nullptr;
  uint64_t v[6] = {};
  for (int i = 1; i < 6; ++i) v[i] = PyLong_AsUnsignedLongLong(a[i]);
  if (PyErr_Occurred()) return nullptr;
  c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, (c10::DeviceIndex)p->device));
  const Tensors t(*p);
  const int err = unlocked([&] {
    return api.topk_run(t.data(), t.count(), t.n, (const int64_t*)v[1], (int)v[2], (float*)v[3], (void*)v[4], (void*)v[5], nullptr, nullptr, t.stream());
  });
  if (err) return cuda_error("solo_topk", err);
  Py_RETURN_NONE;
}

// ---- codecs ------------------------------------------------------------------------------------------------------
// Each returns None where a tensor is not the kernel's case (the caller then takes its general path).

const at::Tensor* tensor_of(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

const at::Tensor* plain(PyObject* o, at::ScalarType type) {
  const at::Tensor* t = tensor_of(o);
  return t && t->is_cuda() && t->scalar_type() == type && t->layout() == at::kStrided && t->is_contiguous() ? t : nullptr;
}

int level_size(at::ScalarType t) { return t == at::kChar ? 1 : t == at::kShort ? 2 : t == at::kInt ? 4 : 0; }
at::ScalarType level_type(int64_t size) { return size == 1 ? at::kChar : size == 2 ? at::kShort : at::kInt; }

// absmax(x, out or None) -> one-element tensor
PyObject* absmax(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 2, "absmax")) return nullptr;
  const at::Tensor* x = plain(a[0], at::kFloat);
  const at::Tensor* given = a[1] == Py_None ? nullptr : plain(a[1], at::kFloat);
  if (!x || x->numel() == 0 || (a[1] != Py_None && !given)) Py_RETURN_NONE;
  const int dev = x->device().index();
  if (dev >= 64 || (given && (given->device() != x->device() || given->numel() < 1))) Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(x->device());
  static at::Tensor scratch[64];           // zeroed once; the kernel leaves it ready for the next call
  if (!scratch[dev].defined()) scratch[dev] = at::zeros({api.absmax_scratch_bytes()}, x->options().dtype(at::kByte));
  void* words = scratch[dev].data_ptr();
  at::Tensor out;
  const int err = unlocked([&] {
    out = given ? *given : at::empty({1}, x->options());
    return api.absmax((const float*)x->data_ptr(), x->numel(), words, (float*)out.data_ptr(), stream_on(dev));
  });
  if (err) return cuda_error("absmax", err);
  return THPVariable_Wrap(out);
}

// quantize(x, norm, s, mode, seed, stream, step, size, out or None) -> levels
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 9, "quantize")) return nullptr;
  const at::Tensor *x = plain(a[0], at::kFloat), *norm = plain(a[1], at::kFloat), *given = a[8] == Py_None ? nullptr : tensor_of(a[8]);
  if (!x || !norm || norm->numel() != 1 || norm->device() != x->device() || x->numel() == 0) Py_RETURN_NONE;
  const int64_t s = as_int(a[2]), mode = as_int(a[3]), size = as_int(a[7]);
  const uint64_t seed = as_bits(a[4]);
  const uint32_t stream = (uint32_t)as_bits(a[5]), step = (uint32_t)as_bits(a[6]);
  if (PyErr_Occurred()) return nullptr;
  if (size != 1 && size != 2 && size != 4) Py_RETURN_NONE;
  if (given && (!given->is_cuda() || !given->is_contiguous() || given->device() != x->device() || level_size(given->scalar_type()) != size ||
                given->numel() < x->numel()))
    Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(x->device());
  at::Tensor out;
  const int err = unlocked([&] {
    out = given ? *given : at::empty({x->numel()}, x->options().dtype(level_type(size)));
    return api.quantize((const float*)x->data_ptr(), x->numel(), (const float*)norm->data_ptr(), (int)s, (int)mode, seed, stream, step, out.data_ptr(), (int)size,
                        stream_on(x->device().index()));
  });
  if (err) return cuda_error("quantize_levels", err);
  return THPVariable_Wrap(out);
}

// quantize_fit(x, norm, s, s_fit, seed, stream, step, size) -> (levels, int8 mask of those that fit s_fit)
PyObject* quantize_fit(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 8, "quantize_fit")) return nullptr;
  const at::Tensor *x = plain(a[0], at::kFloat), *norm = plain(a[1], at::kFloat);
  const int64_t s = as_int(a[2]), fit = as_int(a[3]), size = as_int(a[7]);
  const uint64_t seed = as_bits(a[4]);
  const uint32_t stream = (uint32_t)as_bits(a[5]), step = (uint32_t)as_bits(a[6]);
  if (PyErr_Occurred()) return nullptr;
  if (!x || !norm || norm->numel() != 1 || norm->device() != x->device() || x->numel() == 0 || s >= (1 << 22)) Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(x->device());
  at::Tensor out, mask;
  const int err = unlocked([&] {
    out = at::empty({x->numel()}, x->options().dtype(level_type(size)));
    mask = at::empty({x->numel()}, x->options().dtype(at::kChar));
    return api.quantize_fit((const float*)x->data_ptr(), x->numel(), (const float*)norm->data_ptr(), (int)s, (int)fit, seed, stream, step, out.data_ptr(),
                            (int)size, (int8_t*)mask.data_ptr(), stream_on(x->device().index()));
  });
  if (err) return cuda_error("quantize_fit", err);
  PyObject *po = THPVariable_Wrap(out), *pm = THPVariable_Wrap(mask);
  PyObject* r = PyTuple_Pack(2, po, pm);
  Py_XDECREF(po);
  Py_XDECREF(pm);
  return r;
}

// dequantize(q, mask or None, norm, s, s_other, world, out or None) -> values
PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 7, "dequantize")) return nullptr;
  const at::Tensor *q = tensor_of(a[0]), *mask = a[1] == Py_None ? nullptr : plain(a[1], at::kChar), *norm = plain(a[2], at::kFloat);
  const at::Tensor* given = a[6] == Py_None ? nullptr : plain(a[6], at::kFloat);
  const int64_t s = as_int(a[3]), other = as_int(a[4]), world = as_int(a[5]);
  if (PyErr_Occurred()) return nullptr;
  if (!q || !q->is_cuda() || !q->is_contiguous() || q->numel() == 0 || !level_size(q->scalar_type()) || !norm || norm->numel() != 1 ||
      norm->device() != q->device() || (a[1] != Py_None && (!mask || mask->numel() != q->numel() || mask->device() != q->device())) ||
      (a[6] != Py_None && (!given || given->numel() != q->numel() || given->device() != q->device())))
    Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(q->device());
  at::Tensor out;
  const int err = unlocked([&] {
    out = given ? *given : at::empty({q->numel()}, norm->options());
    const int size = level_size(q->scalar_type());
    void* st = stream_on(q->device().index());
    return mask ? api.dequantize_two(q->data_ptr(), size, (const int8_t*)mask->data_ptr(), q->numel(), (const float*)norm->data_ptr(), (int)s, (int)other, (int)world,
                                     (float*)out.data_ptr(), st)
                : api.dequantize(q->data_ptr(), size, q->numel(), (const float*)norm->data_ptr(), (int)s, (int)world, (float*)out.data_ptr(), st);
  });
  if (err) return cuda_error("dequantize_levels", err);
  return THPVariable_Wrap(out);
}

// ---- inference ---------------------------------------------------------------------------------------------------
// Whether an operator is expected to leave a trace of itself that these calls do not: a tangent of forward-mode differentiation, a
// node of a graph being traced, a functorch transform.  The general path says that it has none.
bool observed(const at::Tensor& t) {
  constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize});
  return t._fw_grad(0).defined() || t.key_set().has_any(wrapped) || torch::jit::tracer::isTracing();
}

// A dense fp32 CUDA activation in channels-last memory order, 16-byte aligned.
const at::Tensor* activation(PyObject* o) {
  const at::Tensor* t = tensor_of(o);
  return t && !observed(*t) && t->is_cuda() && t->scalar_type() == at::kFloat && t->dim() == 4 && t->numel() > 0 && t->is_contiguous(at::MemoryFormat::ChannelsLast) &&
                 ((uintptr_t)t->data_ptr() & 15u) == 0
             ? t
             : nullptr;
}
// Per-channel parameters: c floats on x's device.
const float* channels(PyObject* o, const at::Tensor& x, int64_t c) {
  const at::Tensor* t = plain(o, at::kFloat);
  return t && t->numel() == c && t->device() == x.device() && ((uintptr_t)t->data_ptr() & 15u) == 0 ? (const float*)t->data_ptr() : nullptr;
}
at::Tensor like_activation(const at::Tensor& x, int64_t n, int64_t c, int64_t h, int64_t w) {
  return at::empty({n, c, h, w}, x.options(), at::MemoryFormat::ChannelsLast);
}

// conv_bn_eval(x, w, cbias or None, gamma, beta, mean, var, eps, residual or None, relu, stride, pad, pool, error flag (address)) -> y
PyObject* conv_bn_eval(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 14, "conv_bn_eval")) return nullptr;
  const at::Tensor *x = activation(a[0]), *w = tensor_of(a[1]), *res = a[8] == Py_None ? nullptr : activation(a[8]);
  if (!x || !w || (a[8] != Py_None && !res)) Py_RETURN_NONE;
  if (!w->is_cuda() || w->scalar_type() != at::kFloat || w->dim() != 4 || w->device() != x->device() || w->size(1) != x->size(1) || w->size(2) != w->size(3) ||
      ((uintptr_t)w->data_ptr() & 15u))
    Py_RETURN_NONE;
  const int64_t n = x->size(0), cin = x->size(1), h = x->size(2), wd = x->size(3), cout = w->size(0), r = w->size(2);
  if (!(w->is_contiguous(at::MemoryFormat::ChannelsLast) || (r == 1 && w->is_contiguous()))) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(a[7]);
  const int relu = PyObject_IsTrue(a[9]), stride = (int)as_int(a[10]), pad = (int)as_int(a[11]), pool = PyObject_IsTrue(a[12]);
  int* flag = (int*)PyLong_AsUnsignedLongLong(a[13]);
  if (PyErr_Occurred()) return nullptr;
  const float *cbias = a[2] == Py_None ? nullptr : channels(a[2], *x, cout), *gamma = channels(a[3], *x, cout), *beta = channels(a[4], *x, cout),
              *mean = channels(a[5], *x, cout), *var = channels(a[6], *x, cout);
  if ((a[2] != Py_None && !cbias) || !gamma || !beta || !mean || !var || stride < 1 || n > INT32_MAX || n * h * wd > INT32_MAX) Py_RETURN_NONE;
  const int64_t ho = (h + 2 * pad - r) / stride + 1, wo = (wd + 2 * pad - r) / stride + 1;
  if (ho < 1 || wo < 1 || h + 2 * pad < r || wd + 2 * pad < r || !api.bn_supported(n * ho * wo, (int)cout)) Py_RETURN_NONE;
  if (res && (res->device() != x->device() || res->size(0) != n || res->size(1) != cout || res->size(2) != ho || res->size(3) != wo)) Py_RETURN_NONE;
  if (pool && (res || ((ho | wo) & 1))) Py_RETURN_NONE;
  const int64_t floats = api.conv_bn_eval_scratch((int)n, (int)h, (int)wd, (int)cin, (int)cout, (int)r, stride, pad);
  if (floats < 0) Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(x->device());
  at::Tensor y, pooled;
  const char* what = "conv_bn_eval";
  const int err = unlocked([&] {
    y = like_activation(*x, n, cout, ho, wo);
    at::Tensor scratch;
    if (floats) scratch = at::empty({floats}, x->options());
    void* st = stream_on(x->device().index());
    const int e = api.conv_bn_eval((const float*)x->data_ptr(), (const float*)w->data_ptr(), (float*)y.data_ptr(), cbias, (int)n, (int)h, (int)wd, (int)cin,
                                   (int)cout, (int)r, stride, pad, gamma, beta, mean, var, (float)eps, res ? (const float*)res->data_ptr() : nullptr, relu,
                                   floats ? (float*)scratch.data_ptr() : nullptr, flag, st);
    if (e || !pool) return e;
    what = "max_pool2";
    pooled = like_activation(*x, n, cout, ho / 2, wo / 2);
    return api.max_pool2((const float*)y.data_ptr(), (int)n, (int)ho, (int)wo, (int)cout, (float*)pooled.data_ptr(), st);
  });
  if (err) return cuda_error(what, err);
  return THPVariable_Wrap(pool ? pooled : y);
}

// classify(feature map, weight, bias or None) -> logits of the mean over the map, or None
PyObject* classify(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 3, "classify")) return nullptr;
  const at::Tensor *x = activation(a[0]), *w = tensor_of(a[1]);
  if (!x || !w || !w->is_cuda() || w->scalar_type() != at::kFloat || w->dim() != 2 || !w->is_contiguous() || w->device() != x->device() ||
      w->size(1) != x->size(1) || ((uintptr_t)w->data_ptr() | (uintptr_t)x->data_ptr()) & 15u)
    Py_RETURN_NONE;
  const int64_t n = x->size(0), c = x->size(1), positions = x->size(2) * x->size(3), k = w->size(0);
  const float* bias = a[2] == Py_None ? nullptr : channels(a[2], *x, k);
  if ((a[2] != Py_None && !bias) || n < 1 || n > INT32_MAX || c < 4 || c & 3 || c > 4096 || positions < 1 || positions > INT32_MAX || k < 1 || k > 32)
    Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(x->device());
  at::Tensor logits;
  const int err = unlocked([&] {
    logits = at::empty({n, k}, x->options().memory_format(at::MemoryFormat::Contiguous));
    return api.head_eval((const float*)x->data_ptr(), (int)n, (int)positions, (int)c, (const float*)w->data_ptr(), bias, (int)k, (float*)logits.data_ptr(),
                         stream_on(x->device().index()));
  });
  if (err) return cuda_error("classify", err);
  return THPVariable_Wrap(logits);
}

// logit_metrics(logits, labels) -> (cross-entropy, top-1 rate, top-5 rate), or None
PyObject* logit_metrics(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 2, "logit_metrics")) return nullptr;
  const at::Tensor *z = tensor_of(a[0]), *y = tensor_of(a[1]);
  if (!z || !y || observed(*z) || !z->is_cuda() || z->scalar_type() != at::kFloat || z->dim() != 2 || !z->is_contiguous() || y->scalar_type() != at::kLong ||
      y->dim() != 1 || !y->is_contiguous() || y->device() != z->device() || y->size(0) != z->size(0))
    Py_RETURN_NONE;
  // what the kernel computes (top-5 needs five classes, as torch.topk does); where it is the faster way is the caller's rule
  const int64_t n = z->size(0), k = z->size(1);
  if (n < 1 || n > (1 << 18) || k < 5 || k > 1024 || n * k > (1 << 22)) Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(z->device());
  at::Tensor out;
  const int err = unlocked([&] {
    out = at::empty({3}, z->options());
    return api.logit_metrics((const float*)z->data_ptr(), (const int64_t*)y->data_ptr(), (int)n, (int)k, (float*)out.data_ptr(), stream_on(z->device().index()));
  });
  if (err) return cuda_error("logit_metrics", err);
  PyObject* t = PyTuple_New(3);
  for (int i = 0; t && i < 3; ++i) PyTuple_SET_ITEM(t, i, THPVariable_Wrap(out.select(0, i)));
  return t;
}

// bn_eval(x, gamma, beta, mean, var, eps, residual or None, relu) -> y
PyObject* bn_eval(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (!want(nargs, 8, "bn_eval")) return nullptr;
  const at::Tensor *x = activation(a[0]), *res = a[6] == Py_None ? nullptr : activation(a[6]);
  if (!x || (a[6] != Py_None && (!res || res->sizes() != x->sizes() || res->device() != x->device()))) Py_RETURN_NONE;
  const int64_t c = x->size(1), m = x->numel() / c;
  const float *gamma = channels(a[1], *x, c), *beta = channels(a[2], *x, c), *mean = channels(a[3], *x, c), *var = channels(a[4], *x, c);
  const double eps = PyFloat_AsDouble(a[5]);
  const int relu = PyObject_IsTrue(a[7]);
  if (PyErr_Occurred()) return nullptr;
  if (!gamma || !beta || !mean || !var || !api.bn_supported(m, (int)c)) Py_RETURN_NONE;
  c10::cuda::OptionalCUDAGuard guard(x->device());
  at::Tensor y;
  const int err = unlocked([&] {
    y = like_activation(*x, x->size(0), c, x->size(2), x->size(3));
    return api.bn_eval_apply((const float*)x->data_ptr(), m, (int)c, mean, var, (float)eps, gamma, beta, res ? (const float*)res->data_ptr() : nullptr, relu,
                             (float*)y.data_ptr(), stream_on(x->device().index()));
  });
  if (err) return cuda_error("bn_eval", err);
  return THPVariable_Wrap(y);
}

// bind({name: address}): the kernel library's entry points
PyObject* bind(PyObject*, PyObject* table) {
  for (const Entry& e : entries) {
    PyObject* v = PyDict_GetItemString(table, e.name);
    if (!v) { PyErr_Format(PyExc_KeyError, "%s", e.name); return nullptr; }
    *e.slot = (void*)PyLong_AsUnsignedLongLong(v);
    if (PyErr_Occurred()) return nullptr;
  }
  max_segs = api.solo_max_segs();
  Py_RETURN_NONE;
}

PyObject* names(PyObject*, PyObject*) {
  PyObject* l = PyList_New(0);
  for (const Entry& e : entries) {
    PyObject* s = PyUnicode_FromString(e.name);
    PyList_Append(l, s);
    Py_DECREF(s);
  }
  return l;
}

PyMethodDef methods[] = {
    {"bind", bind, METH_O, "bind(table): addresses of the kernel library's entry points by name"},
    {"names", names, METH_NOARGS, "names() -> the entry points bind() needs"},
    {"plan_new", plan_new, METH_NOARGS, "plan_new() -> a plan, one per reducer"},
    {"solo_maxnorm", method<solo_maxnorm>(), METH_FASTCALL, "QSGD-MaxNorm reduce of a single worker"},
    {"solo_copy", method<solo_copy>(), METH_FASTCALL, "plain mean of a single worker"},
    {"collect", method<collect_py>(), METH_FASTCALL, "reads two lists of tensors into a plan"},
    {"solo_randk", method<solo_randk>(), METH_FASTCALL, "Rand-K reduce of a single worker"},
    {"solo_randk_limit", method<solo_randk_limit>(), METH_FASTCALL, "most coordinates solo_randk takes"},
    {"solo_psgd", method<solo_psgd>(), METH_FASTCALL, "PowerSGD step of a single worker"},
    {"solo_topk", method<solo_topk>(), METH_FASTCALL, "top-k with error feedback of a single worker"},
    {"conv_bn_eval", method<conv_bn_eval>(), METH_FASTCALL, "convolution, batch norm of running statistics, residual, ReLU, pool"},
    {"bn_eval", method<bn_eval>(), METH_FASTCALL, "batch norm of running statistics, residual, ReLU"},
    {"absmax", method<absmax>(), METH_FASTCALL, "largest magnitude"},
    {"classify", method<classify>(), METH_FASTCALL, "logits of a feature map in inference"},
    {"logit_metrics", method<logit_metrics>(), METH_FASTCALL, "cross-entropy, top-1 and top-5 of logits"},
    {"quantize", method<quantize>(), METH_FASTCALL, "levels of a vector"},
    {"quantize_fit", method<quantize_fit>(), METH_FASTCALL, "levels of the higher scale and where they fit the lower one"},
    {"dequantize", method<dequantize>(), METH_FASTCALL, "values of levels of one or two scales"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "gcb200_ext", "native front end of the reducers", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_gcb200_ext() { return PyModule_Create(&module); }
