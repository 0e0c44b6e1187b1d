// The host side of a call in native code: arguments out of Python objects, checks, outputs, the launch.  The same work
// in Python (a ctypes structure of 45 fields, a dozen tensor attribute reads, two allocations) took 20 to 40 us per call,
// as long as the kernels of a decode step or longer; here it is 3 to 5 us.  Everything reaches the GPU through the C ABI
// of jpt_b200.h.  Loaded as jetstream_pytorch_b200._native.
#include <Python.h>

#include <ATen/Context.h>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <optional>
#include <string>
#include <vector>

#include "jpt_b200.h"

namespace {

using at::Tensor;
using c10::ScalarType;

// A Python exception of `type` is raised when this reaches the entry points below.
struct PyFail {
  PyObject* type;
  std::string text;
};
[[noreturn]] void fail(PyObject* type, const char* fmt, ...) {
  char buf[640];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  throw PyFail{type, buf};
}
struct PySet {};  // the Python error is already set

void check(int rc) {
  if (rc == 0) return;
  if (rc < 0) fail(PyExc_ValueError, "libjpt_b200 argument error %d: %s", rc, jpt_last_error_string());
  fail(PyExc_RuntimeError, "libjpt_b200 CUDA error %d: %s", rc, jpt_last_error_string());
}

// ---------------------------------------------------------------- arguments
const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "expected a tensor, got %s", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
const Tensor* maybe(PyObject* o) { return o == Py_None ? nullptr : &tensor(o); }
long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PySet{};
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PySet{};
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PySet{};
  return v != 0;
}
void* ptr(const Tensor& t) {
  if (!t.is_cuda()) fail(PyExc_ValueError, "libjpt_b200 works on CUDA tensors only; got a tensor on %s", t.device().str().c_str());
  return t.data_ptr();
}
void* ptr(const Tensor* t) { return t ? ptr(*t) : nullptr; }
int dtype_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case ScalarType::BFloat16: return JPT_BF16;
    case ScalarType::Float: return JPT_F32;
    case ScalarType::Char: return JPT_INT8;
    default: fail(PyExc_ValueError, "unsupported dtype %s", c10::toString(t.scalar_type()));
  }
}
// (int32, contiguous, on `dev`: what the kernels read positions, lengths and tables as)
Tensor as_i32(const Tensor& t, c10::Device dev) {
  Tensor r = t;
  if (r.device() != dev) r = r.to(dev, /*non_blocking=*/true);
  if (r.scalar_type() != ScalarType::Int) r = r.to(ScalarType::Int);
  return r.contiguous();
}
Tensor dense(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
Tensor empty(at::IntArrayRef sizes, ScalarType type, c10::Device dev) {
  if (!dev.is_cuda()) fail(PyExc_ValueError, "libjpt_b200 works on CUDA tensors only; got a tensor on %s", dev.str().c_str());
  return Tensor(at::detail::empty_cuda(sizes, type, dev, std::nullopt));
}
cudaStream_t stream_of(c10::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
// Launches go to the current device's stream and kernel attributes are per device.
struct OnDevice {
  std::optional<c10::cuda::CUDAGuard> guard;
  explicit OnDevice(c10::Device dev) {
    if (dev.is_cuda() && dev.index() != c10::cuda::current_device()) guard.emplace(dev);
  }
};

PyObject* wrap(const Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None); }
template <typename... Ts>
PyObject* tuple(const Ts&... ts) {
  PyObject* r = PyTuple_New(sizeof...(ts));
  if (!r) throw PySet{};
  Py_ssize_t i = 0;
  (PyTuple_SET_ITEM(r, i++, wrap(ts)), ...);
  return r;
}

// ---------------------------------------------------------------- attention workspaces
// Grow-only attention scratch, one per stream (two launches that share one must not overlap) and one more per device for
// CUDA graph captures, which run on a stream of their own and must not allocate: every eager call keeps that one at
// least as large as its own.  Cleared once when created, as the kernels' arrival counters require.  A graph holds the address
// of the scratch that it was captured with, so one that a capture has been given stays allocated when a larger one takes
// its place; each is at least twice as large as the one before, so that all retired ones together are smaller than it.
struct Workspace {
  c10::DeviceIndex device;
  bool graph;
  cudaStream_t stream;
  Tensor mem;
  bool captured = false, retired = false;  // (graph)
};
std::vector<Workspace>& workspaces() {
  static auto* list = new std::vector<Workspace>();  // (never destroyed: the CUDA context may be gone by then)
  return *list;
}
Workspace* find_workspace(c10::Device dev, cudaStream_t st, bool graph) {
  for (Workspace& e : workspaces())
    if (e.device == dev.index() && e.graph == graph && !e.retired && (graph || e.stream == st)) return &e;
  return nullptr;
}
Workspace& grown_workspace(c10::Device dev, cudaStream_t st, bool graph, size_t bytes) {
  Workspace* w = find_workspace(dev, st, graph);
  if (w && (size_t)w->mem.numel() >= bytes) return *w;
  size_t size = std::max<size_t>(bytes, 8u << 20);
  if (w && w->captured) size = std::max<size_t>(size, 2 * (size_t)w->mem.numel());
  Tensor mem = empty({(int64_t)size}, ScalarType::Byte, dev);
  check(jpt_flash_decode_workspace_init(mem.data_ptr(), (size_t)mem.numel(), st));
  if (w && !w->captured) {
    w->mem = mem;
    return *w;
  }
  if (w) w->retired = true;
  workspaces().push_back({dev.index(), graph, st, mem});
  return workspaces().back();
}
bool is_capturing(cudaStream_t st) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &capturing) == cudaSuccess && capturing != cudaStreamCaptureStatusNone;
}
Tensor workspace(c10::Device dev, cudaStream_t st, size_t bytes) {
  if (!is_capturing(st)) {
    Tensor own = grown_workspace(dev, st, false, bytes).mem;
    grown_workspace(dev, st, true, bytes);
    return own;
  }
  Workspace* w = find_workspace(dev, st, true);
  if (!w || (size_t)w->mem.numel() < bytes)
    fail(PyExc_RuntimeError,
         "the attention workspace for CUDA graphs is too small and cannot grow during capture; call the same shape once before "
         "capturing");
  w->captured = true;
  return w->mem;
}

// ---------------------------------------------------------------- attention
struct Call {  // one attention call; tensors are kept alive until the launch is enqueued
  Tensor q, k, v, ks, vs, start, end, mask, table;
  int mask_mode = JPT_MASK_NONE;
  int64_t kv_b = 0, kv_h = 0, kv_s = 0, sc_b = 0, sc_s = 0, mk_b = 0, mk_r = 0;
  int64_t k_off = 0, sc_off = 0;  // elements from the tensors' start to the selected layer
  int64_t hkv = 0, seq = 0, page_size = 0;
  bool paged = false, want_ml = true, rounding = false, static_scratch = false;
  int num_splits = 0, force_generic = 0;
  double sm_scale = 1.0;
  jpt_new_token* nt = nullptr;
  bool out_f32 = false;  // (with nt)
  Tensor o, m, l;        // outputs; made here when not given
  bool out_given = false;
};

void* offset(const Tensor& t, int64_t elements) {
  return t.defined() ? static_cast<char*>(ptr(t)) + elements * (int64_t)t.element_size() : nullptr;
}

void run_attention(Call& c, at::IntArrayRef out_shape, at::IntArrayRef ml_shape) {
  const c10::Device dev = c.q.device();
  OnDevice on(dev);
  // (a transposed view of a prompt's projection stays as it is where the prefill kernel takes its strides)
  bool strided = c.q.size(2) > 1 && c.q.size(3) == 128 && !c.q.is_contiguous() && c.q.stride(3) == 1;
  if (!strided) c.q = dense(c.q);
  for (const Tensor* t : {&c.k, &c.v, &c.ks, &c.vs, &c.mask})
    if (t->defined() && t->device() != dev)
      fail(PyExc_ValueError, "attention operands live on %s and %s", t->device().str().c_str(), dev.str().c_str());
  const int64_t b = c.q.size(0), hq = c.q.size(1), tq = c.q.size(2), d = c.q.size(3);
  jpt_attn_params p{};
  p.q = ptr(c.q);
  p.q_dtype = dtype_of(c.q);
  p.B = (int)b, p.Hq = (int)hq, p.Hkv = (int)c.hkv, p.Tq = (int)tq, p.D = (int)d;
  p.k = offset(c.k, c.k_off), p.v = offset(c.v, c.k_off), p.kv_dtype = dtype_of(c.k);
  p.paged = c.paged;
  if (c.paged) {
    c.table = as_i32(c.table, dev);
    p.page_table = static_cast<const int32_t*>(ptr(c.table));
    p.max_pages = (int)c.table.size(1);
    p.page_size = (int)c.page_size;
    p.S = (int)(c.table.size(1) * c.page_size);
    p.kv_h = c.k.stride(0), p.kv_page = c.k.stride(1);
  } else {
    p.S = (int)c.seq;
    p.kv_b = c.kv_b, p.kv_h = c.kv_h, p.kv_s = c.kv_s;
  }
  if (c.ks.defined()) {
    if (c.ks.scalar_type() != c.vs.scalar_type()) fail(PyExc_ValueError, "k and v scales must share a dtype");
    p.k_scale = offset(c.ks, c.sc_off), p.v_scale = offset(c.vs, c.sc_off), p.scale_dtype = dtype_of(c.ks);
    p.sc_b = c.sc_b, p.sc_s = c.sc_s;
  }
  p.mask_mode = c.mask_mode;
  if (c.start.defined()) {
    c.start = as_i32(c.start, dev);
    p.start = static_cast<const int32_t*>(ptr(c.start));
  }
  if (c.end.defined()) {
    c.end = as_i32(c.end, dev);
    p.end = static_cast<const int32_t*>(ptr(c.end));
  }
  if (c.mask.defined()) {
    p.mask = ptr(c.mask);
    p.mk_b = c.mk_b, p.mk_r = c.mk_r;
  }
  p.sm_scale = (float)c.sm_scale;
  if (c.out_given) {
    if (c.o.sizes() != c.q.sizes() || c.o.scalar_type() != c.q.scalar_type() || c.o.device() != dev || !c.o.is_contiguous())
      fail(PyExc_ValueError, "out[0] must be a contiguous tensor of the query's shape, dtype and device");
    for (const Tensor* t : {&c.m, &c.l})
      if (t->defined() && (t->numel() != b * hq * tq || t->scalar_type() != ScalarType::Float || t->device() != dev || !t->is_contiguous()))
        fail(PyExc_ValueError, "out[1], out[2] must be contiguous float32 tensors of B*Hq*Tq elements");
    p.o = ptr(c.o);
    if (c.m.defined() && c.l.defined()) p.m = static_cast<float*>(ptr(c.m)), p.l = static_cast<float*>(ptr(c.l));
  } else {
    c.o = empty(out_shape, c.out_f32 ? ScalarType::Float : c.q.scalar_type(), dev);
    p.o = c.o.data_ptr();
    if (c.want_ml) {
      c.m = empty(ml_shape, ScalarType::Float, dev);
      c.l = empty(ml_shape, ScalarType::Float, dev);
      p.m = static_cast<float*>(c.m.data_ptr()), p.l = static_cast<float*>(c.l.data_ptr());
    }
  }
  p.num_splits = c.num_splits, p.force_generic = c.force_generic, p.logit_rounding = c.rounding;
  if (strided && (c.static_scratch || c.nt || !jpt_flash_attend_strided_q_ok(&p, c.q.stride(0), c.q.stride(1), c.q.stride(2)))) {
    c.q = c.q.contiguous();
    strided = false;
    p.q = ptr(c.q);
  }
  const cudaStream_t st = stream_of(dev);
  if (c.static_scratch) {
    if (c.nt) fail(PyExc_ValueError, "the fused update needs a workspace that keeps its contents between calls");
    check(jpt_flash_decode_static(&p, st));
    return;
  }
  Tensor ws;
  if (const size_t need = jpt_flash_decode_workspace_bytes(&p)) {
    if (!c.nt && is_capturing(st)) {
      // A prompt captured before anything ran: the prefill kernel wants only a status word and its table of mask classes, which the
      // scratch built into the library has (the scalar kernel that took such calls before mostly needed none).
      const Workspace* w = find_workspace(dev, st, true);
      if ((!w || (size_t)w->mem.numel() < need) && jpt_flash_attend_strided_q_ok(&p, hq * tq * d, tq * d, d)) {
        c.q = dense(c.q);
        p.q = ptr(c.q);
        check(jpt_flash_decode_static(&p, st));
        return;
      }
    }
    ws = workspace(dev, st, need);
    p.workspace = ws.data_ptr(), p.workspace_bytes = (size_t)ws.numel();
  }
  if (strided)
    check(jpt_flash_attend_strided_q(&p, c.q.stride(0), c.q.stride(1), c.q.stride(2), st));
  else if (c.nt)
    check(jpt_decode_update_attend_out(&p, c.nt, c.out_f32 ? JPT_F32 : JPT_BF16, st));
  else
    check(jpt_flash_decode(&p, st));
}

int64_t layer_index(int64_t layer, int64_t n) {
  const int64_t i = layer < 0 ? layer + n : layer;
  if (i < 0 || i >= n) fail(PyExc_IndexError, "layer %lld of a cache of %lld layers", (long long)layer, (long long)n);
  return i;
}
// Dense K/V [B,H,S,D] or one layer of [NL,B,H,S,D].
void take_kv(Call& c, const Tensor& k, const Tensor& v, int64_t layer) {
  c.k = k, c.v = v;
  if (k.stride(-1) != 1 || v.strides() != k.strides()) {
    if (k.dim() == 5) {
      c.k = k.select(0, layer), c.v = v.select(0, layer);
      c.k = c.k.contiguous(), c.v = c.v.contiguous();
    } else {
      c.k = k.contiguous(), c.v = v.contiguous();
    }
  }
  const int64_t o = c.k.dim() - 4;
  if (o == 1) c.k_off = layer_index(layer, c.k.size(0)) * c.k.stride(0);
  c.kv_b = c.k.stride(o), c.kv_h = c.k.stride(o + 1), c.kv_s = c.k.stride(o + 2);
  c.hkv = c.k.size(o + 1), c.seq = c.k.size(o + 2);
  if (c.hkv < 1) fail(PyExc_ValueError, "a cache without KV heads");
}
// Scales [B,1,S,1] or [B,1,S]; stacked: a leading NL.
void take_scales(Call& c, const Tensor* ks, const Tensor* vs, int64_t layer) {
  if (!ks) return;
  if (!vs) fail(PyExc_ValueError, "k and v scales come together");
  c.ks = *ks, c.vs = *vs;
  const bool stacked = ks->dim() == 5 || (ks->dim() == 4 && ks->size(3) != 1);
  if (vs->strides() != ks->strides()) {
    if (stacked) c.ks = ks->select(0, layer), c.vs = vs->select(0, layer);
    c.ks = c.ks.contiguous(), c.vs = c.vs.contiguous();
    c.sc_b = c.ks.stride(0), c.sc_s = c.ks.stride(2);
    return;
  }
  const int64_t o = stacked ? 1 : 0;
  if (stacked) c.sc_off = layer_index(layer, ks->size(0)) * ks->stride(0);
  c.sc_b = ks->stride(o), c.sc_s = ks->stride(o + 2);
}
// Additive mask [B|1, 1, R|1, S] with R = rep * Tq: what broadcasts against the grouped scores.
void take_mask(Call& c, const Tensor* mask) {
  if (!mask) return;
  const int64_t b = c.q.size(0), rows = c.q.size(1) / c.hkv * c.q.size(2);
  if (mask->dim() != 4 || mask->size(1) != 1 || mask->size(3) != c.seq)
    fail(PyExc_ValueError, "mask must be [B|1, 1, R|1, S] with S = %lld", (long long)c.seq);
  if ((mask->size(0) != 1 && mask->size(0) != b) || (mask->size(2) != 1 && mask->size(2) != rows))
    fail(PyExc_ValueError, "mask [%lld, 1, %lld, %lld] does not broadcast against scores [%lld, %lld, %lld, %lld]",
         (long long)mask->size(0), (long long)mask->size(2), (long long)mask->size(3), (long long)b, (long long)c.hkv, (long long)rows,
         (long long)c.seq);
  c.mask = *mask;
  if (c.mask.scalar_type() != c.q.scalar_type()) c.mask = c.mask.to(c.q.scalar_type());
  if (c.mask.stride(3) != 1) c.mask = c.mask.contiguous();
  c.mask_mode = JPT_MASK_ADD;
  c.mk_b = c.mask.size(0) > 1 ? c.mask.stride(0) : 0;
  c.mk_r = c.mask.size(2) > 1 ? c.mask.stride(2) : 0;
}
void take_options(Call& c, PyObject* const* a) {  // num_splits, force_generic, static_scratch, out (o, m, l)
  c.num_splits = (int)integer(a[0]);
  c.force_generic = (int)integer(a[1]);
  c.static_scratch = truth(a[2]);
  if (a[3] != Py_None) {
    if (!PyTuple_Check(a[3]) || PyTuple_GET_SIZE(a[3]) != 3) fail(PyExc_ValueError, "out is a tuple (o, m, l)");
    c.out_given = true;
    c.o = tensor(PyTuple_GET_ITEM(a[3], 0));
    if (const Tensor* m = maybe(PyTuple_GET_ITEM(a[3], 1))) c.m = *m;
    if (const Tensor* l = maybe(PyTuple_GET_ITEM(a[3], 2))) c.l = *l;
  }
}

using Args = PyObject* const*;
void expect(Py_ssize_t n, Py_ssize_t want, const char* who) {
  if (n != want) fail(PyExc_TypeError, "%s takes %lld arguments, got %lld", who, (long long)want, (long long)n);
}
void head_check(const Tensor& q, const Tensor& k) {
  if (q.dim() != 4) fail(PyExc_ValueError, "queries are [B,Hq,T,D]");
  if (k.dim() != 4 && k.dim() != 5) fail(PyExc_ValueError, "caches are [B,H,S,D] or [NL,B,H,S,D]");
}

// What the kernels of a call over a whole cache take on trust: as many sequences and dims as the queries have, and a scale per token.
void cache_check(const Tensor& q, const Tensor& k) {
  head_check(q, k);
  if (k.size(-1) != q.size(-1) || k.size(-4) != q.size(0)) fail(PyExc_AssertionError, "queries and cache differ in batch or head_dim");
}
void scale_check(const Call& c) {
  if (!c.ks.defined()) return;
  const int64_t o = c.sc_off || c.ks.dim() == 5 || (c.ks.dim() == 4 && c.ks.size(3) != 1) ? 1 : 0;
  if (c.ks.size(o) != c.q.size(0) || c.ks.size(o + 2) != c.seq) fail(PyExc_AssertionError, "scales do not match the cache");
}
// ... and of a step's token: one per sequence and KV head, on the queries' GPU.
void token_check(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& xk, const Tensor& xv) {
  cache_check(q, k);
  if (v.sizes() != k.sizes()) fail(PyExc_ValueError, "K and V caches differ in shape");
  if (q.size(2) != 1) fail(PyExc_ValueError, "a step has one query token, got %lld", (long long)q.size(2));
  const int64_t want[4] = {q.size(0), k.size(-3), 1, q.size(3)};
  for (const Tensor* x : {&xk, &xv})
    if (x->sizes() != at::IntArrayRef(want, 4) || x->device() != q.device())
      fail(PyExc_ValueError, "the step's token must be [%lld, %lld, 1, %lld] on %s", (long long)want[0], (long long)want[1],
           (long long)want[3], q.device().str().c_str());
}

// attend(q, k, v, k_scale, v_scale, page_table, start, end, mask, mask_mode, kv strides (b, h, s), scale strides (b, s), mask
// strides (b, r), hkv, seq, page_size, sm_scale, want_ml, rounding, num_splits, force_generic, static_scratch, out)
PyObject* attend(Args a, Py_ssize_t n) {
  expect(n, 27, "attend");
  Call c;
  c.q = tensor(a[0]), c.k = tensor(a[1]), c.v = tensor(a[2]);
  if (auto t = maybe(a[3])) c.ks = *t;
  if (auto t = maybe(a[4])) c.vs = *t;
  if (c.ks.defined() != c.vs.defined()) fail(PyExc_ValueError, "k and v scales come together");
  if (auto t = maybe(a[5])) c.table = *t, c.paged = true;
  if (auto t = maybe(a[6])) c.start = *t;
  if (auto t = maybe(a[7])) c.end = *t;
  if (auto t = maybe(a[8])) c.mask = *t;
  c.mask_mode = (int)integer(a[9]);
  c.kv_b = integer(a[10]), c.kv_h = integer(a[11]), c.kv_s = integer(a[12]);
  c.sc_b = integer(a[13]), c.sc_s = integer(a[14]);
  c.mk_b = integer(a[15]), c.mk_r = integer(a[16]);
  c.hkv = integer(a[17]), c.seq = integer(a[18]), c.page_size = integer(a[19]);
  c.sm_scale = real(a[20]);
  c.want_ml = truth(a[21]), c.rounding = truth(a[22]);
  take_options(c, a + 23);
  const Tensor q = c.q;
  run_attention(c, q.sizes(), {q.size(0), q.size(1), q.size(2)});
  return tuple(c.o, c.m, c.l);
}

// ragged(q, k, v, layer, start, end, k_scaler, v_scaler, normalize, ring) -> o [B,Hkv,rep T,D], m, l [B,Hkv,rep T]
PyObject* ragged(Args a, Py_ssize_t n) {
  expect(n, 10, "ragged");
  Call c;
  c.q = tensor(a[0]);
  const Tensor &k = tensor(a[1]), &v = tensor(a[2]);
  cache_check(c.q, k);
  const int64_t layer = integer(a[3]);
  const bool ring = truth(a[9]);
  take_kv(c, k, v, layer);
  take_scales(c, maybe(a[6]), maybe(a[7]), layer);
  scale_check(c);
  if (ring) c.start = tensor(a[4]);
  c.end = tensor(a[5]);
  c.mask_mode = ring ? JPT_MASK_RING : JPT_MASK_LENGTH;
  const int64_t b = c.q.size(0), d = c.q.size(3), rt = c.q.size(1) / c.hkv * c.q.size(2);
  c.sm_scale = truth(a[8]) ? 1.0 / std::sqrt((double)d) : 1.0;
  run_attention(c, {b, c.hkv, rt, d}, {b, c.hkv, rt});
  return tuple(c.o, c.m, c.l);
}

// dense(q, k, v, k_scaler, v_scaler, mask) -> o [B,Hq,T,D]
PyObject* dense_attention(Args a, Py_ssize_t n) {
  expect(n, 6, "dense");
  Call c;
  c.q = tensor(a[0]);
  const Tensor &k = tensor(a[1]), &v = tensor(a[2]);
  head_check(c.q, k);
  take_kv(c, k, v, 0);
  take_scales(c, maybe(a[3]), maybe(a[4]), 0);
  take_mask(c, maybe(a[5]));
  c.sm_scale = 1.0 / std::sqrt((double)c.q.size(3));
  // The reference computes the logits of this function as bf16 tensor operations when its inputs are bf16 (matmul,
  // / sqrt(D), * k_scaler, + mask: four roundings); the kernels reproduce those roundings.
  c.rounding = c.q.scalar_type() == ScalarType::BFloat16;
  c.want_ml = false;
  const Tensor q = c.q;
  run_attention(c, q.sizes(), {});
  return wrap(c.o);
}

// flash(q, k, v, layer, k_scaler, v_scaler, mask, normalize) -> o [B,Hq,T,D], m, l [B,Hq,T,1]
PyObject* flash(Args a, Py_ssize_t n) {
  expect(n, 8, "flash");
  Call c;
  c.q = tensor(a[0]);
  const Tensor &k = tensor(a[1]), &v = tensor(a[2]);
  head_check(c.q, k);
  const int64_t layer = integer(a[3]);
  take_kv(c, k, v, layer);
  take_scales(c, maybe(a[4]), maybe(a[5]), layer);
  take_mask(c, maybe(a[6]));
  c.sm_scale = truth(a[7]) ? 1.0 / std::sqrt((double)c.k.size(-1)) : 1.0;
  const Tensor q = c.q;
  run_attention(c, q.sizes(), {q.size(0), q.size(1), q.size(2), 1});
  return tuple(c.o, c.m, c.l);
}

// paged(q [B,Hq,D], k, v, lengths, page_table, sm_scale, k_scaler, v_scaler) -> o [B,Hq,D]
PyObject* paged(Args a, Py_ssize_t n) {
  expect(n, 8, "paged");
  Call c;
  const Tensor& q = tensor(a[0]);
  if (q.dim() != 3) fail(PyExc_ValueError, "paged attention takes queries [B,Hq,D]");
  c.q = q.unsqueeze(2);
  c.k = tensor(a[1]), c.v = tensor(a[2]);
  if (c.k.dim() != 4) fail(PyExc_ValueError, "page pools are [H,P,page,D]");
  c.end = tensor(a[3]), c.table = tensor(a[4]);
  c.paged = true;
  c.hkv = c.k.size(0), c.page_size = c.k.size(2);
  if (c.hkv < 1) fail(PyExc_ValueError, "page pools without KV heads");
  c.sm_scale = real(a[5]);
  if (auto t = maybe(a[6])) c.ks = *t, c.vs = tensor(a[7]);
  c.mask_mode = JPT_MASK_LENGTH;
  c.want_ml = false;
  run_attention(c, q.sizes(), {});
  return wrap(c.o);
}

// ---------------------------------------------------------------- cache updates
struct Positions {  // of a step: a shared host value, or a device array of one or B entries
  Tensor t;
  const int32_t* dev = nullptr;
  int count = 1, host = 0;
};
Positions positions(PyObject* o, c10::Device dev, int64_t batch) {
  Positions p;
  if (PyLong_Check(o)) {
    p.host = (int)integer(o);
    return p;
  }
  p.t = as_i32(tensor(o), dev).reshape({-1});
  p.count = (int)p.t.numel();
  if (p.count != 1 && p.count != batch) fail(PyExc_ValueError, "input_pos has %d entries, expected 1 or %lld", p.count, (long long)batch);
  p.dev = static_cast<const int32_t*>(ptr(p.t));
  return p;
}
struct CacheRef {  // one layer of an int8 cache with its scalers
  int8_t *k = nullptr, *v = nullptr;
  void *ks = nullptr, *vs = nullptr;
  int64_t b = 0, h = 0, s = 0, sb = 0, ss = 0, len = 1;
};
CacheRef cache_ref(const Tensor& k, const Tensor& v, const Tensor& ks, const Tensor& vs, int64_t layer) {
  if (k.stride(-1) != 1) fail(PyExc_ValueError, "cache head_dim axis must be contiguous");
  CacheRef r;
  const int64_t o = k.dim() - 4;
  const int64_t ko = o ? layer_index(layer, k.size(0)) * k.stride(0) : 0, so = o ? layer * ks.stride(0) : 0;
  r.k = static_cast<int8_t*>(offset(k, ko)), r.v = static_cast<int8_t*>(offset(v, ko));
  r.ks = offset(ks, so), r.vs = offset(vs, so);
  r.b = k.stride(o), r.h = k.stride(o + 1), r.s = k.stride(o + 2), r.len = k.size(o + 2);
  r.sb = ks.stride(o), r.ss = ks.stride(o + 2);
  return r;
}
struct Stash {  // where the quantised token is kept: four tensors of one step, or a layer of stacked ones
  Tensor kq, vq, ks, vs;
  int64_t q_off = 0, s_off = 0;
};
Stash stash(PyObject* outs, PyObject* layer, int64_t b, int64_t h, int64_t d, ScalarType type, c10::Device dev) {
  Stash s;
  if (outs == Py_None) {
    s.kq = empty({b, h, 1, d}, ScalarType::Char, dev), s.vq = empty({b, h, 1, d}, ScalarType::Char, dev);
    s.ks = empty({b, 1, 1, 1}, type, dev), s.vs = empty({b, 1, 1, 1}, type, dev);
    return s;
  }
  if (!PyTuple_Check(outs) || PyTuple_GET_SIZE(outs) != 4) fail(PyExc_ValueError, "the kept token is four tensors");
  s.kq = tensor(PyTuple_GET_ITEM(outs, 0)), s.vq = tensor(PyTuple_GET_ITEM(outs, 1));
  s.ks = tensor(PyTuple_GET_ITEM(outs, 2)), s.vs = tensor(PyTuple_GET_ITEM(outs, 3));
  if (s.ks.scalar_type() != type || s.vs.scalar_type() != type)  // the kernel writes the scale in the input's dtype
    fail(PyExc_ValueError, "scale buffers of dtype %s cannot take the scales of %s inputs", c10::toString(s.ks.scalar_type()), c10::toString(type));
  if (s.kq.scalar_type() != ScalarType::Char || s.vq.scalar_type() != ScalarType::Char)
    fail(PyExc_ValueError, "the buffers for the quantised new token must be int8");
  const int64_t layers = s.kq.dim() == 5 ? s.kq.size(0) : 1;
  for (const Tensor* t : {&s.kq, &s.vq, &s.ks, &s.vs})
    if (t->numel() != layers * b * (t == &s.kq || t == &s.vq ? h * d : 1) || !t->is_contiguous() || t->device() != dev)
      fail(PyExc_ValueError, "the buffers for the quantised new token must be contiguous, of %lld sequences and %lld heads", (long long)b, (long long)h);
  if (s.kq.dim() == 5) {
    const int64_t l = layer_index(integer(layer), s.kq.size(0));
    s.q_off = l * s.kq.stride(0), s.s_off = l * s.ks.stride(0);
  }
  return s;
}

// quant_append(xk, xv, cache (k, v, k_scaler, v_scaler) or None, layer, outs or None, pos, amax_in, peers address)
//   -> (kq, vq, ks, vs); with stacked outs: the outs themselves
PyObject* quant_append(Args a, Py_ssize_t n) {
  expect(n, 8, "quant_append");
  const Tensor xk = dense(tensor(a[0])), xv = dense(tensor(a[1]));
  if (xk.dim() != 4 || xk.size(2) != 1) fail(PyExc_ValueError, "the decode cache takes one new token per step");
  const c10::Device dev = xk.device();
  OnDevice on(dev);
  const int64_t b = xk.size(0), h = xk.size(1), d = xk.size(3);
  ptr(xk);
  Stash s = stash(a[4], a[3], b, h, d, xk.scalar_type(), dev);
  CacheRef c;
  Positions p;
  if (a[2] != Py_None) {
    const Tensor& ks = tensor(PyTuple_GET_ITEM(a[2], 2));
    if (ks.scalar_type() != xk.scalar_type())
      fail(PyExc_ValueError, "scaler dtype %s differs from the input dtype %s", c10::toString(ks.scalar_type()), c10::toString(xk.scalar_type()));
    c = cache_ref(tensor(PyTuple_GET_ITEM(a[2], 0)), tensor(PyTuple_GET_ITEM(a[2], 1)), ks, tensor(PyTuple_GET_ITEM(a[2], 3)), integer(a[3]));
    p = positions(a[5], dev, b);
  }
  int8_t *kq = static_cast<int8_t*>(offset(s.kq, s.q_off)), *vq = static_cast<int8_t*>(offset(s.vq, s.q_off));
  void *ks = offset(s.ks, s.s_off), *vs = offset(s.vs, s.s_off);
  if (a[7] != Py_None) {
    if (a[6] != Py_None) fail(PyExc_ValueError, "give either the reduced amax or the peer exchange, not both");
    check(jpt_kv_quant_append_dense_peers(ptr(xk), ptr(xv), dtype_of(xk), c.k, c.v, c.ks, c.vs, kq, vq, ks, vs, p.dev, p.count, p.host,
                                          (int)b, (int)h, (int)c.len, (int)d, c.b, c.h, c.s, c.sb, c.ss,
                                          reinterpret_cast<const jpt_peer_exchange*>(integer(a[7])), stream_of(dev)));
  } else {
    check(jpt_kv_quant_append_dense(ptr(xk), ptr(xv), dtype_of(xk), c.k, c.v, c.ks, c.vs, kq, vq, ks, vs, p.dev, p.count, p.host,
                                    (int)b, (int)h, (int)c.len, (int)d, c.b, c.h, c.s, c.sb, c.ss,
                                    static_cast<const float*>(ptr(maybe(a[6]))), nullptr, stream_of(dev)));
  }
  return tuple(s.kq, s.vq, s.ks, s.vs);
}

// update_attend(xq, xk, xv, (k, v, k_scaler, v_scaler), layer, start, end, ring, pos, write_cache, outs or None, out_f32, out or None,
//               peers address or None) -> (kq, vq, ks, vs, o [B,Hkv,rep,D], m, l); with out_f32: o [B,Hq,T,D] fp32, None, None
PyObject* update_attend(Args a, Py_ssize_t n) {
  expect(n, 14, "update_attend");
  Call c;
  c.q = tensor(a[0]);
  const Tensor xk = dense(tensor(a[1])), xv = dense(tensor(a[2]));
  const c10::Device dev = c.q.device();
  OnDevice on(dev);
  const Tensor &k = tensor(PyTuple_GET_ITEM(a[3], 0)), &v = tensor(PyTuple_GET_ITEM(a[3], 1));
  token_check(c.q, k, v, xk, xv);
  const int64_t layer = integer(a[4]);
  take_kv(c, k, v, layer);
  take_scales(c, maybe(PyTuple_GET_ITEM(a[3], 2)), maybe(PyTuple_GET_ITEM(a[3], 3)), layer);
  scale_check(c);
  const bool ring = truth(a[7]);
  if (ring) c.start = tensor(a[5]);
  c.end = tensor(a[6]);
  c.mask_mode = ring ? JPT_MASK_RING : JPT_MASK_LENGTH;
  const int64_t b = c.q.size(0), d = c.q.size(3), rt = c.q.size(1) / c.hkv * c.q.size(2), h = xk.size(1);
  c.sm_scale = 1.0 / std::sqrt((double)d);
  Stash s = stash(a[10], a[4], b, h, d, xk.scalar_type(), dev);
  Positions p = positions(a[8], dev, b);
  jpt_new_token nt{};
  nt.xk = ptr(xk), nt.xv = ptr(xv), nt.in_dtype = dtype_of(xk);
  nt.write_cache = truth(a[9]);
  nt.k_quant = static_cast<int8_t*>(offset(s.kq, s.q_off)), nt.v_quant = static_cast<int8_t*>(offset(s.vq, s.q_off));
  nt.k_scale = offset(s.ks, s.s_off), nt.v_scale = offset(s.vs, s.s_off);
  nt.pos = p.dev, nt.pos_count = p.count, nt.pos_host = p.host;
  if (a[13] != Py_None) nt.px = reinterpret_cast<const jpt_peer_exchange*>(integer(a[13]));
  c.nt = &nt;
  c.out_f32 = truth(a[11]);
  if (a[12] != Py_None) {
    PyObject* none_options[4] = {PyLong_FromLong(0), PyLong_FromLong(0), Py_False, a[12]};
    take_options(c, none_options);
    Py_DECREF(none_options[0]);
    Py_DECREF(none_options[1]);
    c.out_f32 = false;
  }
  const int64_t hq = c.q.size(1), tq = c.q.size(2);
  c.want_ml = !c.out_f32;
  if (c.out_f32)
    run_attention(c, {b, hq, tq, d}, {});
  else
    run_attention(c, {b, c.hkv, rt, d}, {b, c.hkv, rt});
  return tuple(s.kq, s.vq, s.ks, s.vs, c.o, c.m, c.l);
}

// fused_ok(xq, xk, k_scaler): shapes and types that update_attend takes
PyObject* fused_ok(Args a, Py_ssize_t n) {
  expect(n, 3, "fused_ok");
  const Tensor &q = tensor(a[0]), &k = tensor(a[1]);
  const Tensor* sc = maybe(a[2]);
  const bool ok = q.dim() == 4 && k.dim() == 4 && q.size(3) == 128 && q.size(2) == 1 && k.size(2) == 1 && k.size(1) > 0 && q.size(1) % k.size(1) == 0 &&
                  q.size(1) / k.size(1) <= 8 && (k.scalar_type() == ScalarType::BFloat16 || k.scalar_type() == ScalarType::Float) &&
                  q.scalar_type() == ScalarType::BFloat16 && sc && sc->scalar_type() == k.scalar_type();
  return PyBool_FromLong(ok);
}

// attend_lazy(xq, xk, xv, k, v, layer, end, keep_k or None, keep_v or None) -> out fp32 [B,Hq,1,D]: ragged attention over a
// bf16 / fp32 cache that does not hold the step's token yet, joined by that token, which is kept in layer `layer` of keep_k, keep_v.
PyObject* attend_lazy(Args a, Py_ssize_t n) {
  expect(n, 9, "attend_lazy");
  Call c;
  c.q = dense(tensor(a[0]));
  const Tensor xk = dense(tensor(a[1])), xv = dense(tensor(a[2]));
  const Tensor &k = tensor(a[3]), &v = tensor(a[4]);
  token_check(c.q, k, v, xk, xv);
  const c10::Device dev = c.q.device();
  OnDevice on(dev);
  const int64_t layer = integer(a[5]);
  take_kv(c, k, v, layer);
  c.end = tensor(a[6]);
  c.mask_mode = JPT_MASK_LENGTH;
  const int64_t b = c.q.size(0), hq = c.q.size(1), d = c.q.size(3);
  c.sm_scale = 1.0 / std::sqrt((double)d);
  const Tensor *kk = maybe(a[7]), *kv = maybe(a[8]);
  if ((kk == nullptr) != (kv == nullptr)) fail(PyExc_ValueError, "attend_lazy: kept K and V come together");
  if (xk.scalar_type() != c.q.scalar_type() || xv.scalar_type() != c.q.scalar_type() ||
      (kk && (kk->scalar_type() != xk.scalar_type() || kv->scalar_type() != xk.scalar_type())))
    fail(PyExc_ValueError, "attend_lazy: queries, token and kept rows share a dtype");
  for (const Tensor* t : {kk, kv})
    if (kk && (t->dim() != 5 || t->numel() != t->size(0) * xk.numel() || !t->is_contiguous() || t->device() != dev))
      fail(PyExc_ValueError, "attend_lazy: the kept rows must be contiguous tensors [layers, %lld, %lld, 1, %lld]", (long long)b,
           (long long)xk.size(1), (long long)d);
  const int64_t keep = kk ? layer_index(layer, kk->size(0)) * kk->stride(0) : 0;
  run_attention(c, {b, hq, 1, d}, {b, hq});
  Tensor out = empty({b, hq, 1, d}, ScalarType::Float, dev);
  check(jpt_attend_new_token(ptr(c.q), dtype_of(c.q), ptr(xk), ptr(xv), dtype_of(xk), nullptr, nullptr, 0, ptr(c.o),
                             static_cast<const float*>(ptr(c.m)), static_cast<const float*>(ptr(c.l)),
                             kk ? offset(*kk, keep) : nullptr, kk ? offset(*kv, keep) : nullptr, static_cast<float*>(ptr(out)), (int)b,
                             (int)hq, (int)c.hkv, (int)d, (float)c.sm_scale, stream_of(dev)));
  return wrap(out);
}

// attend_lazy_int8(xq, (k, v, k_scaler, v_scaler), layer, end, kq, vq, ks, vs) -> out fp32 [B,Hq,1,D]: the same over an int8 cache with
// the quantised token of the step (as quant_append returned it: one layer's)
PyObject* attend_lazy_int8(Args a, Py_ssize_t n) {
  expect(n, 8, "attend_lazy_int8");
  Call c;
  c.q = dense(tensor(a[0]));
  const Tensor &k = tensor(PyTuple_GET_ITEM(a[1], 0)), &v = tensor(PyTuple_GET_ITEM(a[1], 1));
  const c10::Device dev = c.q.device();
  OnDevice on(dev);
  const Tensor kq = dense(tensor(a[4])), vq = dense(tensor(a[5])), ks = dense(tensor(a[6])), vs = dense(tensor(a[7]));
  token_check(c.q, k, v, kq, vq);
  for (const Tensor* t : {&ks, &vs})
    if (t->numel() != c.q.size(0) || t->device() != dev || t->scalar_type() != ks.scalar_type())
      fail(PyExc_ValueError, "attend_lazy_int8: the token has a scale per sequence");
  const int64_t layer = integer(a[2]);
  take_kv(c, k, v, layer);
  take_scales(c, maybe(PyTuple_GET_ITEM(a[1], 2)), maybe(PyTuple_GET_ITEM(a[1], 3)), layer);
  scale_check(c);
  c.end = tensor(a[3]);
  c.mask_mode = JPT_MASK_LENGTH;
  const int64_t b = c.q.size(0), hq = c.q.size(1), d = c.q.size(3);
  c.sm_scale = 1.0 / std::sqrt((double)d);
  run_attention(c, {b, hq, 1, d}, {b, hq});
  Tensor out = empty({b, hq, 1, d}, ScalarType::Float, dev);
  check(jpt_attend_new_token(ptr(c.q), dtype_of(c.q), ptr(kq), ptr(vq), dtype_of(kq), ptr(ks), ptr(vs), dtype_of(ks), ptr(c.o),
                             static_cast<const float*>(ptr(c.m)), static_cast<const float*>(ptr(c.l)), nullptr, nullptr,
                             static_cast<float*>(ptr(out)), (int)b, (int)hq, (int)c.hkv, (int)d, (float)c.sm_scale, stream_of(dev)));
  return wrap(out);
}

// scatter_rows(src_k, src_v, dst_k, dst_v, pos, clamp): one row per (layer, slot, head) of dst [NL,B,H,S,D] or [B,H,S,D]
PyObject* scatter_rows(Args a, Py_ssize_t n) {
  expect(n, 6, "scatter_rows");
  const Tensor sk = dense(tensor(a[0])), sv = dense(tensor(a[1]));
  const Tensor &dk = tensor(a[2]), &dv = tensor(a[3]);
  if (dk.stride(-1) != 1) fail(PyExc_ValueError, "cache head_dim axis must be contiguous");
  const c10::Device dev = dk.device();
  OnDevice on(dev);
  const int64_t o = dk.dim() - 4;
  const Positions p = positions(a[4], dev, dk.size(o));
  check(jpt_kv_scatter_rows(ptr(sk), ptr(sv), ptr(dk), ptr(dv), (int)dk.element_size(), p.dev, p.count, p.host, truth(a[5]),
                            o ? (int)dk.size(0) : 1, (int)dk.size(o), (int)dk.size(o + 1), (int)dk.size(o + 2), (int)dk.size(o + 3),
                            o ? dk.stride(0) : 0, dk.stride(o), dk.stride(o + 1), dk.stride(o + 2), stream_of(dev)));
  Py_RETURN_NONE;
}

// finalize_int8(new_k, new_v, new_ks, new_vs, cache_k, cache_v, k_scaler, v_scaler, pos)
PyObject* finalize_int8(Args a, Py_ssize_t n) {
  expect(n, 9, "finalize_int8");
  const Tensor nk = dense(tensor(a[0])), nv = dense(tensor(a[1])), ns = dense(tensor(a[2])), ws = dense(tensor(a[3]));
  const Tensor &ck = tensor(a[4]), &cv = tensor(a[5]), &ks = tensor(a[6]), &vs = tensor(a[7]);
  if (ck.stride(-1) != 1) fail(PyExc_ValueError, "cache head_dim axis must be contiguous");
  const c10::Device dev = ck.device();
  OnDevice on(dev);
  const int64_t o = ck.dim() - 4;
  const Positions p = positions(a[8], dev, ck.size(o));
  check(jpt_kv_finalize_int8(static_cast<const int8_t*>(ptr(nk)), static_cast<const int8_t*>(ptr(nv)), static_cast<int8_t*>(ptr(ck)),
                             static_cast<int8_t*>(ptr(cv)), ptr(ns), ptr(ws), ptr(ks), ptr(vs), (int)ks.element_size(), p.dev, p.count,
                             p.host, o ? (int)ck.size(0) : 1, (int)ck.size(o), (int)ck.size(o + 1), (int)ck.size(o + 2),
                             (int)ck.size(o + 3), o ? ck.stride(0) : 0, ck.stride(o), ck.stride(o + 1), ck.stride(o + 2),
                             o ? ks.stride(0) : 0, ks.stride(o), ks.stride(o + 2), stream_of(dev)));
  Py_RETURN_NONE;
}

// kept_token(cache_k [NL,B,H,S,D], scale dtype of a tensor) -> zeroed new_k, new_v [NL,B,H,1,D] int8 and new_ks, new_vs [NL,B,1,1,1]:
// one allocation and one launch for the four
PyObject* kept_token(Args a, Py_ssize_t n) {
  expect(n, 2, "kept_token");
  const Tensor& ck = tensor(a[0]);
  const bool f32 = truth(a[1]);
  const c10::Device dev = ck.device();
  OnDevice on(dev);
  const int64_t nl = ck.size(0), b = ck.size(1), h = ck.size(2), d = ck.size(4);
  const ScalarType st = f32 ? ScalarType::Float : ScalarType::BFloat16;
  const int64_t rows = (nl * b * h * d + 255) / 256 * 256, es = f32 ? 4 : 2, scales = (nl * b * es + 255) / 256 * 256;
  Tensor all = empty({2 * rows + 2 * scales}, ScalarType::Char, dev);
  check(jpt_zero(all.data_ptr(), (size_t)all.numel(), stream_of(dev)));
  auto part = [&](int64_t byte, at::IntArrayRef sizes, ScalarType type, int64_t bytes_each) {
    Tensor t = empty({0}, type, dev);
    t.set_(all.storage(), byte / bytes_each, sizes, {});
    return t;
  };
  return tuple(part(0, {nl, b, h, 1, d}, ScalarType::Char, 1), part(rows, {nl, b, h, 1, d}, ScalarType::Char, 1),
               part(2 * rows, {nl, b, 1, 1, 1}, st, es), part(2 * rows + scales, {nl, b, 1, 1, 1}, st, es));
}

// append_paged(key, value, pool_k, pool_v, k_scales, v_scales, pti int32 [3,n], n_active or None)
PyObject* append_paged(Args a, Py_ssize_t n) {
  expect(n, 8, "append_paged");
  const Tensor key = dense(tensor(a[0])), value = dense(tensor(a[1]));
  const Tensor &ck = tensor(a[2]), &cv = tensor(a[3]);
  const c10::Device dev = key.device();
  OnDevice on(dev);
  const Tensor pti = as_i32(tensor(a[6]), dev);
  const int64_t cols = pti.size(1);
  check(jpt_kv_append_paged(ptr(key), ptr(value), dtype_of(key), ptr(ck), ptr(cv), dtype_of(ck), ptr(maybe(a[4])), ptr(maybe(a[5])),
                            static_cast<const int32_t*>(ptr(pti)), cols, (int)cols, static_cast<const int32_t*>(ptr(maybe(a[7]))),
                            (int)key.size(0), (int)ck.size(0), (int)ck.size(1), (int)ck.size(2), (int)ck.size(3), stream_of(dev)));
  Py_RETURN_NONE;
}

// page_token_indices(lens, page_table, page_size, slots, pages per slot) -> pti int32 [3,B], n_active [1], new_lengths [B]
PyObject* page_token_indices(Args a, Py_ssize_t n) {
  expect(n, 5, "page_token_indices");
  const c10::Device dev = tensor(a[0]).device();
  OnDevice on(dev);
  const int64_t b = integer(a[3]), pages = integer(a[4]);
  if (tensor(a[0]).numel() < b || tensor(a[1]).numel() < b * pages)
    fail(PyExc_ValueError, "page_token_indices: lengths of %lld slots and a table of %lld pages each are needed", (long long)b, (long long)pages);
  const Tensor lens = as_i32(tensor(a[0]), dev), table = as_i32(tensor(a[1]), dev);
  Tensor pti = empty({3, b}, ScalarType::Int, dev), active = empty({1}, ScalarType::Int, dev), lengths = empty({b}, ScalarType::Int, dev);
  check(jpt_page_token_indices(static_cast<const int32_t*>(ptr(lens)), static_cast<const int32_t*>(ptr(table)), (int)b, (int)pages,
                               (int)integer(a[2]), static_cast<int32_t*>(ptr(pti)), static_cast<int32_t*>(ptr(active)),
                               static_cast<int32_t*>(ptr(lengths)), stream_of(dev)));
  return tuple(pti, active, lengths);
}

// ---------------------------------------------------------------- insert
struct Layers {
  std::vector<jpt_layer_tensors> list;
  std::vector<Tensor> keep;  // copies made for odd layouts
  Tensor pk, ck, ks;         // of the first layer: shapes and strides
};
PyObject* item(PyObject* fast, Py_ssize_t i) { return PySequence_Fast_GET_ITEM(fast, i); }
struct Fast {  // a sequence as a list or tuple
  PyObject* o;
  explicit Fast(PyObject* s) : o(PySequence_Fast(s, "a list of layers was expected")) {
    if (!o) throw PySet{};
  }
  ~Fast() { Py_DECREF(o); }
  Py_ssize_t size() const { return PySequence_Fast_GET_SIZE(o); }
};
// The tensors of every layer; false where a layer's layout differs from the first one's, so that one launch cannot take all.
// `stacked`: caches (and scales) are one pair of stacked tensors.
bool take_layers(Layers& r, PyObject* prefixes, PyObject* caches, PyObject* scales, bool stacked) {
  Fast pre(prefixes), cac(caches);
  const Py_ssize_t n = pre.size();
  if (n < 1 || cac.size() != (stacked ? 1 : n)) return false;
  std::optional<Fast> sca;
  if (scales != Py_None) {
    sca.emplace(scales);
    if (sca->size() < (stacked ? 1 : n)) return false;
  }
  r.list.reserve(n);
  for (Py_ssize_t i = 0; i < n; ++i) {
    Fast p(item(pre.o, i)), c(item(cac.o, stacked ? 0 : i));
    if (p.size() != 2 || c.size() != 2) return false;
    Tensor pk = tensor(item(p.o, 0)), pv = tensor(item(p.o, 1));
    const Tensor &ck = tensor(item(c.o, 0)), &cv = tensor(item(c.o, 1));
    if (pk.stride(-1) != 1 || pv.strides() != pk.strides()) {
      pk = pk.contiguous(), pv = pv.contiguous();
      r.keep.push_back(pk);
      r.keep.push_back(pv);
    }
    const Tensor *ks = nullptr, *vs = nullptr;
    if (sca) {
      Fast s(item(sca->o, stacked ? 0 : i));
      if (s.size() != 2) return false;
      ks = maybe(item(s.o, 0)), vs = maybe(item(s.o, 1));
    }
    if (i == 0) {
      r.pk = pk, r.ck = ck;
      if (ks) r.ks = *ks;
      if (ck.dim() != (stacked ? 5 : 4) || (stacked && ck.size(0) < n)) return false;
      if (ks && (ks->dim() != ck.dim() || (stacked && vs && (ks->size(0) < n || vs->size(0) < n)))) return false;
    }
    if (pk.dim() != 4 || pv.sizes() != pk.sizes() || pk.sizes() != r.pk.sizes() || pk.strides() != r.pk.strides() ||
        pk.scalar_type() != r.pk.scalar_type() || pv.scalar_type() != pk.scalar_type() || pk.device() != r.pk.device() ||
        pv.device() != pk.device() || ck.sizes() != r.ck.sizes() || cv.sizes() != ck.sizes() || ck.strides() != r.ck.strides() ||
        cv.strides() != ck.strides() || ck.scalar_type() != r.ck.scalar_type() || cv.scalar_type() != ck.scalar_type() ||
        ck.device() != r.ck.device() || cv.device() != ck.device() || (ks != nullptr) != r.ks.defined() || (ks != nullptr) != (vs != nullptr))
      return false;
    if (ks && (ks->strides() != r.ks.strides() || vs->strides() != ks->strides() || ks->scalar_type() != pk.scalar_type() ||
               vs->scalar_type() != pk.scalar_type()) && ck.scalar_type() == ScalarType::Char)
      return false;
    const int64_t co = stacked ? i * ck.stride(0) : 0, so = stacked && ks ? i * ks->stride(0) : 0;
    jpt_layer_tensors t{};
    t.prefix_k = ptr(pk), t.prefix_v = ptr(pv);
    t.cache_k = offset(ck, co), t.cache_v = offset(cv, co);
    if (ks) t.k_scaler = offset(*ks, so), t.v_scaler = offset(*vs, so);
    r.list.push_back(t);
  }
  return true;
}

// insert_dense(prefixes, caches, scales or None, slot, pos, wrap, stacked) -> True when done; False: layer by layer
PyObject* insert_dense(Args a, Py_ssize_t n) {
  expect(n, 7, "insert_dense");
  Layers r;
  const bool stacked = truth(a[6]);
  if (!take_layers(r, a[0], a[1], a[2], stacked)) Py_RETURN_FALSE;
  const int64_t o = stacked ? 1 : 0, slot = integer(a[3]);
  const int64_t b = r.ck.size(o), h = r.ck.size(o + 1), s = r.ck.size(o + 2), d = r.ck.size(o + 3);
  if (r.pk.size(1) != h || r.pk.size(3) != d || slot < 0 || slot >= b || r.ck.stride(-1) != 1 || r.pk.device() != r.ck.device() ||
      (r.ck.scalar_type() == ScalarType::Char && r.pk.scalar_type() != ScalarType::Char && !r.ks.defined()))
    Py_RETURN_FALSE;  // (the calls layer by layer say what is wrong, or read the prefix from another GPU)
  OnDevice on(r.ck.device());
  check(jpt_prefill_insert_dense_layers(r.list.data(), (int)r.list.size(), dtype_of(r.pk), dtype_of(r.ck), (int)slot, (int)integer(a[4]),
                                        truth(a[5]), (int)h, (int)r.pk.size(2), (int)s, (int)d, r.pk.stride(1), r.pk.stride(2),
                                        r.ck.stride(o), r.ck.stride(o + 1), r.ck.stride(o + 2), r.ks.defined() ? r.ks.stride(o) : 0,
                                        r.ks.defined() ? r.ks.stride(o + 2) : 0, stream_of(r.ck.device())));
  Py_RETURN_TRUE;
}

// Layers that are views of stacked tensors: every pointer moves by the same step from layer to layer.
bool evenly_spaced(const std::vector<jpt_layer_tensors>& l) {
  auto even = [&](auto member) {
    const auto at = [&](size_t i) { return reinterpret_cast<intptr_t>(l[i].*member); };
    for (size_t i = 2; i < l.size(); ++i)
      if (at(i) - at(i - 1) != at(1) - at(0)) return false;
    return l.size() < 2 || at(1) >= at(0);
  };
  return even(&jpt_layer_tensors::prefix_k) && even(&jpt_layer_tensors::prefix_v) && even(&jpt_layer_tensors::cache_k) &&
         even(&jpt_layer_tensors::cache_v) && even(&jpt_layer_tensors::k_scaler) && even(&jpt_layer_tensors::v_scaler);
}

// insert_paged(prefixes, pools, scales or None, pages: a tensor or a sequence of ints) -> True when done
PyObject* insert_paged(Args a, Py_ssize_t n) {
  expect(n, 4, "insert_paged");
  Layers r;
  if (!take_layers(r, a[0], a[1], a[2], false)) Py_RETURN_FALSE;
  const int64_t h = r.ck.size(0), p = r.ck.size(1), ps = r.ck.size(2), d = r.ck.size(3);
  if (r.pk.size(1) != h || r.pk.size(3) != d || !r.ck.is_contiguous() ||
      (r.ck.scalar_type() == ScalarType::Char && r.pk.scalar_type() != ScalarType::Char && !r.ks.defined()))
    Py_RETURN_FALSE;
  // From four layers on one launch takes them wherever they lie.  Up to three scattered ones keep a launch each, as they had
  // before there was such a launch, not because that were better: 38 to 53 us a call for two or three layers of 37 to 1900
  // tokens, which take 5 to 10 as one launch.
  if (r.list.size() < 4 && !evenly_spaced(r.list)) Py_RETURN_FALSE;
  const c10::Device dev = r.ck.device();
  OnDevice on(dev);
  Tensor upd;
  std::vector<int32_t> pages;
  if (THPVariable_Check(a[3])) {
    upd = as_i32(tensor(a[3]), dev);
  } else {
    Fast list(a[3]);
    if (list.size() > 256) Py_RETURN_FALSE;
    for (Py_ssize_t i = 0; i < list.size(); ++i) pages.push_back((int32_t)integer(item(list.o, i)));
    if (pages.empty()) Py_RETURN_FALSE;
  }
  const int count = upd.defined() ? (int)upd.numel() : (int)pages.size();
  check(jpt_prefill_insert_paged_layers(r.list.data(), (int)r.list.size(), dtype_of(r.pk), dtype_of(r.ck),
                                        upd.defined() ? static_cast<const int32_t*>(ptr(upd)) : nullptr,
                                        upd.defined() ? nullptr : pages.data(), count, (int)h, (int)r.pk.size(2), (int)p, (int)ps, (int)d,
                                        r.pk.stride(1), r.pk.stride(2), stream_of(dev)));
  Py_RETURN_TRUE;
}

// ---------------------------------------------------------------- engine
struct MaskArg {
  void* p = nullptr;
  int dtype = JPT_F32;
  int64_t stride = 0;
};
MaskArg mask_arg(PyObject* o) {
  MaskArg m;
  if (const Tensor* t = maybe(o)) {
    if (t->stride(1) != 1) fail(PyExc_ValueError, "the mask's rows must be contiguous");
    m.p = ptr(*t), m.dtype = dtype_of(*t), m.stride = t->stride(0);
  }
  return m;
}
int32_t* i32(const Tensor& t, const char* what) {
  if (t.scalar_type() != ScalarType::Int || !t.is_contiguous()) fail(PyExc_ValueError, "%s must be a contiguous int32 tensor", what);
  return static_cast<int32_t*>(ptr(t));
}

// engine_begin(start, input_pos, S, block, mask or None, ring, pos) -> next_b, next_i, int32 [B, S / block]
PyObject* engine_begin(Args a, Py_ssize_t n) {
  expect(n, 7, "engine_begin");
  const Tensor &start = tensor(a[0]), &pos = tensor(a[1]);
  const c10::Device dev = start.device();
  OnDevice on(dev);
  const int64_t b = start.size(0), s = integer(a[2]), block = integer(a[3]);
  if (start.numel() != b || pos.numel() != b || pos.device() != dev) fail(PyExc_ValueError, "engine_begin: start and input_pos are one row per slot");
  if (block < 1) fail(PyExc_ValueError, "engine_begin: blocks of %lld tokens", (long long)block);
  if (a[4] != Py_None && (tensor(a[4]).dim() != 2 || tensor(a[4]).size(0) != b || tensor(a[4]).size(1) != s || tensor(a[4]).device() != dev))
    fail(PyExc_ValueError, "engine_begin: the mask is [%lld, %lld]", (long long)b, (long long)s);
  Tensor nb = empty({b, s / block}, ScalarType::Int, dev), ni = empty({b, s / block}, ScalarType::Int, dev);
  const MaskArg m = mask_arg(a[4]);
  check(jpt_engine_begin(i32(start, "start"), i32(pos, "input_pos"), (int)b, (int)s, (int)block, i32(nb, ""), i32(ni, ""), m.p, m.dtype,
                         m.stride, truth(a[5]), (int)integer(a[6]), stream_of(dev)));
  return tuple(nb, ni);
}

// engine_end(logits [B,T,V], tokens, lens, input_pos, S, mask or None, ring, pos) -> next_token [B,1], lens [B,1], input_pos [B], data [B,3]
PyObject* engine_end(Args a, Py_ssize_t n) {
  expect(n, 8, "engine_end");
  const Tensor &lg = tensor(a[0]), &tokens = tensor(a[1]), &lens = tensor(a[2]), &pos = tensor(a[3]);
  const c10::Device dev = lg.device();
  OnDevice on(dev);
  const int64_t b = lg.size(0);
  if (lg.dim() != 3 || lg.size(1) < 1 || lg.stride(2) != 1 || tokens.numel() != b || lens.numel() != b || pos.numel() != b)
    fail(PyExc_ValueError, "engine_end: logits are [B,T,V] with contiguous rows");
  if (tokens.device() != dev || lens.device() != dev || pos.device() != dev || (a[5] != Py_None && tensor(a[5]).device() != dev))
    fail(PyExc_ValueError, "engine_end: logits on %s, the state elsewhere", dev.str().c_str());
  Tensor next = empty({b, 1}, ScalarType::Int, dev), lo = empty(lens.sizes(), ScalarType::Int, dev),
         po = empty(pos.sizes(), ScalarType::Int, dev), data = empty({b, 3}, ScalarType::Int, dev);
  const MaskArg m = mask_arg(a[5]);
  check(jpt_engine_end(offset(lg, (lg.size(1) - 1) * lg.stride(1)), dtype_of(lg), lg.stride(0), (int)lg.size(2), i32(tokens, "tokens"),
                       i32(lens, "lens"), i32(pos, "input_pos"), (int)b, (int)integer(a[4]), truth(a[6]), (int)integer(a[7]), i32(next, ""),
                       i32(lo, ""), i32(po, ""), i32(data, ""), m.p, m.dtype, m.stride, stream_of(dev)));
  return tuple(next, lo, po, data);
}

// engine_slot(mask or None, S, slot, pos, cur, wrap, start value, seq_len, start, input_pos, lens, tokens or None, token or None)
PyObject* engine_slot(Args a, Py_ssize_t n) {
  expect(n, 13, "engine_slot");
  const MaskArg m = mask_arg(a[0]);
  const Tensor *start = maybe(a[8]), *pos = maybe(a[9]), *lens = maybe(a[10]), *tokens = maybe(a[11]), *token = maybe(a[12]);
  const Tensor* any = start ? start : pos ? pos : lens ? lens : a[0] == Py_None ? nullptr : &tensor(a[0]);
  if (!any) Py_RETURN_NONE;
  OnDevice on(any->device());
  check(jpt_engine_insert_slot(m.p, m.dtype, m.stride, (int)integer(a[1]), (int)integer(a[2]), (int)integer(a[3]), (int)integer(a[4]),
                               truth(a[5]), (int)integer(a[6]), (int)integer(a[7]), start ? i32(*start, "start") : nullptr,
                               pos ? i32(*pos, "input_pos") : nullptr, lens ? i32(*lens, "lens") : nullptr,
                               tokens ? i32(*tokens, "tokens") : nullptr, ptr(token), token ? (int)token->element_size() : 4,
                               stream_of(any->device())));
  Py_RETURN_NONE;
}

// ---------------------------------------------------------------- linear layers
Tensor scratch(const Tensor* have, size_t need, c10::Device dev) {
  if (have && (size_t)have->numel() >= need && have->device() == dev) return *have;
  return empty({(int64_t)need}, ScalarType::Byte, dev);
}
std::vector<int64_t> with_last(const Tensor& x, int64_t last) {
  std::vector<int64_t> s = x.sizes().vec();
  s.back() = last;
  return s;
}

// Rows of k features in x.
int64_t rows_of(const Tensor& x, int64_t k) {
  if (k < 1 || x.dim() < 1) fail(PyExc_ValueError, "activations of %lld features", (long long)k);
  return x.numel() / k;
}
// What a layer keeps between its calls is the workspace of up to kKeptRows rows, whose first word its kernels report to.  The scratch of a
// longer prompt (2 M K bytes) goes back to the allocator behind the call, in stream order: kept by every layer it was
// several GB of a model.
constexpr int64_t kKeptRows = 128;
constexpr size_t kStatusBytes = 256;

// linear(x [...,K], weight [N,K], scale [N], workspace or None) -> y [...,N], workspace to keep
PyObject* linear(Args a, Py_ssize_t n) {
  expect(n, 4, "linear");
  const Tensor x = dense(tensor(a[0]));
  const Tensor &w = tensor(a[1]), &sc = tensor(a[2]);
  const c10::Device dev = x.device();
  OnDevice on(dev);
  const int64_t out = w.size(0), k = w.size(1), m = rows_of(x, k);
  const size_t need = jpt_w8a16_linear_workspace_bytes((int)m, (int)out, (int)k);
  Tensor kept = scratch(maybe(a[3]), m > kKeptRows ? kStatusBytes : need, dev);
  Tensor ws = m > kKeptRows ? scratch(nullptr, need, dev) : kept;
  Tensor y = empty(with_last(x, out), ScalarType::BFloat16, dev);
  check(jpt_w8a16_linear_reporting(ptr(x), ptr(w), ptr(sc), ptr(y), (int)m, (int)out, (int)k, ptr(ws), (size_t)ws.numel(),
                                   static_cast<int32_t*>(ptr(kept)), stream_of(dev)));
  return tuple(y, kept);
}

// gate(x [...,K], w1, s1, w3, s3[, workspace or None]) -> h [...,N], workspace to keep: bf16(silu(x w1)) * (x w3)
PyObject* gate(Args a, Py_ssize_t n) {
  if (n != 5) expect(n, 6, "gate");
  const Tensor x = dense(tensor(a[0]));
  const Tensor &w1 = tensor(a[1]), &s1 = tensor(a[2]), &w3 = tensor(a[3]), &s3 = tensor(a[4]);
  const c10::Device dev = x.device();
  OnDevice on(dev);
  const int64_t out = w1.size(0), k = w1.size(1), m = rows_of(x, k);
  if (w3.sizes() != w1.sizes()) fail(PyExc_ValueError, "gate: w1 and w3 differ in shape");
  Tensor kept = scratch(n == 6 ? maybe(a[5]) : nullptr, kStatusBytes, dev);
  Tensor ws = scratch(nullptr, jpt_w8a16_gate_workspace_bytes((int)m, (int)out, (int)k), dev);
  Tensor h = empty(with_last(x, out), ScalarType::BFloat16, dev);
  check(jpt_w8a16_gate_reporting(ptr(x), ptr(w1), ptr(s1), ptr(w3), ptr(s3), ptr(h), (int)m, (int)out, (int)k, ptr(ws), (size_t)ws.numel(),
                                 static_cast<int32_t*>(ptr(kept)), stream_of(dev)));
  return tuple(h, kept);
}

// linear_from_levels(x [...,K] for its shape, levels workspace, weight, scale) -> y
PyObject* linear_from_levels(Args a, Py_ssize_t n) {
  expect(n, 4, "linear_from_levels");
  const Tensor &x = tensor(a[0]), &ws = tensor(a[1]), &w = tensor(a[2]), &sc = tensor(a[3]);
  const c10::Device dev = ws.device();
  OnDevice on(dev);
  const int64_t out = w.size(0), k = w.size(1), m = rows_of(x, k);
  Tensor y = empty(with_last(x, out), ScalarType::BFloat16, dev);
  check(jpt_w8a16_linear_from_levels(ptr(ws), (size_t)ws.numel(), ptr(w), ptr(sc), ptr(y), (int)m, (int)out, (int)k, stream_of(dev)));
  return wrap(y);
}

// rmsnorm(x, weight, eps, with_levels) -> y, levels workspace or None
PyObject* rmsnorm(Args a, Py_ssize_t n) {
  expect(n, 4, "rmsnorm");
  const Tensor x = dense(tensor(a[0]));
  const Tensor& w = tensor(a[1]);
  const c10::Device dev = x.device();
  OnDevice on(dev);
  const int64_t k = x.size(-1), m = rows_of(x, k);
  Tensor y = empty(x.sizes(), ScalarType::BFloat16, dev), ws;
  if (truth(a[3])) ws = scratch(nullptr, jpt_w8a16_linear_workspace_bytes((int)m, 1, (int)k), dev);
  check(jpt_rmsnorm(ptr(x), ptr(w), (float)real(a[2]), ptr(y), (int)m, (int)k, ws.defined() ? ptr(ws) : nullptr,
                    ws.defined() ? (size_t)ws.numel() : 0, stream_of(dev)));
  return tuple(y, ws);
}

// silu_mul(a, b, with_levels) -> h, levels workspace or None
PyObject* silu_mul(Args a, Py_ssize_t n) {
  expect(n, 3, "silu_mul");
  const Tensor x = dense(tensor(a[0])), g = dense(tensor(a[1]));
  const c10::Device dev = x.device();
  OnDevice on(dev);
  const int64_t k = x.size(-1), m = rows_of(x, k);
  Tensor h = empty(x.sizes(), ScalarType::BFloat16, dev), ws;
  if (truth(a[2])) ws = scratch(nullptr, jpt_w8a16_linear_workspace_bytes((int)m, 1, (int)k), dev);
  check(jpt_silu_mul(ptr(x), ptr(g), ptr(h), (int)m, (int)k, ws.defined() ? ptr(ws) : nullptr, ws.defined() ? (size_t)ws.numel() : 0,
                     stream_of(dev)));
  return tuple(h, ws);
}

// attention_workspaces() -> [(device index, stream handle or None, tensor)]
PyObject* attention_workspaces(Args, Py_ssize_t n) {
  expect(n, 0, "attention_workspaces");
  PyObject* list = PyList_New(0);
  if (!list) throw PySet{};
  for (const Workspace& w : workspaces()) {
    PyObject* t = w.graph ? Py_BuildValue("(iON)", (int)w.device, Py_None, wrap(w.mem))
                          : Py_BuildValue("(iKN)", (int)w.device, (unsigned long long)(uintptr_t)w.stream, wrap(w.mem));
    if (!t || PyList_Append(list, t) < 0) throw PySet{};
    Py_DECREF(t);
  }
  return list;
}

// (exceptions of torch's own calls become the Python types that its operators raise: OutOfMemoryError, IndexError and so on)
template <PyObject* (*F)(Args, Py_ssize_t)>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    return F(args, n);
  } catch (const PyFail& f) {
    PyErr_SetString(f.type, f.text.c_str());
    return nullptr;
  } catch (const PySet&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}
#define JPT_METHOD(name, fn) {name, (PyCFunction)(void (*)(void))entry<fn>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    JPT_METHOD("attend", attend), JPT_METHOD("ragged", ragged), JPT_METHOD("dense", dense_attention), JPT_METHOD("flash", flash),
    JPT_METHOD("paged", paged), JPT_METHOD("quant_append", quant_append), JPT_METHOD("update_attend", update_attend),
    JPT_METHOD("fused_ok", fused_ok), JPT_METHOD("attend_lazy", attend_lazy), JPT_METHOD("attend_lazy_int8", attend_lazy_int8), JPT_METHOD("scatter_rows", scatter_rows), JPT_METHOD("finalize_int8", finalize_int8),
    JPT_METHOD("kept_token", kept_token), JPT_METHOD("append_paged", append_paged), JPT_METHOD("page_token_indices", page_token_indices),
    JPT_METHOD("insert_dense", insert_dense), JPT_METHOD("insert_paged", insert_paged), JPT_METHOD("engine_begin", engine_begin),
    JPT_METHOD("engine_end", engine_end), JPT_METHOD("engine_slot", engine_slot), JPT_METHOD("linear", linear),
    JPT_METHOD("gate", gate), JPT_METHOD("linear_from_levels", linear_from_levels), JPT_METHOD("rmsnorm", rmsnorm), JPT_METHOD("silu_mul", silu_mul),
    JPT_METHOD("attention_workspaces", attention_workspaces), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
