// Native call path of the host mirrors: reads the tensors' addresses and strides, fills the argument block of the C entry
// point and launches on torch's current stream, in C++ instead of Python + ctypes.
//
// What bounds it: a decode step is dozens of calls of 5 to 20 us on the device each, so a call that costs the host 10 to
// 45 us (attribute look-ups, stride tuples, ctypes stores, one tensor allocation) leaves the GPU idle between launches.
// Here a call is one foreign function with positional arguments; what is left is the output's allocation and the launch.
//
// Every function handles the ordinary case only and returns None for anything else (operands on several devices or none, an unexpected
// shape or type, a status other than LQ_OK from the library).  The Python caller then takes its general path, which
// makes the same launch through ctypes or raises the error that belongs to it, so error behaviour has one home.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <map>
#include <utility>

#include "../../include/layer_quant_b200.h"

namespace {

struct Library {
  int (*mx_state_update)(const lq_mx_update_args*, void*) = nullptr;
  int (*mx_quantize)(const lq_mx_state*, const void*, int32_t, int64_t, const lq_rounding*, void*) = nullptr;
  int (*counter_add)(uint64_t*, uint64_t, void*) = nullptr;
  int (*int4_kv_append)(const lq_int4_cache*, const void*, const int64_t*, const void*, const int64_t*, int32_t, const int64_t*,
                        int32_t, void*) = nullptr;
  int (*int4_decode_attn)(const lq_int4_decode_args*, void*) = nullptr;
  size_t (*int4_decode_workspace_bytes)(int32_t, int32_t, int32_t, int32_t, int32_t) = nullptr;
  int32_t (*int4_decode_split_count)(const lq_int4_decode_args*) = nullptr;
  int (*int4_prefill_attn)(const lq_int4_prefill_args*, void*) = nullptr;
  int (*dense_state_update)(const lq_dense_update_args*, void*) = nullptr;
  int (*causal_conv1d_update)(const lq_conv1d_update_args*, void*) = nullptr;
} L;

// attribute names, interned once
struct Names {
  PyObject *q_state, *shared_exp, *micro_exp, *format_bits, *step, *layout, *layer, *step_counter, *advances_counter;
  PyObject *k_packed, *v_packed, *k_scale, *v_scale;
} N;

PyObject* none() { Py_RETURN_NONE; }

// An attribute that is a tensor; the object that owns it stays alive through its owner for the length of the call.
struct Attr {
  PyObject* o;
  Attr(PyObject* owner, PyObject* name) : o(PyObject_GetAttr(owner, name)) {
    if (o == nullptr) PyErr_Clear();
  }
  ~Attr() { Py_XDECREF(o); }
  Attr(const Attr&) = delete;
  Attr& operator=(const Attr&) = delete;
};

bool as_long(PyObject* o, int64_t& v) {
  if (o == nullptr || !PyLong_Check(o)) return false;
  int overflow = 0;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

// The truth value of an option; without one (a tensor of several elements) the call is not the ordinary case
bool as_bool(PyObject* o, bool& v) {
  const int r = o == nullptr ? -1 : PyObject_IsTrue(o);
  if (r < 0) PyErr_Clear();
  v = r == 1;
  return r >= 0;
}

// Collects operands: every tensor has to be on one CUDA device and of a type the kernels read.
struct Call {
  int device = -1;
  bool ok = true;

  const at::Tensor* tensor(PyObject* o, int64_t ndim) {
    if (o == nullptr || !THPVariable_Check(o)) return fail();
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.dim() != ndim || t.layout() != at::kStrided) return fail();
    const int d = t.get_device();
    if (device < 0) device = d;
    return d == device ? &t : fail();
  }
  int32_t dtype(const at::Tensor& t) {
    switch (t.scalar_type()) {
      case at::kBFloat16: return LQ_BF16;
      case at::kHalf: return LQ_F16;
      case at::kFloat: return LQ_F32;
      default: ok = false; return -1;
    }
  }
  // pointer, strides and type of an operand; None leaves the null pointer in place
  template <int ND, class P>
  const at::Tensor* operand(PyObject* o, P& ptr, int64_t (&stride)[ND], int32_t& type, bool optional = false) {
    if (optional && o == Py_None) return nullptr;
    const at::Tensor* t = tensor(o, ND);
    if (t == nullptr) return nullptr;
    ptr = t->data_ptr();
    for (int i = 0; i < ND; ++i) stride[i] = t->stride(i);
    type = dtype(*t);
    return t;
  }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream(); }

 private:
  const at::Tensor* fail() {
    ok = false;
    return nullptr;
  }
};

// f(stream) with `device` current, which is where the library's kernels go, and with other Python threads free to run: a launch
// blocks for as long as the queue of launches is full.  Both together cost 0.1 to 0.2 us of a call's 3 to 6.
template <class F>
int launch(int device, F f) {
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != device) guard.set_device(at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
  void* const stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
  PyThreadState* const thread = PyEval_SaveThread();
  const int status = f(stream);
  PyEval_RestoreThread(thread);
  return status;
}

// out: the caller's tensor (shaped like `like`) or a fresh one; returns a new reference in `ref`
bool output(Call& c, PyObject* given, const at::Tensor& like, at::Tensor& out) {
  if (given == Py_None) {
    out = at::empty_like(like);
    return true;
  }
  const at::Tensor* t = c.tensor(given, like.dim());
  if (t == nullptr || t->sizes() != like.sizes()) return false;
  out = *t;
  return true;
}
PyObject* give_back(PyObject* given, at::Tensor&& out) { return given == Py_None ? THPVariable_Wrap(std::move(out)) : Py_NewRef(given); }

bool state_struct(Call& c, const Attr& q, const Attr& e, const Attr& m, int64_t bits, bool packed, lq_mx_state& s) {
  const at::Tensor *tq = c.tensor(q.o, 4), *te = c.tensor(e.o, 4), *tm = c.tensor(m.o, 4);
  if (!c.ok || tq->stride(3) != 1 || te->stride(3) != 1 || tm->stride(3) != 1) return false;
  s.q_state = tq->data_ptr();
  s.shared_exp = static_cast<uint8_t*>(te->data_ptr());
  s.micro_exp = static_cast<uint8_t*>(tm->data_ptr());
  for (int i = 0; i < 3; ++i) {
    s.q_stride[i] = tq->stride(i);
    s.exp_stride[i] = te->stride(i);
    s.micro_stride[i] = tm->stride(i);
  }
  s.batch = tq->size(0);
  s.heads = tq->size(1);
  s.dim = tq->size(2);
  s.dstate = tq->size(3) * (packed && bits == 4 ? 2 : 1);
  s.format_bits = bits;
  s.layout = packed ? LQ_MX_LAYOUT_PACKED : LQ_MX_LAYOUT_REFERENCE;
  return true;
}

bool layout_of(PyObject* o, bool& packed) {
  if (o == nullptr || !PyUnicode_Check(o)) return false;
  packed = PyUnicode_CompareWithASCIIString(o, "packed") == 0;
  return packed || PyUnicode_CompareWithASCIIString(o, "reference") == 0;
}

// mx_update(cache, x, dt, A, B, C, D, z, dt_bias, dt_softplus, stochastic, seed, rng_stream, out)
PyObject* mx_update(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 14 || L.mx_state_update == nullptr) return none();
  PyObject* cache = a[0];
  Attr q(cache, N.q_state), e(cache, N.shared_exp), m(cache, N.micro_exp), bits_o(cache, N.format_bits), step_o(cache, N.step),
      layout_o(cache, N.layout), layer_o(cache, N.layer), counter_o(cache, N.step_counter);
  int64_t bits, step, layer;
  bool packed, softplus, stochastic;
  if (!as_long(bits_o.o, bits) || !as_long(step_o.o, step) || !as_long(layer_o.o, layer) || !layout_of(layout_o.o, packed) ||
      counter_o.o == nullptr || !as_bool(a[9], softplus) || !as_bool(a[10], stochastic) || !PyLong_Check(a[11]) || !PyUnicode_Check(a[12]))
    return none();
  Call c;
  lq_mx_update_args u = {};
  if (!state_struct(c, q, e, m, bits, packed, u.state)) return none();
  const at::Tensor* x = c.operand(a[1], u.x, u.x_stride, u.x_dtype);
  c.operand(a[2], u.dt, u.dt_stride, u.dt_dtype);
  c.operand(a[3], u.A, u.A_stride, u.A_dtype);
  const at::Tensor* B = c.operand(a[4], u.B, u.B_stride, u.B_dtype);
  c.operand(a[5], u.C, u.C_stride, u.C_dtype);
  c.operand(a[6], u.D, u.D_stride, u.D_dtype, true);
  c.operand(a[7], u.z, u.z_stride, u.z_dtype, true);
  c.operand(a[8], u.dt_bias, u.dt_bias_stride, u.dt_bias_dtype, true);
  if (!c.ok || x->size(0) != u.state.batch || x->size(1) != u.state.heads || x->size(2) != u.state.dim) return none();
  // the reference's kernel addresses dt_bias with D's strides
  u.dt_bias_stride[0] = u.D ? u.D_stride[0] : 0;
  u.dt_bias_stride[1] = u.D ? u.D_stride[1] : 0;
  u.ngroups = B->size(1);
  u.dt_softplus = softplus;
  lq_rounding& r = u.rounding;
  r.seed = PyLong_AsUnsignedLongLongMask(a[11]);
  r.layer = static_cast<uint32_t>(layer);
  r.step = static_cast<uint64_t>(step);
  r.rng_offset = static_cast<uint64_t>(step) * static_cast<uint64_t>(u.state.batch) * u.state.heads * u.state.dim * u.state.dstate;
  if (!stochastic) {
    r.mode = LQ_ROUND_HALF_UP;
  } else if (PyUnicode_CompareWithASCIIString(a[12], "layered") == 0) {
    r.mode = LQ_ROUND_PHILOX_LAYERED;
  } else if (PyUnicode_CompareWithASCIIString(a[12], "reference") == 0) {
    r.mode = LQ_ROUND_PHILOX_REF;
  } else if (PyUnicode_CompareWithASCIIString(a[12], "layered4") == 0) {
    r.mode = LQ_ROUND_PHILOX_LAYERED4;
  } else {
    return none();
  }
  if (counter_o.o != Py_None) {
    const at::Tensor* k = c.tensor(counter_o.o, 1);
    if (k == nullptr || k->scalar_type() != at::kLong || k->numel() != 1) return none();
    r.step_counter = static_cast<const uint64_t*>(k->data_ptr());
  }
  bool advances = false;
  if (counter_o.o != Py_None) {
    const Attr advances_o(cache, N.advances_counter);
    if (!as_bool(advances_o.o, advances)) return none();
  }
  at::Tensor out;
  if (!output(c, a[13], *x, out)) return none();
  u.out = out.data_ptr();
  for (int i = 0; i < 3; ++i) u.out_stride[i] = out.stride(i);
  u.out_dtype = c.dtype(out);
  if (!c.ok) return none();
  if (launch(c.device, [&](void* stream) { return L.mx_state_update(&u, stream); }) != LQ_OK) return none();
  if (r.step_counter == nullptr) {
    PyObject* next = PyLong_FromLongLong(step + 1);
    if (next == nullptr || PyObject_SetAttr(cache, N.step, next) != 0) {
      Py_XDECREF(next);
      return nullptr;
    }
    Py_DECREF(next);
  } else {
    if (advances && launch(c.device, [&](void* stream) { return L.counter_add(const_cast<uint64_t*>(r.step_counter), 1, stream); }) != LQ_OK) {
      PyErr_SetString(PyExc_RuntimeError, "the step counter could not be advanced");
      return nullptr;
    }
  }
  return give_back(a[13], std::move(out));
  END_HANDLE_TH_ERRORS
}

// mx_plan_run(address of the prepared lq_mx_update_args, device, step): launches it with this step; the status
PyObject* mx_plan_run(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t device, step;
  void* address = n == 3 ? PyLong_AsVoidPtr(a[0]) : nullptr;
  if (address == nullptr || !as_long(a[1], device) || !as_long(a[2], step)) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "mx_plan_run(address, device, step)");
    return nullptr;
  }
  lq_mx_update_args& u = *static_cast<lq_mx_update_args*>(address);
  u.rounding.step = static_cast<uint64_t>(step);
  u.rounding.rng_offset = static_cast<uint64_t>(step) * static_cast<uint64_t>(u.state.batch) * u.state.heads * u.state.dim * u.state.dstate;
  return PyLong_FromLong(launch(static_cast<int>(device), [&](void* stream) { return L.mx_state_update(&u, stream); }));
  END_HANDLE_TH_ERRORS
}

// int4_plan_launch(address of the prepared lq_int4_decode_args, device): the status
PyObject* int4_plan_launch(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t device;
  void* address = n == 2 ? PyLong_AsVoidPtr(a[0]) : nullptr;
  if (address == nullptr || !as_long(a[1], device)) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "int4_plan_launch(address, device)");
    return nullptr;
  }
  return PyLong_FromLong(launch(static_cast<int>(device), [&](void* stream) { return L.int4_decode_attn(static_cast<const lq_int4_decode_args*>(address), stream); }));
  END_HANDLE_TH_ERRORS
}

// mx_quantize(state [B,H,P,N], format_bits, packed) -> (q_state, shared_exp, micro_exp), rounded half to even
PyObject* mx_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t bits;
  if (n != 3 || L.mx_quantize == nullptr || !as_long(a[1], bits) || (bits != 8 && bits != 4)) return none();
  bool packed;
  if (!as_bool(a[2], packed)) return none();
  Call c;
  const at::Tensor* src = c.tensor(a[0], 4);
  if (src == nullptr) return none();
  const int32_t type = c.dtype(*src);
  const int64_t width = src->size(3);
  if (!c.ok || width % 16 != 0 || !src->is_contiguous() || src->numel() == 0) return none();
  const auto bytes = src->options().dtype(at::kByte);
  const int64_t s0 = src->size(0), s1 = src->size(1), s2 = src->size(2);
  at::Tensor q = packed && bits == 4 ? at::empty({s0, s1, s2, width / 2}, bytes) : at::empty({s0, s1, s2, width}, bytes.dtype(at::kChar));
  at::Tensor e = at::empty({s0, s1, s2, width / 16}, bytes);
  at::Tensor m = at::empty({s0, s1, s2, packed ? width / 16 : width / 2}, bytes);
  lq_mx_state s = {};
  s.q_state = q.data_ptr();
  s.shared_exp = static_cast<uint8_t*>(e.data_ptr());
  s.micro_exp = static_cast<uint8_t*>(m.data_ptr());
  const int64_t rows = s0 * s1 * s2;
  if (rows >= (1ll << 31)) return none();
  s.batch = s.heads = 1;
  s.dim = rows;
  s.dstate = width;
  s.q_stride[2] = q.size(3);
  s.exp_stride[2] = e.size(3);
  s.micro_stride[2] = m.size(3);
  s.q_stride[0] = s.q_stride[1] = rows * q.size(3);
  s.exp_stride[0] = s.exp_stride[1] = rows * e.size(3);
  s.micro_stride[0] = s.micro_stride[1] = rows * m.size(3);
  s.format_bits = bits;
  s.layout = packed ? LQ_MX_LAYOUT_PACKED : LQ_MX_LAYOUT_REFERENCE;
  lq_rounding r = {};
  r.mode = LQ_ROUND_HALF_EVEN;
  if (launch(c.device, [&](void* stream) { return L.mx_quantize(&s, src->data_ptr(), type, width, &r, stream); }) != LQ_OK) return none();
  PyObject* out = PyTuple_New(3);
  if (out == nullptr) return nullptr;
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(q)));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(std::move(e)));
  PyTuple_SET_ITEM(out, 2, THPVariable_Wrap(std::move(m)));
  return out;
  END_HANDLE_TH_ERRORS
}

// ---- INT4 KV cache ---------------------------------------------------------------------------------------------------
bool cache_struct(Call& c, PyObject* cache, int64_t group, lq_int4_cache& s) {
  Attr kp(cache, N.k_packed), vp(cache, N.v_packed), ks(cache, N.k_scale), vs(cache, N.v_scale);
  const at::Tensor *tkp = c.tensor(kp.o, 4), *tvp = c.tensor(vp.o, 4), *tks = c.tensor(ks.o, 4), *tvs = c.tensor(vs.o, 4);
  if (!c.ok) return false;
  s.k_packed = static_cast<uint8_t*>(tkp->data_ptr());
  s.v_packed = static_cast<uint8_t*>(tvp->data_ptr());
  s.k_scale = static_cast<float*>(tks->data_ptr());
  s.v_scale = static_cast<float*>(tvs->data_ptr());
  for (int i = 0; i < 4; ++i) {
    s.kp_stride[i] = tkp->stride(i);
    s.vp_stride[i] = tvp->stride(i);
    s.ks_stride[i] = tks->stride(i);
    s.vs_stride[i] = tvs->stride(i);
  }
  s.batch = tkp->size(0);
  s.kv_heads = tkp->size(1);
  s.capacity = tkp->size(2);
  s.head_dim = tkp->size(3) * 2;
  s.group_size = group;
  return tkp->scalar_type() == at::kByte && tvp->scalar_type() == at::kByte && tks->scalar_type() == at::kFloat &&
         tvs->scalar_type() == at::kFloat && group > 0 && tks->size(3) * group == s.head_dim;
}

// Scratch of the split merge, per (device, stream), zeroed once: the kernels leave the ticket counters at zero.
//
// Calls that run now share one buffer, grown on demand.  It is allocated on the stream that uses it, so one that is replaced by a larger
// one or dropped (the longest unused of more than kMaxWorkspaces) is handed out again by the allocator in stream order only.
// A call that is being recorded must not use it: a graph holds the bare address, and a replay knows nothing of that order.  Each capture
// gets a buffer of its own from the graph's memory pool, where the address stays the graph's, and whose zeroing is recorded ahead of
// its first use.
struct Workspace {
  at::Tensor now, recorded;
  unsigned long long capture = 0;  // the capture that `recorded` belongs to, 0: none
  uint64_t last_use = 0;
};
constexpr size_t kMaxWorkspaces = 64;
std::map<std::pair<int, void*>, Workspace>& workspaces() {
  static auto& all = *new std::map<std::pair<int, void*>, Workspace>;  // never destroyed: the allocator may be gone at exit
  return all;
}

at::Tensor workspace(int device, void* stream, size_t nbytes) {
  static uint64_t uses = 0;
  auto& all = workspaces();
  const auto key = std::make_pair(device, stream);
  if (all.size() >= kMaxWorkspaces && all.find(key) == all.end())
    all.erase(std::min_element(all.begin(), all.end(), [](const auto& a, const auto& b) { return a.second.last_use < b.second.last_use; }));
  Workspace& w = all[key];
  w.last_use = ++uses;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  C10_CUDA_CHECK(cudaStreamGetCaptureInfo(static_cast<cudaStream_t>(stream), &status, &id));
  if (status == cudaStreamCaptureStatusNone) id = 0;
  if (w.capture != id) w.recorded.reset();
  w.capture = id;
  at::Tensor& ws = id != 0 ? w.recorded : w.now;
  if (!ws.defined() || static_cast<size_t>(ws.numel()) < nbytes)
    ws = at::zeros({static_cast<int64_t>(std::max<size_t>(nbytes, 1 << 20))},
                   at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
  return ws;
}

// workspace_for(device, nbytes): the same buffer for prepared launches
PyObject* workspace_for(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t device, nbytes;
  if (n != 2 || !as_long(a[0], device) || !as_long(a[1], nbytes)) return none();
  void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
  return THPVariable_Wrap(workspace(static_cast<int>(device), stream, static_cast<size_t>(nbytes)));
  END_HANDLE_TH_ERRORS
}

// The caller's attention mask as the kernel reads it: 2-D keep flags (the last seq_len columns count) or a 4-D mask's last
// query row, bool or additive.  A batch of one is shared by all sequences.
bool decode_mask(Call& c, PyObject* o, int64_t batch, int64_t seq_len, lq_int4_decode_args& d) {
  if (!THPVariable_Check(o)) return false;
  const at::Tensor& m = THPVariable_Unpack(o);
  if (m.dim() != 2 && m.dim() != 4) return false;
  if (c.tensor(o, m.dim()) == nullptr || (m.size(0) != batch && m.size(0) != 1)) return false;
  const bool four = m.dim() == 4;
  const int64_t width = m.size(four ? 3 : 1), along = m.stride(four ? 3 : 1);
  switch (m.scalar_type()) {
    case at::kBool: d.mask_kind = LQ_MASK_KEEP_U8; break;
    case at::kByte: d.mask_kind = LQ_MASK_KEEP_U8; break;
    case at::kInt: d.mask_kind = LQ_MASK_KEEP_I32; break;
    case at::kLong: d.mask_kind = LQ_MASK_KEEP_I64; break;
    case at::kFloat: d.mask_kind = LQ_MASK_ADD_F32; break;
    case at::kBFloat16: d.mask_kind = LQ_MASK_ADD_BF16; break;
    case at::kHalf: d.mask_kind = LQ_MASK_ADD_F16; break;
    default: return false;
  }
  const bool keeps = d.mask_kind >= LQ_MASK_KEEP_U8;
  // 2-D masks are keep flags of any type (a floating one takes the general path), 4-D ones bool or additive
  if (four ? (keeps && m.scalar_type() != at::kBool) || m.size(1) < 1 || m.size(2) < 1 : !keeps || width < seq_len) return false;
  const int64_t first = four ? (m.size(2) - 1) * m.stride(2) : (width - seq_len) * along;
  d.mask = static_cast<const char*>(m.data_ptr()) + first * m.element_size();
  d.mask_stride_b = m.size(0) == 1 ? 0 : m.stride(0);
  d.mask_stride_k = along;
  d.mask_k_len = static_cast<int32_t>(std::min(width, seq_len));
  return true;
}

// decode_attn(q [B,Hq,1,D], cache, seq_len, query heads per kv head (-1: not checked), group_size, mask, k_new, v_new, splits, counter)
PyObject* decode_attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t seq_len, ratio, group, splits;
  if (n != 10 || L.int4_decode_attn == nullptr || L.int4_decode_split_count == nullptr || !as_long(a[2], seq_len) || !as_long(a[3], ratio) || !as_long(a[4], group) ||
      !as_long(a[8], splits))
    return none();
  Call c;
  lq_int4_decode_args d = {};
  const at::Tensor* q = c.tensor(a[0], 4);
  if (q == nullptr || !cache_struct(c, a[1], group, d.cache)) return none();
  const int64_t batch = q->size(0), heads = q->size(1), dim = q->size(3);
  d.dtype = c.dtype(*q);
  if (!c.ok || q->size(2) != 1 || batch != d.cache.batch || dim != d.cache.head_dim || seq_len < 1 || seq_len > d.cache.capacity ||
      (ratio != -1 && heads != ratio * d.cache.kv_heads))
    return none();
  d.q = q->data_ptr();
  d.q_stride[0] = q->stride(0);
  d.q_stride[1] = q->stride(1);
  d.q_stride[2] = q->stride(3);
  d.q_heads = heads;
  d.seq_len = seq_len;
  if (a[5] != Py_None && !decode_mask(c, a[5], batch, seq_len, d)) return none();
  if (a[6] != Py_None) {
    const at::Tensor *k = c.tensor(a[6], 4), *v = c.tensor(a[7], 4);
    if (!c.ok || k->sizes() != v->sizes() || k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() ||
        k->size(0) != batch || k->size(1) != d.cache.kv_heads || k->size(2) != 1 || k->size(3) != dim)
      return none();
    d.k_new = k->data_ptr();
    d.v_new = v->data_ptr();
    for (int i = 0; i < 3; ++i) {
      d.k_new_stride[i] = k->stride(i + (i == 2));
      d.v_new_stride[i] = v->stride(i + (i == 2));
    }
  }
  if (a[9] != Py_None) {
    const at::Tensor* k = c.tensor(a[9], 1);
    if (k == nullptr || k->scalar_type() != at::kLong || k->numel() != 1) return none();
    d.seq_len_counter = static_cast<const uint64_t*>(k->data_ptr());
  }
  if (splits <= 0) {  // the library's choice, made here once: it costs 0.1 to 0.8 us
    const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(c.device));  // the rule asks for its number of SMs
    splits = L.int4_decode_split_count(&d);
  }
  d.splits = static_cast<int32_t>(std::min<int64_t>(splits, INT32_MAX));
  at::Tensor ws;  // held until the launch is in the stream
  if (splits > 1) {
    ws = workspace(c.device, c.stream(), L.int4_decode_workspace_bytes(batch, heads, d.cache.kv_heads, dim, d.splits));
    d.workspace = ws.data_ptr();
    d.workspace_bytes = ws.numel();
  }
  at::Tensor out = at::empty({batch, heads, dim}, q->options());
  d.out = out.data_ptr();
  for (int i = 0; i < 3; ++i) d.out_stride[i] = out.stride(i);
  if (launch(c.device, [&](void* stream) { return L.int4_decode_attn(&d, stream); }) != LQ_OK) return none();
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// pack_kv(cache, k, v, positions, group_size) -> True
PyObject* pack_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t group;
  if (n != 5 || L.int4_kv_append == nullptr || !as_long(a[4], group)) return none();
  Call c;
  lq_int4_cache s = {};
  const at::Tensor *k = c.tensor(a[1], 4), *v = c.tensor(a[2], 4), *pos = c.tensor(a[3], 1);
  if (!c.ok || !cache_struct(c, a[0], group, s)) return none();
  const int32_t type = c.dtype(*k);
  if (!c.ok || k->sizes() != v->sizes() || k->scalar_type() != v->scalar_type() || pos->scalar_type() != at::kLong || !pos->is_contiguous() ||
      pos->size(0) != k->size(2) || k->size(0) != s.batch || k->size(1) != s.kv_heads || k->size(3) != s.head_dim)
    return none();
  const auto append = [&](void* stream) {
    return L.int4_kv_append(&s, k->data_ptr(), k->strides().data(), v->data_ptr(), v->strides().data(), type,
                            static_cast<const int64_t*>(pos->data_ptr()), static_cast<int32_t>(k->size(2)), stream);
  };
  if (launch(c.device, append) != LQ_OK) return none();
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// prefill_attn(q [B,Hq,Tq,D], cache, query heads per kv head, group_size, first_len, out)
PyObject* prefill_attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t ratio, group, first_len;
  if (n != 6 || L.int4_prefill_attn == nullptr || !as_long(a[2], ratio) || !as_long(a[3], group) || !as_long(a[4], first_len)) return none();
  Call c;
  lq_int4_prefill_args p = {};
  const at::Tensor* q = c.tensor(a[0], 4);
  if (q == nullptr || !cache_struct(c, a[1], group, p.cache)) return none();
  p.dtype = c.dtype(*q);
  if (!c.ok || q->size(0) != p.cache.batch || q->size(3) != p.cache.head_dim || q->size(1) != ratio * p.cache.kv_heads || first_len < 1 ||
      first_len > INT32_MAX)
    return none();
  at::Tensor out;
  if (a[5] == Py_None) {
    out = at::empty(q->sizes(), q->options());
  } else if (!output(c, a[5], *q, out) || out.scalar_type() != q->scalar_type()) {
    return none();
  }
  p.q = q->data_ptr();
  p.out = out.data_ptr();
  for (int i = 0; i < 4; ++i) {
    p.q_stride[i] = q->stride(i);
    p.out_stride[i] = out.stride(i);
  }
  p.q_heads = q->size(1);
  p.q_len = q->size(2);
  p.first_len = static_cast<int32_t>(first_len);
  if (launch(c.device, [&](void* stream) { return L.int4_prefill_attn(&p, stream); }) != LQ_OK) return none();
  return give_back(a[5], std::move(out));
  END_HANDLE_TH_ERRORS
}

// ---- unquantised baselines -------------------------------------------------------------------------------------------
// dense_update(state [B,H,P,N], x, dt, A, B, C, D, z, dt_bias, dt_softplus, out)
PyObject* dense_update(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool softplus;
  if (n != 11 || L.dense_state_update == nullptr || !as_bool(a[9], softplus)) return none();
  Call c;
  lq_dense_update_args u = {};
  const at::Tensor* state = c.operand(a[0], u.state, u.state_stride, u.state_dtype);
  const at::Tensor* x = c.operand(a[1], u.x, u.x_stride, u.x_dtype);
  const at::Tensor* dt = c.operand(a[2], u.dt, u.dt_stride, u.dt_dtype);
  const at::Tensor* A = c.operand(a[3], u.A, u.A_stride, u.A_dtype);
  const at::Tensor* B = c.operand(a[4], u.B, u.B_stride, u.B_dtype);
  const at::Tensor* C = c.operand(a[5], u.C, u.C_stride, u.C_dtype);
  const at::Tensor* D = c.operand(a[6], u.D, u.D_stride, u.D_dtype, true);
  const at::Tensor* z = c.operand(a[7], u.z, u.z_stride, u.z_dtype, true);
  const at::Tensor* bias = c.operand(a[8], u.dt_bias, u.dt_bias_stride, u.dt_bias_dtype, true);
  if (!c.ok) return none();
  const int64_t b = state->size(0), h = state->size(1), p = state->size(2), w = state->size(3), g = B->size(1);
  const auto is3 = [](const at::Tensor* t, int64_t i, int64_t j, int64_t k) { return t->size(0) == i && t->size(1) == j && t->size(2) == k; };
  const auto is2 = [](const at::Tensor* t, int64_t i, int64_t j) { return t == nullptr || (t->size(0) == i && t->size(1) == j); };
  if (!is3(x, b, h, p) || !is3(dt, b, h, p) || !is3(A, h, p, w) || !is3(B, b, g, w) || !is3(C, b, g, w) || g == 0 || h % g != 0 ||
      !is2(D, h, p) || !is2(bias, h, p) || (z != nullptr && !is3(z, b, h, p)))
    return none();
  at::Tensor out;
  if (!output(c, a[10], *x, out)) return none();
  u.out = out.data_ptr();
  for (int i = 0; i < 3; ++i) u.out_stride[i] = out.stride(i);
  u.out_dtype = c.dtype(out);
  u.batch = b;
  u.heads = h;
  u.dim = p;
  u.dstate = w;
  u.ngroups = g;
  u.dt_softplus = softplus;
  if (!c.ok || launch(c.device, [&](void* stream) { return L.dense_state_update(&u, stream); }) != LQ_OK) return none();
  return give_back(a[10], std::move(out));
  END_HANDLE_TH_ERRORS
}

// conv1d_update(x [B,C], conv_state [B,C,W], weight [C,W], bias, silu, out)
PyObject* conv1d_update(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool silu;
  if (n != 6 || L.causal_conv1d_update == nullptr || !as_bool(a[4], silu)) return none();
  Call c;
  lq_conv1d_update_args u = {};
  const at::Tensor* x = c.operand(a[0], u.x, u.x_stride, u.x_dtype);
  const at::Tensor* state = c.operand(a[1], u.conv_state, u.state_stride, u.state_dtype);
  const at::Tensor* weight = c.operand(a[2], u.weight, u.weight_stride, u.weight_dtype);
  const at::Tensor* bias = c.operand(a[3], u.bias, u.bias_stride, u.bias_dtype, true);
  if (!c.ok) return none();
  const int64_t b = x->size(0), ch = x->size(1), w = state->size(2);
  if (state->size(0) != b || state->size(1) != ch || weight->size(0) != ch || weight->size(1) != w || (bias != nullptr && bias->size(0) != ch))
    return none();
  at::Tensor out;
  if (!output(c, a[5], *x, out)) return none();
  u.out = out.data_ptr();
  for (int i = 0; i < 2; ++i) u.out_stride[i] = out.stride(i);
  u.out_dtype = c.dtype(out);
  u.batch = b;
  u.channels = ch;
  u.width = w;
  u.silu = silu;
  if (!c.ok || launch(c.device, [&](void* stream) { return L.causal_conv1d_update(&u, stream); }) != LQ_OK) return none();
  return give_back(a[5], std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind(path): the entry points of the C library at `path` (already loaded by ctypes: the same image)
PyObject* bind(PyObject*, PyObject* path_o) {
  const char* path = PyUnicode_AsUTF8(path_o);
  if (path == nullptr) return nullptr;
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (h == nullptr) {
    PyErr_Format(PyExc_RuntimeError, "cannot load %s: %s", path, dlerror());
    return nullptr;
  }
  bool ok = true;
  const auto find = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(dlsym(h, name));
    if (fn == nullptr) {
      PyErr_Format(PyExc_RuntimeError, "%s does not export %s; rebuild the library", path, name);
      ok = false;
    }
  };
  find(L.mx_state_update, "lq_mx_state_update");
  find(L.mx_quantize, "lq_mx_quantize");
  find(L.counter_add, "lq_counter_add");
  find(L.int4_kv_append, "lq_int4_kv_append");
  find(L.int4_decode_attn, "lq_int4_decode_attn");
  find(L.int4_decode_workspace_bytes, "lq_int4_decode_workspace_bytes");
  find(L.int4_prefill_attn, "lq_int4_prefill_attn");
  find(L.dense_state_update, "lq_dense_state_update");
  find(L.causal_conv1d_update, "lq_causal_conv1d_update");
  if (!ok) return nullptr;
  // (the ctypes binding has seen that the library has it; a stand-in may not, and leaves decode_attn to the general path)
  L.int4_decode_split_count = reinterpret_cast<decltype(L.int4_decode_split_count)>(dlsym(h, "lq_int4_decode_split_count"));
  Py_RETURN_NONE;
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef methods[] = {
    {"bind", bind, METH_O, nullptr},
    {"mx_update", fast(mx_update), METH_FASTCALL, nullptr},
    {"mx_plan_run", fast(mx_plan_run), METH_FASTCALL, nullptr},
    {"int4_plan_launch", fast(int4_plan_launch), METH_FASTCALL, nullptr},
    {"mx_quantize", fast(mx_quantize), METH_FASTCALL, nullptr},
    {"workspace_for", fast(workspace_for), METH_FASTCALL, nullptr},
    {"decode_attn", fast(decode_attn), METH_FASTCALL, nullptr},
    {"pack_kv", fast(pack_kv), METH_FASTCALL, nullptr},
    {"prefill_attn", fast(prefill_attn), METH_FASTCALL, nullptr},
    {"dense_update", fast(dense_update), METH_FASTCALL, nullptr},
    {"conv1d_update", fast(conv1d_update), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "layer_quant_b200._native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  const std::pair<PyObject**, const char*> names[] = {
      {&N.q_state, "q_state"}, {&N.shared_exp, "shared_exp"}, {&N.micro_exp, "micro_exp"}, {&N.format_bits, "format_bits"},
      {&N.step, "step"}, {&N.layout, "layout"}, {&N.layer, "layer"}, {&N.step_counter, "step_counter"},
      {&N.advances_counter, "advances_counter"}, {&N.k_packed, "k_packed"}, {&N.v_packed, "v_packed"}, {&N.k_scale, "k_scale"},
      {&N.v_scale, "v_scale"}};
  for (const auto& [slot, text] : names)
    if ((*slot = PyUnicode_InternFromString(text)) == nullptr) return nullptr;
  return PyModule_Create(&module);
}
