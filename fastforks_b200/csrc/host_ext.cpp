// The repeated call of an operator, in C++: reads the tensors' metadata, allocates the result, fills the C-ABI struct and
// launches. A call of ten microseconds on the GPU spent as long again in Python on keys, checks and ctypes.
//
// Every function returns None for anything but the plain, valid case (other types, broadcast or copied operands, a
// missing workspace, another current device, an error of the library): the Python implementation then runs, checks and
// reports. Nothing is decided here that it would decide otherwise.
#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "../../include/b200_attn.h"

namespace {

constexpr int64_t kHeadDim = 64, kSplitMinKeys = 257;

// Attention workspaces by (device, stream), registered by the Python side when it allocates them.
struct Workspace {
  int64_t device, stream;
  void* ptr;
  int64_t bytes;
};
std::mutex g_workspaces_mutex;
std::vector<Workspace> g_workspaces;

bool find_workspace(int64_t device, int64_t stream, void** ptr, int64_t* bytes) {
  std::lock_guard<std::mutex> lock(g_workspaces_mutex);
  for (const Workspace& w : g_workspaces)
    if (w.device == device && w.stream == stream) {
      *ptr = w.ptr;
      *bytes = w.bytes;
      return true;
    }
  return false;
}

PyObject* py_register_workspace(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4) {
    PyErr_SetString(PyExc_TypeError, "register_workspace(device, stream, pointer, bytes)");
    return nullptr;
  }
  int64_t v[4];
  for (int i = 0; i < 4; ++i) v[i] = static_cast<int64_t>(PyLong_AsUnsignedLongLongMask(args[i]));
  if (PyErr_Occurred()) return nullptr;
  std::lock_guard<std::mutex> lock(g_workspaces_mutex);
  for (Workspace& w : g_workspaces)
    if (w.device == v[0] && w.stream == v[1]) {
      w.ptr = reinterpret_cast<void*>(v[2]);
      w.bytes = v[3];
      Py_RETURN_NONE;
    }
  g_workspaces.push_back(Workspace{v[0], v[1], reinterpret_cast<void*>(v[2]), v[3]});
  Py_RETURN_NONE;
}

const at::Tensor* tensor_of(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

bool half_type(const at::Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }
uint32_t dtype_code(const at::Tensor& t) { return t.scalar_type() == at::kHalf ? B200_ATTN_F16 : B200_ATTN_BF16; }

// A plain strided CUDA tensor (no subclass tricks, nothing lazy) on `device` that needs no gradient.
bool plain(const at::Tensor& t, c10::DeviceIndex device) {
  return t.is_cuda() && t.layout() == at::kStrided && t.device().index() == device && !t.is_conj() && !t.is_neg() &&
         !(t.requires_grad() && at::GradMode::is_enabled()) && t.has_storage();
}

at::Tensor empty_like_type(at::IntArrayRef sizes, const at::Tensor& like) {
  return at::detail::empty_cuda(sizes, like.scalar_type(), like.device(), std::nullopt);
}

// A call of the library, without the interpreter's lock.
template <typename F>
int launched(F&& f) {
  PyThreadState* state = PyEval_SaveThread();
  const int rc = f();
  PyEval_RestoreThread(state);
  return rc;
}

bool number(PyObject* o, double* v) {
  *v = PyFloat_AsDouble(o);
  if (*v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// An int and nothing that converts to one, as ctypes has it for the fields these go to.
bool integer(PyObject* o, int64_t* v) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0 && *v >= INT32_MIN && *v <= INT32_MAX;
}

struct View {  // [batch, tokens, heads, 64] in either layout
  int64_t b, n, h, sb, sn, sh;
};
bool view_of(const at::Tensor& t, bool bnhd, View* v) {
  if (t.dim() != 4 || t.size(3) != kHeadDim || t.stride(3) != 1) return false;
  const int tok = bnhd ? 1 : 2, head = bnhd ? 2 : 1;
  *v = View{t.size(0), t.size(tok), t.size(head), t.stride(0), t.stride(tok), t.stride(head)};
  return v->b > 0 && v->n > 0 && v->h > 0;
}
void set_strides(int64_t* s, const View& v) {
  s[0] = v.sb;
  s[1] = v.sn;
  s[2] = v.sh;
}

// attention(q, k, v, scale | None, bnhd, schedule, out | None, bias | None, rel_h | None, rel_w | None, self_only)
PyObject* py_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 11) Py_RETURN_NONE;
  const at::Tensor *q = tensor_of(args[0]), *k = tensor_of(args[1]), *v = tensor_of(args[2]);
  if (q == nullptr || k == nullptr || v == nullptr) Py_RETURN_NONE;
  const bool bnhd = args[4] == Py_True;
  const c10::DeviceIndex device = c10::cuda::current_device();
  if (!half_type(*q) || k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || !plain(*q, device) || !plain(*k, device) || !plain(*v, device))
    Py_RETURN_NONE;
  View vq, vk, vv;
  if (!view_of(*q, bnhd, &vq) || !view_of(*k, bnhd, &vk) || !view_of(*v, bnhd, &vv)) Py_RETURN_NONE;
  if (vk.b != vq.b || vk.h != vq.h || vv.b != vq.b || vv.h != vq.h || vv.n != vk.n || (args[10] == Py_True && vk.n != vq.n)) Py_RETURN_NONE;
  if (vq.n > INT32_MAX || vk.n > INT32_MAX || vq.b > INT32_MAX || vq.h > INT32_MAX) Py_RETURN_NONE;

  B200AttnArgs a;
  std::memset(&a, 0, sizeof(a));
  a.struct_size = sizeof(a);
  a.dtype = dtype_code(*q);
  a.q = q->data_ptr();
  a.k = k->data_ptr();
  a.v = v->data_ptr();
  set_strides(a.q_stride, vq);
  set_strides(a.k_stride, vk);
  set_strides(a.v_stride, vv);
  a.batch = static_cast<int32_t>(vq.b);
  a.heads = static_cast<int32_t>(vq.h);
  a.q_tokens = static_cast<int32_t>(vq.n);
  a.kv_tokens = static_cast<int32_t>(vk.n);
  a.head_dim = kHeadDim;
  double scale = 0.125;
  if (args[3] != Py_None && !number(args[3], &scale)) Py_RETURN_NONE;
  a.scale = static_cast<float>(scale);
  int64_t schedule = 0;
  if (!integer(args[5], &schedule)) Py_RETURN_NONE;
  a.schedule = static_cast<int32_t>(schedule);

  if (args[7] != Py_None) {  // a 16-bit bias the kernel fetches in tiles; a broadcast dimension has stride 0
    const at::Tensor* bias = tensor_of(args[7]);
    if (bias == nullptr || args[8] != Py_None || !half_type(*bias) || !plain(*bias, device) || bias->dim() > 4 || bias->dim() < 2) Py_RETURN_NONE;
    int64_t size[4] = {1, 1, 1, 1}, stride[4] = {0, 0, 0, 0};
    for (int64_t i = 0, at = 4 - bias->dim(); i < bias->dim(); ++i, ++at) {
      size[at] = bias->size(i);
      stride[at] = bias->stride(i);
    }
    if (size[3] != vk.n || size[2] != vq.n || stride[3] != 1 || (size[0] != 1 && size[0] != vq.b) || (size[1] != 1 && size[1] != vq.h)) Py_RETURN_NONE;
    for (int i = 0; i < 2; ++i)
      if (size[i] == 1) stride[i] = 0;
    if (reinterpret_cast<uintptr_t>(bias->data_ptr()) % 16 != 0 || stride[0] % 8 != 0 || stride[1] % 8 != 0 || stride[2] % 8 != 0 || stride[0] < 0 ||
        stride[1] < 0 || (stride[2] <= 0 && vq.n > 1))
      Py_RETURN_NONE;
    a.bias = bias->data_ptr();
    a.bias_dtype = dtype_code(*bias);
    for (int i = 0; i < 3; ++i) a.bias_stride[i] = stride[i];
  }
  if (args[8] != Py_None) {
    const at::Tensor *rh = tensor_of(args[8]), *rw = tensor_of(args[9]);
    if (rh == nullptr || rw == nullptr || rh->scalar_type() != rw->scalar_type() || (!half_type(*rh) && rh->scalar_type() != at::kFloat) || !plain(*rh, device) ||
        !plain(*rw, device) || rh->dim() != 4 || rw->dim() != 4)
      Py_RETURN_NONE;
    for (const at::Tensor* t : {rh, rw})
      if (t->size(0) != vq.b || t->size(1) != vq.h || t->size(2) != vq.n || t->stride(3) != 1) Py_RETURN_NONE;
    if (rh->size(3) * rw->size(3) != vk.n) Py_RETURN_NONE;
    a.rel_h = rh->data_ptr();
    a.rel_w = rw->data_ptr();
    a.rel_dtype = rh->scalar_type() == at::kFloat ? B200_ATTN_F32 : dtype_code(*rh);
    a.rel_kh = static_cast<int32_t>(rh->size(3));
    a.rel_kw = static_cast<int32_t>(rw->size(3));
    for (int i = 0; i < 3; ++i) {
      a.rel_h_stride[i] = rh->stride(i);
      a.rel_w_stride[i] = rw->stride(i);
    }
  }
  const int64_t stream = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(device).stream());
  if (vk.n >= kSplitMinKeys && !find_workspace(device, stream, &a.workspace, &a.workspace_bytes)) Py_RETURN_NONE;

  at::Tensor out;
  if (args[6] == Py_None) {
    out = empty_like_type({vq.b, vq.n, vq.h, kHeadDim}, *q);
    if (!bnhd) {  // the same memory as [batch, heads, tokens, 64]
      const int64_t sizes[4] = {vq.b, vq.h, vq.n, kHeadDim}, strides[4] = {vq.n * vq.h * kHeadDim, kHeadDim, vq.h * kHeadDim, 1};
      out.unsafeGetTensorImpl()->set_sizes_and_strides(c10::IntArrayRef(sizes), c10::IntArrayRef(strides));
    }
  } else {
    const at::Tensor* given = tensor_of(args[6]);
    if (given == nullptr || given->scalar_type() != q->scalar_type() || !given->is_cuda() || given->device().index() != device || given->sizes() != q->sizes())
      Py_RETURN_NONE;
    out = *given;
  }
  View vo;
  if (!view_of(out, bnhd, &vo)) Py_RETURN_NONE;
  a.o = out.data_ptr();
  set_strides(a.o_stride, vo);
  if (launched([&] { return b200_attn_fwd(&a, reinterpret_cast<void*>(stream)); }) != B200_ATTN_OK) Py_RETURN_NONE;
  return THPVariable_Wrap(out);
}

// Row stride of `t` as [m, n] rows; false where the Python side has to look closer.
bool rows_of(const at::Tensor& t, int64_t m, int64_t n, int64_t* stride) {
  if (t.dim() < 1 || t.size(t.dim() - 1) != n || t.numel() != m * n) return false;
  if (t.is_contiguous()) {
    *stride = n;
    return true;
  }
  if (t.dim() != 2 || t.stride(1) != 1) return false;
  *stride = t.stride(0);
  return true;
}

// gemm(x, w, bias | None, act, scale | None, res | None, out | None)
PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 7) Py_RETURN_NONE;
  const at::Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]);
  if (x == nullptr || w == nullptr) Py_RETURN_NONE;
  const c10::DeviceIndex device = c10::cuda::current_device();
  if (!half_type(*x) || w->scalar_type() != x->scalar_type() || !plain(*x, device) || !plain(*w, device) || x->dim() < 1 || x->numel() == 0 || w->dim() != 2 ||
      !w->is_contiguous())
    Py_RETURN_NONE;
  const int64_t k = x->size(x->dim() - 1), m = x->numel() / k, cols = w->size(0);
  if (w->size(1) != k || m > INT32_MAX || cols > INT32_MAX || k > INT32_MAX) Py_RETURN_NONE;
  B200GemmArgs a;
  std::memset(&a, 0, sizeof(a));
  a.struct_size = sizeof(a);
  a.dtype = dtype_code(*x);
  a.m = static_cast<int32_t>(m);
  a.n = static_cast<int32_t>(cols);
  a.k = static_cast<int32_t>(k);
  int64_t act = 0;
  if (!integer(args[3], &act)) Py_RETURN_NONE;
  a.act = static_cast<int32_t>(act);
  if (!rows_of(*x, m, k, &a.lda)) Py_RETURN_NONE;
  a.x = x->data_ptr();
  a.w = w->data_ptr();
  if (args[2] != Py_None) {
    const at::Tensor* b = tensor_of(args[2]);
    if (b == nullptr || b->scalar_type() != x->scalar_type() || !plain(*b, device) || b->dim() != 1 || b->size(0) != cols || b->stride(0) != 1) Py_RETURN_NONE;
    a.bias = b->data_ptr();
  }
  if (args[4] != Py_None) {
    const at::Tensor* s = tensor_of(args[4]);
    if (s == nullptr || s->scalar_type() != at::kFloat || !plain(*s, device) || s->dim() != 1 || s->size(0) != cols || s->stride(0) != 1) Py_RETURN_NONE;
    a.scale = static_cast<const float*>(s->data_ptr());
  }
  if (args[5] != Py_None) {
    const at::Tensor* r = tensor_of(args[5]);
    if (r == nullptr || r->scalar_type() != x->scalar_type() || !plain(*r, device) || !rows_of(*r, m, cols, &a.lres)) Py_RETURN_NONE;
    a.res = r->data_ptr();
  }
  at::Tensor out;
  if (args[6] == Py_None) {
    c10::SmallVector<int64_t, 5> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = cols;
    out = empty_like_type(sizes, *x);
  } else {
    const at::Tensor* given = tensor_of(args[6]);
    if (given == nullptr || given->scalar_type() != x->scalar_type() || !plain(*given, device)) Py_RETURN_NONE;
    out = *given;
  }
  if (!rows_of(out, m, cols, &a.ldy)) Py_RETURN_NONE;
  a.y = out.data_ptr();
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(device);
  if (launched([&] { return b200_gemm(&a, stream.stream()); }) != B200_ATTN_OK) Py_RETURN_NONE;
  return THPVariable_Wrap(out);
}

// rope_qk_(qkv, cs, q_scale) -> whether it was launched
PyObject* py_rope(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) Py_RETURN_FALSE;
  const at::Tensor *x = tensor_of(args[0]), *cs = tensor_of(args[1]);
  if (x == nullptr || cs == nullptr) Py_RETURN_FALSE;
  const c10::DeviceIndex device = c10::cuda::current_device();
  if (!half_type(*x) || !plain(*x, device) || !plain(*cs, device) || x->dim() != 5 || x->size(2) != 3 || x->size(4) != kHeadDim || x->stride(4) != 1 ||
      x->numel() == 0 || cs->scalar_type() != at::kFloat || cs->dim() != 3 || cs->size(1) != 2 || cs->size(2) != kHeadDim / 2 || !cs->is_contiguous() ||
      cs->size(0) > x->size(1) || x->size(0) > INT32_MAX || x->size(1) > INT32_MAX || x->size(3) > INT32_MAX)
    Py_RETURN_FALSE;
  double scale = 1;
  if (!number(args[2], &scale)) Py_RETURN_FALSE;
  B200RopeArgs a;
  std::memset(&a, 0, sizeof(a));
  a.struct_size = sizeof(a);
  a.dtype = dtype_code(*x);
  a.q = x->data_ptr();
  a.k = static_cast<char*>(x->data_ptr()) + 2 * x->stride(2);
  for (int64_t* s : {a.q_stride, a.k_stride}) {
    s[0] = x->stride(0);
    s[1] = x->stride(1);
    s[2] = x->stride(3);
  }
  a.cs = static_cast<const float*>(cs->data_ptr());
  a.batch = static_cast<int32_t>(x->size(0));
  a.heads = static_cast<int32_t>(x->size(3));
  a.tokens = static_cast<int32_t>(x->size(1));
  a.prefix = static_cast<int32_t>(x->size(1) - cs->size(0));
  a.head_dim = kHeadDim;
  a.q_scale = static_cast<float>(scale);
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(device);
  if (launched([&] { return b200_rope_qk(&a, stream.stream()); }) != B200_ATTN_OK) Py_RETURN_FALSE;
  Py_RETURN_TRUE;
}

// sam_rel_terms(q, rel_pos_h, rel_pos_w, side)
PyObject* py_rel_terms(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4) Py_RETURN_NONE;
  const at::Tensor *q = tensor_of(args[0]), *ph = tensor_of(args[1]), *pw = tensor_of(args[2]);
  int64_t side = 0;
  if (q == nullptr || ph == nullptr || pw == nullptr || !integer(args[3], &side)) Py_RETURN_NONE;
  const c10::DeviceIndex device = c10::cuda::current_device();
  View v;
  if (!half_type(*q) || !plain(*q, device) || !view_of(*q, true, &v) || side < 2 || side > 64 || v.n != side * side || v.b > INT32_MAX || v.h > INT32_MAX) Py_RETURN_NONE;
  for (const at::Tensor* t : {ph, pw})
    if (t->scalar_type() != q->scalar_type() || !plain(*t, device) || t->dim() != 2 || t->size(0) != 2 * side - 1 || t->size(1) != kHeadDim || !t->is_contiguous())
      Py_RETURN_NONE;
  at::Tensor rel_h = empty_like_type({v.b, v.h, v.n, side}, *q), rel_w = empty_like_type({v.b, v.h, v.n, side}, *q);
  B200RelTermsArgs a;
  std::memset(&a, 0, sizeof(a));
  a.struct_size = sizeof(a);
  a.dtype = dtype_code(*q);
  a.q = q->data_ptr();
  set_strides(a.q_stride, v);
  a.rel_pos_h = ph->data_ptr();
  a.rel_pos_w = pw->data_ptr();
  a.rel_h = rel_h.data_ptr();
  a.rel_w = rel_w.data_ptr();
  a.batch = static_cast<int32_t>(v.b);
  a.heads = static_cast<int32_t>(v.h);
  a.side = static_cast<int32_t>(side);
  a.head_dim = kHeadDim;
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(device);
  if (launched([&] { return b200_sam_rel_terms(&a, stream.stream()); }) != B200_ATTN_OK) Py_RETURN_NONE;
  PyObject *h = THPVariable_Wrap(rel_h), *w = THPVariable_Wrap(rel_w);
  PyObject* pair = PyTuple_Pack(2, h, w);
  Py_DECREF(h);
  Py_DECREF(w);
  return pair;
}

// What an encoder's table of parameter addresses was made from (encoder.py: Snapshot). The tensors are held, so an address
// cannot come to mean another one while it is compared with.
struct Fact {
  at::Tensor tensor;
  const void* ptr;
  c10::SmallVector<int64_t, 4> sizes, strides;
};
using Facts = std::vector<Fact>;
constexpr const char* kFactsName = "_b200host.snapshot";

void free_facts(PyObject* capsule) { delete static_cast<Facts*>(PyCapsule_GetPointer(capsule, kFactsName)); }

// Calls f(tensor) for every value of every dictionary in the tuple `dicts`; false as soon as f says so or one is no tensor.
template <typename F>
bool for_each_tensor(PyObject* dicts, F&& f) {
  if (!PyTuple_Check(dicts)) return false;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(dicts); ++i) {
    PyObject* d = PyTuple_GET_ITEM(dicts, i);
    if (!PyDict_Check(d)) return false;
    PyObject *key = nullptr, *value = nullptr;
    for (Py_ssize_t at = 0; PyDict_Next(d, &at, &key, &value);) {
      const at::Tensor* t = tensor_of(value);
      if (t == nullptr || !t->has_storage() || !f(*t)) return false;
    }
  }
  return true;
}

// snapshot(dicts) -> capsule, or None for anything but dictionaries of plain tensors
PyObject* py_snapshot(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 1) Py_RETURN_NONE;
  auto facts = std::make_unique<Facts>();
  const auto take = [&](const at::Tensor& t) {
    facts->push_back(Fact{t, t.const_data_ptr(), {t.sizes().begin(), t.sizes().end()}, {t.strides().begin(), t.strides().end()}});
    return true;
  };
  if (!for_each_tensor(args[0], take)) Py_RETURN_NONE;
  PyObject* capsule = PyCapsule_New(facts.get(), kFactsName, free_facts);
  if (capsule != nullptr) facts.release();
  return capsule;
}

// unchanged(capsule, dicts): the same tensors in the same places
PyObject* py_unchanged(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2 || !PyCapsule_IsValid(args[0], kFactsName)) Py_RETURN_FALSE;
  const Facts& facts = *static_cast<Facts*>(PyCapsule_GetPointer(args[0], kFactsName));
  size_t i = 0;
  const auto same = [&](const at::Tensor& t) {
    if (i >= facts.size()) return false;
    const Fact& f = facts[i++];
    return t.is_same(f.tensor) && t.const_data_ptr() == f.ptr && t.sizes().equals(f.sizes) && t.strides().equals(f.strides);
  };
  if (for_each_tensor(args[1], same) && i == facts.size()) Py_RETURN_TRUE;
  Py_RETURN_FALSE;
}

// C++ exceptions (an allocation that fails) must not cross into the interpreter: the Python side runs and reports.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  try {
    return F(self, args, n);
  } catch (...) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<F>));
}

PyMethodDef methods[] = {
    {"attention", fast<py_attention>(), METH_FASTCALL, nullptr},
    {"gemm", fast<py_gemm>(), METH_FASTCALL, nullptr},
    {"rope_qk_", fast<py_rope>(), METH_FASTCALL, nullptr},
    {"sam_rel_terms", fast<py_rel_terms>(), METH_FASTCALL, nullptr},
    {"snapshot", fast<py_snapshot>(), METH_FASTCALL, nullptr},
    {"unchanged", fast<py_unchanged>(), METH_FASTCALL, nullptr},
    {"register_workspace", fast<py_register_workspace>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

#ifndef B200_SOURCE_HASH
#define B200_SOURCE_HASH "0000000000000000"
#endif
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_b200host", "b200attn-src:" B200_SOURCE_HASH, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200host(void) { return PyModule_Create(&module_def); }
