// Steady-state host path of the eager operators: one native call from Python per convolution.
//
// A conv2d call used to spend 20-25 us of host time in Python (argument checks, a plan key of twenty tuples, ctypes
// marshalling of fourteen arguments), more than the small layers' kernels take: a 53-convolution network of small
// images was bound by it (1250 us of host time for 530 us of kernels).  Here the tensors' metadata is read through
// torch's C++ API, the plan is looked up by its value, the output is allocated and the C ABI is called.
//
// Every function answers None for a call it does not take (wrong types, devices or shapes, tensor subclasses, string
// padding, empty results, a residual that cannot be fused); the Python implementation then runs, raises the
// documented errors, or takes the slow route.  Nothing is remembered about tensors: plans are kept by geometry,
// strides and alignment (at most kMaxPlans of them), and filters that need packing are either packed into a buffer of
// this call (small ones of NCHW layers, by the launch that relays x out) or looked up by the Python-side cache through the
// callback given to bind().
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/core/DeviceGuard.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <cstring>
#include <unordered_map>

#include "../../../include/flagdnn_b200.h"

namespace {

using QueryFn = int (*)(const fdnn_conv_desc*, const void*, const void*, const void*, fdnn_conv_plan*);
using FwdFn = int (*)(const fdnn_conv_desc*, const void*, const void*, const void*, const void*, const void*, const void*,
                      int, void*, void*, int64_t, void*, int64_t, void*);
QueryFn g_query = nullptr;
FwdFn g_fwd = nullptr;
using FwdUnpackedFn = int (*)(const fdnn_conv_desc*, const void*, const void*, void*, int64_t, const void*, const void*, const void*,
                              int, void*, void*, int64_t, void*);
FwdUnpackedFn g_fwd_unpacked = nullptr;
PyObject* g_packed_weight = nullptr;   // (weight, address of desc, address of plan, stream, y address) -> packed tensor

// The descriptor (all plain integers), the alignment of x, w and y, and the device.
struct PlanKey {
  fdnn_conv_desc desc;
  int32_t align[3];
  int32_t device;
  bool operator==(const PlanKey& o) const { return std::memcmp(this, &o, sizeof *this) == 0; }
};
struct PlanHash {
  size_t operator()(const PlanKey& k) const {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&k);
    uint64_t h = 0x9e3779b97f4a7c15ull;
    for (size_t i = 0; i < sizeof(PlanKey) / 4; ++i) h = (h ^ w[i]) * 0x100000001b3ull;
    return size_t(h ^ (h >> 29));
  }
};
static_assert(sizeof(fdnn_conv_desc) % 4 == 0 && sizeof(PlanKey) % 4 == 0, "hashed and compared by words");
constexpr size_t kMaxPlans = 1024;
// Packing a filter of up to a megabyte in the launch that relays an NCHW x out costs less than the look-up of a kept one, which
// is Python code, as long as the GPU is done before the host: calls of 64 -> 64 3x3 bf16 on one 14 x 14 image 8.6 us against
// 10.5, on 4 x 56 x 56 8.7 and 10.6, 128 -> 128 on 8 x 28 x 28 10.4 and 11.4, fp32 64 -> 64 on 4 x 56 x 56 through a graph 13.7 and 15.8.
// Beyond some 12 us of GPU time the look-up is hidden and the packing is not: 128 -> 128 on 32 x 28 x 28 16.5 and 15.5, fp32
// 64 -> 64 on 8 x 56 x 56 21.9 and 20.9.
constexpr int64_t kPackAlways = 1 << 20;
// Under capture they are packed on the way at any size: replays then read the filter as it is, not as it was.
bool pack_on_the_way(const fdnn_conv_plan& plan, int dtype) {
  if (plan.packed_weight_bytes > kPackAlways) return false;
  return (plan.bytes <= 1e7 && plan.flops <= (dtype == FDNN_F32 ? 1e9 : 3e9)) ||
         c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
}
std::unordered_map<PlanKey, fdnn_conv_plan, PlanHash>& plans() {   // used with the GIL held
  static auto* m = new std::unordered_map<PlanKey, fdnn_conv_plan, PlanHash>();
  return *m;
}

// nullptr: not a plain strided CUDA tensor (subclasses and other layouts take the Python route).  The tensors belong to
// the caller's arguments, which outlive the call.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_conj() || t.is_neg())
    return nullptr;   // (tensors without storage: wrappers of function transforms)
  return &t;
}

// An int, or two of them.
bool pair_of(PyObject* o, int64_t (&v)[2]) {
  auto one = [](PyObject* p, int64_t* out) {
    if (!PyLong_Check(p)) return false;
    *out = PyLong_AsLongLong(p);
    if (*out == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    return *out >= 0 && *out <= 1 << 30;
  };
  if (PyLong_Check(o)) {
    if (!one(o, &v[0])) return false;
    v[1] = v[0];
    return true;
  }
  if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 2) return false;
  return one(PyTuple_GET_ITEM(o, 0), &v[0]) && one(PyTuple_GET_ITEM(o, 1), &v[1]);
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return FDNN_F16;
    case at::kBFloat16: return FDNN_BF16;
    case at::kFloat: return FDNN_F32;
    default: return -1;
  }
}

int64_t out_dim(int64_t in, int64_t pad, int64_t dil, int64_t k, int64_t stride) {
  const int64_t span = in + 2 * pad - dil * (k - 1) - 1;
  return span < 0 ? 0 : span / stride + 1;
}

// A per-channel vector: nullptr pointer for None; false if the call is not ours.
bool vector_of(PyObject* o, const at::Tensor& x, int64_t k, const void** ptr) {
  *ptr = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = plain(o);
  if (t == nullptr || t->dim() != 1 || t->numel() != k || t->scalar_type() != x.scalar_type() ||
      t->device() != x.device() || !t->is_contiguous())
    return false;
  *ptr = t->const_data_ptr();
  return true;
}

PyObject* none() { Py_RETURN_NONE; }

// Other Python threads may run while this one allocates and launches (an allocation can wait for the device).
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// Runs one planned convolution; `weight_obj` is the tensor the packed-filter cache knows, or nullptr when the filter is
// a view made for this call (packed into a buffer of this call then).  Returns 0 or the C ABI's status; -1 with a Python
// error set.
int launch(const fdnn_conv_desc& d, const at::Tensor& x, const at::Tensor& w, PyObject* weight_obj, const void* bias,
           const void* scale, const void* residual, int act, const at::Tensor& y) {
  const void *xp = x.const_data_ptr(), *wp = w.const_data_ptr();
  void* yp = y.mutable_data_ptr();
  PlanKey key;
  std::memset(&key, 0, sizeof key);
  key.desc = d;
  key.align[0] = int(reinterpret_cast<uintptr_t>(xp) % 16);
  key.align[1] = int(reinterpret_cast<uintptr_t>(wp) % 16);
  key.align[2] = int(reinterpret_cast<uintptr_t>(yp) % 16);
  key.device = x.get_device();
  auto& cache = plans();
  auto it = cache.find(key);
  if (it == cache.end()) {
    fdnn_conv_plan plan;
    const int st = g_query(&d, xp, wp, yp, &plan);
    if (st != FDNN_OK) return st;
    if (cache.size() >= kMaxPlans) cache.clear();
    it = cache.emplace(key, plan).first;
  }
  const fdnn_conv_plan plan = it->second;   // a copy: the callback below may run other Python code
  void* stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
  at::Tensor scratch;
  PyObject* held = nullptr;
  const void* packed_ptr = nullptr;
  if (plan.algo != FDNN_ALGO_DIRECT && plan.w_packed) {
    const bool in_relayout = plan.x_repacked && d.groups == 1 && plan.low_channel == 0 && plan.pixel_group <= 1 && d.c >= 8 &&
                             d.x_strides[3] == 1 && d.x_strides[1] != 1 && d.w > 1 && pack_on_the_way(plan, d.dtype);
    if (weight_obj == nullptr || in_relayout) {
      WithoutGil free;
      const int64_t ws_bytes = (plan.workspace_bytes + 255) / 256 * 256, bytes = ws_bytes + plan.packed_weight_bytes;
      scratch = at::empty({bytes}, x.options().dtype(at::kByte));
      char* base = static_cast<char*>(scratch.mutable_data_ptr());
      return g_fwd_unpacked(&d, xp, wp, base + ws_bytes, plan.packed_weight_bytes, bias, scale, residual, act, yp, base, bytes, stream);
    }
    held = PyObject_CallFunction(g_packed_weight, "OKKKK", weight_obj, (unsigned long long)(uintptr_t)&d,
                                 (unsigned long long)(uintptr_t)&plan, (unsigned long long)(uintptr_t)stream,
                                 (unsigned long long)(uintptr_t)yp);
    if (held == nullptr) return -1;
    packed_ptr = THPVariable_Unpack(held).const_data_ptr();
  }
  int st;
  try {
    WithoutGil free;
    void* ws = nullptr;
    if (plan.workspace_bytes > 0) {
      // from the caching allocator, which hands the block out again in this stream's order
      scratch = at::empty({plan.workspace_bytes}, x.options().dtype(at::kByte));
      ws = scratch.mutable_data_ptr();
    }
    st = g_fwd(&d, xp, wp, packed_ptr, bias, scale, residual, act, yp, ws, plan.workspace_bytes, nullptr, 0, stream);
  } catch (...) {
    Py_XDECREF(held);
    throw;
  }
  Py_XDECREF(held);
  return st;
}

PyObject* finish(int status, at::Tensor&& y) {
  if (status == -1) return nullptr;
  if (status != FDNN_OK) return PyLong_FromLong(status);   // the caller raises with the C ABI's message
  return THPVariable_Wrap(std::move(y));
}

// conv(input, weight, bias, scale, residual, stride, padding, dilation, groups, algo, activation)
PyObject* fast_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS   // C++ exceptions leave as the Python types torch gives them (torch.OutOfMemoryError among them)
  if (n != 11 || g_fwd_unpacked == nullptr) return none();
    const at::Tensor *x = plain(a[0]), *w = plain(a[1]);
    if (x == nullptr || w == nullptr || x->dim() != 4 || w->dim() != 4) return none();
    const int dtype = dtype_code(x->scalar_type());
    if (dtype < 0 || w->scalar_type() != x->scalar_type() || w->device() != x->device()) return none();
    int64_t stride[2], pad[2], dil[2];
    if (!pair_of(a[5], stride) || !pair_of(a[6], pad) || !pair_of(a[7], dil) || !PyLong_Check(a[8])) return none();
    const int64_t groups = PyLong_AsLongLong(a[8]);
    if (stride[0] < 1 || stride[1] < 1 || dil[0] < 1 || dil[1] < 1 || groups < 1) {
      PyErr_Clear();
      return none();
    }
    const auto xs = x->sizes(), ws = w->sizes();
    const int64_t k = ws[0];
    for (int i = 0; i < 4; ++i)
      if (xs[i] < 1 || ws[i] < 1 || xs[i] > 0x7fffffff || ws[i] > 0x7fffffff) return none();
    if (xs[1] % groups != 0 || k % groups != 0 || ws[1] != xs[1] / groups) return none();
    const int64_t oh = out_dim(xs[2], pad[0], dil[0], ws[2], stride[0]), ow = out_dim(xs[3], pad[1], dil[1], ws[3], stride[1]);
    if (oh < 1 || ow < 1) return none();
    const void *bias, *scale, *residual = nullptr;
    if (!vector_of(a[2], *x, k, &bias) || !vector_of(a[3], *x, k, &scale)) return none();
    const int64_t algo = PyLong_AsLongLong(a[9]), act = PyLong_AsLongLong(a[10]);

    c10::DeviceGuard guard(x->device());
    at::Tensor y;
    {
      WithoutGil free;
      y = at::empty({xs[0], k, oh, ow}, x->options().requires_grad(false),
                    x->stride(1) == 1 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::Contiguous);
    }
    if (a[4] != Py_None) {
      const at::Tensor* r = plain(a[4]);
      if (r == nullptr || r->scalar_type() != y.scalar_type() || r->device() != y.device() || r->sizes() != y.sizes() ||
          r->strides() != y.strides())
        return none();
      residual = r->const_data_ptr();
      if (reinterpret_cast<uintptr_t>(residual) % 16 != reinterpret_cast<uintptr_t>(y.const_data_ptr()) % 16) return none();
      if (xs[1] <= 4) return none();   // the low-channel path adds a residual in a second step
    }
    fdnn_conv_desc d;
    std::memset(&d, 0, sizeof d);
    d.dtype = dtype;
    d.n = int(xs[0]); d.c = int(xs[1]); d.h = int(xs[2]); d.w = int(xs[3]);
    d.k = int(k); d.r = int(ws[2]); d.s = int(ws[3]);
    d.stride_h = int(stride[0]); d.stride_w = int(stride[1]);
    d.pad_top = d.pad_bottom = int(pad[0]);
    d.pad_left = d.pad_right = int(pad[1]);
    d.dil_h = int(dil[0]); d.dil_w = int(dil[1]);
    d.groups = int(groups);
    d.algo = int(algo);
    for (int i = 0; i < 4; ++i) {
      d.x_strides[i] = x->stride(i);
      d.w_strides[i] = w->stride(i);
      d.y_strides[i] = y.stride(i);
    }
    const int st = launch(d, *x, *w, a[1], bias, scale, residual, int(act), y);
    return finish(st, std::move(y));
  END_HANDLE_TH_ERRORS
}

// conv1d(input [N, C, L], weight, bias, stride, padding, dilation, groups, algo): the 2-D call with H = R = 1
PyObject* fast_conv1d(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS   // C++ exceptions leave as the Python types torch gives them (torch.OutOfMemoryError among them)
  if (n != 8 || g_fwd_unpacked == nullptr) return none();
    const at::Tensor *x = plain(a[0]), *w = plain(a[1]);
    if (x == nullptr || w == nullptr || x->dim() != 3 || w->dim() != 3) return none();
    const int dtype = dtype_code(x->scalar_type());
    if (dtype < 0 || w->scalar_type() != x->scalar_type() || w->device() != x->device()) return none();
    if (x->requires_grad() || w->requires_grad()) return none();
    int64_t v[4];
    for (int i = 0; i < 4; ++i) {
      if (!PyLong_Check(a[3 + i])) return none();
      v[i] = PyLong_AsLongLong(a[3 + i]);
      if (PyErr_Occurred()) {
        PyErr_Clear();
        return none();
      }
    }
    const int64_t stride = v[0], pad = v[1], dil = v[2], groups = v[3];
    if (stride < 1 || pad < 0 || dil < 1 || groups < 1 || stride > 1 << 30 || pad > 1 << 30 || dil > 1 << 30) return none();
    const auto xs = x->sizes(), ws = w->sizes();
    for (int i = 0; i < 3; ++i)
      if (xs[i] < 1 || ws[i] < 1 || xs[i] > 0x7fffffff || ws[i] > 0x7fffffff) return none();
    if (xs[1] % groups != 0 || ws[0] % groups != 0 || ws[1] != xs[1] / groups) return none();
    const int64_t k = ws[0], ol = out_dim(xs[2], pad, dil, ws[2], stride);
    if (ol < 1) return none();
    const void* bias;
    if (!vector_of(a[2], *x, k, &bias)) return none();
    if (a[2] != Py_None && THPVariable_Unpack(a[2]).requires_grad()) return none();
    const int64_t algo = PyLong_AsLongLong(a[7]);

    c10::DeviceGuard guard(x->device());
    const bool rows = x->stride(1) == 1;   // channels contiguous: so are y's
    at::Tensor y;
    {
      WithoutGil free;
      y = rows ? at::empty_strided({xs[0], k, ol}, {ol * k, 1, k}, x->options()) : at::empty({xs[0], k, ol}, x->options());
    }
    fdnn_conv_desc d;
    std::memset(&d, 0, sizeof d);
    d.dtype = dtype;
    d.n = int(xs[0]); d.c = int(xs[1]); d.h = 1; d.w = int(xs[2]);
    d.k = int(k); d.r = 1; d.s = int(ws[2]);
    d.stride_h = 1; d.stride_w = int(stride);
    d.pad_left = d.pad_right = int(pad);
    d.dil_h = 1; d.dil_w = int(dil);
    d.groups = int(groups);
    d.algo = int(algo);
    const at::Tensor* t[3] = {x, w, &y};
    int64_t* to[3] = {d.x_strides, d.w_strides, d.y_strides};
    for (int i = 0; i < 3; ++i) {
      to[i][0] = t[i]->stride(0);
      to[i][1] = t[i]->stride(1);
      to[i][2] = t[i]->size(2) * t[i]->stride(2);
      to[i][3] = t[i]->stride(2);
    }
    const int st = launch(d, *x, *w, nullptr, bias, nullptr, nullptr, FDNN_ACT_NONE, y);
    return finish(st, std::move(y));
  END_HANDLE_TH_ERRORS
}

// mm(a [M, K], b [K, N], algo): a 1x1 convolution over one row of M pixels whose filter is b transposed
PyObject* fast_mm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS   // C++ exceptions leave as the Python types torch gives them (torch.OutOfMemoryError among them)
  if (n != 3 || g_fwd_unpacked == nullptr) return none();
    const at::Tensor *x = plain(a[0]), *w = plain(a[1]);
    if (x == nullptr || w == nullptr || x->dim() != 2 || w->dim() != 2) return none();
    const int dtype = dtype_code(x->scalar_type());
    if (dtype < 0 || w->scalar_type() != x->scalar_type() || w->device() != x->device()) return none();
    const int64_t m = x->size(0), k = x->size(1), nn = w->size(1);
    if (w->size(0) != k || m < 1 || k < 1 || nn < 1 || m > 0x7fffffff || k > 0x7fffffff || nn > 0x7fffffff) return none();
    const int64_t algo = PyLong_AsLongLong(a[2]);
    c10::DeviceGuard guard(x->device());
    at::Tensor y;
    {
      WithoutGil free;
      y = at::empty({m, nn}, x->options().requires_grad(false));
    }
    fdnn_conv_desc d;
    std::memset(&d, 0, sizeof d);
    d.dtype = dtype;
    d.n = 1; d.c = int(k); d.h = 1; d.w = int(m);
    d.k = int(nn); d.r = 1; d.s = 1;
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1;
    d.groups = 1;
    d.algo = int(algo);
    d.x_strides[0] = d.x_strides[2] = m * x->stride(0);
    d.x_strides[1] = x->stride(1);
    d.x_strides[3] = x->stride(0);
    d.w_strides[0] = w->stride(1);
    d.w_strides[1] = w->stride(0);
    d.w_strides[2] = d.w_strides[3] = 1;
    d.y_strides[0] = d.y_strides[2] = m * nn;
    d.y_strides[1] = 1;
    d.y_strides[3] = nn;
    const int st = launch(d, *x, *w, nullptr, nullptr, nullptr, nullptr, FDNN_ACT_NONE, y);
    return finish(st, std::move(y));
  END_HANDLE_TH_ERRORS
}

// bind(query, pack, fwd: addresses of the C ABI's functions, packed_weight: callback, version of the loaded library and the
// sizes of the two structures as the caller knows them): refuses a library or caller of another ABI than this file's.
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long q, p, f, desc_bytes, plan_bytes;
  int version;
  PyObject* cb;
  if (!PyArg_ParseTuple(args, "KKKOiKK", &q, &p, &f, &cb, &version, &desc_bytes, &plan_bytes)) return nullptr;
  if (version != FDNN_ABI_VERSION || desc_bytes != sizeof(fdnn_conv_desc) || plan_bytes != sizeof(fdnn_conv_plan)) {
    PyErr_Format(PyExc_ImportError, "compiled for version %d of the C ABI (structures of %zu and %zu bytes), given %d (%llu and %llu)",
                 FDNN_ABI_VERSION, sizeof(fdnn_conv_desc), sizeof(fdnn_conv_plan), version, desc_bytes, plan_bytes);
    return nullptr;
  }
  Py_INCREF(cb);
  Py_XDECREF(g_packed_weight);
  g_packed_weight = cb;
  (void)p;   // fdnn_conv2d_pack_weight: the packed-filter callback calls it
  g_query = reinterpret_cast<QueryFn>(uintptr_t(q));
  g_fwd = reinterpret_cast<FwdFn>(uintptr_t(f));
  return none();
}

// bind_unpacked(address of fdnn_conv2d_fwd_unpacked), after bind()
PyObject* bind_unpacked(PyObject*, PyObject* arg) {
  const unsigned long long f = PyLong_AsUnsignedLongLong(arg);
  if (PyErr_Occurred()) return nullptr;
  g_fwd_unpacked = reinterpret_cast<FwdUnpackedFn>(uintptr_t(f));
  return none();
}

PyMethodDef kMethods[] = {
    {"conv", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fast_conv)), METH_FASTCALL, nullptr},
    {"conv1d", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fast_conv1d)), METH_FASTCALL, nullptr},
    {"mm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fast_mm)), METH_FASTCALL, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {"bind_unpacked", bind_unpacked, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// `built_for`: the torch this was compiled against (the build compares it with the installed one, and the loader too).
PyMODINIT_FUNC PyInit__fastcall() {
  PyObject* m = PyModule_Create(&kModule);
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", FDNN_HOST_TAG) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
