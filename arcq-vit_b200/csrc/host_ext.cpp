// Host path of the package in native code: a CPython extension over libarcq_b200 that takes torch tensors.
//
// A packed linear is two short kernels; called from Python, argument checks, stream and allocator look-ups and ctypes
// marshalling took 35 us a layer around 8 us of GPU work, and an eager ViT forward (about 250 calls) 5.5 ms around 0.7 ms.  Here
// a layer is one call (about 6 us, launches included) and the forward of a packed ViT one call that launches every kernel.
//
// Every function returns None for what it does not take (other dtypes, devices, layouts, shapes); the Python code it
// shortcuts then runs as before and raises what it always raised.  Module parameters are not copied or cached: a call
// reads the tensors out of the modules' own dictionaries, so moved, replaced or re-typed parameters are seen.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/Context.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/arcq_b200.h"

namespace {

void check(int rc, const char* what) {
  if (rc != ARCQ_OK)
    throw std::runtime_error(std::string(what) + " failed (" + std::to_string(rc) + "): " + arcq_last_error_string());
}

// Other Python threads run while a call allocates and launches: with a full launch queue that waits for the GPU.  What the call
// reads out of Python objects is read, and held, before.
struct WithoutGil {
  PyThreadState* const state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};
template <typename F> auto without_gil(F work) {
  const WithoutGil released;
  return work();
}
// The Python tensors that a call reads, kept from being replaced under it (references counted with the lock held: cheaper than
// copies of the tensors, 0.5 us a layer).
class Held {
 public:
  Held() = default;
  Held(const Held&) = delete;
  ~Held() {
    for (PyObject* o : objects_) Py_DECREF(o);
  }
  void add(PyObject* o) {
    Py_INCREF(o);
    objects_.push_back(o);
  }

 private:
  c10::SmallVector<PyObject*, 16> objects_;
};

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return ARCQ_DT_F32;
    case at::kHalf: return ARCQ_DT_F16;
    case at::kBFloat16: return ARCQ_DT_BF16;
    default: return -1;
  }
}

at::Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType t, c10::Device dev) {
  return at::detail::empty_cuda(sizes, t, dev, std::nullopt);
}

// A plain torch.Tensor or Parameter; subclasses, functorch wrappers and the like have behaviour of their own.
const at::Tensor* tensor_of(PyObject* o) {
  if (o == nullptr || !THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  using K = c10::DispatchKey;
  constexpr c10::DispatchKeySet wrappers({K::Python, K::Functionalize, K::FuncTorchBatched, K::FuncTorchGradWrapper, K::BatchedNestedTensor,
                                          K::NestedTensor});
  return t.key_set().has_any(wrappers) ? nullptr : &t;
}

// Arguments of another Python type than these are left to the Python code, which takes or refuses them as ever.
long int_of(PyObject* o) {               // -1: not an int, or out of range
  int overflow = 0;
  const long v = PyLong_Check(o) ? PyLong_AsLongAndOverflow(o, &overflow) : -1;
  return overflow != 0 ? -1 : v;
}
bool all_bools(PyObject* const* args, std::initializer_list<int> which) {
  for (int i : which)
    if (!PyBool_Check(args[i])) return false;
  return true;
}

PyObject* g_oom_error = nullptr;    // torch.OutOfMemoryError
PyObject* g_key[16];
enum Key { kPacked, kCenter, kScale, kCodeSum, kWCodebook, kACodebook, kAThresholds, kBiasTensor, kBias, kWeight, kKeys };
const char* const kKeyNames[kKeys] = {"packed_weight_codes", "weight_center", "weight_scale", "weight_code_sum", "weight_codebook",
                                      "activation_codebook", "activation_thresholds", "bias_tensor", "bias", "weight"};

// A contiguous CUDA tensor of the given type out of a module's dictionary, or null.
const at::Tensor* device_tensor(PyObject* dict, PyObject* key, at::ScalarType t, const c10::Device& dev, Held* held) {
  PyObject* const o = PyDict_GetItemWithError(dict, key);
  const at::Tensor* v = tensor_of(o);
  if (v == nullptr || v->scalar_type() != t || v->device() != dev || !v->is_contiguous()) return nullptr;
  held->add(o);
  return v;
}

// The kernels' view of one packed linear.
struct Linear {
  int64_t N, K;
  int bits;
  const float *th, *acb, *bias;
  arcq_unpack_job job;
  int64_t weight_elems() const { return N * K; }
  // 3-bit rows of an odd number of groups: the operands are those of arcq_packed_gemm, activations rebuilt with one fma
  bool one_fma() const { return K * bits / 8 % 16 != 0; }
};

bool read_linear(PyObject* buffers, Key bias_key, const c10::Device& dev, Linear* l, Held* held) {
  if (!PyDict_Check(buffers)) return false;
  const at::Tensor* codes = device_tensor(buffers, g_key[kPacked], at::kByte, dev, held);
  const at::Tensor* f[6];
  const Key keys[6] = {kCenter, kScale, kCodeSum, kWCodebook, kACodebook, kAThresholds};
  for (int i = 0; i < 6; ++i)
    if ((f[i] = device_tensor(buffers, g_key[keys[i]], at::kFloat, dev, held)) == nullptr) return false;
  if (codes == nullptr || codes->dim() != 2 || f[0]->dim() != 2) return false;
  const int64_t levels = f[3]->numel();
  l->bits = levels == 16 ? 4 : levels == 8 ? 3 : levels == 4 ? 2 : 0;
  l->N = f[0]->size(0);
  l->K = f[0]->size(1) * 64;
  if (l->bits == 0 || l->N % 16 != 0 || l->N == 0 || l->K == 0 || codes->size(0) != l->N || codes->size(1) != l->K * l->bits / 8 ||
      f[1]->numel() != f[0]->numel() || f[2]->numel() != f[0]->numel() || f[4]->numel() != levels || f[5]->numel() != levels - 1)
    return false;
  PyObject* const bias = PyDict_GetItemWithError(buffers, g_key[bias_key]);
  const at::Tensor* b = tensor_of(bias);
  if (b == nullptr) return false;                          // no bias is an empty tensor; not among the buffers: a parameter, say
  l->bias = nullptr;
  if (b->numel() > 0) {
    if (b->scalar_type() != at::kFloat || b->device() != dev || !b->is_contiguous() || b->numel() != l->N) return false;
    l->bias = b->const_data_ptr<float>();
  }
  l->acb = f[4]->const_data_ptr<float>();
  l->th = f[5]->const_data_ptr<float>();
  l->job = arcq_unpack_job{codes->const_data_ptr<uint8_t>(), f[0]->const_data_ptr<float>(), f[1]->const_data_ptr<float>(),
                           f[2]->const_data_ptr<float>(), f[3]->const_data_ptr<float>(), nullptr, l->N, l->K, l->bits};
  held->add(bias);
  return (reinterpret_cast<uintptr_t>(l->job.packed) & 3u) == 0;
}

// ---------------------------------------------------------------- one packed linear
// linear(buffers, x, bias key 0 "bias_tensor" / 1 "bias", fp32 output, pre_gelu, pre_quantized) -> y or None
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  const at::Tensor* x = n == 6 ? tensor_of(args[1]) : nullptr;
  if (x == nullptr || !x->is_cuda() || x->dim() < 1 || !x->is_contiguous() || !all_bools(args, {2, 3, 4, 5})) Py_RETURN_NONE;
  const bool float_chain = args[3] == Py_True, pre_gelu = args[4] == Py_True, ready = args[5] == Py_True;
  const int xt = dtype_code(x->scalar_type());
  if (xt < 0 || (!float_chain && xt != ARCQ_DT_F16) || ((pre_gelu || ready) && xt != ARCQ_DT_F16)) Py_RETURN_NONE;
  Linear l;
  Held held;
  if (!read_linear(args[0], args[2] == Py_True ? kBias : kBiasTensor, x->device(), &l, &held)) Py_RETURN_NONE;
  const int64_t numel = x->numel();
  if (x->size(-1) != l.K || numel == 0 || !aligned16(x->const_data_ptr()) || (ready && l.one_fma())) Py_RETURN_NONE;
  const int64_t M = numel / l.K;
  at::Tensor y = without_gil([&] {
    const c10::cuda::CUDAGuard guard(x->device());
    void* const st = c10::cuda::getCurrentCUDAStream().stream();
    c10::SmallVector<int64_t, 5> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = l.N;
    const auto out = [&] { return empty_cuda(sizes, float_chain ? at::kFloat : at::kHalf, x->device()); };
    const int yt = float_chain ? ARCQ_DT_F32 : ARCQ_DT_F16;
    // few rows: one launch, no scratch; in a graph, which has no host time to save, only where the GPU needs less for it (the default
    // stream cannot be captured: 0.2 us for the question)
    if (!ready && arcq_packed_linear_small_applies(M, l.N, l.K) &&
        (st == nullptr || c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None ||
         arcq_packed_linear_small_applies_captured(M, l.N, l.K))) {
      at::Tensor y = out();
      check(arcq_packed_linear_small(pre_gelu, x->const_data_ptr(), xt, M, l.th, l.acb, l.one_fma(), &l.job, l.bias, y.mutable_data_ptr(), yt, st),
            "arcq_packed_linear_small");
      return y;
    }
    // the reconstructed activation and the unpacked weight, given back to the caching allocator on return
    const at::Tensor scratch = empty_cuda({(ready ? 0 : numel) + l.weight_elems() + 8}, at::kHalf, x->device());
    at::Half* const w16 = scratch.mutable_data_ptr<at::Half>();
    const void* xhat = x->const_data_ptr();
    l.job.out = w16;
    if (ready) {
      check(arcq_unpack_weight_f16(l.job.packed, l.job.mu, l.job.sigma, l.job.codesum, l.job.codebook, l.bits, 64, l.N, l.K, w16, st),
            "arcq_unpack_weight_f16");
    } else {
      void* const xh = w16 + l.weight_elems();
      check(arcq_act_quant_unpack(pre_gelu, xhat, xt, M, l.K, l.th, l.acb, l.bits, 64, xh, ARCQ_DT_F16, l.one_fma(), &l.job, 1, st),
            "arcq_act_quant");
      xhat = xh;
    }
    at::Tensor y = out();
    check(arcq_dense_weight_gemm(xhat, w16, l.bias, M, l.N, l.K, y.mutable_data_ptr(), yt, st), "arcq_dense_weight_gemm");
    return y;
  });
  return THPVariable_Wrap(std::move(y));
}

// ---------------------------------------------------------------- operators
// quantize_activation(x, thresholds, codebook, bits, want_code_sum, pre_gelu) -> (packed, center, scale, code_sum) or None
PyObject* quantize_activation(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6) Py_RETURN_NONE;
  const at::Tensor *x = tensor_of(args[0]), *th = tensor_of(args[1]), *cb = tensor_of(args[2]);
  if (x == nullptr || th == nullptr || cb == nullptr || !x->is_cuda() || x->dim() != 2 || !x->is_contiguous()) Py_RETURN_NONE;
  const long bits = int_of(args[3]);
  const int xt = dtype_code(x->scalar_type());
  for (const at::Tensor* t : {th, cb})
    if (t->scalar_type() != at::kFloat || t->device() != x->device() || !t->is_contiguous()) Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1);
  if (xt < 0 || bits < 2 || bits > 4 || cb->numel() != (1 << bits) || th->numel() != (1 << bits) - 1 || M == 0 || K == 0 || K % 64 != 0)
    Py_RETURN_NONE;
  if (!all_bools(args, {4, 5})) Py_RETURN_NONE;
  const bool want_cs = args[4] == Py_True, pre_gelu = args[5] == Py_True;
  at::Tensor packed, mu, sg, cs;
  without_gil([&] {
    const c10::cuda::CUDAGuard guard(x->device());
    packed = empty_cuda({M, K * bits / 8}, at::kByte, x->device());
    mu = empty_cuda({M, K / 64}, at::kFloat, x->device());
    sg = empty_cuda({M, K / 64}, at::kFloat, x->device());
    if (want_cs) cs = empty_cuda({M, K / 64}, at::kFloat, x->device());
    check((pre_gelu ? arcq_gelu_act_quant : arcq_act_quant)(
              x->const_data_ptr(), xt, M, K, th->const_data_ptr<float>(), cb->const_data_ptr<float>(), static_cast<int>(bits), 64,
              packed.mutable_data_ptr<uint8_t>(), mu.mutable_data_ptr<float>(), sg.mutable_data_ptr<float>(),
              want_cs ? cs.mutable_data_ptr<float>() : nullptr, nullptr, 0, c10::cuda::getCurrentCUDAStream().stream()),
          "arcq_act_quant");
  });
  PyObject* out = PyTuple_New(4);
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(packed)));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(std::move(mu)));
  PyTuple_SET_ITEM(out, 2, THPVariable_Wrap(std::move(sg)));
  if (want_cs) {
    PyTuple_SET_ITEM(out, 3, THPVariable_Wrap(std::move(cs)));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(out, 3, Py_None);
  }
  return out;
}

// dequant(packed, center, scale, code_sum, codebook, bits, fp32 output) -> [R, K] or None (group size 64)
PyObject* dequant(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 7) Py_RETURN_NONE;
  const at::Tensor* t[5];
  for (int i = 0; i < 5; ++i) {
    t[i] = tensor_of(args[i]);
    if (t[i] == nullptr || !t[i]->is_cuda() || !t[i]->is_contiguous() || t[i]->scalar_type() != (i == 0 ? at::kByte : at::kFloat) ||
        t[i]->device() != t[0]->device())
      Py_RETURN_NONE;
  }
  const long bits = int_of(args[5]);
  if (bits < 2 || bits > 4 || t[0]->dim() != 2 || t[1]->dim() != 2) Py_RETURN_NONE;
  const int64_t R = t[1]->size(0), K = t[1]->size(1) * 64;
  if (R == 0 || K == 0 || t[0]->size(0) != R || t[0]->size(1) != K * bits / 8 || t[2]->numel() != t[1]->numel() ||
      t[3]->numel() != t[1]->numel() || t[4]->numel() != (1 << bits))
    Py_RETURN_NONE;
  if (!all_bools(args, {6})) Py_RETURN_NONE;
  const bool f32 = args[6] == Py_True;
  at::Tensor out = without_gil([&] {
    const c10::cuda::CUDAGuard guard(t[0]->device());
    at::Tensor out = empty_cuda({R, K}, f32 ? at::kFloat : at::kHalf, t[0]->device());
    check(arcq_dequant(t[0]->const_data_ptr<uint8_t>(), t[1]->const_data_ptr<float>(), t[2]->const_data_ptr<float>(),
                       t[3]->const_data_ptr<float>(), t[4]->const_data_ptr<float>(), static_cast<int>(bits), 64, R, K,
                       out.mutable_data_ptr(), f32 ? ARCQ_DT_F32 : ARCQ_DT_F16, c10::cuda::getCurrentCUDAStream().stream()),
          "arcq_dequant");
    return out;
  });
  return THPVariable_Wrap(std::move(out));
}

// ---------------------------------------------------------------- the library's attention
// Whether nothing was chosen about it: all back ends allowed, in the order that the framework settles on.  It does so when it is first
// asked for a back end, whatever the order was until then; after that, the order that it starts with is a choice like any other.  So
// where that order stands it is asked, once, about tensors without elements.
bool back_ends_as_they_come() {
  using B = at::SDPBackend;
  using Order = std::array<B, at::num_sdp_backends>;
  constexpr Order initial = {B::flash_attention, B::efficient_attention, B::math, B::cudnn_attention, B::overrideable};
  constexpr Order settled = {B::cudnn_attention, B::flash_attention, B::efficient_attention, B::math, B::overrideable};
  at::Context& ctx = at::globalContext();
  if (!ctx.userEnabledFlashSDP() || !ctx.userEnabledMemEfficientSDP() || !ctx.userEnabledMathSDP() || !ctx.userEnabledCuDNNSDP())
    return false;
  if (ctx.sDPPriorityOrder() == initial) {
    if (c10::cuda::device_count() == 0) return true;
    static std::once_flag asked;
    std::call_once(asked, [] {
      const c10::impl::ExcludeDispatchKeyGuard unseen(c10::python_ks);       // no operator of the program's
      const at::Tensor none = at::empty({1, 1, 0, 64}, at::TensorOptions().dtype(at::kHalf).device(at::kCUDA));
      at::_fused_sdp_choice(none, none, none);
    });
  }
  return ctx.sDPPriorityOrder() == settled;
}
// attention_back_ends_as_they_come() -> bool
PyObject* attention_back_ends_as_they_come(PyObject*, PyObject* const*, Py_ssize_t) { return PyBool_FromLong(back_ends_as_they_come()); }

// ---------------------------------------------------------------- the forward of a packed ViT
// The data of a framework operator's fp16 result, which the kernels read as a dense matrix.
const void* half_matrix(const at::Tensor& t, int64_t elems, const c10::Device& dev) {
  TORCH_CHECK(t.scalar_type() == at::kHalf && t.device() == dev && t.is_contiguous() && t.numel() == elems,
              "a framework operator of the ViT forward returned ", t.scalar_type(), " ", t.sizes(), " on ", t.device());
  return t.const_data_ptr();
}

// What a plan holds are references to the dictionaries of the model's modules and, in `watch`, every plain value and module that
// it was made from; no tensors.  A call compares all of `watch` first, so that a plan is never used for another model than the
// one it describes.
struct Norm {
  PyObject* params;             // _parameters of the LayerNorm
  double eps;
};
struct VitBlock {
  Norm norm1, norm2;
  PyObject *qkv, *proj, *fc1, *fc2;   // _buffers
};
struct VitPlan {
  int64_t dim, heads, patch;
  PyObject *own, *patch_params, *head_params;      // _parameters of the model, of patch_embed.proj and of head
  std::vector<VitBlock> blocks;
  Norm norm;
  std::vector<PyObject*> watch;       // (dict, key, expected value) triples; None: absent or None
  std::vector<PyObject*> empty;       // hook dictionaries that have to be empty
  std::vector<PyObject*> refs;
  ~VitPlan() {
    for (PyObject* o : refs) Py_XDECREF(o);
  }
};

// The kernels' view of one LayerNorm, parameters as the module holds them.
struct NormView {
  const void *gamma, *beta;
  int dtype;
};
bool read_norm(const Norm& n, const c10::Device& dev, int64_t dim, NormView* v, Held* held) {
  const void* p[2];
  for (int i = 0; i < 2; ++i) {
    PyObject* const o = PyDict_GetItemWithError(n.params, g_key[i ? kBias : kWeight]);
    const at::Tensor* t = tensor_of(o);
    if (t == nullptr || t->device() != dev || t->numel() != dim || !t->is_contiguous() || !aligned16(t->const_data_ptr())) return false;
    const int d = dtype_code(t->scalar_type());
    if (d < 0 || (i == 1 && d != v->dtype)) return false;
    v->dtype = d;
    held->add(o);
    p[i] = t->const_data_ptr();
  }
  v->gamma = p[0];
  v->beta = p[1];
  return true;
}

void free_plan(PyObject* capsule) { delete static_cast<VitPlan*>(PyCapsule_GetPointer(capsule, "arcq_vit_plan")); }

// vit_plan(dim, heads, patch, own params, patch params, head params, final norm (params, eps),
//          blocks [(norm1 params, eps, norm2 params, eps, qkv, proj, fc1, fc2 buffers)], watch [dict, key, value, ...], empty [dict])
PyObject* vit_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 11) {
    PyErr_SetString(PyExc_TypeError, "vit_plan takes 11 arguments");
    return nullptr;
  }
  auto* p = new VitPlan;
  auto keep = [&](PyObject* o) {
    Py_INCREF(o);
    p->refs.push_back(o);
    return o;
  };
  p->dim = PyLong_AsLongLong(a[0]);
  p->heads = PyLong_AsLongLong(a[1]);
  p->patch = PyLong_AsLongLong(a[2]);
  p->own = keep(a[3]);
  p->patch_params = keep(a[4]);
  p->head_params = keep(a[5]);
  p->norm.params = keep(a[6]);
  p->norm.eps = PyFloat_AsDouble(a[7]);
  for (Py_ssize_t i = 0; i < PyList_Size(a[8]); ++i) {
    PyObject* t = PyList_GetItem(a[8], i);
    VitBlock b;
    b.norm1.params = keep(PyTuple_GetItem(t, 0));
    b.norm1.eps = PyFloat_AsDouble(PyTuple_GetItem(t, 1));
    b.norm2.params = keep(PyTuple_GetItem(t, 2));
    b.norm2.eps = PyFloat_AsDouble(PyTuple_GetItem(t, 3));
    b.qkv = keep(PyTuple_GetItem(t, 4));
    b.proj = keep(PyTuple_GetItem(t, 5));
    b.fc1 = keep(PyTuple_GetItem(t, 6));
    b.fc2 = keep(PyTuple_GetItem(t, 7));
    p->blocks.push_back(std::move(b));
  }
  for (Py_ssize_t i = 0; i < PyList_Size(a[9]); ++i) p->watch.push_back(keep(PyList_GetItem(a[9], i)));
  for (Py_ssize_t i = 0; i < PyList_Size(a[10]); ++i) p->empty.push_back(keep(PyList_GetItem(a[10], i)));
  if (PyErr_Occurred()) {
    delete p;
    return nullptr;
  }
  return PyCapsule_New(p, "arcq_vit_plan", free_plan);
}

// vit_forward(plan, images) -> logits; None: not a call the plan covers; False: the model has changed, the plan is void
PyObject* vit_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) Py_RETURN_NONE;
  auto* p = static_cast<VitPlan*>(PyCapsule_GetPointer(args[0], "arcq_vit_plan"));
  if (p == nullptr) return nullptr;
  for (size_t i = 0; i < p->watch.size(); i += 3) {
    PyObject* const got = PyDict_GetItemWithError(p->watch[i], p->watch[i + 1]);
    if (got != p->watch[i + 2] && !(got == nullptr && p->watch[i + 2] == Py_None)) Py_RETURN_FALSE;
  }
  const at::Tensor* img = tensor_of(args[1]);
  if (img == nullptr || !img->is_cuda() || img->scalar_type() != at::kHalf || img->dim() != 4 || !img->is_contiguous() ||
      img->numel() == 0 || !aligned16(img->const_data_ptr()))
    Py_RETURN_NONE;
  // autocast to another type changes what the framework's linear and attention below take and give
  if (at::autocast::is_autocast_enabled(at::kCUDA) && at::autocast::get_autocast_dtype(at::kCUDA) != at::kHalf) Py_RETURN_NONE;
  for (PyObject* d : p->empty)
    if (PyDict_Size(d) != 0) Py_RETURN_NONE;
  const c10::Device dev = img->device();
  const int64_t B = img->size(0), C = img->size(1), H = img->size(2), W = img->size(3), P = p->patch, D = p->dim;
  if (H % P != 0 || W % P != 0) Py_RETURN_NONE;
  const int64_t T = (H / P) * (W / P) + 1, M = B * T;

  static PyObject* const k_cls = PyUnicode_InternFromString("cls_token");
  static PyObject* const k_pos = PyUnicode_InternFromString("pos_embed");
  Held held;
  const at::Tensor *cls = device_tensor(p->own, k_cls, at::kHalf, dev, &held), *pos = device_tensor(p->own, k_pos, at::kHalf, dev, &held);
  const at::Tensor* pw = device_tensor(p->patch_params, g_key[kWeight], at::kHalf, dev, &held);
  const at::Tensor* pb = device_tensor(p->patch_params, g_key[kBias], at::kHalf, dev, &held);
  const at::Tensor* hw = device_tensor(p->head_params, g_key[kWeight], at::kHalf, dev, &held);
  const at::Tensor* hb = device_tensor(p->head_params, g_key[kBias], at::kHalf, dev, &held);
  for (const at::Tensor* t : {cls, pos})
    if (t == nullptr || !aligned16(t->const_data_ptr())) Py_RETURN_NONE;
  if (pw == nullptr || pb == nullptr || hw == nullptr || hb == nullptr || cls->numel() != D || pos->numel() != T * D ||
      pw->numel() != D * C * P * P)
    Py_RETURN_NONE;
  const size_t depth = p->blocks.size();
  std::vector<Linear> lin(4 * depth);
  std::vector<NormView> norms(2 * depth + 1);
  int64_t scratch_elems[2] = {0, 0};                       // qkv + proj, fc1 + fc2
  for (size_t i = 0; i < depth; ++i) {
    VitBlock& b = p->blocks[i];
    PyObject* const d[4] = {b.qkv, b.proj, b.fc1, b.fc2};
    const int64_t shape[4][2] = {{3 * D, D}, {D, D}, {4 * D, D}, {D, 4 * D}};
    for (int k = 0; k < 4; ++k) {
      Linear& l = lin[4 * i + k];
      if (!read_linear(d[k], kBiasTensor, dev, &l, &held)) Py_RETURN_NONE;
      // any hidden width, the rest as the block's structure fixes it
      if (k < 2 ? (l.N != shape[k][0] || l.K != shape[k][1]) : k == 2 ? l.K != D : (l.N != D || l.K != lin[4 * i + 2].N)) Py_RETURN_NONE;
    }
    scratch_elems[0] = std::max(scratch_elems[0], lin[4 * i].weight_elems() + lin[4 * i + 1].weight_elems());
    scratch_elems[1] = std::max(scratch_elems[1], lin[4 * i + 2].weight_elems() + lin[4 * i + 3].weight_elems());
    if (!read_norm(b.norm1, dev, D, &norms[2 * i], &held) || !read_norm(b.norm2, dev, D, &norms[2 * i + 1], &held)) Py_RETURN_NONE;
  }
  if (!read_norm(p->norm, dev, D, &norms[2 * depth], &held)) Py_RETURN_NONE;
  // The attention kernel, which also quantises for proj, instead of the library's attention and a quantizer launch: a whole forward
  // of DeiT-S batch 64 1552 -> 1466 us, batch 8 679 -> 634, batch 1 488 -> 467, DeiT-T batch 37 785 -> 724, DeiT-B batch 256 14.14 ->
  // 13.89 ms.  The library's where a sequence is too long for the kernel, and where its back ends were chosen among.
  const bool own_attention = T <= 256 && D == 64 * p->heads && back_ends_as_they_come();
  int64_t hidden = 0;
  for (size_t i = 0; i < depth; ++i) hidden = std::max(hidden, lin[4 * i + 2].N);

  at::Tensor logits = without_gil([&] {
    const c10::cuda::CUDAGuard guard(dev);
    void* const st = c10::cuda::getCurrentCUDAStream().stream();
    // one workspace: residual stream (two, written in turn), reconstruction, branch output, qkv / fc1 output, fc2 input, weights
    const int64_t wide = std::max<int64_t>(3 * D, hidden);
    const at::Tensor ws = empty_cuda({M * (4 * D + wide + hidden) + scratch_elems[0] + scratch_elems[1] + 64}, at::kHalf, dev);
    at::Half* at_ptr = ws.mutable_data_ptr<at::Half>();
    auto take = [&](int64_t elems) {
      at::Half* r = at_ptr;
      at_ptr += (elems + 7) / 8 * 8;
      return r;
    };
    at::Half *x = take(M * D), *x_next = take(M * D), *xhat = take(M * D), *branch = take(M * D), *mid = take(M * wide), *xhat4 = take(M * hidden);
    at::Half *w_attn = take(scratch_elems[0]), *w_mlp = take(scratch_elems[1]);
    for (size_t i = 0; i < depth; ++i) {
      lin[4 * i].job.out = w_attn;
      lin[4 * i + 1].job.out = w_attn + lin[4 * i].weight_elems();
      lin[4 * i + 2].job.out = w_mlp;
      lin[4 * i + 3].job.out = w_mlp + lin[4 * i + 2].weight_elems();
    }
    // Where the weights of a half block (qkv + proj, fc1 + fc2) are unpacked.  Few rows: by the GEMM that ends the half block
    // before, on the SMs it leaves idle, while it reads the other scratch matrix; what has no room there by the half block's own
    // first GEMM (its second weight) or the LayerNorm.  Many rows: the GEMMs fill the machine, and extra blocks of the LayerNorm
    // + quantizer launch do it.
    const bool beside_gemm = arcq_unpack_beside_gemm(M, D) != 0;
    int done = 0;                        // of the next half block's two weights
    auto jobs_of = [&](const Linear* half, int from, int to, arcq_unpack_job (&jobs)[2]) {
      for (int k = from; k < to; ++k) jobs[k - from] = half[k].job;
      return to - from;
    };
    // what the GEMM of a layer can take along, asked once per shape
    struct Room {
      int64_t N, K, values;
      int gelu_quant;
    };
    std::vector<Room> rooms;
    auto room_of = [&](const Linear& l, int gelu_quant) {
      for (const Room& r : rooms)
        if (r.N == l.N && r.K == l.K && r.gelu_quant == gelu_quant) return r.values;
      rooms.push_back({l.N, l.K, arcq_dense_weight_gemm_unpack_room(M, l.N, l.K, gelu_quant), gelu_quant});
      return rooms.back().values;
    };
    // how far the weights of `half` from `from` on fit into what the GEMM of `l` can take along
    auto fits = [&](const Linear* half, int from, const Linear& l, int gelu_quant) {
      if (!beside_gemm || half == nullptr) return from;
      int64_t room = room_of(l, gelu_quant);
      while (from < 2 && half[from].weight_elems() <= room) room -= half[from++].weight_elems();
      return from;
    };
    auto norm_quant = [&](const at::Half* y, const NormView& nv, double eps, const Linear* half, int gelu_quant) {
      // the first weight has to be there before the half block's first GEMM, the second may be that GEMM's job
      const int first = std::max(done, 1), to = fits(half, first, half[0], gelu_quant) == 2 ? first : 2;
      arcq_unpack_job jobs[2];
      const int n = jobs_of(half, done, to, jobs);
      check(arcq_add_layernorm_act_quant_unpack(x, y, nv.gamma, nv.beta, nv.dtype, static_cast<float>(eps), M, D, half[0].th, half[0].acb,
                                                half[0].bits, 64, y != nullptr ? x_next : nullptr, nullptr, xhat, half[0].one_fma(), jobs,
                                                n, st),
            "arcq_add_layernorm_act_quant");
      if (y != nullptr) std::swap(x, x_next);
      done = to;
    };
    auto gemm = [&](const at::Half* a, const Linear& l, at::Half* y, const arcq_unpack_job* jobs, int n) {
      check(arcq_dense_weight_gemm_unpack(a, l.job.out, l.bias, M, l.N, l.K, y, ARCQ_DT_F16, jobs, n, st), "arcq_dense_weight_gemm");
    };
    // The last GEMM of a half block; next: the linears of the next one, or null.  Both weights in two rounds of the idle SMs'
    // threads, or the second one left to the next GEMM if that has room.
    auto last_gemm = [&](const at::Half* a, const Linear& l, at::Half* y, const Linear* next, int next_gelu_quant) {
      arcq_unpack_job jobs[2];
      done = fits(next, 0, l, 0);
      if (done == 2 && next[0].weight_elems() + next[1].weight_elems() > room_of(l, 0) * 2 / 5 && fits(next, 1, next[0], next_gelu_quant) == 2)
        done = 1;
      gemm(a, l, y, jobs, jobs_of(next, 0, done, jobs));
    };

    {
      const at::Tensor rows = empty_cuda({B * (T - 1), C * P * P}, at::kHalf, dev);
      check(arcq_patchify(img->const_data_ptr(), B, C, H, W, static_cast<int>(P), rows.mutable_data_ptr(), st), "arcq_patchify");
      const at::Tensor patches = at::linear(rows, pw->view({D, C * P * P}), *pb);
      check(arcq_assemble_tokens(half_matrix(patches, B * (T - 1) * D, dev), cls->const_data_ptr(), pos->const_data_ptr(), B, T - 1, D, x,
                                 st),
            "arcq_assemble_tokens");
    }
    const at::Half* y = nullptr;
    int64_t asked[2] = {0, 0};            // the shape of fc1 that `applies` holds for
    bool applies = false;
    for (size_t i = 0; i < depth; ++i) {
      const VitBlock& b = p->blocks[i];
      const Linear *qkv = &lin[4 * i], *proj = qkv + 1, *fc1 = qkv + 2, *fc2 = qkv + 3;
      if (asked[0] != fc1->N || asked[1] != fc1->K) {
        applies = arcq_dense_weight_gemm_gelu_quant_applies(M, fc1->N, fc1->K) != 0;
        asked[0] = fc1->N;
        asked[1] = fc1->K;
      }
      const bool fused = applies && !fc2->one_fma();     // the fused form reconstructs in three steps only
      arcq_unpack_job jobs[2];
      norm_quant(y, norms[2 * i], b.norm1.eps, qkv, 0);
      gemm(xhat, *qkv, mid, jobs, jobs_of(qkv, done, 2, jobs));
      if (own_attention) {
        check(arcq_attention_act_quant_form(mid, B, T, p->heads, 64, proj->th, proj->acb, proj->bits, 64, xhat, proj->one_fma(), st),
              "arcq_attention_act_quant");
      } else {
        const at::Tensor t = at::from_blob(mid, {B, T, 3, p->heads, D / p->heads}, at::TensorOptions().dtype(at::kHalf).device(dev));
        const at::Tensor r = t.permute({2, 0, 3, 1, 4});
        const at::Tensor o = at::scaled_dot_product_attention(r[0], r[1], r[2]).transpose(1, 2).reshape({M, D}).contiguous();
        check(arcq_act_quant_unpack(0, half_matrix(o, M * D, dev), ARCQ_DT_F16, M, D, proj->th, proj->acb, proj->bits, 64, xhat,
                                    ARCQ_DT_F16, proj->one_fma(), nullptr, 0, st),
              "arcq_act_quant");
      }
      last_gemm(xhat, *proj, branch, fc1, fused);
      norm_quant(branch, norms[2 * i + 1], b.norm2.eps, fc1, fused);
      const int n = jobs_of(fc1, done, 2, jobs);
      if (fused) {
        check(arcq_dense_weight_gemm_gelu_quant(xhat, fc1->job.out, fc1->bias, M, fc1->N, fc1->K, fc2->th, fc2->acb, fc2->bits, 64, xhat4,
                                                jobs, n, st),
              "arcq_dense_weight_gemm_gelu_quant");
      } else {
        gemm(xhat, *fc1, mid, jobs, n);
        check(arcq_act_quant_unpack(1, mid, ARCQ_DT_F16, M, fc2->K, fc2->th, fc2->acb, fc2->bits, 64, xhat4, ARCQ_DT_F16, fc2->one_fma(),
                                    nullptr, 0, st),
              "arcq_gelu_act_quant");
      }
      last_gemm(xhat4, *fc2, branch, i + 1 < depth ? qkv + 4 : nullptr, 0);
      y = branch;
    }
    // the head reads the class token of every image only
    const at::Tensor h = empty_cuda({B, D}, at::kHalf, dev);
    const NormView& nv = norms[2 * depth];
    check(arcq_add_layernorm_strided(x, y, nv.gamma, nv.beta, nv.dtype, static_cast<float>(p->norm.eps), B, D, T * D, nullptr,
                                     h.mutable_data_ptr(), st),
          "arcq_add_layernorm");
    return at::linear(h, *hw, *hb);
  });
  return THPVariable_Wrap(std::move(logits));
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  if (F != &vit_plan && F != &attention_back_ends_as_they_come && c10::impl::TorchDispatchModeTLS::any_modes_set()) Py_RETURN_NONE;      // the mode wants to see the operators
  try {
    return F(self, args, n);
  } catch (const c10::OutOfMemoryError& e) {
    PyErr_SetString(g_oom_error, e.what_without_backtrace());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}
#define ARCQ_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<f>)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {ARCQ_METHOD(linear), ARCQ_METHOD(quantize_activation), ARCQ_METHOD(dequant), ARCQ_METHOD(vit_plan),
                           ARCQ_METHOD(vit_forward), ARCQ_METHOD(attention_back_ends_as_they_come), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_arcq_host", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__arcq_host() {
  for (int i = 0; i < kKeys; ++i)
    if ((g_key[i] = PyUnicode_InternFromString(kKeyNames[i])) == nullptr) return nullptr;
  PyObject* const torch = PyImport_ImportModule("torch");
  if (torch == nullptr || (g_oom_error = PyObject_GetAttrString(torch, "OutOfMemoryError")) == nullptr) return nullptr;
  Py_DECREF(torch);
  return PyModule_Create(&g_module);
}
