// Python binding of the hot entry points: the tensor checks, the output allocation and the call into the C ABI of
// include/b200_attn.h as compiled code.
//
// What bounds a small call is the host: done in Python, one layer of an eager decode step (two checked calls through
// ctypes) costs 29 us while its two kernels take about 11 us on the GPU.  Every function here takes its arguments
// positionally (METH_FASTCALL), reads sizes and strides from the TensorImpl, allocates the output without going
// through the dispatcher and releases the GIL around the launch.  The rules checked, and the exception types, are
// those of the Python layer (AssertionError for a tensor that does not fit, RuntimeError for a CPU tensor,
// B200AttnError for a status of the library).
#include <Python.h>

#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <utility>
#include <vector>

#include "../../include/b200_attn.h"

namespace {

using at::Tensor;

#define REQUIRE(cond, msg)                            \
  do {                                                \
    if (!(cond)) {                                    \
      PyErr_SetString(PyExc_AssertionError, msg);     \
      return nullptr;                                 \
    }                                                 \
  } while (0)

#define NEED_ARGS(n, name)                                                                           \
  do {                                                                                               \
    if (nargs != (n)) {                                                                              \
      PyErr_Format(PyExc_TypeError, name "() takes %d arguments (%zd given)", (n), nargs);           \
      return nullptr;                                                                                \
    }                                                                                                \
  } while (0)

// The tensor behind a Python object, or nullptr with TypeError set.
const Tensor* tensor_of(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor, not %s", what, Py_TYPE(o)->tp_name);
    return nullptr;
  }
  return &THPVariable_Unpack(o);
}

bool all_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t && !t->is_cuda()) {
      PyErr_SetString(PyExc_RuntimeError, "nanovllm_b200 kernels take CUDA tensors only (there is no CPU path)");
      return false;
    }
  return true;
}

// A non-zero status of the library as nanovllm_b200._lib.B200AttnError (the message is kept per thread).
PyObject* raise_status(int rc) {
  PyObject* mod = PyImport_ImportModule("nanovllm_b200._lib");
  if (!mod) return nullptr;
  PyObject* r = PyObject_CallMethod(mod, "check", "i", rc);
  Py_DECREF(mod);
  if (r) {
    Py_DECREF(r);
    PyErr_Format(PyExc_RuntimeError, "libb200attn status %d", rc);
  }
  return nullptr;
}

void* stream_ptr() { return static_cast<void*>(c10::cuda::getCurrentCUDAStream().stream()); }

Tensor empty_like_rows(at::IntArrayRef sizes, const Tensor& like) {
  return at::detail::empty_cuda(sizes, like.scalar_type(), like.device(), std::nullopt);
}

#define LAUNCH(call)                       \
  do {                                     \
    int rc_;                               \
    Py_BEGIN_ALLOW_THREADS                 \
    rc_ = (call);                          \
    Py_END_ALLOW_THREADS                   \
    if (rc_ != 0) return raise_status(rc_); \
  } while (0)

// The functions below return non-null on success; the returned value is a borrowed marker.
PyObject* const kFine = Py_None;

// ---- store_kvcache (nanovllm/layers/attention.py:33-40) ------------------------------------------------------
PyObject* check_store(const Tensor& key, const Tensor& value, const Tensor& kc, const Tensor& vc, const Tensor& slots) {
  if (key.dim() != 3) {
    PyErr_SetString(PyExc_ValueError, "store_kvcache: key must be (tokens, kv heads, head_dim)");
    return nullptr;
  }
  const int64_t d = key.size(2), row = key.size(1) * d;
  REQUIRE(value.dim() == 3 && key.stride(2) == 1 && value.stride(2) == 1, "key and value rows must be contiguous");
  REQUIRE(key.stride(1) == d && value.stride(1) == d, "key and value heads must be contiguous");
  REQUIRE(kc.dim() > 1 && vc.dim() > 1 && kc.stride(1) == row && vc.stride(1) == row, "cache rows must be kv heads x head_dim");
  REQUIRE(slots.numel() == key.size(0), "slot_mapping must have one entry per token");
  REQUIRE(key.scalar_type() == value.scalar_type() && key.scalar_type() == kc.scalar_type() &&
              key.scalar_type() == vc.scalar_type(), "key, value and caches must have one dtype");
  REQUIRE(slots.scalar_type() == at::kInt, "slot_mapping must be int32");
  return all_cuda({&key, &value, &kc, &vc, &slots}) ? kFine : nullptr;
}

PyObject* do_store(const Tensor& key, const Tensor& value, const Tensor& kc, const Tensor& vc, const Tensor& slots) {
  if (!check_store(key, value, kc, vc, slots)) return nullptr;
  const int64_t n = key.size(0), row = key.size(1) * key.size(2);
  if (n == 0) return kFine;
  LAUNCH(b200_store_kvcache(key.data_ptr(), value.data_ptr(), key.stride(0), value.stride(0), kc.data_ptr(), vc.data_ptr(),
                            static_cast<const int32_t*>(slots.data_ptr()), static_cast<int32_t>(n), static_cast<int32_t>(row),
                            static_cast<int32_t>(key.element_size()), kc.numel() / row, stream_ptr()));
  return kFine;
}

// ---- decode (nanovllm/layers/attention.py:71-74) -------------------------------------------------------------
constexpr int kDecodeWorkspaceBatch = 512;   // the library splits larger batches into launches of at most this many

// One zero-initialised workspace per (device, query heads per kv head); layers run back to back on a stream and share
// it.  Allocated on first use (the engine's eager warm-up precedes graph capture); the GIL guards the table, which
// lives until the process ends.
const Tensor* decode_workspace(const Tensor& q, int h, int hkv, int d) {
  static auto* table = new std::map<std::pair<int, int>, Tensor>();
  const std::pair<int, int> key(q.get_device(), hkv > 0 ? h / hkv : 0);
  auto it = table->find(key);
  if (it == table->end()) {
    const int64_t bytes = b200_decode_workspace_bytes(kDecodeWorkspaceBatch, h, hkv, d);
    if (bytes < 0) {
      raise_status(static_cast<int>(bytes));
      return nullptr;
    }
    it = table->emplace(key, at::zeros({bytes}, at::TensorOptions().dtype(at::kByte).device(q.device()))).first;
  }
  return &it->second;
}

// `slots` given: the step's rows k and v (one per sequence) go to the caches first.
PyObject* do_decode(const Tensor& q, const Tensor& kc, const Tensor& vc, const Tensor& lens, const Tensor& bt, double scale,
                    int hkv, const Tensor* k, const Tensor* v, const Tensor* slots, Tensor* result) {
  if (slots && !check_store(*k, *v, kc, vc, *slots)) return nullptr;
  if (q.dim() != 3) {
    PyErr_SetString(PyExc_ValueError, "decode_attention: q must be (batch, heads, head_dim)");
    return nullptr;
  }
  if (!all_cuda({&q, &kc, &vc, &lens, &bt})) return nullptr;
  const int64_t b = q.size(0), h = q.size(1), d = q.size(2);
  REQUIRE(q.scalar_type() == at::kBFloat16 && kc.scalar_type() == at::kBFloat16 && vc.scalar_type() == at::kBFloat16,
          "q and caches must be bf16");
  REQUIRE(q.stride(2) == 1 && q.stride(1) == d, "query heads must be contiguous");
  REQUIRE(kc.dim() == 4 && kc.is_contiguous() && vc.is_contiguous(), "caches must be contiguous (blocks, block size, kv heads, head_dim)");
  REQUIRE(lens.scalar_type() == at::kInt && bt.scalar_type() == at::kInt, "context_lens and block_tables must be int32");
  REQUIRE(bt.dim() == 2 && bt.stride(1) == 1 && lens.dim() == 1 && lens.stride(0) == 1, "context_lens and block-table rows must be contiguous");
  Tensor out = empty_like_rows({b, 1, h, d}, q);
  if (b > 0) {
    const Tensor* ws = decode_workspace(q, static_cast<int>(h), hkv, static_cast<int>(d));
    if (!ws) return nullptr;
    if (slots) {
      LAUNCH(b200_store_decode_attn(q.data_ptr(), q.stride(0), k->data_ptr(), v->data_ptr(), k->stride(0), v->stride(0),
                                    static_cast<const int32_t*>(slots->data_ptr()), kc.data_ptr(), vc.data_ptr(), kc.size(0),
                                    static_cast<int32_t>(kc.size(1)), static_cast<const int32_t*>(bt.data_ptr()), bt.stride(0),
                                    static_cast<int32_t>(bt.size(1)), static_cast<const int32_t*>(lens.data_ptr()), out.data_ptr(),
                                    ws->data_ptr(), ws->numel(), static_cast<int32_t>(b), static_cast<int32_t>(h), hkv,
                                    static_cast<int32_t>(d), static_cast<float>(scale), stream_ptr()));
      *result = std::move(out);
      return kFine;
    }
    LAUNCH(b200_decode_attn(q.data_ptr(), q.stride(0), kc.data_ptr(), vc.data_ptr(), kc.size(0), static_cast<int32_t>(kc.size(1)),
                            static_cast<const int32_t*>(bt.data_ptr()), bt.stride(0), static_cast<int32_t>(bt.size(1)),
                            static_cast<const int32_t*>(lens.data_ptr()), out.data_ptr(), ws->data_ptr(), ws->numel(),
                            static_cast<int32_t>(b), static_cast<int32_t>(h), hkv, static_cast<int32_t>(d),
                            static_cast<float>(scale), stream_ptr()));
  }
  *result = std::move(out);
  return kFine;
}

// ---- prefill (nanovllm/layers/attention.py:64-70) ------------------------------------------------------------
// `slots` given (dense K/V): k and v also go to the caches kc and vc.
PyObject* do_prefill(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu_q, const Tensor& cu_k, int max_q,
                     int max_k, double scale, int hkv, const Tensor* bt, int variant, const Tensor* kc, const Tensor* vc,
                     const Tensor* slots, Tensor* result) {
  if (slots && !check_store(k, v, *kc, *vc, *slots)) return nullptr;
  if (q.dim() != 3) {
    PyErr_SetString(PyExc_ValueError, "prefill_attention: q must be (tokens, heads, head_dim)");
    return nullptr;
  }
  if (!all_cuda({&q, &k, &v, &cu_q, &cu_k, bt})) return nullptr;
  const int64_t tq = q.size(0), h = q.size(1), d = q.size(2);
  REQUIRE(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16,
          "q, k and v must be bf16");
  REQUIRE(q.stride(2) == 1 && q.stride(1) == d, "query heads must be contiguous");
  REQUIRE(cu_q.scalar_type() == at::kInt && cu_k.scalar_type() == at::kInt, "cu_seqlens must be int32");
  Tensor out = empty_like_rows({tq, h, d}, q);
  const int64_t batch = cu_q.numel() - 1;
  if (slots && (tq == 0 || batch <= 0)) {
    if (!do_store(k, v, *kc, *vc, *slots)) return nullptr;
  } else if (tq > 0 && batch > 0) {
    const int32_t* cq = static_cast<const int32_t*>(cu_q.data_ptr());
    const int32_t* ck = static_cast<const int32_t*>(cu_k.data_ptr());
    if (bt) {
      REQUIRE(bt->scalar_type() == at::kInt && bt->dim() == 2 && bt->stride(1) == 1, "block_tables must be int32 with contiguous rows");
      REQUIRE(k.is_contiguous() && v.is_contiguous() && k.dim() == 4, "caches must be contiguous (blocks, block size, kv heads, head_dim)");
      LAUNCH(b200_prefill_attn(q.data_ptr(), q.stride(0), nullptr, nullptr, 0, 0, 0, k.data_ptr(), v.data_ptr(), k.size(0),
                               static_cast<int32_t>(k.size(1)), static_cast<const int32_t*>(bt->data_ptr()), bt->stride(0),
                               static_cast<int32_t>(bt->size(1)), cq, ck, static_cast<int32_t>(batch), static_cast<int32_t>(tq),
                               max_q, max_k, out.data_ptr(), static_cast<int32_t>(h), hkv, static_cast<int32_t>(d),
                               static_cast<float>(scale), variant, stream_ptr()));
    } else {
      REQUIRE(k.dim() == 3 && v.dim() == 3 && k.stride(2) == 1 && v.stride(2) == 1 && k.stride(1) == d && v.stride(1) == d,
              "key and value heads must be contiguous");
      if (slots) {
        const int64_t row = k.size(1) * d;
        LAUNCH(b200_store_prefill_attn(q.data_ptr(), q.stride(0), k.data_ptr(), v.data_ptr(), k.stride(0), v.stride(0), k.size(0),
                                       kc->data_ptr(), vc->data_ptr(), static_cast<const int32_t*>(slots->data_ptr()), kc->numel() / row,
                                       cq, ck, static_cast<int32_t>(batch), static_cast<int32_t>(tq), max_q, max_k, out.data_ptr(),
                                       static_cast<int32_t>(h), hkv, static_cast<int32_t>(d), static_cast<float>(scale), stream_ptr()));
        *result = std::move(out);
        return kFine;
      }
      LAUNCH(b200_prefill_attn(q.data_ptr(), q.stride(0), k.data_ptr(), v.data_ptr(), k.stride(0), v.stride(0), k.size(0),
                               nullptr, nullptr, 0, 0, nullptr, 0, 0, cq, ck, static_cast<int32_t>(batch),
                               static_cast<int32_t>(tq), max_q, max_k, out.data_ptr(), static_cast<int32_t>(h), hkv,
                               static_cast<int32_t>(d), static_cast<float>(scale), variant, stream_ptr()));
    }
  }
  *result = std::move(out);
  return kFine;
}

// ---- module functions ----------------------------------------------------------------------------------------
bool as_int(PyObject* o, int* v) {
  const long x = PyLong_AsLong(o);
  if (x == -1 && PyErr_Occurred()) {
    // what int() takes and __index__ does not (a float, a 0-dim tensor)
    PyErr_Clear();
    PyObject* i = PyNumber_Long(o);
    if (!i) return false;
    const long y = PyLong_AsLong(i);
    Py_DECREF(i);
    if (y == -1 && PyErr_Occurred()) return false;
    *v = static_cast<int>(y);
    return true;
  }
  *v = static_cast<int>(x);
  return true;
}
bool as_double(PyObject* o, double* v) {
  *v = PyFloat_AsDouble(o);
  return !(*v == -1.0 && PyErr_Occurred());
}

PyObject* py_store_kvcache(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(5, "store_kvcache");
  const Tensor* t[5];
  static const char* names[5] = {"key", "value", "k_cache", "v_cache", "slot_mapping"};
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = tensor_of(a[i], names[i]))) return nullptr;
  if (!do_store(*t[0], *t[1], *t[2], *t[3], *t[4])) return nullptr;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* py_decode_attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(7, "decode_attention");
  const Tensor* t[5];
  static const char* names[5] = {"q", "k_cache", "v_cache", "context_lens", "block_tables"};
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = tensor_of(a[i], names[i]))) return nullptr;
  double scale;
  int hkv;
  if (!as_double(a[5], &scale) || !as_int(a[6], &hkv)) return nullptr;
  Tensor out;
  if (!do_decode(*t[0], *t[1], *t[2], *t[3], *t[4], scale, hkv, nullptr, nullptr, nullptr, &out)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyObject* py_prefill_attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(11, "prefill_attention");
  const Tensor* t[5];
  static const char* names[5] = {"q", "k", "v", "cu_seqlens_q", "cu_seqlens_k"};
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = tensor_of(a[i], names[i]))) return nullptr;
  int max_q, max_k, hkv, variant;
  double scale;
  const Tensor* bt = nullptr;
  if (!as_int(a[5], &max_q) || !as_int(a[6], &max_k) || !as_double(a[7], &scale) || !as_int(a[8], &hkv)) return nullptr;
  if (a[9] != Py_None && !(bt = tensor_of(a[9], "block_tables"))) return nullptr;
  if (!as_int(a[10], &variant)) return nullptr;
  Tensor out;
  if (!do_prefill(*t[0], *t[1], *t[2], *t[3], *t[4], max_q, max_k, scale, hkv, bt, variant, nullptr, nullptr, nullptr, &out)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// A new reference released at scope end.
struct Ref {
  PyObject* o;
  explicit Ref(PyObject* p) : o(p) {}
  ~Ref() { Py_XDECREF(o); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};

PyObject *s_is_prefill, *s_cu_q, *s_cu_k, *s_max_q, *s_max_k, *s_slots, *s_lens, *s_bt;

// attention_forward(q, k, v, k_cache, v_cache, context, scale, num_kv_heads, already_stored): the body of
// Attention.forward, the step's metadata read from `context` (nanovllm/utils/context.py).
PyObject* py_attention_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(9, "attention_forward");
  const Tensor* t[5];
  static const char* names[5] = {"q", "k", "v", "k_cache", "v_cache"};
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = tensor_of(a[i], names[i]))) return nullptr;
  PyObject* ctx = a[5];
  double scale;
  int hkv;
  if (!as_double(a[6], &scale) || !as_int(a[7], &hkv)) return nullptr;
  const int stored = PyObject_IsTrue(a[8]);
  if (stored < 0) return nullptr;
  Ref is_prefill(PyObject_GetAttr(ctx, s_is_prefill)), bt_o(PyObject_GetAttr(ctx, s_bt));
  if (!is_prefill.o || !bt_o.o) return nullptr;
  const int prefill = PyObject_IsTrue(is_prefill.o);
  if (prefill < 0) return nullptr;
  const bool store = !stored && t[3]->numel() && t[4]->numel();
  Ref slots_o(store ? PyObject_GetAttr(ctx, s_slots) : nullptr);
  const Tensor* slots = nullptr;
  if (store) {
    if (!slots_o.o || !(slots = tensor_of(slots_o.o, "slot_mapping"))) return nullptr;
    // (bf16 with the layer's own head count stores and attends in one call: dense prefill, and decode with a row per sequence)
    const bool together = (prefill ? bt_o.o == Py_None : t[1]->dim() == 3 && t[0]->dim() == 3 && t[1]->size(0) == t[0]->size(0) && t[1]->size(0) > 0 && t[3]->dim() == 4 && t[3]->size(2) == hkv) &&
                          t[1]->dim() == 3 && t[1]->size(1) == hkv && t[0]->dim() == 3 && t[0]->size(2) == t[1]->size(2) &&
                          t[1]->scalar_type() == at::kBFloat16 && t[0]->scalar_type() == at::kBFloat16;
    if (!together) {
      if (!do_store(*t[1], *t[2], *t[3], *t[4], *slots)) return nullptr;
      slots = nullptr;
    }
  }
  Tensor out;
  if (prefill) {
    Ref cu_q_o(PyObject_GetAttr(ctx, s_cu_q)), cu_k_o(PyObject_GetAttr(ctx, s_cu_k));
    Ref max_q_o(PyObject_GetAttr(ctx, s_max_q)), max_k_o(PyObject_GetAttr(ctx, s_max_k));
    if (!cu_q_o.o || !cu_k_o.o || !max_q_o.o || !max_k_o.o) return nullptr;
    const Tensor *cu_q = tensor_of(cu_q_o.o, "cu_seqlens_q"), *cu_k = cu_q ? tensor_of(cu_k_o.o, "cu_seqlens_k") : nullptr;
    int max_q, max_k;
    if (!cu_k || !as_int(max_q_o.o, &max_q) || !as_int(max_k_o.o, &max_k)) return nullptr;
    const Tensor* bt = nullptr;
    if (bt_o.o != Py_None && !(bt = tensor_of(bt_o.o, "block_tables"))) return nullptr;
    // prefix cache: keys and values come from the cache
    if (!do_prefill(*t[0], bt ? *t[3] : *t[1], bt ? *t[4] : *t[2], *cu_q, *cu_k, max_q, max_k, scale, hkv, bt, 0, t[3], t[4], slots,
                    &out))
      return nullptr;
  } else {
    Ref lens_o(PyObject_GetAttr(ctx, s_lens));
    if (!lens_o.o) return nullptr;
    const Tensor *lens = tensor_of(lens_o.o, "context_lens"), *bt = lens ? tensor_of(bt_o.o, "block_tables") : nullptr;
    if (!bt || !do_decode(*t[0], *t[3], *t[4], *lens, *bt, scale, hkv, t[1], t[2], slots, &out)) return nullptr;
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// qk_norm_rope_store(qkv, positions, q_weight, k_weight, cos_sin_cache, eps, num_heads, num_kv_heads, k_cache, v_cache,
// slot_mapping) -> (q, k, v); the last three may be None.
PyObject* py_qk_norm_rope_store(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(11, "qk_norm_rope_store");
  const Tensor* t[5];
  static const char* names[5] = {"qkv", "positions", "q_weight", "k_weight", "cos_sin_cache"};
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = tensor_of(a[i], names[i]))) return nullptr;
  double eps;
  int h, hkv;
  if (!as_double(a[5], &eps) || !as_int(a[6], &h) || !as_int(a[7], &hkv)) return nullptr;
  const Tensor *kc = nullptr, *vc = nullptr, *slots = nullptr;
  if (a[8] != Py_None && !(kc = tensor_of(a[8], "k_cache"))) return nullptr;
  if (a[9] != Py_None && !(vc = tensor_of(a[9], "v_cache"))) return nullptr;
  if (a[10] != Py_None && !(slots = tensor_of(a[10], "slot_mapping"))) return nullptr;
  const Tensor &qkv = *t[0], &pos = *t[1], &table = *t[4];
  if (!all_cuda({t[0], t[1], t[2], t[3], t[4]})) return nullptr;
  constexpr int64_t d = 128;
  const int64_t width = (h + 2 * static_cast<int64_t>(hkv)) * d;
  REQUIRE(qkv.dim() == 2 && qkv.size(1) == width && qkv.stride(1) == 1, "qkv must be (N, (H + 2 Hkv) * 128), rows contiguous");
  const int64_t n = qkv.size(0);
  REQUIRE(qkv.scalar_type() == at::kBFloat16 && t[2]->scalar_type() == at::kBFloat16 && t[3]->scalar_type() == at::kBFloat16,
          "qkv and norm weights must be bf16");
  REQUIRE(table.scalar_type() == at::kFloat && table.is_contiguous() && table.dim() > 0 && table.size(table.dim() - 1) == d,
          "cos_sin_cache must be contiguous float32 rows of 128");
  REQUIRE(pos.scalar_type() == at::kLong && pos.numel() == n && pos.is_contiguous(), "positions must be int64, one per token");
  REQUIRE(t[2]->numel() == d && t[3]->numel() == d, "norm weights must have 128 elements");
  const bool have = kc && vc && kc->numel() && vc->numel();
  int64_t n_slots = 0;
  if (have) {
    const int64_t row = hkv * d, kd = kc->dim(), vd = vc->dim();
    REQUIRE(kd > 2 && kc->stride(kd - 1) == 1 && kc->stride(kd - 2) == d && kc->stride(1) == row, "k_cache rows must be kv heads x 128, contiguous");
    REQUIRE(vd > 2 && vc->stride(vd - 1) == 1 && vc->stride(vd - 2) == d && vc->stride(1) == row, "v_cache rows must be kv heads x 128, contiguous");
    REQUIRE(slots && slots->numel() == n && slots->scalar_type() == at::kInt, "slot_mapping must be int32, one per token");
    n_slots = kc->numel() / row;
  }
  Tensor q = empty_like_rows({n, h, d}, qkv), k = empty_like_rows({n, hkv, d}, qkv);
  Tensor v = qkv.as_strided({n, hkv, d}, {qkv.stride(0), d, 1}, qkv.storage_offset() + (h + static_cast<int64_t>(hkv)) * d);
  LAUNCH(b200_qk_norm_rope_store(qkv.data_ptr(), qkv.stride(0), static_cast<const int64_t*>(pos.data_ptr()), t[2]->data_ptr(),
                                 t[3]->data_ptr(), static_cast<const float*>(table.data_ptr()), static_cast<int32_t>(table.size(0)),
                                 static_cast<float>(eps), q.data_ptr(), k.data_ptr(), have ? kc->data_ptr() : nullptr,
                                 have ? vc->data_ptr() : nullptr, have ? static_cast<const int32_t*>(slots->data_ptr()) : nullptr,
                                 n_slots, static_cast<int32_t>(n), h, hkv, static_cast<int32_t>(d), stream_ptr()));
  PyObject* res = PyTuple_New(3);
  if (!res) return nullptr;
  PyTuple_SET_ITEM(res, 0, THPVariable_Wrap(std::move(q)));
  PyTuple_SET_ITEM(res, 1, THPVariable_Wrap(std::move(k)));
  PyTuple_SET_ITEM(res, 2, THPVariable_Wrap(std::move(v)));
  return res;
  END_HANDLE_TH_ERRORS
}

// ---- decode metadata (engine/decode_metadata.py) -------------------------------------------------------------
PyObject *s_block_table, *s_last_token;

// pack_decode(seqs, record, max_batch, max_blocks, block_size) -> (batch, table width).  `record` is the int32 pinned
// tensor the step's metadata is written to; the layout is b200_unpack_decode_metadata's.
PyObject* py_pack_decode(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(5, "pack_decode");
  const Tensor* rec = tensor_of(a[1], "record");
  int max_batch, max_blocks, block_size;
  if (!rec || !as_int(a[2], &max_batch) || !as_int(a[3], &max_blocks) || !as_int(a[4], &block_size)) return nullptr;
  // A tuple of our own: the calls below run Python code, during which another thread may change the caller's list.
  Ref seqs(PySequence_Tuple(a[0]));
  if (!seqs.o) return nullptr;
  const Py_ssize_t bs = PyTuple_GET_SIZE(seqs.o);
  if (bs > max_batch) {
    PyErr_Format(PyExc_ValueError, "decode batch %zd exceeds the stager's capacity %d", bs, max_batch);
    return nullptr;
  }
  REQUIRE(rec->scalar_type() == at::kInt && rec->is_contiguous() && !rec->is_cuda() &&
              rec->numel() >= static_cast<int64_t>(max_batch) * (6 + static_cast<int64_t>(max_blocks)), "record too small");
  // First sweep: the scheduler's Python objects into C++ (the block tables as flat ids), because where the tables lie
  // in the record depends on the longest one.
  // (The vectors' memory is kept between calls; a call that comes in through one of the objects' own methods finds none.)
  static thread_local std::vector<int32_t> kept_flat, kept_count;
  std::vector<int32_t> flat(std::move(kept_flat)), count(std::move(kept_count));
  flat.clear();
  count.clear();
  int32_t* const base = static_cast<int32_t*>(rec->data_ptr());
  int64_t* const ids = reinterpret_cast<int64_t*>(base);
  int64_t* const pos = ids + bs;
  int32_t *const slot = base + 4 * bs, *const len = slot + bs, *const tables = len + bs;
  Py_ssize_t width = 0;
  for (Py_ssize_t i = 0; i < bs; ++i) {
    PyObject* s = PyTuple_GET_ITEM(seqs.o, i);
    Ref table(PyObject_GetAttr(s, s_block_table)), last(PyObject_GetAttr(s, s_last_token));
    if (!table.o || !last.o) return nullptr;
    const Py_ssize_t n = PyObject_Size(s);
    if (n < 0) return nullptr;
    const long long token = PyLong_AsLongLong(last.o);
    if (token == -1 && PyErr_Occurred()) return nullptr;
    Ref blocks(PySequence_Fast(table.o, "block_table must be a sequence"));
    if (!blocks.o) return nullptr;
    const Py_ssize_t nb = PySequence_Fast_GET_SIZE(blocks.o);
    if (nb > max_blocks) {
      PyErr_Format(PyExc_ValueError, "block table of %zd blocks exceeds the stager's capacity %d", nb, max_blocks);
      return nullptr;
    }
    if (nb == 0) {
      PyErr_SetString(PyExc_IndexError, "a decoding sequence has an empty block table");
      return nullptr;
    }
    for (Py_ssize_t j = 0; j < nb; ++j) {
      PyObject* item = PySequence_Fast_GET_ITEM(blocks.o, j);
      long id;
      if (PyLong_CheckExact(item)) {
        id = PyLong_AsLong(item);
      } else {
        // It is asked for its value, which may run Python code: held meanwhile, and the table looked at again.
        Py_INCREF(item);
        id = PyLong_AsLong(item);
        Py_DECREF(item);
        if (PySequence_Fast_GET_SIZE(blocks.o) < nb) {
          if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "a block table was shortened while it was read");
          return nullptr;
        }
      }
      if (id == -1 && PyErr_Occurred()) return nullptr;
      if (id != static_cast<int32_t>(id)) {
        PyErr_SetString(PyExc_OverflowError, "block id does not fit 32 bits");
        return nullptr;
      }
      flat.push_back(static_cast<int32_t>(id));
    }
    count.push_back(static_cast<int32_t>(nb));
    width = nb > width ? nb : width;
    ids[i] = token;
    pos[i] = n - 1;
    // Sequence.last_block_num_tokens (nanovllm/engine/sequence.py:60-62) with num_blocks = ceil(len / block_size)
    const int64_t in_last = n - ((n + block_size - 1) / block_size - 1) * static_cast<int64_t>(block_size);
    slot[i] = static_cast<int32_t>(flat.back() * static_cast<int64_t>(block_size) + in_last - 1);
    len[i] = static_cast<int32_t>(n);
  }
  const int32_t* src = flat.data();
  for (Py_ssize_t i = 0; i < bs; ++i) {
    int32_t* row = tables + i * width;
    const int32_t nb = count[i];
    std::memcpy(row, src, nb * sizeof(int32_t));
    std::fill(row + nb, row + width, -1);
    src += nb;
  }
  kept_flat = std::move(flat);
  kept_count = std::move(count);
  return Py_BuildValue("nn", bs, width);
  END_HANDLE_TH_ERRORS
}

// upload_record(host, device, words) -> device[:words]: one asynchronous copy of a pinned record.
PyObject* py_upload_record(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(3, "upload_record");
  const Tensor *host = tensor_of(a[0], "host"), *dev = host ? tensor_of(a[1], "device") : nullptr;
  int n;
  if (!dev || !as_int(a[2], &n)) return nullptr;
  REQUIRE(dev->is_cuda() && !host->is_cuda() && n >= 0 && n <= host->numel() && n <= dev->numel() &&
              host->scalar_type() == dev->scalar_type(), "host and device records do not match");
  const auto stream = c10::cuda::getCurrentCUDAStream();
  if (n > 0) {
    cudaError_t e;
    Py_BEGIN_ALLOW_THREADS
    e = cudaMemcpyAsync(dev->data_ptr(), host->data_ptr(), n * host->element_size(), cudaMemcpyHostToDevice, stream.stream());
    Py_END_ALLOW_THREADS
    if (e != cudaSuccess) {
      PyErr_Format(PyExc_RuntimeError, "upload_record: %s", cudaGetErrorString(e));
      return nullptr;
    }
    // the pinned block must not be handed out again while the copy is in flight (a no-op for ordinary memory)
    at::getHostAllocator(at::kCUDA)->record_event(host->data_ptr(), host->storage().data_ptr().get_context(), stream.unwrap());
  }
  return THPVariable_Wrap(dev->as_strided({n}, {1}, dev->storage_offset()));
  END_HANDLE_TH_ERRORS
}

// unpack_decode_metadata(record, batch, width, input_ids, positions, slot_mapping, context_lens, block_tables)
PyObject* py_unpack(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(8, "unpack_decode_metadata");
  const Tensor* rec = tensor_of(a[0], "record");
  int batch, width;
  if (!rec || !as_int(a[1], &batch) || !as_int(a[2], &width)) return nullptr;
  const Tensor* t[5];
  static const char* names[5] = {"input_ids", "positions", "slot_mapping", "context_lens", "block_tables"};
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = tensor_of(a[3 + i], names[i]))) return nullptr;
  REQUIRE(t[4]->dim() == 2 && t[4]->stride(1) == 1 && t[0]->scalar_type() == at::kLong && t[1]->scalar_type() == at::kLong,
          "block-table rows must be contiguous, input_ids and positions int64");
  REQUIRE(t[2]->numel() == t[3]->numel() && t[0]->numel() >= batch, "the graph buffers do not fit the batch");
  LAUNCH(b200_unpack_decode_metadata(rec->data_ptr(), batch, width, static_cast<int32_t>(t[2]->numel()),
                                     static_cast<int32_t>(t[4]->stride(0)), static_cast<int64_t*>(t[0]->data_ptr()),
                                     static_cast<int64_t*>(t[1]->data_ptr()), static_cast<int32_t*>(t[2]->data_ptr()),
                                     static_cast<int32_t*>(t[3]->data_ptr()), static_cast<int32_t*>(t[4]->data_ptr()),
                                     stream_ptr()));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FAST("store_kvcache", py_store_kvcache),
    FAST("decode_attention", py_decode_attention),
    FAST("prefill_attention", py_prefill_attention),
    FAST("attention_forward", py_attention_forward),
    FAST("qk_norm_rope_store", py_qk_norm_rope_store),
    FAST("pack_decode", py_pack_decode),
    FAST("upload_record", py_upload_record),
    FAST("unpack_decode_metadata", py_unpack),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  s_is_prefill = PyUnicode_InternFromString("is_prefill");
  s_cu_q = PyUnicode_InternFromString("cu_seqlens_q");
  s_cu_k = PyUnicode_InternFromString("cu_seqlens_k");
  s_max_q = PyUnicode_InternFromString("max_seqlen_q");
  s_max_k = PyUnicode_InternFromString("max_seqlen_k");
  s_slots = PyUnicode_InternFromString("slot_mapping");
  s_lens = PyUnicode_InternFromString("context_lens");
  s_bt = PyUnicode_InternFromString("block_tables");
  s_block_table = PyUnicode_InternFromString("block_table");
  s_last_token = PyUnicode_InternFromString("last_token");
  return PyModule_Create(&module_def);
}
