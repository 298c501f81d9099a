// CPython extension adamas_b200._native: the operators a decode loop calls once per layer, from torch tensors to
// the C ABI of libadamas_b200.so (include/adamas_b200.h).
//
// Why it exists: the same checks and the same call, written in Python over ctypes, cost 35-45 us per decode_step and
// 10-20 us per single operator, two to three times what the GPU needs for them; a loop that launches call by call
// ran at the speed of its host.  Here a call costs its launches (about 3 us each) and about 1 us more.
// adamas_b200/_kernels.py keeps the public signatures and forwards to these functions positionally.  What a check
// rejects raises RuntimeError, as the reference's TORCH_CHECK does.  Launches go to torch's current CUDA stream of
// the current device; the interpreter lock is released around the native call.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <stdexcept>
#include <string>

#include "../../include/adamas_b200.h"

namespace {

struct PyFailure {};   // a Python exception is already set

[[noreturn]] void reject(const char* fmt, ...) {
  char msg[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(msg, sizeof(msg), fmt, ap);
  va_end(ap);
  throw std::runtime_error(msg);
}
#define REQUIRE(cond, ...) \
  do {                     \
    if (!(cond)) reject(__VA_ARGS__); \
  } while (0)

// ---- arguments ----------------------------------------------------------------------------------------------
inline bool given(PyObject* o) { return o != nullptr && o != Py_None; }

const at::Tensor& tensor(PyObject* o, const char* name) {
  REQUIRE(o && THPVariable_Check(o), "%s must be a tensor", name);
  return THPVariable_Unpack(o);
}
const at::Tensor& input(PyObject* o, const char* name, int dim = -1) {
  const at::Tensor& t = tensor(o, name);
  REQUIRE(t.is_cuda(), "%s must be a CUDA tensor", name);
  REQUIRE(t.is_contiguous(), "%s must be contiguous", name);
  REQUIRE(dim < 0 || t.dim() == dim, "%s must be a %dD tensor", name, dim);
  return t;
}
// 2-D with dense rows; the row stride may exceed the row length or be 0 (one row shared by all heads)
const at::Tensor& rows(PyObject* o, const char* name) {
  REQUIRE(o && THPVariable_Check(o) && THPVariable_Unpack(o).is_cuda(), "%s must be a CUDA tensor", name);
  const at::Tensor& t = THPVariable_Unpack(o);
  REQUIRE(t.dim() == 2, "%s must be a 2D tensor", name);
  REQUIRE(t.size(1) <= 1 || t.stride(1) == 1, "%s must have unit stride along its rows", name);
  REQUIRE(t.size(0) <= 1 || t.stride(0) == 0 || t.stride(0) >= t.size(1), "%s has overlapping rows", name);
  return t;
}
inline void* ptr(const at::Tensor& t) { return t.data_ptr(); }
template <typename T>
inline T* ptr_as(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }

long long integer(PyObject* o) {
  long long v = PyLong_Check(o) ? PyLong_AsLongLong(o) : 0;
  if (!PyLong_Check(o)) {
    PyObject* i = PyNumber_Long(o);
    if (!i) throw PyFailure{};
    v = PyLong_AsLongLong(i);
    Py_DECREF(i);
  }
  if (v == -1 && PyErr_Occurred()) throw PyFailure{};
  return v;
}
int int32(PyObject* o) {
  const long long v = integer(o);
  REQUIRE(v >= INT32_MIN && v <= INT32_MAX, "integer argument out of range");
  return static_cast<int>(v);
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyFailure{};
  return v;
}
bool truth(PyObject* o) {   // (an object may refuse to be a truth value, as a tensor of several elements does)
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyFailure{};
  return v != 0;
}
float scale_or_default(PyObject* o) { return static_cast<float>(given(o) ? real(o) : 1.0 / std::sqrt(128.0)); }

int dtype_code(const at::Tensor& t, const char* what) {
  if (t.scalar_type() == at::kHalf) return ADAMAS_F16;
  if (t.scalar_type() == at::kBFloat16) return ADAMAS_BF16;
  reject("%s failed to dispatch with dtype %s", what, c10::toString(t.scalar_type()));
}
bool is_int16(const at::Tensor& t) { return t.scalar_type() == at::kShort || t.scalar_type() == at::kUInt16; }
int value_format(const at::Tensor& t, const char* what) {
  if (t.scalar_type() == at::kHalf) return ADAMAS_VAL_F16;
  if (is_int16(t)) return ADAMAS_VAL_U16;
  reject("%s failed to dispatch with dtype %s", what, c10::toString(t.scalar_type()));
}

struct ThresholdsArg {
  float v[3];
  const float* p = nullptr;
  explicit ThresholdsArg(PyObject* o) {
    if (!given(o)) return;
    PyObject* seq = PySequence_Fast(o, "thresholds must be a sequence of three numbers");
    if (!seq) throw PyFailure{};
    const bool ok = PySequence_Fast_GET_SIZE(seq) == 3;
    for (int i = 0; ok && i < 3; ++i) v[i] = static_cast<float>(PyFloat_AsDouble(PySequence_Fast_GET_ITEM(seq, i)));
    Py_DECREF(seq);
    if (PyErr_Occurred()) throw PyFailure{};
    REQUIRE(ok, "thresholds must be a sequence of three numbers");
    p = v;
  }
};

// None | (rope_scale, rope_theta) | {"inv_freq": float32 CUDA tensor [64], "mscale": float}
struct RopeArg {
  bool on = false;
  float scale = 0.f, theta = 0.f, mscale = 1.f;
  const float* inv_freq = nullptr;
  explicit RopeArg(PyObject* o) {
    if (!given(o)) return;
    on = true;
    if (PyDict_Check(o)) {
      PyObject* t = PyDict_GetItemString(o, "inv_freq");
      if (!t) {
        PyErr_SetString(PyExc_KeyError, "inv_freq");
        throw PyFailure{};
      }
      const at::Tensor& f = tensor(t, "rope inv_freq");
      REQUIRE(f.is_cuda() && f.scalar_type() == at::kFloat && f.is_contiguous() && f.numel() == 64,
              "rope inv_freq must be a contiguous float32 CUDA tensor of 64 elements");
      inv_freq = ptr_as<const float>(f);
      if (PyObject* m = PyDict_GetItemString(o, "mscale")) mscale = static_cast<float>(real(m));
      return;
    }
    PyObject* seq = PySequence_Fast(o, "rope must be (rope_scale, rope_theta) or a dict with inv_freq");
    if (!seq) throw PyFailure{};
    const bool ok = PySequence_Fast_GET_SIZE(seq) >= 2;
    if (ok) {
      scale = static_cast<float>(PyFloat_AsDouble(PySequence_Fast_GET_ITEM(seq, 0)));
      theta = static_cast<float>(PyFloat_AsDouble(PySequence_Fast_GET_ITEM(seq, 1)));
    }
    Py_DECREF(seq);
    if (PyErr_Occurred()) throw PyFailure{};
    REQUIRE(ok, "rope must be (rope_scale, rope_theta) or a dict with inv_freq");
  }
};

inline adamas_stream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Calls `f`, a function of the C ABI, without the interpreter lock; a non-zero status becomes RuntimeError.  The arguments
// (pointers of tensors, the current stream) are formed by the caller, before the lock is given up: forming them may throw,
// or warn through Python (a tensor without memory of its own, no driver), and both need the lock.
template <typename... P, typename... A>
void call(const char* what, int (*f)(P...), A... args) {
  PyThreadState* st = PyEval_SaveThread();
  const int rc = f(args...);
  PyEval_RestoreThread(st);
  REQUIRE(rc == ADAMAS_OK, "%s failed: %s", what, adamas_last_error());
}

template <typename F>
PyObject* guarded(const char* name, Py_ssize_t n, Py_ssize_t want, F f) {
  if (n != want) {
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given)", name, want, n);
    return nullptr;
  }
  try {
    return f();
  } catch (const PyFailure&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}
PyObject* none() { Py_RETURN_NONE; }

// ---- shared checks ------------------------------------------------------------------------------------------
struct Caches {
  int heads, page_size;
  const at::Tensor *kv_data, *kv_indices, *code_data, *code_indices;
};

Caches check_append(PyObject* k_, PyObject* v_, PyObject* kv_data_, PyObject* kv_idx_, PyObject* code_data_, PyObject* code_idx_,
                    int layout) {
  REQUIRE(layout == 0, "only the NHD layout is implemented (the reference's controller always uses it)");
  const at::Tensor& k = input(k_, "k", 3);
  const at::Tensor& v = input(v_, "v", 3);
  const at::Tensor& kv = input(kv_data_, "kv_data", 5);
  const at::Tensor& ki = input(kv_idx_, "kv_indices", 1);
  const at::Tensor& cd = input(code_data_, "hadamard_data", 5);
  const at::Tensor& ci = input(code_idx_, "hadamard_indices", 1);
  REQUIRE(ki.scalar_type() == at::kInt, "kv_indices must be int32");
  REQUIRE(ci.scalar_type() == at::kInt, "hadamard_indices must be int32");
  REQUIRE(v.sizes() == k.sizes(), "k and v must have the same shape");
  const int64_t h = k.size(1), d = k.size(2), ps = kv.size(2);
  REQUIRE(kv.size(1) == 2 && kv.size(3) == h && kv.size(4) == d, "kv_data must be [pages, 2, page_size, num_heads, head_dim]");
  REQUIRE(cd.size(1) == 1 && cd.size(2) == ps && cd.size(3) == h && cd.size(4) == d / 8,
          "hadamard_data must be [pages, 1, page_size, num_heads, head_dim/8]");
  REQUIRE(kv.scalar_type() == k.scalar_type() && v.scalar_type() == k.scalar_type(), "k, v and kv_data must share a dtype");
  REQUIRE(cd.element_size() == 2, "hadamard_data must have 16-bit elements");
  return Caches{static_cast<int>(h), static_cast<int>(ps), &kv, &ki, &cd, &ci};
}

int query_heads(const at::Tensor& q, const at::Tensor& k, const char* name) {
  REQUIRE(q.dim() == 3 && q.size(0) == 1 && q.size(2) == k.size(2) && q.scalar_type() == k.scalar_type() &&
              q.size(1) >= k.size(1) && q.size(1) % k.size(1) == 0,
          "%s: q must be [1, Hq, D] in k.dtype with Hq a multiple of the cache's heads", name);
  return static_cast<int>(q.size(1));
}

uint32_t* histogram(PyObject* o, int64_t heads) {
  if (!given(o)) return nullptr;
  const at::Tensor& t = tensor(o, "hist");
  REQUIRE(t.is_cuda() && t.is_contiguous() && t.scalar_type() == at::kInt && t.numel() >= heads * ADAMAS_HIST_WORDS_PER_HEAD,
          "hist must be a contiguous int32 CUDA tensor made by histogram_scratch(H)");
  return ptr_as<uint32_t>(t);
}

float* lse_ptr(PyObject* o) { return given(o) ? ptr_as<float>(tensor(o, "lse")) : nullptr; }

// ---- operators ----------------------------------------------------------------------------------------------
PyObject* py_hadamard_transform(PyObject*, PyObject* const* a, Py_ssize_t n) {   // x, inplace, scale
  return guarded("hadamard_transform", n, 3, [&]() -> PyObject* {
    const at::Tensor& x = input(a[0], "x");
    REQUIRE(x.dim() >= 1 && x.size(-1) == 128, "hadamard_transform supports a last dimension of 128");
    const bool inplace = truth(a[1]);
    const float s = scale_or_default(a[2]);
    const int dt = dtype_code(x, "hadamard_transform");
    at::Tensor y = inplace ? x : at::empty_like(x);
    const int64_t count = x.numel() / 128;
    call("hadamard_transform", adamas_hadamard_transform, ptr(x), ptr(y), count, 128, s, dt, stream());
    if (inplace) {
      Py_INCREF(a[0]);
      return a[0];
    }
    return THPVariable_Wrap(std::move(y));
  });
}

PyObject* py_apply_rope(PyObject*, PyObject* const* a, Py_ssize_t n) {   // q, k, past_kv_len, rope_scale, rope_theta
  return guarded("apply_rope_in_place", n, 5, [&]() -> PyObject* {
    const at::Tensor& q = input(a[0], "q", 3);
    const at::Tensor& k = input(a[1], "k", 3);
    REQUIRE(q.size(0) == k.size(0) && q.size(2) == 128 && k.size(2) == 128 && q.scalar_type() == k.scalar_type(),
            "q and k must be [N, H, 128] of one dtype");
    const int64_t past = integer(a[2]);
    const float rs = static_cast<float>(real(a[3])), rt = static_cast<float>(real(a[4]));
    const int dt = dtype_code(q, "apply_rope_in_place");
    call("apply_rope_in_place", adamas_apply_rope_in_place, ptr(q), ptr(k), q.size(0), static_cast<int>(q.size(1)),
         static_cast<int>(k.size(1)), 128, past, rs, rt, dt, stream());
    return none();
  });
}

// k, v, h, o, kv_data, kv_indices, kv_last_page_len, hadamard_data, hadamard_indices, hadamard_last_page_len, layout, thresholds
PyObject* py_append_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("append_kv_cache_decode", n, 12, [&]() -> PyObject* {
    const Caches c = check_append(a[0], a[1], a[4], a[5], a[7], a[8], int32(a[10]));
    const at::Tensor &k = THPVariable_Unpack(a[0]), &v = THPVariable_Unpack(a[1]);
    const at::Tensor& h = input(a[2], "h", 3);
    const at::Tensor& o = input(a[3], "o", 3);
    REQUIRE(k.size(0) == 1 && v.size(0) == 1 && h.size(0) == 2 && o.size(0) == 1, "decode appends one token");
    REQUIRE(h.size(1) == c.heads && h.size(2) == k.size(2) && h.scalar_type() == k.scalar_type(), "h must be [2, H, D] in k.dtype");
    REQUIRE(o.size(1) == c.heads && o.size(2) == k.size(2) / 8 && o.element_size() == 2, "o must be [1, H, D/8] 16-bit");
    const int kl = int32(a[6]), cl = int32(a[9]), dt = dtype_code(k, "Append_kv_cache_decode");
    const ThresholdsArg th(a[11]);
    call("Append_kv_cache_decode", adamas_append_decode, ptr(k), ptr(v), ptr(h), ptr(o), ptr(*c.kv_data),
         ptr_as<int32_t>(*c.kv_indices), static_cast<int>(c.kv_indices->numel()), kl, ptr(*c.code_data),
         ptr_as<int32_t>(*c.code_indices), static_cast<int>(c.code_indices->numel()), cl, c.heads, static_cast<int>(k.size(2)),
         c.page_size, th.p, dt, stream());
    return none();
  });
}

// q, k, v, o, kv_data, kv_indices, kv_last_page_len, hadamard_data, hadamard_indices, hadamard_last_page_len, layout,
// scale, thresholds, rope
PyObject* py_append_decode_fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("append_kv_cache_decode_fused", n, 14, [&]() -> PyObject* {
    const Caches c = check_append(a[1], a[2], a[4], a[5], a[7], a[8], int32(a[10]));
    const at::Tensor &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
    const at::Tensor& q = input(a[0], "q", 3);
    const at::Tensor& o = input(a[3], "o", 3);
    REQUIRE(k.size(0) == 1, "k, v must be [1, H, D]");
    const int hq = query_heads(q, k, "append_kv_cache_decode_fused"), d = static_cast<int>(k.size(2));
    REQUIRE(o.size(1) == hq && o.size(2) == d / 8 && o.element_size() == 2, "o must be [1, Hq, D/8] 16-bit");
    const int kl = int32(a[6]), cl = int32(a[9]);
    const float s = scale_or_default(a[11]);
    const ThresholdsArg th(a[12]);
    const RopeArg rope(a[13]);
    if (rope.on) {
      const int dt = dtype_code(k, "append_kv_cache_decode_rope_fused");
      call("append_kv_cache_decode_rope_fused", adamas_append_decode_rope_fused, ptr(q), ptr(k), ptr(v), ptr(o), ptr(*c.kv_data),
           ptr_as<int32_t>(*c.kv_indices), static_cast<int>(c.kv_indices->numel()), kl, ptr(*c.code_data),
           ptr_as<int32_t>(*c.code_indices), static_cast<int>(c.code_indices->numel()), cl, c.heads, hq, d, c.page_size, s, th.p,
           rope.inv_freq ? 1.f : rope.scale, rope.inv_freq ? 1e4f : rope.theta, rope.inv_freq, rope.mscale, dt, stream());
    } else {
      const int dt = dtype_code(k, "append_kv_cache_decode_fused");
      call("append_kv_cache_decode_fused", adamas_append_decode_fused, ptr(q), ptr(k), ptr(v), ptr(o), ptr(*c.kv_data),
           ptr_as<int32_t>(*c.kv_indices), static_cast<int>(c.kv_indices->numel()), kl, ptr(*c.code_data),
           ptr_as<int32_t>(*c.code_indices), static_cast<int>(c.code_indices->numel()), cl, c.heads, hq, d, c.page_size, s, th.p,
           dt, stream());
    }
    return none();
  });
}

// k, v, h or None, kv_data, kv_indices, kv_last_page_len, hadamard_data, hadamard_indices, hadamard_last_page_len, layout,
// scale, thresholds
PyObject* py_append_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("append_kv_cache_prefill", n, 12, [&]() -> PyObject* {
    const Caches c = check_append(a[0], a[1], a[3], a[4], a[6], a[7], int32(a[9]));
    const at::Tensor &k = THPVariable_Unpack(a[0]), &v = THPVariable_Unpack(a[1]);
    const void* h = nullptr;
    if (given(a[2])) {
      const at::Tensor& t = input(a[2], "h", 3);
      REQUIRE(t.sizes() == k.sizes() && t.scalar_type() == k.scalar_type(), "h must match k");
      h = ptr(t);
    }
    const int kl = int32(a[5]), cl = int32(a[8]), dt = dtype_code(k, "Append_kv_cache_prefill");
    const float s = scale_or_default(a[10]);
    const ThresholdsArg th(a[11]);
    call("Append_kv_cache_prefill", adamas_append_prefill, ptr(k), ptr(v), h, k.size(0), ptr(*c.kv_data),
         ptr_as<int32_t>(*c.kv_indices), static_cast<int>(c.kv_indices->numel()), kl, ptr(*c.code_data),
         ptr_as<int32_t>(*c.code_indices), static_cast<int>(c.code_indices->numel()), cl, c.heads, static_cast<int>(k.size(2)),
         c.page_size, s, th.p, dt, stream());
    return none();
  });
}

// q, o, code_data, code_indices, last_page_len, layout, metric (0 L1, 1 XOR), exclude_last, hist, hist_slices
PyObject* py_estimate(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("estimate_attn_score", n, 10, [&]() -> PyObject* {
    REQUIRE(integer(a[5]) == 0, "only the NHD layout is implemented (the reference's controller always uses it)");
    const at::Tensor& q = input(a[0], "q", 3);
    const at::Tensor& o = rows(a[1], "o");
    const at::Tensor& cd = input(a[2], "hadamard_data", 5);
    const at::Tensor& ci = input(a[3], "hadamard_indices", 1);
    REQUIRE(q.size(0) == 1, "q.size(0) must be 1");
    REQUIRE(ci.scalar_type() == at::kInt, "hadamard_indices must be int32");
    const int64_t hq = q.size(1), words = q.size(2), ps = cd.size(2), h = cd.size(3);
    REQUIRE(hq >= h && h >= 1 && hq % h == 0 && cd.size(4) == words && words == 16,
            "hadamard_data must be [pages, 1, page_size, num_heads, 16], q [1, Hq, 16]");
    REQUIRE(q.element_size() == 2 && cd.element_size() == 2, "codes must be 16-bit words");
    const int last = int32(a[4]), metric = int32(a[6]), exclude = truth(a[7]) ? 1 : 0;
    const int64_t cols = (ci.numel() - 1) * ps + last - exclude;
    REQUIRE(o.size(0) == hq && o.size(1) == cols, "o must be [%lld, %lld]", static_cast<long long>(hq), static_cast<long long>(cols));
    const int fmt = value_format(o, "Estimate_attn_score"), slices = int32(a[9]);
    uint32_t* hist = histogram(a[8], hq);
    call("Estimate_attn_score", adamas_estimate, ptr(q), ptr(cd), ptr_as<int32_t>(ci), static_cast<int>(ci.numel()), last,
         static_cast<int>(ps), static_cast<int>(h), static_cast<int>(hq), 128, ptr(o), o.stride(0), fmt, metric, exclude, hist,
         slices, stream());
    return none();
  });
}

// estimated_value, estimated_indices, d_out, indices_out, page_budget
PyObject* py_topk_filtering(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("topk_filtering", n, 5, [&]() -> PyObject* {
    const at::Tensor& v = rows(a[0], "estimated_value");
    const at::Tensor& vi = rows(a[1], "estimated_indices");
    const at::Tensor& d = rows(a[2], "d_out");
    const at::Tensor& oi = rows(a[3], "indices_out");
    REQUIRE(d.stride(0) == oi.stride(0), "d_out and indices_out must share a row stride");
    const int64_t count = v.size(0), cols = v.size(1), k = integer(a[4]);
    REQUIRE(vi.sizes() == v.sizes(), "estimated_indices must match estimated_value");
    REQUIRE(vi.scalar_type() == at::kInt && oi.scalar_type() == at::kInt, "indices must be int32");
    REQUIRE(cols >= k, "num_pages must be >= page_budget");
    REQUIRE(d.size(1) == k && oi.size(1) == k, "outputs must have page_budget columns");
    REQUIRE(d.size(0) == count && oi.size(0) == count, "outputs must have one row per head");
    REQUIRE(d.scalar_type() == v.scalar_type(), "d_out must have the dtype of estimated_value");
    const int fmt = value_format(v, "Top-k filtering");
    call("Top-k filtering", adamas_topk, ptr(v), fmt, v.stride(0), static_cast<int>(cols), ptr_as<int32_t>(vi), vi.stride(0), 1,
         static_cast<int>(count), static_cast<int>(k), ptr(d), ptr_as<int32_t>(oi), oi.stride(0), stream());
    return none();
  });
}

// values, k, indices_out, values_out or None, page_table or None, page_size
PyObject* py_topk_select(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("topk_select", n, 6, [&]() -> PyObject* {
    const at::Tensor& v = rows(a[0], "values");
    const at::Tensor& oi = rows(a[2], "indices_out");
    const int64_t count = v.size(0), cols = v.size(1), k = integer(a[1]), ps = integer(a[5]);
    REQUIRE(oi.scalar_type() == at::kInt && oi.size(0) == count && oi.size(1) >= k, "indices_out must be int32 [rows, >=k]");
    void* vo = nullptr;
    if (given(a[3])) {
      const at::Tensor& t = rows(a[3], "values_out");
      REQUIRE(t.scalar_type() == v.scalar_type() && t.stride(0) == oi.stride(0),
              "values_out must match values.dtype and the row stride of indices_out");
      vo = ptr(t);
    }
    int32_t* table = nullptr;
    if (given(a[4])) {
      const at::Tensor& t = input(a[4], "page_table", 1);
      REQUIRE(t.scalar_type() == at::kInt && t.numel() * ps >= cols, "page_table too short");
      table = ptr_as<int32_t>(t);
    }
    const int fmt = value_format(v, "topk_select");
    call("topk_select", adamas_topk, ptr(v), fmt, v.stride(0), static_cast<int>(cols), table, 0, static_cast<int>(ps),
         static_cast<int>(count), static_cast<int>(k), vo, ptr_as<int32_t>(oi), oi.stride(0), stream());
    return none();
  });
}

// handle, q, o, lse or None, kv_data, indices, last_page_len, last_page_idx, token_granular, num_q_heads, num_kv_heads, head_dim,
// page_size, dtype, planned_tokens, batch, tail_len or None -> tokens the handler is planned for
PyObject* py_decode_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("decode_forward", n, 17, [&]() -> PyObject* {
    auto* handle = static_cast<adamas_decode_handler_t*>(PyLong_AsVoidPtr(a[0]));
    const at::Tensor& q = input(a[1], "q", 3);
    const at::Tensor& o = input(a[2], "o", 3);
    const at::Tensor& kv = input(a[4], "paged_kv_data", 5);
    const at::Tensor& idx = rows(a[5], "paged_kv_indices");
    const int last_len = int32(a[6]), last_idx = int32(a[7]), token_granular = truth(a[8]);
    const int hq = int32(a[9]), hkv = int32(a[10]), d = int32(a[11]), ps = int32(a[12]), dt = int32(a[13]), batch = int32(a[15]);
    int64_t planned = integer(a[14]);
    REQUIRE(q.size(0) == 1 && q.size(1) == hq && q.size(2) == d, "q must be [1, H, D]");
    REQUIRE(o.sizes() == q.sizes() && o.scalar_type() == q.scalar_type(), "o must match q");
    REQUIRE(kv.size(1) == 2 && kv.size(2) == ps && kv.size(3) == hkv && kv.size(4) == d,
            "paged_kv_data must be [pages, 2, page_size, H_kv, D]");
    REQUIRE(idx.size(0) == hq && idx.scalar_type() == at::kInt, "paged_kv_indices must be int32 [H, n]");
    REQUIRE(dtype_code(q, "BatchDecodeWithPagedKVCache") == dt && kv.scalar_type() == q.scalar_type(),
            "dtype differs from begin_forward");
    const int64_t n_idx = idx.size(1), unit = token_granular ? 1 : ps;
    const int64_t tail = given(a[16]) ? integer(a[16]) : (token_granular ? 1 : last_len);
    const int64_t tokens = n_idx * unit + tail;
    float* lse = nullptr;
    if (given(a[3])) {
      const at::Tensor& t = tensor(a[3], "lse");
      REQUIRE(t.is_cuda() && t.scalar_type() == at::kFloat && t.numel() == hq && t.is_contiguous(),
              "lse must be a contiguous float32 CUDA tensor of H elements");
      lse = ptr_as<float>(t);
    }
    if (tokens > planned) {
      call("BatchDecodeWithPagedKVCache", adamas_decode_begin_forward, handle, tokens, batch, hkv, hq, d, ps, dt, stream());
      planned = tokens;
    }
    const float sm_scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(d)));
    call("BatchDecodeWithPagedKVCache", adamas_decode_forward, handle, ptr(q), ptr(o), lse, ptr(kv), ptr_as<int32_t>(idx),
         idx.stride(0), static_cast<int>(n_idx), static_cast<int>(unit), last_idx, last_len, static_cast<int>(tail), sm_scale,
         stream());
    return PyLong_FromLongLong(planned);
  });
}

struct StepArgs {
  Caches c;
  const at::Tensor *q, *k, *v, *o, *code, *dist;
  int hq, d, dt, budget;
  int32_t* out_idx = nullptr;
  int64_t out_stride = 0;
};
// The checks decode_step and decode_step_dev share; `name` in their messages.
StepArgs check_step(const char* name, PyObject* q, PyObject* k, PyObject* v, PyObject* o, PyObject* code, PyObject* kv_data,
                    PyObject* kv_idx, PyObject* code_data, PyObject* code_idx, PyObject* budget, PyObject* dist, PyObject* out_idx) {
  StepArgs s;
  s.c = check_append(k, v, kv_data, kv_idx, code_data, code_idx, 0);
  s.k = &THPVariable_Unpack(k);
  s.v = &THPVariable_Unpack(v);
  s.q = &input(q, "q", 3);
  s.o = &input(o, "o", 3);
  s.code = &input(code, "q_code", 3);
  s.dist = &rows(dist, "dist_scratch");
  s.hq = query_heads(*s.q, *s.k, name);
  s.d = static_cast<int>(s.k->size(2));
  s.dt = dtype_code(*s.k, name);
  s.budget = int32(budget);
  REQUIRE(s.q->sizes() == s.o->sizes() && s.k->size(0) == 1, "q, o must be [1, Hq, D], k, v [1, H, D]");
  REQUIRE(s.code->element_size() == 2 && s.code->numel() == static_cast<int64_t>(s.hq) * s.d / 8, "q_code must be [1, Hq, D/8] 16-bit");
  REQUIRE(s.dist->element_size() == 2 && s.dist->size(0) == s.hq, "dist_scratch must be 16-bit [Hq, n]");
  if (given(out_idx)) {
    const at::Tensor& t = rows(out_idx, "indices_out");
    REQUIRE(t.scalar_type() == at::kInt && t.size(0) == s.hq && t.size(1) >= s.budget - 1, "indices_out must be int32 [Hq, >=budget-1]");
    s.out_idx = ptr_as<int32_t>(t);
    s.out_stride = t.stride(0);
  }
  return s;
}

// q, k, v, o, q_code, kv_data, kv_indices, kv_last_page_len, kv_last_page_idx, hadamard_data, hadamard_indices,
// hadamard_last_page_len, budget, dist_scratch, hist, indices_out, lse, scale, thresholds, rope
PyObject* py_decode_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("decode_step", n, 20, [&]() -> PyObject* {
    const StepArgs s = check_step("decode_step", a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[9], a[10], a[12], a[13], a[15]);
    const int kl = int32(a[7]), ki = int32(a[8]), cl = int32(a[11]);
    uint32_t* hist = histogram(a[14], s.hq);
    float* lse = lse_ptr(a[16]);
    const float scale = scale_or_default(a[17]), sm_scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(s.d)));
    const ThresholdsArg th(a[18]);
    const RopeArg rope(a[19]);
    call("decode_step", adamas_decode_step, ptr(*s.q), ptr(*s.k), ptr(*s.v), ptr(*s.o), lse, ptr(*s.code), ptr(*s.c.kv_data),
         ptr_as<int32_t>(*s.c.kv_indices), static_cast<int>(s.c.kv_indices->numel()), kl, ki, ptr(*s.c.code_data),
         ptr_as<int32_t>(*s.c.code_indices), static_cast<int>(s.c.code_indices->numel()), cl, s.c.heads, s.hq, s.d, s.c.page_size,
         s.dt, s.budget, ptr(*s.dist), s.dist->stride(0), hist, s.out_idx, s.out_stride, scale, th.p, rope.scale, rope.theta,
         rope.inv_freq, rope.mscale, sm_scale, stream());
    return none();
  });
}

// q, k, v, o, q_code, kv_data, kv_indices, hadamard_data, hadamard_indices, seq_len, max_seq_len, budget, dist_scratch, hist,
// indices_out, lse, scale, thresholds, rope
PyObject* py_decode_step_dev(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded("decode_step_dev", n, 19, [&]() -> PyObject* {
    const StepArgs s = check_step("decode_step_dev", a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[11], a[12], a[14]);
    const at::Tensor& len = tensor(a[9], "seq_len");
    REQUIRE(len.is_cuda() && len.scalar_type() == at::kInt && len.is_contiguous() && len.numel() == 1,
            "seq_len must be a contiguous int32 CUDA tensor of 1 element(s)");
    const int max_len = int32(a[10]);
    REQUIRE(s.dist->size(1) >= max_len - 1, "dist_scratch must be 16-bit [Hq, >= max_seq_len - 1]");
    REQUIRE(s.c.kv_indices->numel() * s.c.page_size >= max_len && s.c.code_indices->numel() * s.c.page_size >= max_len,
            "the page tables must have room for max_seq_len tokens");
    uint32_t* hist = histogram(a[13], s.hq);
    float* lse = lse_ptr(a[15]);
    const float scale = scale_or_default(a[16]), sm_scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(s.d)));
    const ThresholdsArg th(a[17]);
    const RopeArg rope(a[18]);
    call("decode_step_dev", adamas_decode_step_dev, ptr(*s.q), ptr(*s.k), ptr(*s.v), ptr(*s.o), lse, ptr(*s.code),
         ptr(*s.c.kv_data), ptr_as<int32_t>(*s.c.kv_indices), ptr(*s.c.code_data), ptr_as<int32_t>(*s.c.code_indices),
         ptr_as<int32_t>(len), max_len, s.c.heads, s.hq, s.d, s.c.page_size, s.dt, s.budget, ptr(*s.dist), s.dist->stride(0),
         hist, s.out_idx, s.out_stride, scale, th.p, rope.scale, rope.theta, rope.inv_freq, rope.mscale, sm_scale, stream());
    return none();
  });
}

#define METHOD(name, f) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    METHOD("hadamard_transform", py_hadamard_transform),
    METHOD("apply_rope_in_place", py_apply_rope),
    METHOD("append_kv_cache_decode", py_append_decode),
    METHOD("append_kv_cache_decode_fused", py_append_decode_fused),
    METHOD("append_kv_cache_prefill", py_append_prefill),
    METHOD("estimate_attn_score", py_estimate),
    METHOD("topk_filtering", py_topk_filtering),
    METHOD("topk_select", py_topk_select),
    METHOD("decode_forward", py_decode_forward),
    METHOD("decode_step", py_decode_step),
    METHOD("decode_step_dev", py_decode_step_dev),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  if (adamas_abi_version() != ADAMAS_ABI_VERSION) {
    PyErr_SetString(PyExc_ImportError, "adamas_b200._native was built for another version of libadamas_b200.so; rebuild both");
    return nullptr;
  }
  return PyModule_Create(&kModule);
}
