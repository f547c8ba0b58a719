// The host path of the operators, in native code: argument checks, allocation of the results
// and the call into libmosaicist_sm100a.so.  An operator of this library runs for 5 - 50 us on
// the GPU in a decode step, and the same work written in Python (a dozen attribute look-ups and
// checks per tensor, ctypes argument conversion, stream and allocator calls through Python) took
// 14 us for a GEMM and 170 us for the masked MoE layer as a torch operator: the GPU waited for
// the host.  Here a GEMM call costs about 4 us, most of it the launch itself.
//
// Two fronts over the same functions on at::Tensor:
//   - a CPython module (METH_FASTCALL, positional arguments only): mosaicist_b200.ops and
//     mosaicist_b200.moe keep their documented signatures and pass everything on;
//   - kernels of the torch operators mosaicist_sm100a::* (mosaicist_b200.torch_ops has their schemas
//     and shape functions).
// The library is not linked: its entry points come as addresses from mosaicist_b200._lib, which
// decides which build is loaded and raises if there is none.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <string.h>

#include <atomic>
#include <deque>
#include <initializer_list>
#include <memory>
#include <optional>
#include <tuple>

#include "../../include/mosaicist_sm100a.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// ---- the library's entry points ---------------------------------------------------------------

#define MSC_ENTRY_POINTS(X)                                                                      \
  X(msc_abi) X(msc_last_error) X(msc_grouped_gemm_nvfp4) X(msc_grouped_gemm_nvfp4_ragged)                   \
  X(msc_grouped_gemm_nvfp4_swiglu_ragged) X(msc_grouped_gemm_mxfp8_ragged) X(msc_quantize_rows)  \
  X(msc_amax_global_scale) X(msc_gemm_f16) X(msc_int4_dequant_bf16)                              \
  X(msc_grouped_gemm_bf16_ragged) X(msc_grouped_gemm_bf16_int4_ragged) X(msc_moe_route_topk)     \
  X(msc_moe_plan) X(msc_moe_permute_quantize) X(msc_moe_unpermute)                               \
  X(msc_moe_masked_workspace) X(msc_moe_masked)

struct Lib {
#define X(name) decltype(&::name) name = nullptr;
  MSC_ENTRY_POINTS(X)
#undef X
};
// Set once, when it is complete: a thread without the GIL sees all of the table or none of it.
std::atomic<const Lib*> g_lib{nullptr};

struct Gil {
  PyGILState_STATE s = PyGILState_Ensure();
  ~Gil() { PyGILState_Release(s); }
};

// Carries the Python error that has just been set out of this call, whichever front made it.
[[noreturn]] void raise() {
  python_error e;
  e.persist();
  throw e;
}

// Fetches the addresses on first use: mosaicist_b200._lib.addresses() loads the library.  Threads that
// meet here each fetch them (the GIL may change hands during the import, so nobody waits for another
// thread while holding it); the first table stays.
const Lib* bind() {
  Gil gil;
  PyObject* mod = PyImport_ImportModule("mosaicist_b200._lib");
  if (!mod) raise();
  PyObject* table = PyObject_CallMethod(mod, "addresses", nullptr);
  Py_DECREF(mod);
  if (!table) raise();
  auto lib = std::make_unique<Lib>();
#define X(name)                                                                        \
  {                                                                                    \
    PyObject* a = PyDict_GetItemString(table, #name);                                  \
    lib->name = a ? reinterpret_cast<decltype(&::name)>(PyLong_AsVoidPtr(a)) : nullptr; \
    if (!lib->name) {                                                                  \
      Py_DECREF(table);                                                                \
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "no address for " #name); \
      raise();                                                            \
    }                                                                                  \
  }
  MSC_ENTRY_POINTS(X)
#undef X
  Py_DECREF(table);
#ifdef MSC_ABI
  const char* abi = lib->msc_abi();
  if (abi && *abi && strcmp(abi, MSC_ABI) != 0) {
    PyErr_SetString(PyExc_RuntimeError, "libmosaicist_sm100a and the host path were built from different headers: "
                                        "run `python -m mosaicist_b200.build`");
    raise();
  }
#endif
  const Lib* seen = nullptr;
  if (!g_lib.compare_exchange_strong(seen, lib.get(), std::memory_order_acq_rel, std::memory_order_acquire)) return seen;
  return lib.release();
}

const Lib& lib() {
  const Lib* l = g_lib.load(std::memory_order_acquire);
  return C10_LIKELY(l != nullptr) ? *l : *bind();
}

// Raises mosaicist_b200._lib.MscError for a status other than MSC_OK.
void check(int code) {
  if (C10_LIKELY(code == MSC_OK)) return;
  Gil gil;
  PyObject* mod = PyImport_ImportModule("mosaicist_b200._lib");
  if (mod) {
    const char* text = lib().msc_last_error();
    PyObject* type = PyObject_GetAttrString(mod, "MscError");
    PyObject* exc = type ? PyObject_CallFunction(type, "is", code, text && *text ? text : "libmosaicist_sm100a call failed") : nullptr;
    if (exc) PyErr_SetObject(type, exc);
    Py_XDECREF(exc);
    Py_XDECREF(type);
    Py_DECREF(mod);
  }
  raise();
}

[[noreturn]] void value_error(const std::string& text) {
  Gil gil;
  PyErr_SetString(PyExc_ValueError, text.c_str());
  raise();
}

// The launch itself runs without the GIL: a full launch queue must not stop other threads.
template <class F>
void launch(F&& f) {
  int code;
  if (PyGILState_Check()) {
    Py_BEGIN_ALLOW_THREADS
    code = f();
    Py_END_ALLOW_THREADS
  } else {
    code = f();
  }
  check(code);
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// ---- argument checks ---------------------------------------------------------------------------

enum Types { kBytes, kF32, kI32, kBf16, kBf16F32, kU8, kPackedInt };

bool type_ok(at::ScalarType t, Types want) {
  switch (want) {
    case kBytes:
      return t == at::kByte || t == at::kChar || t == at::ScalarType::Float8_e4m3fn ||
             t == at::ScalarType::Float8_e8m0fnu || t == at::ScalarType::Float4_e2m1fn_x2;
    case kF32: return t == at::kFloat;
    case kI32: return t == at::kInt;
    case kBf16: return t == at::kBFloat16;
    case kBf16F32: return t == at::kBFloat16 || t == at::kFloat;
    case kU8: return t == at::kByte;
    case kPackedInt: return t == at::kByte || t == at::kChar;
  }
  return false;
}
const char* type_names(Types want) {
  switch (want) {
    case kBytes: return "an 8-bit type";
    case kF32: return "float32";
    case kI32: return "int32";
    case kBf16: return "bfloat16";
    case kBf16F32: return "bfloat16 or float32";
    case kU8: return "uint8";
    case kPackedInt: return "uint8 or int8";
  }
  return "";
}
std::string shape_text(at::IntArrayRef s) {
  std::string t = "(";
  for (size_t i = 0; i < s.size(); ++i) t += (i ? ", " : "") + std::to_string(s[i]);
  return t + (s.size() == 1 ? ",)" : ")");
}

void need(const Tensor& t, const char* name, Types types) {
  if (C10_UNLIKELY(!t.is_cuda())) value_error(std::string(name) + " must be a CUDA tensor");
  if (C10_UNLIKELY(!t.is_contiguous())) value_error(std::string(name) + " must be contiguous");
  if (C10_UNLIKELY(!type_ok(t.scalar_type(), types)))
    value_error(std::string(name) + " has dtype " + c10::toString(t.scalar_type()) + ", expected " + type_names(types));
}
void need(const Tensor& t, const char* name, Types types, std::initializer_list<int64_t> shape) {
  need(t, name, types);
  if (C10_UNLIKELY(t.sizes() != at::IntArrayRef(shape.begin(), shape.size())))
    value_error(std::string(name) + " has shape " + shape_text(t.sizes()) + ", expected " +
                shape_text(at::IntArrayRef(shape.begin(), shape.size())));
}
// A buffer of the caller's that a kernel reads or writes `elements` of, whatever shape it has.
void need_room(const Tensor& t, const char* name, Types types, int64_t elements) {
  need(t, name, types);
  if (C10_UNLIKELY(t.numel() < elements))
    value_error(std::string(name) + " holds " + std::to_string(t.numel()) + " elements, the call needs " + std::to_string(elements));
}
void need_dim(const Tensor& t, const char* name, int64_t dim) {
  if (C10_UNLIKELY(t.dim() != dim))
    value_error(std::string(name) + " must have " + std::to_string(dim) + " dimensions, got shape " + shape_text(t.sizes()));
}

template <class T = void>
const T* ptr(const OptTensor& t) { return t ? static_cast<const T*>(t->data_ptr()) : nullptr; }
template <class T = void>
const T* ptr(const Tensor& t) { return static_cast<const T*>(t.data_ptr()); }

Tensor empty(at::IntArrayRef shape, at::ScalarType type, const Tensor& like) {
  return at::detail::empty_cuda(shape, type, like.device(), std::nullopt);
}

int dt(const Tensor& x) { return x.scalar_type() == at::kBFloat16 ? 0 : 1; }

// ---- the operators on tensors ------------------------------------------------------------------

// NVFP4 over padded batches: (l, m, k/2) by (l, n, k/2).
Tensor gemm_masked(const Tensor& a_q, const Tensor& a_sf, const Tensor& b_q, const Tensor& b_sf,
                   const OptTensor& alpha, const OptTensor& masked_m, const msc_gemm_cfg& cfg, OptTensor out) {
  need(a_q, "a_q", kBytes);
  need_dim(a_q, "a_q", 3);
  need(b_q, "b_q", kBytes);
  need_dim(b_q, "b_q", 3);
  const int64_t l = a_q.size(0), m = a_q.size(1), kh = a_q.size(2), n = b_q.size(1), k = kh * 2;
  need(b_q, "b_q", kBytes, {l, n, kh});
  need(a_sf, "a_sf", kBytes, {l, m / 128, k / 64, 32, 16});
  need(b_sf, "b_sf", kBytes, {l, n / 128, k / 64, 32, 16});
  if (alpha) need(*alpha, "alpha", kF32, {l});
  if (masked_m) need(*masked_m, "masked_m", kI32, {l});
  if (out) need(*out, "out", kBf16, {l, m, n});
  else out = empty({l, m, n}, at::kBFloat16, a_q);
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_grouped_gemm_nvfp4(ptr(a_q), ptr(a_sf), ptr(b_q), ptr(b_sf), ptr<float>(alpha), ptr<int32_t>(masked_m),
                                    out->data_ptr(), l, m, n, k, &cfg, st);
  });
  return *out;
}

// Row-concatenated groups, NVFP4 or MXFP8: `chunk` K-elements share a 512-byte piece of the scale tiling.
Tensor gemm_ragged(bool mxfp8, const Tensor& a_q, const Tensor& a_sf, const Tensor& b_q, const Tensor& b_sf,
                   const Tensor& offsets, const Tensor& rows, const OptTensor& alpha, const OptTensor& row_scale,
                   msc_gemm_cfg cfg, OptTensor out) {
  need(a_q, "a_q", kBytes);
  need_dim(a_q, "a_q", 2);
  need(b_q, "b_q", kBytes);
  need_dim(b_q, "b_q", 3);
  const int64_t total = a_q.size(0), kbytes = a_q.size(1), l = b_q.size(0), n = b_q.size(1);
  const int64_t k = mxfp8 ? kbytes : 2 * kbytes, chunk = mxfp8 ? 128 : 64;
  need(b_q, "b_q", kBytes, {l, n, kbytes});
  need(a_sf, "a_sf", kBytes, {(total + 127) / 128, k / chunk, 32, 16});
  need(b_sf, "b_sf", kBytes, {l, n / 128, k / chunk, 32, 16});
  need(offsets, "group_offsets", kI32, {l});
  need(rows, "group_rows", kI32, {l});
  if (alpha) need(*alpha, "alpha", kF32, {l});
  if (row_scale) need(*row_scale, "row_scale", kF32, {total});
  if (out) need(*out, "out", kBf16, {total, n});
  else out = empty({total, n}, at::kBFloat16, a_q);
  cfg.epilogue = row_scale ? MSC_EPI_ROW_SCALE : MSC_EPI_PLAIN;
  const Lib& f = lib();
  void* st = stream();
  const auto fn = mxfp8 ? f.msc_grouped_gemm_mxfp8_ragged : f.msc_grouped_gemm_nvfp4_ragged;
  launch([&] {
    return fn(ptr(a_q), ptr(a_sf), ptr(b_q), ptr(b_sf), ptr<float>(alpha), ptr<int32_t>(offsets), ptr<int32_t>(rows),
              ptr<float>(row_scale), out->data_ptr(), l, total, n, k, &cfg, st);
  });
  return *out;
}

std::tuple<Tensor, Tensor> swiglu_ragged(const Tensor& a_q, const Tensor& a_sf, const Tensor& w1_q, const Tensor& w1_sf,
                                         const Tensor& offsets, const Tensor& rows, const Tensor& alpha, const Tensor& gs,
                                         const msc_gemm_cfg& cfg, OptTensor d_q, OptTensor d_sf) {
  need(a_q, "a_q", kBytes);
  need_dim(a_q, "a_q", 2);
  need(w1_q, "w1_q", kBytes);
  need_dim(w1_q, "w1_q", 3);
  const int64_t total = a_q.size(0), kh = a_q.size(1), k = 2 * kh, l = w1_q.size(0), n2 = w1_q.size(1), n = n2 / 2;
  need(w1_q, "w1_q", kBytes, {l, n2, kh});
  need(a_sf, "a_sf", kBytes, {(total + 127) / 128, k / 64, 32, 16});
  need(w1_sf, "w1_sf", kBytes, {l, n2 / 128, k / 64, 32, 16});
  need(offsets, "group_offsets", kI32, {l});
  need(rows, "group_rows", kI32, {l});
  need(alpha, "alpha", kF32, {l});
  need(gs, "out_global_scale", kF32, {l});
  if (d_q) {
    need(*d_q, "d_q", kU8, {total, n / 2});
    need(*d_sf, "d_sf", kU8, {(total + 127) / 128, n / 64, 32, 16});
  } else {
    d_q = empty({total, n / 2}, at::kByte, a_q);
    d_sf = at::zeros({(total + 127) / 128, n / 64, 32, 16}, a_q.options().dtype(at::kByte));
  }
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_grouped_gemm_nvfp4_swiglu_ragged(ptr(a_q), ptr(a_sf), ptr(w1_q), ptr(w1_sf), ptr<float>(alpha),
                                                  ptr<int32_t>(offsets), ptr<int32_t>(rows), ptr<float>(gs), d_q->data_ptr(),
                                                  d_sf->data_ptr(), l, total, n2, k, &cfg, st);
  });
  return {*d_q, *d_sf};
}

// (l, m, k), or with silu (l, m, 2k) gate | up.  Scales of rows at or beyond masked_m are zero.
std::tuple<Tensor, Tensor> quantize_nvfp4(const Tensor& x, const Tensor& gs, const OptTensor& masked_m, bool tiled, bool silu) {
  const char* name = silu ? "gateup" : "x";
  need(x, name, silu ? kBf16 : kBf16F32);
  need_dim(x, name, 3);
  const int64_t l = x.size(0), m = x.size(1), k = silu ? x.size(2) / 2 : x.size(2);
  need(gs, "global_scale", kF32, {l});
  if (masked_m) need(*masked_m, "masked_m", kI32, {l});
  Tensor q = empty({l, m, k / 2}, at::kByte, x);
  Tensor sf = tiled ? empty({l, m / 128, k / 64, 32, 16}, at::kByte, x) : empty({l, m, k / 16}, at::kByte, x);
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_quantize_rows(0, ptr(x), silu ? 2 : dt(x), ptr<float>(gs), nullptr, ptr<int32_t>(masked_m), q.data_ptr(),
                               sf.data_ptr(), (tiled ? 1 : 0) | MSC_SF_ZERO_REST, nullptr, l, l * m, m, k, st);
  });
  return {q, sf};
}

std::tuple<Tensor, Tensor> quantize_nvfp4_ragged(const Tensor& x, const Tensor& gs, const Tensor& offsets, const Tensor& rows,
                                                 bool silu, OptTensor q, OptTensor sf) {
  need(x, "x", kBf16F32);
  need_dim(x, "x", 2);
  const int64_t total = x.size(0), k = silu ? x.size(1) / 2 : x.size(1), l = gs.size(0);
  need(gs, "global_scale", kF32, {l});
  need(offsets, "group_offsets", kI32, {l});
  need(rows, "group_rows", kI32, {l});
  if (silu && x.scalar_type() != at::kBFloat16) value_error("the fused SiLU form takes bf16 input");
  const bool fresh = !q;
  if (fresh) {
    q = empty({total, k / 2}, at::kByte, x);
    sf = empty({(total + 127) / 128, k / 64, 32, 16}, at::kByte, x);
  } else {
    need(*q, "q", kU8, {total, k / 2});
    need(*sf, "sf", kU8, {(total + 127) / 128, k / 64, 32, 16});
  }
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_quantize_rows(0, ptr(x), silu ? 2 : dt(x), ptr<float>(gs), ptr<int32_t>(offsets), ptr<int32_t>(rows),
                               q->data_ptr(), sf->data_ptr(), 1 | (fresh ? MSC_SF_ZERO_REST : 0), nullptr, l, total, 0, k, st);
  });
  return {*q, *sf};
}

Tensor global_scale_for(const Tensor& x, double numerator, OptTensor out) {
  need(x, "x", kBf16F32);
  if (x.dim() < 1 || x.size(0) < 1) value_error("x must have at least one group");
  const int64_t l = x.size(0);
  if (out) need(*out, "out", kF32, {l});
  else out = empty({l}, at::kFloat, x);
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_amax_global_scale(ptr(x), dt(x), l, x.numel() / l, (float)numerator, static_cast<float*>(out->data_ptr()), st);
  });
  return *out;
}

std::tuple<Tensor, Tensor> quantize_mxfp8(const Tensor& x, bool tiled, const OptTensor& offsets, const OptTensor& rows,
                                          OptTensor q, OptTensor sf) {
  need(x, "x", kBf16F32);
  need_dim(x, "x", 2);
  const int64_t total = x.size(0), k = x.size(1);
  if (offsets && !tiled) value_error("the ragged form writes tiled scales");
  int64_t l = 0;
  if (offsets) {
    l = offsets->size(0);
    need(*offsets, "group_offsets", kI32, {l});
    if (!rows) value_error("group_rows is required with group_offsets");
    need(*rows, "group_rows", kI32, {l});
  }
  const bool fresh = !q;
  if (fresh) {
    q = empty({total, k}, at::kByte, x);
    sf = tiled ? empty({(total + 127) / 128, k / 128, 32, 16}, at::kByte, x) : empty({total, k / 32}, at::kByte, x);
  } else {
    need_room(*q, "q", kBytes, total * k);
    need_room(*sf, "sf", kBytes, tiled ? (total + 127) / 128 * (k / 128) * 512 : total * (k / 32));
  }
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_quantize_rows(1, ptr(x), dt(x), nullptr, ptr<int32_t>(offsets), offsets ? ptr<int32_t>(rows) : nullptr,
                               q->data_ptr(), sf->data_ptr(), (tiled ? 1 : 0) | (fresh ? MSC_SF_ZERO_REST : 0), nullptr, l,
                               total, 0, k, st);
  });
  return {*q, *sf};
}

Tensor gemm_f16(const Tensor& a, const Tensor& b, OptTensor out, int max_ctas) {
  const at::ScalarType t = a.scalar_type();
  if (t != b.scalar_type() || (t != at::kHalf && t != at::kBFloat16))
    value_error("a and b must both be float16 or both bfloat16");
  if (a.dim() != 2 || b.dim() != 2 || a.size(1) != b.size(0))
    value_error("shapes " + shape_text(a.sizes()) + " and " + shape_text(b.sizes()) + " do not multiply");
  if (!a.is_cuda() || !b.is_cuda() || a.stride(1) != 1 || b.stride(1) != 1)
    value_error("a and b must be CUDA tensors with unit stride along their rows");
  const int64_t m = a.size(0), k = a.size(1), n = b.size(1);
  if (!out) out = empty({m, n}, t, a);
  else if (!out->is_cuda() || out->scalar_type() != t || out->dim() != 2 || out->size(0) != m || out->size(1) != n || out->stride(1) != 1)
    value_error("out must be an (m, n) CUDA tensor in the input dtype with unit stride along rows");
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_gemm_f16(ptr(a), ptr(b), out->data_ptr(), m, n, k, a.stride(0), b.stride(0), out->stride(0),
                          t == at::kHalf ? 0 : 1, max_ctas, st);
  });
  return *out;
}

Tensor dequant_int4(const Tensor& b_q, const Tensor& scales, int64_t group_size, OptTensor out) {
  need(b_q, "b_q", kPackedInt);
  need_dim(b_q, "b_q", 3);
  const int64_t l = b_q.size(0), n = b_q.size(1), k = b_q.size(2) * 2;
  if (group_size <= 0) value_error("group_size must be positive");
  need(scales, "scales", kBf16, {l, n, k / group_size});
  if (!out) out = empty({l, n, k}, at::kBFloat16, b_q);
  else need_room(*out, "out", kBf16, l * n * k);
  const Lib& f = lib();
  void* st = stream();
  launch([&] { return f.msc_int4_dequant_bf16(ptr(b_q), ptr(scales), out->data_ptr(), l, n, k, group_size, st); });
  return *out;
}

Tensor gemm_bf16_ragged(const Tensor& a, const Tensor& b, const Tensor& offsets, const Tensor& rows, const OptTensor& alpha,
                        OptTensor out, int max_ctas) {
  need(a, "a", kBf16);
  need_dim(a, "a", 2);
  need_dim(b, "b", 3);
  const int64_t total = a.size(0), k = a.size(1), l = b.size(0), n = b.size(1);
  need(b, "b", kBf16, {l, n, k});
  need(offsets, "group_offsets", kI32, {l});
  need(rows, "group_rows", kI32, {l});
  if (alpha) need(*alpha, "alpha", kF32, {l});
  if (!out) out = empty({total, n}, at::kBFloat16, a);
  else need_room(*out, "out", kBf16, total * n);
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_grouped_gemm_bf16_ragged(ptr(a), ptr(b), ptr<float>(alpha), ptr<int32_t>(offsets), ptr<int32_t>(rows),
                                          out->data_ptr(), l, total, n, k, max_ctas, st);
  });
  return *out;
}

// fused: -1 = choose.
Tensor gemm_int4_ragged(const Tensor& a, const Tensor& b_q, const Tensor& scales, const Tensor& offsets, const Tensor& rows,
                        const OptTensor& alpha, int64_t group_size, const OptTensor& workspace, OptTensor out, int fused,
                        int max_ctas) {
  need(b_q, "b_q", kPackedInt);
  need_dim(b_q, "b_q", 3);
  const int64_t l = b_q.size(0), n = b_q.size(1), k = b_q.size(2) * 2;
  if (group_size <= 0) value_error("group_size must be positive");
  const bool can_fuse = k % 64 == 0 && group_size % 64 == 0 && k % group_size == 0;
  if (fused < 0) fused = can_fuse && !workspace;
  if (!fused) {
    const Tensor b = dequant_int4(b_q, scales, group_size, workspace);
    return gemm_bf16_ragged(a, b, offsets, rows, alpha, out, max_ctas);
  }
  if (!can_fuse) value_error("the fused kernel needs k and group_size to be multiples of 64");
  need(a, "a", kBf16);
  need_dim(a, "a", 2);
  const int64_t total = a.size(0);
  need(a, "a", kBf16, {total, k});
  need(scales, "scales", kBf16, {l, n, k / group_size});
  need(offsets, "group_offsets", kI32, {l});
  need(rows, "group_rows", kI32, {l});
  if (alpha) need(*alpha, "alpha", kF32, {l});
  if (!out) out = empty({total, n}, at::kBFloat16, a);
  else need_room(*out, "out", kBf16, total * n);
  const Lib& f = lib();
  void* st = stream();
  launch([&] {
    return f.msc_grouped_gemm_bf16_int4_ragged(ptr(a), ptr(b_q), ptr(scales), ptr<float>(alpha), ptr<int32_t>(offsets),
                                               ptr<int32_t>(rows), out->data_ptr(), l, total, n, k, group_size, max_ctas, st);
  });
  return *out;
}

// Whether a factor of the masked layer is what msc_moe_masked reads: one fp32 per expert.
bool per_expert(const OptTensor& t, int64_t l) {
  return t && t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->dim() == 1 && t->size(0) == l;
}

// The masked MoE layer in one call; zero_rest: rows at or beyond masked_m come back as zeros.  Nothing
// is returned for the forms that only the layer's separate steps take (mosaicist_b200.moe): fp32
// activations, global scales and alphas that have to be broadcast, converted or copied first, a
// second weight whose rows are not hidden's columns, sizes the fused call is not built for.
OptTensor moe_masked(const Tensor& hidden, const Tensor& w1_q, const Tensor& w1_sf, const OptTensor& w1_gs, const OptTensor& w1_alpha,
                     const Tensor& w2_q, const Tensor& w2_sf, const OptTensor& w2_gs, const OptTensor& w2_alpha,
                     const Tensor& masked_m, const Tensor& in_gs, const Tensor& a2_gs, const OptTensor& g1_alpha,
                     const OptTensor& g2_alpha, bool zero_rest) {
  if (hidden.scalar_type() != at::kBFloat16 || hidden.dim() != 3 || w1_q.dim() != 3 || w2_q.dim() != 3) return std::nullopt;
  const int64_t l = hidden.size(0), m = hidden.size(1), k = hidden.size(2), n2 = w1_q.size(1), n = n2 / 2;
  if (m % 128 || k % 128 || n % 64 || w2_q.size(1) != k) return std::nullopt;
  if (g1_alpha || g2_alpha) {
    if (!per_expert(g1_alpha, l) || !per_expert(g2_alpha, l)) return std::nullopt;
  } else if (!per_expert(w1_gs, l) || !per_expert(w1_alpha, l) || !per_expert(w2_gs, l) || !per_expert(w2_alpha, l)) {
    return std::nullopt;
  }
  need(hidden, "x", kBf16);
  need(in_gs, "global_scale", kF32, {l});
  need(masked_m, "masked_m", kI32, {l});
  need(w1_q, "w1_q", kBytes, {l, n2, k / 2});
  need(w1_sf, "w1_sf", kBytes, {l, n2 / 128, k / 64, 32, 16});
  need(w2_q, "b_q", kBytes, {l, k, n / 2});
  need(w2_sf, "b_sf", kBytes, {l, k / 128, n / 64, 32, 16});
  need(a2_gs, "out_global_scale", kF32, {l});
  const Lib& f = lib();
  const size_t bytes = f.msc_moe_masked_workspace(l, m, k, n);
  Tensor ws = empty({(int64_t)bytes}, at::kByte, hidden);
  Tensor out = empty({l, m, k}, at::kBFloat16, hidden);
  void* st = stream();
  launch([&] {
    return f.msc_moe_masked(ptr(hidden), ptr(w1_q), ptr(w1_sf), ptr<float>(w1_gs), ptr<float>(w1_alpha), ptr(w2_q), ptr(w2_sf),
                            ptr<float>(w2_gs), ptr<float>(w2_alpha), ptr<int32_t>(masked_m), ptr<float>(in_gs),
                            ptr<float>(a2_gs), ptr<float>(g1_alpha), ptr<float>(g2_alpha), ws.data_ptr(), bytes,
                            out.data_ptr(), zero_rest ? 1 : 0, l, m, k, n, st);
  });
  return out;
}

// The layer's separate steps, written in Python: the torch operator's way for what moe_masked leaves.
Tensor moe_masked_steps(std::initializer_list<Tensor> args) {
  Gil gil;
  PyObject* mod = PyImport_ImportModule("mosaicist_b200.moe");
  PyObject* fn = mod ? PyObject_GetAttrString(mod, "moe_masked_steps") : nullptr;
  Py_XDECREF(mod);
  PyObject* tuple = fn ? PyTuple_New(args.size()) : nullptr;
  Py_ssize_t i = 0;
  bool ok = tuple != nullptr;
  for (const Tensor& t : args) {
    if (!ok) break;
    PyObject* o = THPVariable_Wrap(t);
    ok = o != nullptr;
    if (ok) PyTuple_SET_ITEM(tuple, i++, o);
  }
  PyObject* out = ok ? PyObject_CallObject(fn, tuple) : nullptr;
  Py_XDECREF(tuple);
  Py_XDECREF(fn);
  if (!out) raise();
  const Tensor result = THPVariable_Unpack(out);
  Py_DECREF(out);
  return result;
}

// ---- the CPython module ------------------------------------------------------------------------

const Tensor& tensor(PyObject* o, const char* name) {
  if (C10_UNLIKELY(!THPVariable_Check(o))) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor, got %s", name, Py_TYPE(o)->tp_name);
    raise();
  }
  return THPVariable_Unpack(o);
}
OptTensor opt_tensor(PyObject* o, const char* name) {
  if (o == Py_None) return std::nullopt;
  return tensor(o, name);
}
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) raise();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) raise();
  return v != 0;
}
void arity(Py_ssize_t got, Py_ssize_t want, const char* name) {
  if (got == want) return;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, got);
  raise();
}
PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap(const std::tuple<Tensor, Tensor>& t) {
  PyObject* a = wrap(std::get<0>(t));
  PyObject* b = a ? wrap(std::get<1>(t)) : nullptr;
  if (!b) {
    Py_XDECREF(a);
    raise();
  }
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, a);
  PyTuple_SET_ITEM(r, 1, b);
  return r;
}
// (q, sf) or None
void opt_pair(PyObject* o, OptTensor& q, OptTensor& sf) {
  if (o == Py_None) return;
  PyObject* seq = PySequence_Fast(o, "out must be a pair of tensors");
  if (!seq) raise();
  if (PySequence_Fast_GET_SIZE(seq) != 2) {
    Py_DECREF(seq);
    value_error("out must be a pair of tensors");
  }
  q = tensor(PySequence_Fast_GET_ITEM(seq, 0), "q");
  sf = tensor(PySequence_Fast_GET_ITEM(seq, 1), "sf");
  Py_DECREF(seq);
}
// ops.GemmConfig -> the C structure
msc_gemm_cfg config(PyObject* o) {
  static PyObject* const names[] = {
      PyUnicode_InternFromString("tile_n"),   PyUnicode_InternFromString("stages"),   PyUnicode_InternFromString("raster"),
      PyUnicode_InternFromString("max_ctas"), PyUnicode_InternFromString("cta_pair"), PyUnicode_InternFromString("sf_warps")};
  msc_gemm_cfg c = {};
  int* const fields[] = {&c.tile_n, &c.stages, &c.raster, &c.max_ctas, &c.cta_pair, &c.sf_warps};
  for (int i = 0; i < 6; ++i) {
    PyObject* v = PyObject_GetAttr(o, names[i]);
    if (!v) raise();
    *fields[i] = (int)PyLong_AsLong(v);
    Py_DECREF(v);
    if (PyErr_Occurred()) raise();
  }
  return c;
}

#define PY_FUNCTION(name, count)                                                     \
  PyObject* name##_body(PyObject* const* a);                                         \
  PyObject* py_##name(PyObject*, PyObject* const* a, Py_ssize_t n) {                 \
    HANDLE_TH_ERRORS                                                                 \
    arity(n, count, #name);                                                          \
    return name##_body(a);                                                           \
    END_HANDLE_TH_ERRORS                                                             \
  }                                                                                  \
  PyObject* name##_body(PyObject* const* a)

PY_FUNCTION(masked_grouped_gemm, 8) {
  return wrap(gemm_masked(tensor(a[0], "a_q"), tensor(a[1], "a_sf"), tensor(a[2], "b_q"), tensor(a[3], "b_sf"),
                          opt_tensor(a[4], "alpha"), opt_tensor(a[5], "masked_m"), config(a[6]), opt_tensor(a[7], "out")));
}
PY_FUNCTION(ragged_grouped_gemm, 11) {
  return wrap(gemm_ragged(truth(a[0]), tensor(a[1], "a_q"), tensor(a[2], "a_sf"), tensor(a[3], "b_q"), tensor(a[4], "b_sf"),
                          tensor(a[5], "group_offsets"), tensor(a[6], "group_rows"), opt_tensor(a[7], "alpha"),
                          opt_tensor(a[8], "row_scale"), config(a[9]), opt_tensor(a[10], "out")));
}
PY_FUNCTION(ragged_gemm1_swiglu_quantize, 10) {
  OptTensor q, sf;
  opt_pair(a[9], q, sf);
  return wrap(swiglu_ragged(tensor(a[0], "a_q"), tensor(a[1], "a_sf"), tensor(a[2], "w1_q"), tensor(a[3], "w1_sf"),
                            tensor(a[4], "group_offsets"), tensor(a[5], "group_rows"), tensor(a[6], "alpha"),
                            tensor(a[7], "out_global_scale"), config(a[8]), q, sf));
}
PY_FUNCTION(quantize_nvfp4, 5) {
  return wrap(quantize_nvfp4(tensor(a[0], "x"), tensor(a[1], "global_scale"), opt_tensor(a[2], "masked_m"), truth(a[3]),
                             truth(a[4])));
}
PY_FUNCTION(quantize_nvfp4_ragged, 6) {
  OptTensor q, sf;
  opt_pair(a[5], q, sf);
  return wrap(quantize_nvfp4_ragged(tensor(a[0], "x"), tensor(a[1], "global_scale"), tensor(a[2], "group_offsets"),
                                    tensor(a[3], "group_rows"), truth(a[4]), q, sf));
}
PY_FUNCTION(global_scale_for, 3) {
  const double numerator = PyFloat_AsDouble(a[1]);
  if (numerator == -1.0 && PyErr_Occurred()) raise();
  return wrap(global_scale_for(tensor(a[0], "x"), numerator, opt_tensor(a[2], "out")));
}
PY_FUNCTION(quantize_mxfp8, 5) {
  OptTensor q, sf;
  opt_pair(a[4], q, sf);
  return wrap(quantize_mxfp8(tensor(a[0], "x"), truth(a[1]), opt_tensor(a[2], "group_offsets"), opt_tensor(a[3], "group_rows"), q, sf));
}
PY_FUNCTION(gemm_f16, 4) {
  return wrap(gemm_f16(tensor(a[0], "a"), tensor(a[1], "b"), opt_tensor(a[2], "out"), (int)integer(a[3])));
}
PY_FUNCTION(dequant_int4, 4) {
  return wrap(dequant_int4(tensor(a[0], "b_q"), tensor(a[1], "scales"), integer(a[2]), opt_tensor(a[3], "out")));
}
PY_FUNCTION(ragged_grouped_gemm_bf16, 7) {
  return wrap(gemm_bf16_ragged(tensor(a[0], "a"), tensor(a[1], "b"), tensor(a[2], "group_offsets"), tensor(a[3], "group_rows"),
                               opt_tensor(a[4], "alpha"), opt_tensor(a[5], "out"), (int)integer(a[6])));
}
PY_FUNCTION(mixed_grouped_gemm_int4, 11) {
  return wrap(gemm_int4_ragged(tensor(a[0], "a"), tensor(a[1], "b_q"), tensor(a[2], "scales"), tensor(a[3], "group_offsets"),
                               tensor(a[4], "group_rows"), opt_tensor(a[5], "alpha"), integer(a[6]), opt_tensor(a[7], "workspace"),
                               opt_tensor(a[8], "out"), a[9] == Py_None ? -1 : (int)truth(a[9]), (int)integer(a[10])));
}
// -> the result, or None where the separate steps have to be taken
PY_FUNCTION(moe_masked, 14) {
  const OptTensor out =
      moe_masked(tensor(a[0], "x"), tensor(a[1], "w1_q"), tensor(a[2], "w1_sf"), opt_tensor(a[3], "w1_gs"),
                 opt_tensor(a[4], "w1_alpha"), tensor(a[5], "w2_q"), tensor(a[6], "w2_sf"), opt_tensor(a[7], "w2_gs"),
                 opt_tensor(a[8], "w2_alpha"), tensor(a[9], "masked_m"), tensor(a[10], "global_scale"),
                 tensor(a[11], "a2_global_scale"), opt_tensor(a[12], "folded alpha"), opt_tensor(a[13], "folded alpha"), false);
  if (out) return wrap(*out);
  Py_RETURN_NONE;
}

// ---- the routed layer (mosaicist_b200.moe.MegaMoE) ----------------------------------------------
// The layer object owns its workspaces; its attributes are read by name on every call, as the
// Python form of the same steps does, so whoever replaces one of them is heard.

struct Layer {
  PyObject* self;
  std::deque<Tensor> held;    // what the call uses stays alive until it returns, whoever rebinds the attribute
  int64_t num(PyObject* name) {
    PyObject* v = get(name);
    const long long n = PyLong_AsLongLong(v);
    Py_DECREF(v);
    if (n == -1 && PyErr_Occurred()) raise();
    return n;
  }
  // null where the attribute is None
  const Tensor* opt(PyObject* name) {
    PyObject* v = get(name);
    const bool none = v == Py_None, tensor = !none && THPVariable_Check(v);
    if (tensor) held.push_back(THPVariable_Unpack(v));
    Py_DECREF(v);
    if (none) return nullptr;
    if (!tensor) value_error("a buffer of the layer is not a tensor");
    return &held.back();
  }
  const Tensor& t(PyObject* name) {
    const Tensor* v = opt(name);
    if (!v) value_error("a buffer of the layer is missing");
    return *v;
  }
  template <class T>
  T* p(PyObject* name) { return static_cast<T*>(t(name).data_ptr()); }

 private:
  PyObject* get(PyObject* name) const {
    PyObject* v = PyObject_GetAttr(self, name);
    if (!v) raise();
    return v;
  }
};
#define ATTR(name) static PyObject* const s_##name = PyUnicode_InternFromString(#name)

void route(Layer& layer, const Tensor& logits) {
  ATTR(ids); ATTR(weights); ATTR(topk);
  need_dim(logits, "logits", 2);
  const int64_t tokens = logits.size(0), experts = logits.size(1), topk = layer.num(s_topk);
  need_room(logits, "logits", kF32, tokens * experts);
  need_room(layer.t(s_ids), "ids", kI32, tokens * topk);
  need_room(layer.t(s_weights), "weights", kF32, tokens * topk);
  int32_t* ids = layer.p<int32_t>(s_ids);
  float* weights = layer.p<float>(s_weights);
  const Lib& f = lib();
  void* st = stream();
  launch([&] { return f.msc_moe_route_topk(ptr<float>(logits), ids, weights, tokens, experts, topk, st); });
}

// route(self, logits)
PY_FUNCTION(moe_route, 2) {
  Layer layer{a[0]};
  route(layer, tensor(a[1], "logits"));
  Py_RETURN_NONE;
}

// dispatch(self, tokens, logits or None): routing, plan, gather + quantise into a_q / a_sf
PY_FUNCTION(moe_dispatch, 3) {
  ATTR(ids); ATTR(weights); ATTR(rank); ATTR(group_rows); ATTR(group_offsets); ATTR(total_rows); ATTR(scratch); ATTR(topk);
  ATTR(E); ATTR(expert_first); ATTR(input_gs); ATTR(h); ATTR(a_q); ATTR(a_sf); ATTR(row_weight); ATTR(row_token); ATTR(sf_rows);
  ATTR(rows_cap);
  Layer layer{a[0]};
  const Tensor& tokens = tensor(a[1], "tokens");
  if (tokens.dim() < 1) value_error("tokens must have a dimension of tokens");
  const int64_t T = tokens.size(0), K = layer.num(s_topk), E = layer.num(s_E), first = layer.num(s_expert_first);
  const int64_t h = layer.num(s_h), cap = layer.num(s_rows_cap);
  need(tokens, "tokens", kBf16);
  if (tokens.numel() != T * h) value_error("tokens has shape " + shape_text(tokens.sizes()) + ", expected " + shape_text({T, h}));
  for (PyObject* name : {s_ids, s_rank}) need_room(layer.t(name), "ids / rank", kI32, T * K);
  if (a[2] != Py_None) route(layer, tensor(a[2], "logits"));
  int32_t *ids = layer.p<int32_t>(s_ids), *rank = layer.p<int32_t>(s_rank), *rows = layer.p<int32_t>(s_group_rows);
  int32_t *offsets = layer.p<int32_t>(s_group_offsets), *total = layer.p<int32_t>(s_total_rows), *scratch = layer.p<int32_t>(s_scratch);
  const Tensor* staged = layer.opt(s_sf_rows);
  void* sf_rows = staged ? staged->data_ptr() : nullptr;
  const float *weights = layer.p<float>(s_weights), *gs = layer.p<float>(s_input_gs);
  void *a_q = layer.p<void>(s_a_q), *a_sf = layer.p<void>(s_a_sf);
  float* row_weight = layer.p<float>(s_row_weight);
  int32_t* row_token = layer.p<int32_t>(s_row_token);
  const Lib& f = lib();
  void* st = stream();
  launch([&] { return f.msc_moe_plan(ids, T * K, first, E, rank, rows, offsets, total, scratch, st); });
  launch([&] {
    return f.msc_moe_permute_quantize(ptr(tokens), ids, weights, rank, offsets, gs, T, h, K, first, E, a_q, a_sf, row_weight,
                                      row_token, sf_rows, cap, total, st);
  });
  Py_RETURN_NONE;
}

// combine(self, tokens, out or None) -> out: the sum of each token's expert rows
PY_FUNCTION(moe_combine, 3) {
  ATTR(y); ATTR(ids); ATTR(rank); ATTR(group_offsets); ATTR(h); ATTR(topk); ATTR(expert_first); ATTR(E);
  Layer layer{a[0]};
  const Tensor& tokens = tensor(a[1], "tokens");
  const int64_t T = tokens.size(0), h = layer.num(s_h);
  OptTensor out = opt_tensor(a[2], "out");
  if (!out) out = empty({T, h}, at::kBFloat16, tokens);
  else need_room(*out, "out", kBf16, T * h);
  const int64_t K = layer.num(s_topk), first = layer.num(s_expert_first), E = layer.num(s_E);
  const void* y = layer.p<void>(s_y);
  const int32_t *ids = layer.p<int32_t>(s_ids), *rank = layer.p<int32_t>(s_rank), *offsets = layer.p<int32_t>(s_group_offsets);
  const Lib& f = lib();
  void* st = stream();
  launch([&] { return f.msc_moe_unpermute(y, ids, rank, offsets, out->data_ptr(), T, h, K, first, E, st); });
  return wrap(*out);
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {METHOD(masked_grouped_gemm),
                          METHOD(ragged_grouped_gemm),
                          METHOD(ragged_gemm1_swiglu_quantize),
                          METHOD(quantize_nvfp4),
                          METHOD(quantize_nvfp4_ragged),
                          METHOD(global_scale_for),
                          METHOD(quantize_mxfp8),
                          METHOD(gemm_f16),
                          METHOD(dequant_int4),
                          METHOD(ragged_grouped_gemm_bf16),
                          METHOD(mixed_grouped_gemm_int4),
                          METHOD(moe_masked),
                          METHOD(moe_route),
                          METHOD(moe_dispatch),
                          METHOD(moe_combine),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

// ---- torch operators ---------------------------------------------------------------------------
// Operators return fresh tensors: rows that a call has nothing to say about come back as zeros.

OptTensor zeros(at::IntArrayRef shape, const Tensor& like) { return at::zeros(shape, like.options().dtype(at::kBFloat16)); }

void zero_dead_rows(Tensor& q, const OptTensor& masked_m) {
  if (!masked_m) return;
  const Tensor rows = at::arange(q.size(1), masked_m->options());
  q.masked_fill_(rows.view({1, -1, 1}).ge(masked_m->view({-1, 1, 1})), 0);
}

Tensor op_grouped_gemm_nvfp4(const Tensor& a_q, const Tensor& a_sf, const Tensor& b_q, const Tensor& b_sf,
                             const OptTensor& alpha, const OptTensor& masked_m) {
  need_dim(a_q, "a_q", 3);
  need_dim(b_q, "b_q", 3);
  OptTensor out;
  if (masked_m) out = zeros({a_q.size(0), a_q.size(1), b_q.size(1)}, a_q);
  return gemm_masked(a_q, a_sf, b_q, b_sf, alpha, masked_m, msc_gemm_cfg{}, out);
}
Tensor op_grouped_gemm_nvfp4_ragged(const Tensor& a_q, const Tensor& a_sf, const Tensor& b_q, const Tensor& b_sf,
                                    const Tensor& offsets, const Tensor& rows, const OptTensor& alpha, const OptTensor& row_scale) {
  need_dim(a_q, "a_q", 2);
  need_dim(b_q, "b_q", 3);
  return gemm_ragged(false, a_q, a_sf, b_q, b_sf, offsets, rows, alpha, row_scale, msc_gemm_cfg{}, zeros({a_q.size(0), b_q.size(1)}, a_q));
}
Tensor op_grouped_gemm_mxfp8_ragged(const Tensor& a_q, const Tensor& a_sf, const Tensor& b_q, const Tensor& b_sf,
                                    const Tensor& offsets, const Tensor& rows, const OptTensor& alpha, const OptTensor& row_scale) {
  need_dim(a_q, "a_q", 2);
  need_dim(b_q, "b_q", 3);
  return gemm_ragged(true, a_q, a_sf, b_q, b_sf, offsets, rows, alpha, row_scale, msc_gemm_cfg{}, zeros({a_q.size(0), b_q.size(1)}, a_q));
}
std::tuple<Tensor, Tensor> op_quantize_nvfp4(const Tensor& x, const Tensor& gs, const OptTensor& masked_m) {
  auto r = quantize_nvfp4(x, gs, masked_m, true, false);
  zero_dead_rows(std::get<0>(r), masked_m);
  return r;
}
std::tuple<Tensor, Tensor> op_silu_mul_quantize_nvfp4(const Tensor& gateup, const Tensor& gs, const OptTensor& masked_m) {
  auto r = quantize_nvfp4(gateup, gs, masked_m, true, true);
  zero_dead_rows(std::get<0>(r), masked_m);
  return r;
}
Tensor op_global_scale_for(const Tensor& x) { return global_scale_for(x, 2688.0, std::nullopt); }
std::tuple<Tensor, Tensor> op_quantize_mxfp8(const Tensor& x) {
  return quantize_mxfp8(x, true, std::nullopt, std::nullopt, std::nullopt, std::nullopt);
}
Tensor op_gemm_f16(const Tensor& a, const Tensor& b) { return gemm_f16(a, b, std::nullopt, 0); }
Tensor op_grouped_gemm_bf16_int4_ragged(const Tensor& a, const Tensor& b_q, const Tensor& scales, const Tensor& offsets,
                                        const Tensor& rows, const OptTensor& alpha, int64_t group_size) {
  need_dim(a, "a", 2);
  need_dim(b_q, "b_q", 3);
  return gemm_int4_ragged(a, b_q, scales, offsets, rows, alpha, group_size, std::nullopt, zeros({a.size(0), b_q.size(1)}, a), -1, 0);
}
Tensor op_moe_masked(const Tensor& hidden, const Tensor& w1_q, const Tensor& w1_sf, const Tensor& w1_gs, const Tensor& w1_alpha,
                     const Tensor& w2_q, const Tensor& w2_sf, const Tensor& w2_gs, const Tensor& w2_alpha,
                     const Tensor& masked_m, const Tensor& in_gs, const Tensor& a2_gs) {
  const OptTensor out = moe_masked(hidden, w1_q, w1_sf, w1_gs, w1_alpha, w2_q, w2_sf, w2_gs, w2_alpha, masked_m, in_gs, a2_gs,
                                   std::nullopt, std::nullopt, true);
  if (out) return *out;
  Tensor r = moe_masked_steps({hidden, w1_q, w1_sf, w1_gs, w1_alpha, w2_q, w2_sf, w2_gs, w2_alpha, masked_m, in_gs, a2_gs});
  zero_dead_rows(r, masked_m);
  return r;
}

// The operators' schemas are in mosaicist_b200.torch_ops.
TORCH_LIBRARY_IMPL(mosaicist_sm100a, CUDA, m) {
  m.impl("grouped_gemm_nvfp4", op_grouped_gemm_nvfp4);
  m.impl("grouped_gemm_nvfp4_ragged", op_grouped_gemm_nvfp4_ragged);
  m.impl("quantize_nvfp4", op_quantize_nvfp4);
  m.impl("silu_mul_quantize_nvfp4", op_silu_mul_quantize_nvfp4);
  m.impl("global_scale_for", op_global_scale_for);
  m.impl("quantize_mxfp8", op_quantize_mxfp8);
  m.impl("grouped_gemm_mxfp8_ragged", op_grouped_gemm_mxfp8_ragged);
  m.impl("gemm_f16", op_gemm_f16);
  m.impl("grouped_gemm_bf16_int4_ragged", op_grouped_gemm_bf16_int4_ragged);
  m.impl("moe_masked", op_moe_masked);
}
// No operator has a derivative: a backward pass through one raises.  (Without a kernel under this
// key torch only warns and leaves the operator's share out of the gradients.)
TORCH_LIBRARY_IMPL(mosaicist_sm100a, Autograd, m) {
  for (const char* name : {"grouped_gemm_nvfp4", "grouped_gemm_nvfp4_ragged", "quantize_nvfp4", "silu_mul_quantize_nvfp4",
                           "global_scale_for", "quantize_mxfp8", "grouped_gemm_mxfp8_ragged", "gemm_f16",
                           "grouped_gemm_bf16_int4_ragged", "moe_masked"})
    m.impl(name, torch::autograd::autogradNotImplementedFallback());
}

}  // namespace

PyMODINIT_FUNC PyInit__host_ops(void) { return PyModule_Create(&kModule); }
