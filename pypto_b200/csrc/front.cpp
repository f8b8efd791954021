// Native front end of the operator entry points: argument checks, workspace and the C call in one step.
//
// A decode step is a handful of calls whose kernels take a few microseconds each, so what the host does per call counts:
// checking two dozen tensors one by one in Python took longer (40-130 us a call) than the kernels ran.  Every function
// here takes an entry point's tensors as they are, checks dtype, shape, contiguity and device against a short pattern,
// takes the workspace from torch's caching allocator (stream-ordered, as torch.empty would), fills the argument block
// and enqueues the operator on the current stream: 8-17 us a call with its two to four launches.  A call that does not fit its pattern -- a
// wrong argument, a tensor on another device than the current one, a layout only the Python layer accepts -- is
// declined (False / None) before anything is enqueued, and the Python layer, which knows every accepted form and every
// error message, takes it from there.
//
// The library's entry points arrive as addresses from the ctypes binding (bind()), so there is one loaded library.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <algorithm>
#include <cstring>
#include <initializer_list>

#include "../../include/dsv32_b200.h"

namespace {

constexpr int kMaxDevices = 64;
uint32_t* g_status[kMaxDevices] = {};   // device status words, set by the Python layer when it creates them
PyObject* g_on_error = nullptr;         // _lib.check

// Entry points of the library, by the names of the header.
#define FRONT_ENTRIES(X)                                                                                              \
  X(dsv32_sfa_workspace_bytes) X(dsv32_sfa_quant) X(dsv32_sfa_bf16_cache) X(dsv32_sparse_attention_antiquant)         \
  X(dsv32_indexer_workspace_bytes) X(dsv32_indexer_topk) X(dsv32_prolog_workspace_bytes) X(dsv32_indexer_prolog)      \
  X(dsv32_mla_prolog_workspace_bytes) X(dsv32_mla_prolog) X(dsv32_mla_indexer_prolog)                                 \
  X(dsv32_prolog_v4_workspace_bytes) X(dsv32_indexer_prolog_v4) X(dsv32_hc_pre_workspace_bytes) X(dsv32_hc_pre)       \
  X(dsv32_scfa_workspace_bytes) X(dsv32_sparse_compress_attention)                                                    \
  X(dsv32_mla_prolog_v4_workspace_bytes) X(dsv32_mla_prolog_v4) X(dsv32_compressor_workspace_bytes) X(dsv32_compressor) \
  X(dsv32_pg_indexer_prolog_workspace_bytes) X(dsv32_pg_indexer_prolog)
#define DECLARE_ENTRY(name) decltype(&::name) p_##name = nullptr;
FRONT_ENTRIES(DECLARE_ENTRY)
#undef DECLARE_ENTRY
bool g_bound = false;

constexpr auto BF16 = at::kBFloat16;
constexpr auto F16 = at::kHalf;
constexpr auto F32 = at::kFloat;
constexpr auto I8 = at::kChar;
constexpr auto U8 = at::kByte;
constexpr auto I32 = at::kInt;
constexpr auto I64 = at::kLong;

// Dimension patterns: a size, ANY, or a variable A..F that takes the size it meets first and has to meet it again.
constexpr int64_t ANY = -1;
enum : int64_t { A = -2, B = -3, C_ = -4, D = -5, E = -6, F = -7 };

struct Call {
  bool ok;
  int dev = -1;
  int64_t var[6] = {-1, -1, -1, -1, -1, -1};

  Call() : ok(g_bound) {}
  int64_t operator[](int64_t v) const { return var[-2 - v]; }

  bool no() {
    ok = false;
    return false;
  }
  // The tensor of `o` if it is a CUDA tensor of type `dt` on the call's device; layout is up to the caller.
  const at::Tensor* any(PyObject* o, at::ScalarType dt) {
    if (!ok) return nullptr;
    if (!THPVariable_Check(o)) {
      no();
      return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.scalar_type() != dt) {
      no();
      return nullptr;
    }
    const int d = t.device().index();
    if (dev < 0) dev = d;
    if (d != dev) {
      no();
      return nullptr;
    }
    return &t;
  }
  // Data pointer of a contiguous tensor whose sizes fit the pattern.
  void* ten(PyObject* o, at::ScalarType dt, std::initializer_list<int64_t> dims) {
    const at::Tensor* t = any(o, dt);
    if (t == nullptr) return nullptr;
    if (t->dim() != static_cast<int64_t>(dims.size()) || !t->is_contiguous()) {
      no();
      return nullptr;
    }
    int i = 0;
    for (const int64_t d : dims) {
      const int64_t s = t->size(i++);
      if (d >= 0) {
        if (s != d) no();
      } else if (d != ANY) {
        int64_t& v = var[-2 - d];
        if (v < 0) v = s;
        else if (v != s) no();
      }
    }
    return ok ? t->data_ptr() : nullptr;
  }
  // Contiguous tensor of a given number of elements, whatever its shape.
  void* flat(PyObject* o, at::ScalarType dt, int64_t numel) {
    const at::Tensor* t = any(o, dt);
    if (t == nullptr) return nullptr;
    if (t->numel() != numel || !t->is_contiguous()) {
      no();
      return nullptr;
    }
    return t->data_ptr();
  }
  int64_t integer(PyObject* o) {
    if (!ok) return 0;
    if (!PyLong_Check(o)) {
      no();
      return 0;
    }
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      no();
    }
    if (v > INT32_MAX || v < INT32_MIN) no();
    return v;
  }
  double number(PyObject* o) {
    if (!ok) return 0.0;
    if (PyFloat_Check(o)) return PyFloat_AS_DOUBLE(o);
    return static_cast<double>(integer(o));
  }
  // All arguments seen: is the call's device the current one, and has it a status word?
  bool ready() {
    if (!ok) return false;
    if (dev < 0 || dev >= kMaxDevices || g_status[dev] == nullptr) return no();
    if (c10::cuda::current_device() != dev) return no();
    return true;
  }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream(); }
  at::Tensor make(at::IntArrayRef sizes, at::ScalarType dt) const {
    return at::empty(sizes, at::TensorOptions().dtype(dt).device(at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(dev))));
  }
};

// Scratch memory of one call; given back to the stream-ordered allocator when the call has been enqueued.
struct Scratch {
  c10::DataPtr mem;
  size_t bytes;
  explicit Scratch(size_t n) : bytes(n) {
    if (n > 0) mem = c10::cuda::CUDACachingAllocator::get()->allocate(n);
  }
  void* ptr() const { return mem.get(); }
};

bool fail(int rc, const char* what) {   // raises through _lib.check; true when an exception is set
  if (rc == 0) return false;
  PyObject* r = PyObject_CallFunction(g_on_error, "is", rc, what);
  if (r != nullptr) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, what);
  }
  return true;
}

PyObject* done(int rc, const char* what) {
  if (fail(rc, what)) return nullptr;
  Py_RETURN_TRUE;
}

template <class T>
T* as(void* p) {
  return static_cast<T*>(p);
}


// ---- V3.2 attention ------------------------------------------------------------------------------------------------
// sfa(query_nope, query_rope, key_nope, key_rope, scales, topk_indices, block_table, act_seqs, out, nq, n_kv, scale,
//     topk, block_size, max_blocks, kv_splits)
PyObject* sfa(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 16) Py_RETURN_FALSE;
  Dsv32SfaArgs g{};
  const int64_t nq = c.integer(a[9]), n_kv = c.integer(a[10]), topk = c.integer(a[12]), bs = c.integer(a[13]);
  const int64_t mb = c.integer(a[14]), splits = c.integer(a[15]);
  g.softmax_scale = static_cast<float>(c.number(a[11]));
  if (!c.ok || n_kv != 1 || nq < 1 || topk < 1 || !THPVariable_Check(a[2])) Py_RETURN_FALSE;
  const bool quant = THPVariable_Unpack(a[2]).scalar_type() == I8;
  g.query_nope = c.ten(a[0], BF16, {A, 512});
  g.query_rope = c.ten(a[1], BF16, {A, 64});
  g.key_nope = c.ten(a[2], quant ? I8 : BF16, {B, 512});
  g.key_rope = c.ten(a[3], BF16, {B, 64});
  if (quant) g.k_nope_scales = as<const float>(c.ten(a[4], F32, {B, 4}));
  g.topk_indices = as<const int32_t>(c.ten(a[5], I32, {C_, topk}));
  g.block_table = as<const int32_t>(c.ten(a[6], I32, {D, mb}));
  g.kv_act_seqs = as<const int32_t>(c.ten(a[7], I32, {D}));
  g.attention_out = c.ten(a[8], BF16, {D, E, nq, 512});
  if (!c.ready() || c[D] < 1 || c[E] < 1 || c[D] * c[E] != c[C_] || c[A] != c[C_] * nq) Py_RETURN_FALSE;
  g.rows = c[B];
  g.b = static_cast<int32_t>(c[D]); g.s1 = static_cast<int32_t>(c[E]); g.n_q = static_cast<int32_t>(nq);
  g.topk = static_cast<int32_t>(topk); g.block_size = static_cast<int32_t>(bs); g.max_blocks = static_cast<int32_t>(mb);
  g.kv_splits = static_cast<int32_t>(splits);
  Scratch ws(p_dsv32_sfa_workspace_bytes(g.b, g.s1, g.n_q, g.topk, g.kv_splits));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  return done((quant ? p_dsv32_sfa_quant : p_dsv32_sfa_bf16_cache)(&g, c.stream()), "sparse_flash_attention_quant");
  END_HANDLE_TH_ERRORS
}

// sa_antiquant(query_nope, query_rope, cache, topk_indices, block_table, act_seqs, out, nq, n_kv, scale, topk, block_size,
//              max_blocks, kv_splits)
PyObject* sa_antiquant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 14) Py_RETURN_FALSE;
  Dsv32SaAntiquantArgs g{};
  const int64_t nq = c.integer(a[7]), n_kv = c.integer(a[8]), topk = c.integer(a[10]), bs = c.integer(a[11]);
  const int64_t mb = c.integer(a[12]), splits = c.integer(a[13]);
  g.softmax_scale = static_cast<float>(c.number(a[9]));
  if (!c.ok || n_kv != 1 || nq < 1 || topk < 1) Py_RETURN_FALSE;
  g.query_nope = c.ten(a[0], BF16, {A, 512});
  g.query_rope = c.ten(a[1], BF16, {A, 64});
  g.nope_cache = c.ten(a[2], I8, {B, DSV32_ANTIQUANT_ROW_BYTES});
  g.topk_indices = as<const int32_t>(c.ten(a[3], I32, {C_, topk}));
  g.block_table = as<const int32_t>(c.ten(a[4], I32, {D, mb}));
  g.kv_act_seqs = as<const int32_t>(c.ten(a[5], I32, {D}));
  g.attention_out = c.ten(a[6], BF16, {D, E, nq, 512});
  if (!c.ready() || c[D] < 1 || c[E] < 1 || c[D] * c[E] != c[C_] || c[A] != c[C_] * nq) Py_RETURN_FALSE;
  g.rows = c[B];
  g.b = static_cast<int32_t>(c[D]); g.s1 = static_cast<int32_t>(c[E]); g.n_q = static_cast<int32_t>(nq);
  g.topk = static_cast<int32_t>(topk); g.block_size = static_cast<int32_t>(bs); g.max_blocks = static_cast<int32_t>(mb);
  g.kv_splits = static_cast<int32_t>(splits);
  Scratch ws(p_dsv32_sfa_workspace_bytes(g.b, g.s1, g.n_q, g.topk, g.kv_splits));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  return done(p_dsv32_sparse_attention_antiquant(&g, c.stream()), "sparse_attention_antiquant");
  END_HANDLE_TH_ERRORS
}

// ---- lightning indexer ---------------------------------------------------------------------------------------------
// indexer(idx_query, query_scale, key_cache, key_scale, weight, act_seq, block_table, topk_res, selected_count)
PyObject* indexer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 9) Py_RETURN_FALSE;
  Dsv32IndexerArgs g{};
  const int64_t k = c.integer(a[8]);
  if (!c.ok || k < 1) Py_RETURN_FALSE;
  g.idx_query = as<const int8_t>(c.ten(a[0], I8, {A, 64, 128}));
  g.idx_query_scale = c.flat(a[1], F16, c.ok ? c[A] * 64 : 0);
  g.idx_key_cache = as<const int8_t>(c.ten(a[2], I8, {B, 128, 1, 128}));
  g.idx_key_scale = c.flat(a[3], F16, c.ok ? c[B] * 128 : 0);
  g.idx_weight = c.ten(a[4], F16, {A, 64});
  g.act_seq_key = as<const int32_t>(c.ten(a[5], I32, {C_}));
  g.block_table = as<const int32_t>(c.ten(a[6], I32, {C_, D}));
  g.topk_res = as<int32_t>(c.ten(a[7], I32, {A, 1, k}));
  if (!c.ready() || c[C_] < 1 || c[A] < 1 || c[D] < 1 || c[A] % c[C_] != 0) Py_RETURN_FALSE;
  g.num_blocks = c[B];
  g.b = static_cast<int32_t>(c[C_]); g.s1 = static_cast<int32_t>(c[A] / c[C_]); g.block_size = 128;
  g.max_blocks = static_cast<int32_t>(c[D]); g.selected_count = static_cast<int32_t>(k);
  g.score_ld = g.max_blocks * 128;
  g.key_begin = 0;
  g.key_end = INT32_MAX;
  Scratch ws(p_dsv32_indexer_workspace_bytes(g.b, g.s1, g.max_blocks, 128));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  return done(p_dsv32_indexer_topk(&g, c.stream()), "lightning_indexer_decode");
  END_HANDLE_TH_ERRORS
}

// ---- V3.2 prologs --------------------------------------------------------------------------------------------------
// The indexer half: w_qb, w_qb_scale, wk, w_proj, ln_gamma, ln_beta, hadamard_q, hadamard_k, k_cache, k_scale of `in` and
// q_int8, q_scale, k_cache, k_scale, weights of `out`.
void fill_prolog(Call& c, Dsv32PrologArgs& g, PyObject* const* in, PyObject* const* out) {
  g.w_qb = as<const int8_t>(c.ten(in[0], I8, {1536, 8192}));
  g.w_qb_scale = as<const float>(c.flat(in[1], F32, 8192));
  g.wk = c.ten(in[2], BF16, {7168, 128});
  g.w_proj = c.ten(in[3], BF16, {7168, 64});
  g.ln_gamma_k = c.ten(in[4], BF16, {128});
  g.ln_beta_k = c.ten(in[5], BF16, {128});
  g.hadamard_q = c.ten(in[6], BF16, {128, 128});
  g.hadamard_k = c.ten(in[7], BF16, {128, 128});
  g.k_cache = as<int8_t>(c.ten(in[8], I8, {B, C_, 1, 128}));
  g.k_scale_cache = c.ten(in[9], F16, {B, C_, 1, 1});
  g.q_int8 = as<int8_t>(c.ten(out[0], I8, {A, 64, 128}));
  g.q_scale = c.ten(out[1], F16, {A, 64, 1});
  if (c.ten(out[2], I8, {B, C_, 1, 128}) != g.k_cache || c.ten(out[3], F16, {B, C_, 1, 1}) != g.k_scale_cache) c.no();
  g.weights = c.ten(out[4], F16, {A, 64});
  if (!c.ok) return;
  g.cache_rows = c[B] * c[C_];
  g.t = static_cast<int32_t>(c[A]);
}

// indexer_prolog(x, q_norm, q_norm_scale, w_qb, w_qb_scale, wk, w_proj, ln_gamma, ln_beta, cos, sin, hadamard_q, hadamard_k,
//                k_cache, k_scale, cache_index, q_int8, q_scale, k_cache, k_scale, weights, eps)
PyObject* indexer_prolog(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 22) Py_RETURN_FALSE;
  Dsv32PrologArgs g{};
  g.ln_eps = static_cast<float>(c.number(a[21]));
  g.x = c.ten(a[0], BF16, {A, 7168});
  g.q_norm = as<const int8_t>(c.ten(a[1], I8, {A, 1536}));
  g.q_norm_scale = as<const float>(c.ten(a[2], F32, {A, 1}));
  g.cos_idx_rope = c.ten(a[9], BF16, {A, 64});
  g.sin_idx_rope = c.ten(a[10], BF16, {A, 64});
  g.k_cache_index = as<const int64_t>(c.ten(a[15], I64, {A}));
  if (!c.ok || THPVariable_Check(a[4]) == 0 || THPVariable_Unpack(a[4]).dim() != 2 || THPVariable_Unpack(a[4]).size(1) != 1)
    Py_RETURN_FALSE;
  PyObject* in[10] = {a[3], a[4], a[5], a[6], a[7], a[8], a[11], a[12], a[13], a[14]};
  fill_prolog(c, g, in, a + 16);
  if (!c.ready() || g.t < 1) Py_RETURN_FALSE;
  Scratch ws(p_dsv32_prolog_workspace_bytes(g.t));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  return done(p_dsv32_indexer_prolog(&g, c.stream()), "lightning_indexer_prolog_quant");
  END_HANDLE_TH_ERRORS
}

// The MLA half's inputs, from token_x to the three caches, and query_nope, query_rope and the caches of `out`.
void fill_mla(Call& c, Dsv32MlaPrologArgs& g, PyObject* const* in, PyObject* const* out) {
  g.x = c.ten(in[0], BF16, {A, 7168});
  g.w_dq = c.ten(in[1], BF16, {7168, 1536});
  g.w_uq_qr = as<const int8_t>(c.ten(in[2], I8, {1536, 24576}));
  g.w_qb_scale = as<const float>(c.flat(in[3], F32, 24576));
  g.w_uk = c.ten(in[4], BF16, {128, 128, 512});
  g.w_dkv_kr = c.ten(in[5], BF16, {7168, 576});
  g.gamma_cq = c.ten(in[6], BF16, {1536});
  g.gamma_ckv = c.ten(in[7], BF16, {512});
  g.cos = c.ten(in[8], BF16, {A, 64});
  g.sin = c.ten(in[9], BF16, {A, 64});
  g.cache_index = as<const int64_t>(c.ten(in[10], I64, {A}));
  g.kv_cache = as<int8_t>(c.ten(in[11], I8, {D, E, 1, 512}));
  g.kr_cache = c.ten(in[12], BF16, {D, E, 1, 64});
  g.k_scale_cache = as<float>(c.ten(in[13], F32, {D, E, 1, 4}));
  g.query_nope = c.ten(out[0], BF16, {A, 128, 512});
  g.query_rope = c.ten(out[1], BF16, {A, 128, 64});
  // the caches are updated in place: only the storage of the "out" arguments is looked at
  if (c.ok && (!THPVariable_Check(out[2]) || !THPVariable_Check(out[3]) || !THPVariable_Check(out[4]) ||
               THPVariable_Unpack(out[2]).data_ptr() != g.kv_cache || THPVariable_Unpack(out[3]).data_ptr() != g.kr_cache ||
               THPVariable_Unpack(out[4]).data_ptr() != g.k_scale_cache))
    c.no();
  if (!c.ok) return;
  g.cache_rows = c[D] * c[E];
  g.t = static_cast<int32_t>(c[A]);
}

bool cache_mode_ok(PyObject* o) {
  return PyUnicode_Check(o) && (PyUnicode_CompareWithASCIIString(o, "PA_BSND") == 0 || PyUnicode_CompareWithASCIIString(o, "BSND") == 0 ||
                                PyUnicode_CompareWithASCIIString(o, "PA_NZ") == 0);
}

// mla_prolog(14 inputs, q_norm, q_norm_scale, query_nope, query_rope, 3 caches, eps_cq, eps_ckv, cache_mode)
PyObject* mla_prolog(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 24 || !cache_mode_ok(a[23])) Py_RETURN_FALSE;
  Dsv32MlaPrologArgs g{};
  g.eps_cq = static_cast<float>(c.number(a[21]));
  g.eps_ckv = static_cast<float>(c.number(a[22]));
  fill_mla(c, g, a, a + 16);
  g.q_norm = as<int8_t>(c.ten(a[14], I8, {A, 1536}));
  g.q_norm_scale = as<float>(c.ten(a[15], F32, {A, 1}));
  if (!c.ready() || g.t < 1) Py_RETURN_FALSE;
  Scratch ws(p_dsv32_mla_prolog_workspace_bytes(g.t));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  return done(p_dsv32_mla_prolog(&g, c.stream()), "mla_prolog_quant");
  END_HANDLE_TH_ERRORS
}

// mla_indexer_prolog(24 inputs, 10 outputs, eps_cq, eps_ckv, cache_mode, indexer eps)
PyObject* mla_indexer_prolog(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 38 || !cache_mode_ok(a[36])) Py_RETURN_FALSE;
  Dsv32FusedPrologArgs f{};
  f.mla.eps_cq = static_cast<float>(c.number(a[34]));
  f.mla.eps_ckv = static_cast<float>(c.number(a[35]));
  f.indexer.ln_eps = static_cast<float>(c.number(a[37]));
  fill_mla(c, f.mla, a, a + 24);
  fill_prolog(c, f.indexer, a + 14, a + 29);
  if (!c.ready() || f.mla.t < 1) Py_RETURN_FALSE;
  const int t = f.mla.t;
  f.indexer.x = f.mla.x;
  f.indexer.cos_idx_rope = f.mla.cos;
  f.indexer.sin_idx_rope = f.mla.sin;
  f.indexer.k_cache_index = f.mla.cache_index;
  // one allocation: q_norm [t, 1536], q_norm_scale [t], then the workspace (the MLA half's serves both)
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  const size_t o_scale = up(static_cast<size_t>(t) * 1536), o_mla = o_scale + up(static_cast<size_t>(t) * 4);
  const size_t n_mla = p_dsv32_mla_prolog_workspace_bytes(t);
  Scratch ws(o_mla + n_mla);
  char* base = as<char>(ws.ptr());
  f.mla.q_norm = reinterpret_cast<int8_t*>(base);
  f.mla.q_norm_scale = reinterpret_cast<float*>(base + o_scale);
  f.mla.workspace = base + o_mla;
  f.mla.workspace_bytes = n_mla;
  f.indexer.q_norm = f.mla.q_norm;
  f.indexer.q_norm_scale = f.mla.q_norm_scale;
  f.mla.status = f.indexer.status = g_status[c.dev];
  return done(p_dsv32_mla_indexer_prolog(&f, c.stream()), "mla_indexer_prolog_quant");
  END_HANDLE_TH_ERRORS
}

// pg_prolog(format, 16 inputs, 5 outputs, eps): caches are strided views, pages contiguous
PyObject* pg_prolog(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 23) Py_RETURN_FALSE;
  Dsv32PgPrologArgs g{};
  g.format = static_cast<int32_t>(c.integer(a[0]));
  g.eps = static_cast<float>(c.number(a[22]));
  const bool mx = g.format == DSV32_PG_FORMAT_MXFP8;
  if (!c.ok || !THPVariable_Check(a[2])) Py_RETURN_FALSE;
  const at::ScalarType code = (mx && THPVariable_Unpack(a[2]).scalar_type() == at::kFloat8_e4m3fn) ? at::kFloat8_e4m3fn : U8;
  g.x = c.ten(a[1], BF16, {A, B});
  g.q_norm = as<const uint8_t>(c.ten(a[2], code, {A, C_}));
  g.w_qb = as<const uint8_t>(c.ten(a[4], code, {C_, D}));
  g.wk = c.ten(a[6], BF16, {B, 128});
  g.w_proj = c.ten(a[7], BF16, {B, E});
  if (!c.ok || c[D] != c[E] * 128) Py_RETURN_FALSE;
  if (mx) {
    if (!THPVariable_Check(a[3]) || c[C_] % 64 != 0) Py_RETURN_FALSE;
    const at::ScalarType e8 = THPVariable_Unpack(a[3]).scalar_type() == U8 ? U8 : at::kFloat8_e8m0fnu;
    g.q_norm_scale = c.flat(a[3], e8, c[A] * (c[C_] / 32));
    g.w_qb_scale = c.ten(a[5], e8, {c[C_] / 64, D, 2});
  } else {
    g.q_norm_scale = c.ten(a[3], F32, {A, 1});
    g.w_qb_scale = c.ten(a[5], F32, {1, D});
  }
  g.gamma_k = c.flat(a[8], BF16, 128);
  g.cos_idx_rope = c.ten(a[9], BF16, {A, 64});
  g.sin_idx_rope = c.ten(a[10], BF16, {A, 64});
  g.hadamard_q = c.ten(a[11], BF16, {128, 128});
  g.hadamard_k = c.ten(a[12], BF16, {128, 128});
  g.k_cache_index = as<const int64_t>(c.ten(a[15], I64, {A, 1}));
  g.k_scale_cache_index = as<const int64_t>(c.ten(a[16], I64, {A, 1}));
  if (!c.ok) Py_RETURN_FALSE;
  g.q_quant = as<uint8_t>(c.ten(a[17], code, {c[A] * c[E], 128}));
  g.q_scale = as<float>(c.ten(a[18], F32, {c[A] * c[E], 1}));
  g.weights = c.ten(a[21], BF16, {A, E});
  const at::Tensor* kin = c.any(a[13], code);
  const at::Tensor* ksin = c.any(a[14], F32);
  const at::Tensor* k = c.any(a[19], code);
  const at::Tensor* ks = c.any(a[20], F32);
  if (!c.ready() || c[A] < 1) Py_RETURN_FALSE;
  for (const at::Tensor* t : {k, ks}) {
    const int64_t last = t == k ? 128 : 1;
    if (t->dim() != 4 || t->size(0) < 1 || t->size(2) != 1 || t->size(3) != last || t->stride(3) != 1 || t->stride(2) != last ||
        t->stride(1) != last || t->stride(0) < t->size(1) * last)
      Py_RETURN_FALSE;
  }
  if (ks->size(0) != k->size(0) || ks->size(1) != k->size(1) || kin->data_ptr() != k->data_ptr() || kin->strides() != k->strides() ||
      kin->sizes() != k->sizes() || ksin->data_ptr() != ks->data_ptr() || ksin->strides() != ks->strides() || ksin->sizes() != ks->sizes())
    Py_RETURN_FALSE;
  g.k_cache = as<uint8_t>(k->data_ptr());
  g.k_scale_cache = as<float>(ks->data_ptr());
  g.block_size = static_cast<int32_t>(k->size(1));
  g.cache_rows = k->size(0) * k->size(1);
  g.k_block_stride = k->size(0) > 1 ? k->stride(0) : k->size(1) * 128;
  g.k_scale_block_stride = (ks->size(0) > 1 ? ks->stride(0) : ks->size(1)) * 4;
  g.t = static_cast<int32_t>(c[A]); g.h = static_cast<int32_t>(c[B]); g.q_lora = static_cast<int32_t>(c[C_]);
  g.heads = static_cast<int32_t>(c[E]);
  Scratch ws(p_dsv32_pg_indexer_prolog_workspace_bytes(g.t, g.h, g.q_lora, g.heads));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  return done(p_dsv32_pg_indexer_prolog(&g, c.stream()), "lightning_indexer_prolog_quant (page-grouped)");
  END_HANDLE_TH_ERRORS
}

// ---- DeepSeek-V4 ---------------------------------------------------------------------------------------------------
// indexer_prolog_v4(9 inputs): (q, weights, q_scale), or None when declined; with the three outputs given, True / False
PyObject* indexer_prolog_v4(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 9 && n != 12) Py_RETURN_NONE;
  Dsv32PrologV4Args g{};
  g.qr = as<const int8_t>(c.ten(a[0], I8, {A, 1024}));
  g.idx_wq_b = as<const int8_t>(c.ten(a[1], I8, {1024, 8192}));
  g.x = c.ten(a[2], BF16, {A, B});
  g.weights_proj = c.ten(a[3], BF16, {B, 64});
  g.cos = c.ten(a[4], BF16, {A, 64});
  g.sin = c.ten(a[5], BF16, {A, 64});
  g.hadamard = c.ten(a[6], BF16, {128, 128});
  g.qr_scale = as<const float>(c.ten(a[7], F32, {A, 1}));
  g.idx_wq_b_scale = as<const float>(c.ten(a[8], F32, {8192, 1}));
  if (n == 12) {
    g.q = as<int8_t>(c.ten(a[9], I8, {A, 64, 128}));
    g.weights = c.ten(a[10], F16, {A, 64});
    g.q_scale = c.ten(a[11], F16, {A, 64});
  }
  if (!c.ready() || c[A] < 1) {
    if (n == 12) Py_RETURN_FALSE;
    Py_RETURN_NONE;
  }
  g.t = static_cast<int32_t>(c[A]); g.h = static_cast<int32_t>(c[B]);
  at::Tensor q, w, s;
  if (n == 9) {
    q = c.make({c[A], 64, 128}, I8);
    w = c.make({c[A], 64}, F16);
    s = c.make({c[A], 64}, F16);
    g.q = as<int8_t>(q.data_ptr());
    g.weights = w.data_ptr();
    g.q_scale = s.data_ptr();
  }
  Scratch ws(p_dsv32_prolog_v4_workspace_bytes(g.t, g.h));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  if (fail(p_dsv32_indexer_prolog_v4(&g, c.stream()), "quant_lightning_indexer_prolog")) return nullptr;
  if (n == 12) Py_RETURN_TRUE;
  return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(q)), THPVariable_Wrap(std::move(w)), THPVariable_Wrap(std::move(s)));
  END_HANDLE_TH_ERRORS
}

// mla_prolog_v4(x, wq_a, wq_b, wkv, cos, sin, gamma_cq, gamma_ckv, wq_b_scale or None, eps): (q, kv, qr[, qr_scale]), or None
// when declined; with the outputs between wq_b_scale and eps, True / False
PyObject* mla_prolog_v4(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  Dsv32MlaPrologV4Args g{};
  const bool quant = n > 8 && a[8] != Py_None;
  const int outs = quant ? 4 : 3;
  const bool given = n == 10 + outs;
  if (n != 10 && !given) Py_RETURN_NONE;
  g.eps = static_cast<float>(c.number(a[n - 1]));
  g.x = c.ten(a[0], BF16, {A, B});
  g.wq_a = c.ten(a[1], BF16, {B, 1024});
  g.wq_b = c.ten(a[2], quant ? I8 : BF16, {1024, C_});
  g.wkv = c.ten(a[3], BF16, {B, 512});
  g.cos = c.ten(a[4], BF16, {A, 64});
  g.sin = c.ten(a[5], BF16, {A, 64});
  g.gamma_cq = c.ten(a[6], BF16, {1024});
  g.gamma_ckv = c.ten(a[7], BF16, {512});
  if (c.ok && (c[C_] < 512 || c[C_] % 512 != 0 || c[A] < 1 || c[B] < 8 || c[B] % 8 != 0)) c.no();
  const int64_t heads = c.ok ? c[C_] / 512 : 0;
  if (quant && c.ok) {
    if (!THPVariable_Check(a[8]) || THPVariable_Unpack(a[8]).dim() > 2 || THPVariable_Unpack(a[8]).dim() < 1 ||
        (THPVariable_Unpack(a[8]).dim() == 2 && THPVariable_Unpack(a[8]).size(0) != 1 && THPVariable_Unpack(a[8]).size(1) != 1))
      c.no();
    g.wq_b_scale = as<const float>(c.flat(a[8], F32, c[C_]));
  }
  if (given) {
    g.q_out = c.ten(a[9], BF16, {A, heads, 512});
    g.kv_out = c.ten(a[10], BF16, {A, 512});
    g.qr = c.ten(a[11], quant ? I8 : BF16, {A, 1024});
    if (quant) g.qr_scale = as<float>(c.ten(a[12], F32, {A, 1}));
  }
  auto aligned = [](const void* p, unsigned to) { return reinterpret_cast<uintptr_t>(p) % to == 0; };
  if (!c.ready() || !aligned(g.cos, 4) || !aligned(g.sin, 4) || !aligned(g.q_out, 16) || !aligned(g.qr, 16)) {
    if (given) Py_RETURN_FALSE;
    Py_RETURN_NONE;
  }
  g.t = static_cast<int32_t>(c[A]); g.h = static_cast<int32_t>(c[B]); g.heads = static_cast<int32_t>(heads);
  g.quant = quant ? 1 : 0;
  at::Tensor q, kv, qr, qs;
  if (!given) {
    q = c.make({c[A], heads, 512}, BF16);
    kv = c.make({c[A], 512}, BF16);
    qr = c.make({c[A], 1024}, quant ? I8 : BF16);
    g.q_out = q.data_ptr();
    g.kv_out = kv.data_ptr();
    g.qr = qr.data_ptr();
    if (quant) {
      qs = c.make({c[A], 1}, F32);
      g.qr_scale = as<float>(qs.data_ptr());
    }
  }
  Scratch ws(p_dsv32_mla_prolog_v4_workspace_bytes(g.t, g.h));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  if (fail(p_dsv32_mla_prolog_v4(&g, c.stream()), "mla_prolog_v4")) return nullptr;
  if (given) Py_RETURN_TRUE;
  if (quant)
    return Py_BuildValue("(NNNN)", THPVariable_Wrap(std::move(q)), THPVariable_Wrap(std::move(kv)), THPVariable_Wrap(std::move(qr)),
                         THPVariable_Wrap(std::move(qs)));
  return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(q)), THPVariable_Wrap(std::move(kv)), THPVariable_Wrap(std::move(qr)));
  END_HANDLE_TH_ERRORS
}

// hc_pre(x, hc_fn, hc_scale, hc_base, hc_mult, iters, hc_eps): (y, post, comb), or None when declined; with the outputs
// between the inputs and hc_mult, True / False
PyObject* hc_pre(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 7 && n != 10) Py_RETURN_NONE;
  PyObject* const* tail = a + (n - 3);
  Dsv32HcPreArgs g{};
  g.hc_mult = static_cast<int32_t>(c.integer(tail[0]));
  g.iters = static_cast<int32_t>(c.integer(tail[1]));
  g.hc_eps = static_cast<float>(c.number(tail[2]));
  g.x = c.ten(a[0], BF16, {A, 4, 4096});
  g.hc_fn = as<const float>(c.ten(a[1], F32, {24, 16384}));
  g.hc_scale = as<const float>(c.ten(a[2], F32, {3}));
  g.hc_base = as<const float>(c.ten(a[3], F32, {24}));
  if (n == 10) {
    g.y = c.ten(a[4], BF16, {A, 4096});
    g.post = as<float>(c.ten(a[5], F32, {A, 4}));
    g.comb = as<float>(c.ten(a[6], F32, {A, 4, 4}));
  }
  if (!c.ready() || g.hc_mult != 4 || g.iters < 1 || c[A] < 1) {
    if (n == 10) Py_RETURN_FALSE;
    Py_RETURN_NONE;
  }
  g.t = static_cast<int32_t>(c[A]);
  g.d = 4096;
  g.norm_eps = 1e-6f;
  at::Tensor y, post, comb;
  if (n == 7) {
    y = c.make({c[A], 4096}, BF16);
    post = c.make({c[A], 4}, F32);
    comb = c.make({c[A], 4, 4}, F32);
    g.y = y.data_ptr();
    g.post = as<float>(post.data_ptr());
    g.comb = as<float>(comb.data_ptr());
  }
  Scratch ws(p_dsv32_hc_pre_workspace_bytes(g.t));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  if (fail(p_dsv32_hc_pre(&g, c.stream()), "hc_pre")) return nullptr;
  if (n == 10) Py_RETURN_TRUE;
  return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(y)), THPVariable_Wrap(std::move(post)), THPVariable_Wrap(std::move(comb)));
  END_HANDLE_TH_ERRORS
}

// compressor(x, kv_state, score_state, kv_block_table, score_block_table, sin, cos, wkv, wgate, ape, weight, hadamard, start_pos,
//            ratio, rope_head_dim, rotate): out, or None when declined
PyObject* compressor(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 16 || !PyBool_Check(a[15])) Py_RETURN_NONE;
  Dsv32CompressorOpArgs g{};
  const int64_t ratio = c.integer(a[13]);
  if (c.integer(a[14]) != 64 || (ratio != 4 && ratio != 128)) Py_RETURN_NONE;
  g.weight = as<const float>(c.ten(a[10], F32, {D}));
  if (!c.ok || c[D] < 64 || c[D] > 512 || c[D] % 2 != 0) Py_RETURN_NONE;
  const int64_t d = c[D], cd = ratio == 4 ? 2 * d : d;
  g.x = c.ten(a[0], BF16, {A, B, C_});
  g.kv_state = as<float>(c.ten(a[1], F32, {ANY, 128, cd}));
  g.score_state = as<float>(c.ten(a[2], F32, {ANY, 128, cd}));
  g.kv_block_table = as<const int32_t>(c.ten(a[3], I32, {A, E}));
  g.score_block_table = as<const int32_t>(c.ten(a[4], I32, {A, F}));
  if (!c.ok || c[A] < 1 || c[B] < 1 || c[C_] < 8 || c[C_] % 8 != 0 || c[E] < 1 || c[F] < 1) Py_RETURN_NONE;
  const int64_t t = c[A] * c[B], rows = std::min(t, t / ratio + c[A]);
  g.sin = c.ten(a[5], BF16, {rows, 64});
  g.cos = c.ten(a[6], BF16, {rows, 64});
  g.wkv = c.ten(a[7], BF16, {cd, C_});
  g.wgate = c.ten(a[8], BF16, {cd, C_});
  g.ape = as<const float>(c.ten(a[9], F32, {ratio, cd}));
  const void* had = c.ten(a[11], BF16, {d, d});
  g.hadamard = a[15] == Py_True ? had : nullptr;
  g.start_pos = as<const int32_t>(c.ten(a[12], I32, {A}));
  if (!c.ready() || t > INT32_MAX) Py_RETURN_NONE;
  g.kv_blocks = THPVariable_Unpack(a[1]).size(0);
  g.score_blocks = THPVariable_Unpack(a[2]).size(0);
  g.b = static_cast<int32_t>(c[A]); g.s1 = static_cast<int32_t>(c[B]); g.d = static_cast<int32_t>(d);
  g.ratio = static_cast<int32_t>(ratio); g.h = static_cast<int32_t>(c[C_]); g.out_rows = static_cast<int32_t>(rows);
  g.kv_cols = static_cast<int32_t>(c[E]); g.score_cols = static_cast<int32_t>(c[F]);
  g.eps = 1e-6f;
  at::Tensor out = c.make({rows, d}, BF16);
  g.out = out.data_ptr();
  Scratch ws(p_dsv32_compressor_workspace_bytes(g.b * g.s1, g.h, static_cast<int32_t>(cd)));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  if (fail(p_dsv32_compressor(&g, c.stream()), "compressor")) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// window_attention(query, seq_q, ori_kv, cmp_kv, ori_table, cmp_table, sink, seqused, indices, out, nq, scale, topk,
//                  block_size, win_size, cmp_ratio, cmp_mode): seq_q (None: tokens split
//                  evenly), cmp_kv, cmp_table, indices may be None
PyObject* window_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c;
  if (n != 17) Py_RETURN_FALSE;
  Dsv32ScfaArgs g{};
  const int64_t nq = c.integer(a[10]), topk = c.integer(a[12]), bs = c.integer(a[13]), win = c.integer(a[14]);
  const int64_t ratio = c.integer(a[15]), mode = c.integer(a[16]);
  g.softmax_scale = static_cast<float>(c.number(a[11]));
  if (!c.ok || nq < 1 || topk < 0) Py_RETURN_FALSE;
  g.query = c.ten(a[0], BF16, {A, 512});
  g.ori_kv = c.ten(a[2], BF16, {B, 512});
  g.ori_block_table = as<const int32_t>(c.ten(a[4], I32, {C_, D}));
  if (!c.ok || c[A] % nq != 0) Py_RETURN_FALSE;
  const int64_t t = c[A] / nq, b = c[C_];
  if (a[1] != Py_None) g.actual_seq_q = as<const int32_t>(c.ten(a[1], I32, {b + 1}));
  else if (b < 1 || t % b != 0) c.no();
  g.seqused_kv = as<const int32_t>(c.ten(a[7], I32, {b}));
  g.atten_sink = as<const float>(c.ten(a[6], F32, {nq}));
  g.attention_out = c.ten(a[9], BF16, {A, 512});
  if (topk > 0) {
    g.cmp_kv = c.ten(a[3], BF16, {E, 512});
    g.cmp_block_table = as<const int32_t>(c.ten(a[5], I32, {b, F}));
    if (mode == DSV32_SCFA_SELECTED) g.cmp_sparse_indices = as<const int32_t>(c.ten(a[8], I32, {t, topk}));
  }
  if (!c.ready() || t < 1 || b < 1) Py_RETURN_FALSE;
  g.ori_rows = c[B];
  g.cmp_rows = topk > 0 ? c[E] : 0;
  g.t = static_cast<int32_t>(t); g.b = static_cast<int32_t>(b); g.n_q = static_cast<int32_t>(nq);
  g.topk = static_cast<int32_t>(topk); g.block_size = static_cast<int32_t>(bs); g.win_size = static_cast<int32_t>(win);
  g.cmp_ratio = static_cast<int32_t>(ratio); g.cmp_mode = static_cast<int32_t>(mode);
  g.ori_max_blocks = static_cast<int32_t>(c[D]);
  g.cmp_max_blocks = topk > 0 ? static_cast<int32_t>(c[F]) : 0;
  Scratch ws(p_dsv32_scfa_workspace_bytes(g.t, g.topk, g.win_size));
  g.workspace = ws.ptr();
  g.workspace_bytes = ws.bytes;
  g.status = g_status[c.dev];
  return done(p_dsv32_sparse_compress_attention(&g, c.stream()), "sparse_compress_flash_attention");
  END_HANDLE_TH_ERRORS
}

// ---- binding -------------------------------------------------------------------------------------------------------
// bind({name: address}, on_error)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyDict_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "bind(addresses, on_error)");
    return nullptr;
  }
#define BIND_ENTRY(name)                                                                     \
  {                                                                                          \
    PyObject* v = PyDict_GetItemString(a[0], #name);                                         \
    void* p = v != nullptr ? PyLong_AsVoidPtr(v) : nullptr;                                  \
    if (p == nullptr) {                                                                      \
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, #name);                         \
      return nullptr;                                                                        \
    }                                                                                        \
    p_##name = reinterpret_cast<decltype(p_##name)>(p);                                      \
  }
  FRONT_ENTRIES(BIND_ENTRY)
#undef BIND_ENTRY
  Py_INCREF(a[1]);
  Py_XDECREF(g_on_error);
  g_on_error = a[1];
  g_bound = true;
  Py_RETURN_NONE;
}

// set_status(device index, address): the status word of a device
PyObject* set_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "set_status(device, address)");
    return nullptr;
  }
  const long dev = PyLong_AsLong(a[0]);
  void* p = PyLong_AsVoidPtr(a[1]);
  if (PyErr_Occurred()) return nullptr;
  if (dev >= 0 && dev < kMaxDevices) g_status[dev] = static_cast<uint32_t*>(p);
  Py_RETURN_NONE;
}

#define FRONT_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FRONT_METHOD(bind),         FRONT_METHOD(set_status),     FRONT_METHOD(sfa),
                         FRONT_METHOD(sa_antiquant), FRONT_METHOD(indexer),        FRONT_METHOD(indexer_prolog),
                         FRONT_METHOD(mla_prolog),   FRONT_METHOD(mla_indexer_prolog), FRONT_METHOD(pg_prolog),
                         FRONT_METHOD(indexer_prolog_v4), FRONT_METHOD(hc_pre),    FRONT_METHOD(window_attention),
                         FRONT_METHOD(mla_prolog_v4), FRONT_METHOD(compressor),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_front", "Native front end of the operator entry points.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

// What this file was compiled for: its argument blocks follow the header of that version, its calls torch's of that release.
PyMODINIT_FUNC PyInit__front(void) {
  PyObject* m = PyModule_Create(&module);
  if (m == nullptr || PyModule_AddIntConstant(m, "ABI_VERSION", DSV32_ABI_VERSION) != 0 ||
      PyModule_AddStringConstant(m, "TORCH_VERSION", TORCH_VERSION) != 0) {
    Py_XDECREF(m);
    return nullptr;
  }
  return m;
}
