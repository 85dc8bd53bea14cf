// Host path of the per-layer operators in native code (a CPython module over libhqkv's C ABI).
//
// A decode step calls these once per layer; the two kernels of a call take 10 - 20 us at batch 1, and walking the
// 42-slot tuple, filling a ctypes descriptor and allocating the results from Python took 18 - 25 us.  Here the tuple
// is read directly (40 pointer loads, no memo to look up or to keep valid), the results come from torch's allocator
// and the library is called through its function pointers: 5 - 6 us.
//
// Every function returns None for arguments it does not take as they are (non-contiguous tiers, wrong types, CPU
// tensors, an error status): the Python operator then goes its general way, which copies or raises.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <vector>

#include "hqkv.h"

#ifndef HQKV_BUILD_ID
#define HQKV_BUILD_ID "unstamped"
#endif
static const char g_build_stamp[] = "HQKV_BUILD_ID=" HQKV_BUILD_ID;

namespace {

// entry points of the library that _lib.py has loaded (it may be another build of it, so nothing is linked here)
struct Lib {
  decltype(&hqkv_decode_workspace_bytes) decode_workspace_bytes;
  decltype(&hqkv_decode_attention) decode_attention;
  decltype(&hqkv_decode_attention_headsum) decode_attention_headsum;
  decltype(&hqkv_quantize_pack) quantize_pack;
  decltype(&hqkv_dequantize_unpack) dequantize_unpack;
  decltype(&hqkv_head_sum) head_sum;
  decltype(&hqkv_token_importance) token_importance;
  decltype(&hqkv_block_rank) block_rank;
  decltype(&hqkv_flush_workspace_bytes) flush_workspace_bytes;
  decltype(&hqkv_flush_prepare) flush_prepare;
  decltype(&hqkv_flush_join) flush_join;
  decltype(&hqkv_flush_tiers_beside) flush_tiers_beside;
  decltype(&hqkv_flush_finish) flush_finish;
  decltype(&hqkv_flush_evict) flush_evict;
} L;
PyObject* g_workspace_fn = nullptr;  // _lib.decode_workspace(device, bytes, stream): owns the scratch buffers
bool g_bound = false;

constexpr int kSlotK[HQKV_NUM_TIERS] = {0, 4, 12, 20, 28}, kSlotV[HQKV_NUM_TIERS] = {2, 8, 16, 24, 32};
constexpr int kBits[HQKV_NUM_TIERS] = {16, 8, 4, 2, 1};
constexpr int kSlotNorm = 38, kSlotNewK = 39, kSlotNewV = 40, kSlotSeqLen = 41, kSlots = 42;

// a slot as a contiguous CUDA tensor: false if it is something else; *t stays null for None
inline bool slot(PyObject* o, const at::Tensor** t) {
  if (o == Py_None) {
    *t = nullptr;
    return true;
  }
  if (!THPVariable_Check(o)) return false;
  const at::Tensor& v = THPVariable_Unpack(o);
  if (!v.is_cuda() || !v.is_contiguous()) return false;
  *t = &v;
  return true;
}
inline void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }

PyObject* none() { Py_RETURN_NONE; }

PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long a[14];
  PyObject* fn;
  if (!PyArg_ParseTuple(args, "KKKKKKKKKKKKKKO", &a[0], &a[1], &a[2], &a[3], &a[4], &a[5], &a[6], &a[7], &a[8], &a[9], &a[10],
                        &a[11], &a[12], &a[13], &fn))
    return nullptr;
  int i = 0;
  auto take = [&](auto& f) { f = reinterpret_cast<std::decay_t<decltype(f)>>(a[i++]); };
  take(L.decode_workspace_bytes);
  take(L.decode_attention);
  take(L.decode_attention_headsum);
  take(L.quantize_pack);
  take(L.dequantize_unpack);
  take(L.head_sum);
  take(L.token_importance);
  take(L.block_rank);
  take(L.flush_workspace_bytes);
  take(L.flush_prepare);
  take(L.flush_join);
  take(L.flush_tiers_beside);
  take(L.flush_finish);
  take(L.flush_evict);
  Py_INCREF(fn);
  Py_XDECREF(g_workspace_fn);
  g_workspace_fn = fn;
  g_bound = true;
  Py_RETURN_NONE;
}

// ---- scratch of the decode call: the buffers belong to _lib.decode_workspace, one per (device, stream), and are
//      never released; here only their addresses are remembered (under the GIL)
struct Scratch {
  int dev;
  cudaStream_t stream;
  void* p;
  size_t bytes;
};
std::vector<Scratch> g_scratch;

bool scratch(int dev, cudaStream_t st, size_t need, PyObject* any_tensor, void** p, size_t* bytes) {
  for (const Scratch& s : g_scratch)
    if (s.dev == dev && s.stream == st && s.bytes >= need) {
      *p = s.p;
      *bytes = s.bytes;
      return true;
    }
  PyObject* device = PyObject_GetAttrString(any_tensor, "device");
  if (!device) return false;
  PyObject* buf = PyObject_CallFunction(g_workspace_fn, "OKK", device, static_cast<unsigned long long>(need),
                                        static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(st)));
  Py_DECREF(device);
  if (!buf) return false;
  const at::Tensor& t = THPVariable_Unpack(buf);
  Scratch s{dev, st, t.data_ptr(), static_cast<size_t>(t.numel())};
  Py_DECREF(buf);
  bool known = false;
  for (Scratch& o : g_scratch)
    if (o.dev == dev && o.stream == st) {
      o = s;
      known = true;
    }
  if (!known) g_scratch.push_back(s);
  *p = s.p;
  *bytes = s.bytes;
  return true;
}

inline cudaStream_t current_stream(const at::Tensor& t) {
  return c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

PyObject* pack(std::initializer_list<at::Tensor> ts) {
  PyObject* out = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  if (!out) return nullptr;
  Py_ssize_t i = 0;
  for (const at::Tensor& t : ts) {
    PyObject* w = THPVariable_Wrap(t);
    if (!w) {
      Py_DECREF(out);
      return nullptr;
    }
    PyTuple_SET_ITEM(out, i++, w);
  }
  return out;
}

// decode(q, cache, block_size, group_size, low_codec, head_sum_row | None) -> (attn_weights, attn_output) | None
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  if (!g_bound || na != 6 || !THPVariable_Check(a[0]) || !PyTuple_Check(a[1]) || PyTuple_GET_SIZE(a[1]) != kSlots)
    return none();
  const at::Tensor& q_in = THPVariable_Unpack(a[0]);
  if (!q_in.is_cuda() || q_in.scalar_type() != at::kHalf || q_in.dim() != 4 || q_in.size(2) != 1) return none();
  PyObject* cache = a[1];
  hqkv_cache_desc_t d = {};
  d.group_k = static_cast<int32_t>(PyLong_AsLong(a[2]));
  d.group_v = static_cast<int32_t>(PyLong_AsLong(a[3]));
  const int low_codec = static_cast<int>(PyLong_AsLong(a[4]));
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return none();
  }
  int64_t B = 0, H = 0, D = 0, n_k = 0;
  const at::Tensor* where = nullptr;
  for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
    const at::Tensor *k[4] = {}, *v[4] = {};
    const int parts = t == 0 ? 2 : 4;
    for (int i = 0; i < parts; ++i)
      if (!slot(PyTuple_GET_ITEM(cache, kSlotK[t] + i), &k[i]) || !slot(PyTuple_GET_ITEM(cache, kSlotV[t] + i), &v[i]))
        return none();
    hqkv_tier_t& T = d.tier[t];
    T.bits = kBits[t];
    T.codec = kBits[t] == 1 ? low_codec : 0;
    for (const at::Tensor* idx : {k[1], v[1]})
      if (idx && idx->scalar_type() != at::kLong) return none();
    T.n_k = k[1] ? static_cast<int32_t>(k[1]->numel()) : 0;
    T.n_v = v[1] ? static_cast<int32_t>(v[1]->numel()) : 0;
    n_k += T.n_k;
    T.k_data = ptr(k[0]);
    T.k_idx = static_cast<const int64_t*>(ptr(k[1]));
    T.k_scale = ptr(k[2]);
    T.k_zero = ptr(k[3]);
    T.v_data = ptr(v[0]);
    T.v_idx = static_cast<const int64_t*>(ptr(v[1]));
    T.v_scale = ptr(v[2]);
    T.v_zero = ptr(v[3]);
    if (v[0]) {
      if (v[0]->dim() != 4) return none();
      B = v[0]->size(0);
      H = v[0]->size(1);
      D = v[0]->size(3) * (t == 0 ? 1 : 32 / kBits[t]);
      where = v[0];
    }
  }
  const at::Tensor *nk, *nv;
  if (!slot(PyTuple_GET_ITEM(cache, kSlotNewK), &nk) || !slot(PyTuple_GET_ITEM(cache, kSlotNewV), &nv)) return none();
  if (nv) {
    if (nv->dim() != 4 || (where && (nv->size(0) != B || nv->size(1) != H || nv->size(3) != D))) return none();
    B = nv->size(0);
    H = nv->size(1);
    D = nv->size(3);
    d.n_new = static_cast<int32_t>(nv->size(2));
    where = nv;
  }
  if (!where || where->device() != q_in.device() || q_in.size(0) != B || q_in.size(3) != D) return none();
  d.new_k = ptr(nk);
  d.new_v = ptr(nv);
  const int64_t nh_q = q_in.size(1), len = n_k + d.n_new;
  d.B = static_cast<int32_t>(B);
  d.H = static_cast<int32_t>(H);
  d.D = static_cast<int32_t>(D);
  d.nh_q = static_cast<int32_t>(nh_q);
  d.softmax_scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(D)));
  void* row = nullptr;
  if (a[5] != Py_None) {
    if (!THPVariable_Check(a[5])) return none();
    const at::Tensor& r = THPVariable_Unpack(a[5]);
    if (r.scalar_type() != at::kHalf || r.device() != q_in.device() || r.dim() != 1 || r.numel() < len || r.stride(0) != 1)
      return none();
    row = r.data_ptr();
  }
  const size_t need = L.decode_workspace_bytes(&d);
  if (need == 0) return none();
  const c10::cuda::OptionalCUDAGuard guard(q_in.device());
  const cudaStream_t st = current_stream(q_in);
  void* ws;
  size_t ws_bytes;
  if (!scratch(q_in.device().index(), st, need, a[0], &ws, &ws_bytes)) return nullptr;
  const at::Tensor q = q_in.contiguous();
  at::Tensor weights = at::empty({B, nh_q, 1, len}, q.options());
  at::Tensor out = at::empty({B, nh_q, 1, D}, q.options());
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = row ? L.decode_attention_headsum(&d, q.data_ptr(), weights.data_ptr(), out.data_ptr(), row, ws, ws_bytes, st)
           : L.decode_attention(&d, q.data_ptr(), weights.data_ptr(), out.data_ptr(), ws, ws_bytes, st);
  Py_END_ALLOW_THREADS
  return rc ? none() : pack({weights, out});
  END_HANDLE_TH_ERRORS
}

// quantize_pack(data, group_size, bit) -> (code, scale, mn) | None
PyObject* quantize_pack(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  if (!g_bound || na != 3 || !THPVariable_Check(a[0])) return none();
  at::Tensor x = THPVariable_Unpack(a[0]);
  const int64_t group = PyLong_AsLong(a[1]), bit = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return none();
  }
  if (!x.is_cuda() || x.scalar_type() != at::kHalf || x.dim() != 4 || group <= 0 || x.size(3) % group ||
      (bit != 8 && bit != 4 && bit != 2 && bit != 1))
    return none();
  const int64_t B = x.size(0), nh = x.size(1), D = x.size(2), T = x.size(3);
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  const bool collapsible = B == 1 || x.stride(0) == nh * x.stride(1);
  if (!(collapsible && (x.stride(3) == 1 || x.stride(2) == 1)) || D == 1 || T == 1) x = x.contiguous();
  const auto opt = x.options();
  at::Tensor code = at::empty({B, nh, D, T * bit / 32}, opt.dtype(at::kInt));
  at::Tensor scale = at::empty({B, nh, D, T / group}, opt), mn = at::empty({B, nh, D, T / group}, opt);
  const cudaStream_t st = current_stream(x);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = L.quantize_pack(x.data_ptr(), B * nh * D, T, D, x.stride(1), x.stride(2), x.stride(3), static_cast<int>(group),
                       static_cast<int>(bit), code.data_ptr(), scale.data_ptr(), mn.data_ptr(), st);
  Py_END_ALLOW_THREADS
  return rc ? none() : pack({code, scale, mn});
  END_HANDLE_TH_ERRORS
}

// dequantize_unpack(code, scale, mn, group_size, bit) -> values | None
PyObject* dequantize_unpack(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  const at::Tensor *code, *scale, *mn;
  if (!g_bound || na != 5 || !slot(a[0], &code) || !slot(a[1], &scale) || !slot(a[2], &mn) || !code || !scale || !mn)
    return none();
  const int64_t group = PyLong_AsLong(a[3]), bit = PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return none();
  }
  if (code->dim() != 4 || (bit != 8 && bit != 4 && bit != 2 && bit != 1)) return none();
  const int64_t B = code->size(0), nh = code->size(1), D = code->size(2), T = code->size(3) * (32 / bit);
  const c10::cuda::OptionalCUDAGuard guard(code->device());
  at::Tensor out = at::empty({B, nh, D, T}, code->options().dtype(at::kHalf));
  const cudaStream_t st = current_stream(*code);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = L.dequantize_unpack(code->data_ptr(), scale->data_ptr(), mn->data_ptr(), B * nh * D, T, static_cast<int>(group),
                           static_cast<int>(bit), out.data_ptr(), st);
  Py_END_ALLOW_THREADS
  return rc ? none() : THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// head_sum(attn_weights [B, nh, 1, L], ring [rows, cap], row) -> True | None
PyObject* head_sum(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  const at::Tensor *w, *ring;
  if (!g_bound || na != 3 || !slot(a[0], &w) || !slot(a[1], &ring) || !w || !ring) return none();
  const int64_t row = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return none();
  }
  if (w->dim() != 4 || w->size(2) != 1 || w->scalar_type() != at::kHalf || ring->scalar_type() != at::kHalf || ring->dim() != 2 ||
      row < 0 || row >= ring->size(0) || w->size(3) > ring->size(1) || w->device() != ring->device())
    return none();
  const c10::cuda::OptionalCUDAGuard guard(w->device());
  const int64_t len = w->size(3);
  void* out = static_cast<at::Half*>(ring->data_ptr()) + row * ring->size(1);
  const cudaStream_t st = current_stream(*w);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = L.head_sum(w->data_ptr(), static_cast<int>(w->size(0)), static_cast<int>(w->size(1)), len, len, out, st);
  Py_END_ALLOW_THREADS
  if (rc) return none();
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// token_importance(ring [rows, cap], rows, L) -> [L] | None
PyObject* token_importance(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  const at::Tensor* ring;
  if (!g_bound || na != 3 || !slot(a[0], &ring) || !ring) return none();
  const int64_t rows = PyLong_AsLong(a[1]), len = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return none();
  }
  if (ring->dim() != 2 || ring->scalar_type() != at::kHalf || rows <= 0 || rows > ring->size(0) || len < 0 || len > ring->size(1))
    return none();
  const c10::cuda::OptionalCUDAGuard guard(ring->device());
  at::Tensor out = at::empty({len}, ring->options());
  const int rc = L.token_importance(ring->data_ptr(), static_cast<int>(rows), ring->size(1), len, out.data_ptr(), current_stream(*ring));
  return rc ? none() : THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// block_rank(importance, range | None, block_size, block_num) -> ids | None
PyObject* block_rank(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  const at::Tensor *imp, *range;
  if (!g_bound || na != 4 || !slot(a[0], &imp) || !slot(a[1], &range) || !imp) return none();
  const int64_t block = PyLong_AsLong(a[2]), num = PyLong_AsLong(a[3]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return none();
  }
  if (imp->scalar_type() != at::kHalf || block <= 0 || num < 0 || imp->numel() != block * num ||
      (range && (range->scalar_type() != at::kHalf || range->device() != imp->device())))
    return none();
  const c10::cuda::OptionalCUDAGuard guard(imp->device());
  at::Tensor ids = at::empty({block * num}, imp->options().dtype(at::kLong));
  const int rc = L.block_rank(imp->data_ptr(), ptr(range), static_cast<int>(block), static_cast<int>(num), ids.data_ptr<int64_t>(),
                              current_stream(*imp));
  return rc ? none() : THPVariable_Wrap(ids);
  END_HANDLE_TH_ERRORS
}

// Tensors of one allocation.  The parts of a tier (codes, ids, scales, zeros) live and die together; an allocation of their
// own for each of them took more host time than anything else in a flush.
struct Slab {
  // Larger tiers get an allocation per part: there the microseconds do not count (5 of 147 us with tiers of 40 MB), and blocks
  // of a tier's whole size leave holes that nothing else fits when the memory is nearly full (32 layers of 2.7 GB at batch 64
  // of 128 k tokens: 21 GB of holes and out of memory, 5 GB with separate parts).
  static constexpr int64_t kSlabMax = 128 << 20;
  std::vector<std::pair<at::Tensor*, std::vector<int64_t>>> parts;
  std::vector<at::ScalarType> types;
  void add(at::Tensor* t, std::initializer_list<int64_t> sizes, at::ScalarType type) {
    parts.emplace_back(t, sizes);
    types.push_back(type);
  }
  void allocate(const at::TensorOptions& opt) {
    auto bytes = [&](size_t i) {
      int64_t n = static_cast<int64_t>(c10::elementSize(types[i]));
      for (int64_t d : parts[i].second) n *= d;
      return (n + 511) & ~int64_t{511};
    };
    int64_t total = 0;
    for (size_t i = 0; i < parts.size(); ++i) total += bytes(i);
    if (total == 0) return;
    if (total >= kSlabMax) {
      for (size_t i = 0; i < parts.size(); ++i) *parts[i].first = at::empty(parts[i].second, opt.dtype(types[i]));
      return;
    }
    const at::Tensor base = at::empty({total}, opt.dtype(at::kByte));
    int64_t at = 0;
    for (size_t i = 0; i < parts.size(); ++i) {
      at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(base.storage()), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                              c10::scalarTypeToTypeMeta(types[i]));
      t.unsafeGetTensorImpl()->set_storage_offset(at / static_cast<int64_t>(c10::elementSize(types[i])));
      t.unsafeGetTensorImpl()->set_sizes_contiguous(parts[i].second);
      *parts[i].first = std::move(t);
      at += bytes(i);
    }
  }
};

bool six_counts(PyObject* list, int64_t (&cum)[6]) {
  if (!PyList_Check(list) || PyList_GET_SIZE(list) != 6) return false;
  int64_t run = 0;
  for (int i = 0; i < 6; ++i) {
    run += PyLong_AsLong(PyList_GET_ITEM(list, i));
    cum[i] = run;
  }
  if (!PyErr_Occurred()) return true;
  PyErr_Clear();
  return false;
}

// flush(cache, compress, history, K_sorted_idx, K counts, V counts, token_importance, low_codec, ring | None, block, group,
//       times_range) -> new cache | None
// One launch per step and side, outputs allocated while the GPU works: 430 us of host time became 90.
PyObject* flush(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  if (!g_bound || na != 12 || !PyTuple_Check(a[0]) || PyTuple_GET_SIZE(a[0]) != kSlots) return none();
  PyObject* cache = a[0];
  const at::Tensor *k_sorted, *imp, *ring, *nk, *nv, *norm;
  if (!slot(a[3], &k_sorted) || !slot(a[6], &imp) || !slot(a[8], &ring) || !k_sorted || !imp ||
      !slot(PyTuple_GET_ITEM(cache, kSlotNewK), &nk) || !slot(PyTuple_GET_ITEM(cache, kSlotNewV), &nv) || !nk || !nv ||
      !slot(PyTuple_GET_ITEM(cache, kSlotNorm), &norm))
    return none();
  hqkv_flush_t f = {};
  f.compress = PyLong_AsLong(a[1]);
  f.hist = PyLong_AsLong(a[2]);
  const int low_codec = static_cast<int>(PyLong_AsLong(a[7]));
  f.block = static_cast<int32_t>(PyLong_AsLong(a[9]));
  f.group = static_cast<int32_t>(PyLong_AsLong(a[10]));
  f.times_range = PyObject_IsTrue(a[11]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return none();
  }
  const int64_t total = f.hist + f.compress;
  const at::Device dev = nk->device();
  if (nk->dim() != 4 || nk->scalar_type() != at::kHalf || nv->scalar_type() != at::kHalf || nv->sizes() != nk->sizes() ||
      nv->device() != dev || nk->size(3) != 128 || f.compress <= 0 || f.hist < 0 || f.compress > nk->size(2) || f.block <= 0 ||
      total % f.block || !six_counts(a[4], f.k_cum) || !six_counts(a[5], f.v_cum) || k_sorted->scalar_type() != at::kLong ||
      k_sorted->device() != dev || k_sorted->numel() < f.k_cum[5] || imp->scalar_type() != at::kHalf || imp->device() != dev ||
      imp->numel() != total || (norm ? norm->scalar_type() != at::kHalf || norm->device() != dev || norm->numel() != f.hist : f.hist != 0) ||
      (ring && (ring->dim() != 2 || ring->scalar_type() != at::kHalf || ring->device() != dev || ring->size(1) < total)))
    return none();
  const int64_t B = nk->size(0), H = nk->size(1), D = 128, window = nk->size(2);
  f.B = static_cast<int32_t>(B);
  f.H = static_cast<int32_t>(H);
  f.D = static_cast<int32_t>(D);
  f.rest = window - f.compress;
  f.importance = imp->data_ptr();
  f.k_sorted = k_sorted->data_ptr<int64_t>();
  for (int side = 0; side < 2; ++side) {
    hqkv_flush_src_t& src = side ? f.v : f.k;
    const int* slots = side ? kSlotV : kSlotK;
    src.low_codec = low_codec;
    for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
      const at::Tensor* x[4] = {};
      for (int i = 0; i < (t == 0 ? 2 : 4); ++i)
        if (!slot(PyTuple_GET_ITEM(cache, slots[t] + i), &x[i]) || (x[i] && x[i]->device() != dev)) return none();
      if (x[1] && (x[1]->scalar_type() != at::kLong || !x[0] || (t > 0 && (!x[2] || !x[3])))) return none();
      src.data[t] = ptr(x[0]);
      src.scale[t] = ptr(x[2]);
      src.zero[t] = ptr(x[3]);
      src.n[t] = x[1] ? static_cast<int32_t>(x[1]->numel()) : 0;
      (side ? f.v_idx : f.k_idx)[t] = static_cast<const int64_t*>(ptr(x[1]));
    }
    src.residual = side ? nv->data_ptr() : nk->data_ptr();
    src.residual_b_stride = H * window * D;
    src.residual_h_stride = window * D;
  }
  const c10::cuda::OptionalCUDAGuard guard(dev);
  const cudaStream_t st = current_stream(*nk);
  const auto half = nk->options();
  at::Tensor norm_out = at::empty({total}, half);
  at::Tensor ws = at::empty({static_cast<int64_t>(L.flush_workspace_bytes(total))}, half.dtype(at::kByte));
  f.norm_old = ptr(norm);
  f.norm_out = norm_out.data_ptr();
  int32_t counts[16];
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = L.flush_prepare(&f, ws.data_ptr(), static_cast<size_t>(ws.numel()), counts, st);
  Py_END_ALLOW_THREADS
  if (rc) return none();
  struct Join {  // the V side and the builds run on other streams: this one waits for them before the call's memory is let go
    cudaStream_t st;
    int32_t* counts;
    bool done = false;
    int now() {
      done = true;
      return L.flush_join(counts, st);
    }
    ~Join() {
      if (!done) L.flush_join(nullptr, st);
      L.flush_finish(st);
    }
  } join{st, counts};
  for (int t = 0; t < HQKV_NUM_TIERS; ++t)
    if (counts[t] % f.block) return none();
  at::Tensor out[kSlots];
  for (int side = 0; side < 2; ++side) {
    const int* slots = side ? kSlotV : kSlotK;
    const int64_t group = side ? f.group : f.block;
    void *data[HQKV_NUM_TIERS] = {}, *scale[HQKV_NUM_TIERS] = {}, *zero[HQKV_NUM_TIERS] = {};
    int64_t* ids[HQKV_NUM_TIERS] = {};
    if (side) {  // the K build has its work, the counts of V are needed now
      Py_BEGIN_ALLOW_THREADS
      rc = join.now();
      Py_END_ALLOW_THREADS
      if (rc) return none();
    }
    for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
      const int64_t n = counts[8 * side + t], bits = kBits[t];
      if (n == 0) continue;
      at::Tensor* o = out + slots[t];
      Slab slab;
      if (t == 0) {
        if (side) slab.add(&o[0], {B, H, n, D}, at::kHalf);
        else slab.add(&o[0], {B, H, D, n}, at::kHalf);
      } else if (side) {
        slab.add(&o[0], {B, H, n, D * bits / 32}, at::kInt);
        slab.add(&o[2], {B, H, n, D / group}, at::kHalf);
        slab.add(&o[3], {B, H, n, D / group}, at::kHalf);
      } else {
        slab.add(&o[0], {B, H, D, n * bits / 32}, at::kInt);
        slab.add(&o[2], {B, H, D, n / group}, at::kHalf);
        slab.add(&o[3], {B, H, D, n / group}, at::kHalf);
      }
      slab.add(&o[1], {n}, at::kLong);
      slab.allocate(half);
      data[t] = o[0].data_ptr();
      ids[t] = o[1].data_ptr<int64_t>();
      if (t) scale[t] = o[2].data_ptr(), zero[t] = o[3].data_ptr();
    }
    at::Tensor& rest = out[side ? kSlotNewV : kSlotNewK];
    if (f.rest) rest = at::empty({B, H, f.rest, D}, half);
    rc = L.flush_tiers_beside(&f, side, ws.data_ptr(), counts, data, scale, zero, ids, f.rest ? rest.data_ptr() : nullptr, st);
    if (rc) return none();
  }
  out[kSlotNorm] = norm_out;
  if (counts[14]) {  // something was evicted on the V side: compact the range vector and the ring (beside the builds)
    out[kSlotNorm] = at::empty({counts[13]}, half);
    rc = L.flush_evict(&f, ws.data_ptr(), counts[13], out[kSlotNorm].data_ptr(), ptr(ring), ring ? ring->size(1) : 0,
                       ring ? static_cast<int>(ring->size(0)) : 0, st);
    if (rc) return none();
  }
  if (L.flush_finish(st)) return none();
  PyObject* res = PyTuple_New(kSlots);
  if (!res) return nullptr;
  for (int i = 0; i < kSlots; ++i) {
    PyObject* o;
    if (i == 36 || i == 37 || i == kSlotSeqLen) {
      o = PyTuple_GET_ITEM(cache, i);
      Py_INCREF(o);
    } else if (out[i].defined()) {
      o = THPVariable_Wrap(out[i]);
    } else {
      o = none();
    }
    if (!o) {
      Py_DECREF(res);
      return nullptr;
    }
    PyTuple_SET_ITEM(res, i, o);
  }
  return res;
  END_HANDLE_TH_ERRORS
}

PyObject* build_id(PyObject*, PyObject*) { return PyUnicode_FromString(g_build_stamp + 14); }

template <typename F>
PyCFunction fast(F f) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, "addresses of the library's entry points, and the owner of the decode scratch"},
    {"build_id", build_id, METH_NOARGS, "hash of the sources this module was compiled from"},
    {"decode", fast(decode), METH_FASTCALL, nullptr},
    {"quantize_pack", fast(quantize_pack), METH_FASTCALL, nullptr},
    {"dequantize_unpack", fast(dequantize_unpack), METH_FASTCALL, nullptr},
    {"head_sum", fast(head_sum), METH_FASTCALL, nullptr},
    {"token_importance", fast(token_importance), METH_FASTCALL, nullptr},
    {"block_rank", fast(block_rank), METH_FASTCALL, nullptr},
    {"flush", fast(flush), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
