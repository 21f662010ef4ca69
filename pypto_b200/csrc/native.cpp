// Host path of the operators: what `ops.py` does for an ordinary call (argument checks, workspace look-up, stream, the C
// entry point), in one native function per entry point. A decode loop called from Python spends more time here than on
// the GPU: checking 29 tensors and passing 31 arguments through ctypes took 40 of the 64 us of a prolog call.
//
// Every function takes the operator's tensors (torch tensors or `from_torch` handles) and scalars and returns True when
// the call has been enqueued. Anything out of the ordinary (a wrong dtype, shape or device, a tensor subclass, a
// workspace that does not exist yet) returns False before anything has happened: `ops.py` then goes through its own
// checks, which raise the operator's errors or allocate.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cuda_runtime_api.h>

#include <exception>

// (the C declarations take a cudaStream_t through pto_stream_t)
#include "../../include/pypto_b200.h"

namespace {

PyObject* g_handle_type = nullptr;  // compat.Tensor
PyObject* g_handle_attr = nullptr;  // "_t"
PyObject* g_workspaces = nullptr;   // ops._workspaces: {(device, stream): uint8 tensor}
PyObject* g_check = nullptr;        // _lib.check: raises PtoError for a return code

constexpr auto kI8 = at::kChar;
constexpr auto kI32 = at::kInt;
constexpr auto kI64 = at::kLong;
constexpr auto kF16 = at::kHalf;
constexpr auto kBf16 = at::kBFloat16;
constexpr auto kF32 = at::kFloat;

// The tensors of one call: all contiguous, all on one CUDA device.
class Call {
 public:
  const at::Tensor* take(PyObject* o) {
    if (!ok_) return nullptr;
    const at::Tensor* t = nullptr;
    if (THPVariable_CheckExact(o)) {
      t = &THPVariable_Unpack(o);
    } else if (reinterpret_cast<PyObject*>(Py_TYPE(o)) == g_handle_type) {
      PyObject* inner = PyObject_GetAttr(o, g_handle_attr);  // the handle keeps it alive
      if (inner == nullptr) {
        PyErr_Clear();
        return refuse();
      }
      if (THPVariable_CheckExact(inner)) t = &THPVariable_Unpack(inner);
      Py_DECREF(inner);
    }
    if (t == nullptr || !t->is_cuda() || !t->is_contiguous()) return refuse();
    const int d = t->device().index();
    if (dev_ < 0) dev_ = d;
    if (d != dev_) return refuse();
    return t;
  }
  // a tensor of a dtype and element count
  void* flat(PyObject* o, at::ScalarType dt, int64_t numel) {
    const at::Tensor* t = take(o);
    if (t == nullptr) return nullptr;
    if (t->scalar_type() != dt || t->numel() != numel) return refuse();
    return t->data_ptr();
  }
  void need(bool cond) { ok_ = ok_ && cond; }
  bool ok() const { return ok_; }
  int device() const { return dev_; }

 private:
  std::nullptr_t refuse() {
    ok_ = false;
    return nullptr;
  }
  bool ok_ = true;
  int dev_ = -1;
};

// The current stream's workspace if it exists and is large enough. `*ws` is a reference of the caller's own: another thread on
// the same stream that needs a larger workspace replaces the entry as soon as the interpreter lock is let go, and with the
// entry goes the last other reference.
bool find_workspace(const Call& c, size_t bytes, at::Tensor* ws, cudaStream_t* stream) {
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(c.device())).stream();
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;  // (a workspace that a capture records is kept: `ops._workspace`)
  if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) return false;
  PyObject* key = Py_BuildValue("(iK)", c.device(), static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(s)));
  if (key == nullptr) {
    PyErr_Clear();
    return false;
  }
  PyObject* t = PyDict_GetItemWithError(g_workspaces, key);  // borrowed
  Py_DECREF(key);
  if (t == nullptr || !THPVariable_Check(t)) {
    PyErr_Clear();
    return false;
  }
  const at::Tensor& w = THPVariable_Unpack(t);
  if (static_cast<size_t>(w.numel()) < bytes) return false;
  *ws = w;
  *stream = s;
  return true;
}

// Lets go of the interpreter lock for a scope; an exception takes it again on its way out.
class WithoutLock {
 public:
  WithoutLock() : state_(PyEval_SaveThread()) {}
  ~WithoutLock() { PyEval_RestoreThread(state_); }
  WithoutLock(const WithoutLock&) = delete;
  WithoutLock& operator=(const WithoutLock&) = delete;

 private:
  PyThreadState* state_;
};

// Runs `f(workspace, bytes, stream)` on the call's device without the interpreter lock. Throws, if at all, before `f`: what has
// been enqueued is not enqueued again by the caller's other path.
template <typename F>
PyObject* launch(const Call& c, size_t bytes, F&& f) {
  at::Tensor ws;  // (let go with the lock held, after the last use)
  cudaStream_t stream = nullptr;
  if (!c.ok() || c.device() < 0 || !find_workspace(c, bytes, &ws, &stream)) Py_RETURN_FALSE;
  void* const base = ws.data_ptr();
  const size_t have = static_cast<size_t>(ws.numel());
  int rc = 0;
  {
    const WithoutLock without_lock;
    const c10::cuda::CUDAGuard device(static_cast<c10::DeviceIndex>(c.device()));  // (its destructor does not throw)
    rc = f(base, have, reinterpret_cast<pto_stream_t>(stream));
  }
  if (rc != 0) {
    PyObject* r = PyObject_CallFunction(g_check, "i", rc);  // raises
    Py_XDECREF(r);
    if (PyErr_Occurred()) return nullptr;
  }
  Py_RETURN_TRUE;
}

bool as_int(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsLongLong(o);
  if (*v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return *v >= INT32_MIN && *v <= INT32_MAX;
}
bool as_float(PyObject* o, double* v) {
  if (PyFloat_CheckExact(o)) {
    *v = PyFloat_AS_DOUBLE(o);
    return true;
  }
  return false;
}

// ---- pieces shared by the entry points ---------------------------------------------------------------

struct Indexer {
  const void *q, *qs, *kc, *ks, *w, *act, *bt;
  int t, b, block_num, max_blocks, scale_dtype;
};

// int8 indexer: q [t, 64, 128], scales / weights [t, 64], key cache [blocks, 128, 1, 128] with its scales
void take_indexer(Call& c, PyObject* const* a, Indexer& x) {
  const at::Tensor *q = c.take(a[0]), *qs = c.take(a[1]), *kc = c.take(a[2]), *ks = c.take(a[3]), *w = c.take(a[4]),
                   *act = c.take(a[5]), *bt = c.take(a[6]);
  if (!c.ok()) return;
  c.need(q->scalar_type() == kI8 && q->dim() == 3 && q->size(1) == 64 && q->size(2) == 128);
  c.need(kc->scalar_type() == kI8 && kc->dim() == 4 && kc->size(1) == 128 && kc->size(2) == 1 && kc->size(3) == 128);
  c.need(act->scalar_type() == kI32 && act->dim() == 1 && bt->scalar_type() == kI32 && bt->dim() == 2);
  if (!c.ok()) return;
  const int64_t t = q->size(0), b = act->size(0);
  const auto sd = qs->scalar_type();
  c.need(b >= 1 && t % b == 0 && bt->size(0) == b && t <= INT32_MAX);
  c.need((sd == kF16 || sd == kF32) && ks->scalar_type() == sd && w->scalar_type() == sd);
  c.need(qs->dim() == 2 && qs->size(0) == t && qs->size(1) == 64 && w->dim() == 2 && w->size(0) == t && w->size(1) == 64);
  c.need(ks->numel() == kc->size(0) * 128);
  if (!c.ok()) return;
  x = {q->data_ptr(), qs->data_ptr(), kc->data_ptr(), ks->data_ptr(), w->data_ptr(), act->data_ptr(), bt->data_ptr(),
       static_cast<int>(t), static_cast<int>(b), static_cast<int>(kc->size(0)), static_cast<int>(bt->size(1)),
       sd == kF16 ? PTO_DT_F16 : PTO_DT_F32};
}

struct IndexerBf16 {
  const void *q, *kc, *w, *act, *bt;
  int t, b, block_num, max_blocks;
};

void take_indexer_bf16(Call& c, PyObject* const* a, IndexerBf16& x) {
  const at::Tensor *q = c.take(a[0]), *kc = c.take(a[1]), *w = c.take(a[2]), *act = c.take(a[3]), *bt = c.take(a[4]);
  if (!c.ok()) return;
  c.need(q->scalar_type() == kBf16 && q->numel() % (64 * 128) == 0);
  c.need(kc->scalar_type() == kBf16 && kc->dim() == 4 && kc->size(1) == 128 && kc->size(2) == 1 && kc->size(3) == 128);
  c.need(act->scalar_type() == kI32 && act->dim() == 1 && bt->scalar_type() == kI32 && bt->dim() == 2);
  if (!c.ok()) return;
  const int64_t t = q->numel() / (64 * 128), b = act->size(0);
  c.need(w->scalar_type() == kBf16 && w->numel() == t * 64 && b >= 1 && t % b == 0 && bt->size(0) == b && t <= INT32_MAX);
  if (!c.ok()) return;
  x = {q->data_ptr(), kc->data_ptr(), w->data_ptr(), act->data_ptr(), bt->data_ptr(),
       static_cast<int>(t), static_cast<int>(b), static_cast<int>(kc->size(0)), static_cast<int>(bt->size(1))};
}

struct Attention {
  void *qn, *qr, *ti, *bt, *act, *out;
  int t, b, max_blocks;
};

// a: query_nope, query_rope, topk_indices, block_table, kv_act_seqs, attention_out; nq = rows per token in memory
void take_attention(Call& c, PyObject* qn_, PyObject* qr_, PyObject* ti_, PyObject* bt_, PyObject* act_, PyObject* out_,
                    int64_t nq, int64_t topk, Attention& x) {
  const at::Tensor *qn = c.take(qn_), *qr = c.take(qr_), *ti = c.take(ti_), *bt = c.take(bt_), *act = c.take(act_),
                   *out = c.take(out_);
  if (!c.ok()) return;
  c.need(nq > 0 && qn->scalar_type() == kBf16 && qn->dim() == 2 && qn->size(1) == 512 && qn->size(0) % nq == 0);
  c.need(qr->scalar_type() == kBf16 && qr->dim() == 2 && qr->size(0) == qn->size(0) && qr->size(1) == 64);
  c.need(act->scalar_type() == kI32 && act->dim() == 1 && act->size(0) >= 1);
  c.need(bt->scalar_type() == kI32 && bt->dim() == 2);
  if (!c.ok()) return;
  const int64_t t = qn->size(0) / nq, b = act->size(0);
  c.need(ti->scalar_type() == kI32 && ti->numel() == t * topk && t % b == 0 && bt->size(0) == b && t <= INT32_MAX);
  c.need(out->scalar_type() == kBf16 && out->numel() == t * nq * 512);
  if (!c.ok()) return;
  x = {qn->data_ptr(), qr->data_ptr(), ti->data_ptr(), bt->data_ptr(), act->data_ptr(), out->data_ptr(),
       static_cast<int>(t), static_cast<int>(b), static_cast<int>(bt->size(1))};
}

#define PTO_GUARD_BEGIN try {
#define PTO_GUARD_END                     \
  }                                       \
  catch (const std::exception&) {         \
    if (PyErr_Occurred()) return nullptr; \
    Py_RETURN_FALSE;                      \
  }

// idx_query, idx_query_scale, idx_key_cache, idx_key_scale, idx_weight, act_seq_key, block_table, topk_res, selected_count, flags
PyObject* li_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  int64_t k = 0, flags = 0;
  if (n != 10 || !as_int(a[8], &k) || !as_int(a[9], &flags) || k < 1 || k > 2048) Py_RETURN_FALSE;
  Call c;
  Indexer x{};
  take_indexer(c, a, x);
  if (!c.ok()) Py_RETURN_FALSE;
  void* out = c.flat(a[7], kI32, x.t * k);
  return launch(c, pto_li_workspace_bytes(x.t, x.max_blocks, 128), [&](void* ws, size_t have, pto_stream_t s) {
    return pto_li_decode(static_cast<const int8_t*>(x.q), x.qs, static_cast<const int8_t*>(x.kc), x.ks, x.w, x.scale_dtype,
                         static_cast<const int32_t*>(x.act), static_cast<const int32_t*>(x.bt), static_cast<int32_t*>(out), x.b,
                         x.t / x.b, 64, 128, 128, x.block_num, x.max_blocks, static_cast<int>(k), static_cast<int>(flags), ws,
                         have, s);
  });
  PTO_GUARD_END
}

// idx_query, idx_key_cache, idx_weight, act_seq_key, block_table, topk_res, selected_count, flags
PyObject* li_decode_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  int64_t k = 0, flags = 0;
  if (n != 8 || !as_int(a[6], &k) || !as_int(a[7], &flags) || k < 1 || k > 2048) Py_RETURN_FALSE;
  Call c;
  IndexerBf16 x{};
  take_indexer_bf16(c, a, x);
  if (!c.ok()) Py_RETURN_FALSE;
  void* out = c.flat(a[5], kI32, x.t * k);
  return launch(c, pto_li_workspace_bytes(x.t, x.max_blocks, 128), [&](void* ws, size_t have, pto_stream_t s) {
    return pto_li_decode_bf16(x.q, x.kc, x.w, static_cast<const int32_t*>(x.act), static_cast<const int32_t*>(x.bt),
                              static_cast<int32_t*>(out), x.b, x.t / x.b, 64, 128, 128, x.block_num, x.max_blocks,
                              static_cast<int>(k), static_cast<int>(flags), ws, have, s);
  });
  PTO_GUARD_END
}

// query_nope, query_rope, key_nope_2d, key_rope_2d, k_nope_scales, topk_indices, block_table, kv_act_seqs, attention_out, nq, n_kv,
// softmax_scale, topk, block_size, max_blocknum_perbatch, head_begin, nq_total (None: nq)
PyObject* sfa(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  int64_t nq = 0, n_kv = 0, topk = 0, bs = 0, mb = 0, h0 = 0, nt = 0;
  double scale = 0;
  if (n != 17 || !as_int(a[9], &nq) || !as_int(a[10], &n_kv) || !as_float(a[11], &scale) || !as_int(a[12], &topk) ||
      !as_int(a[13], &bs) || !as_int(a[14], &mb) || !as_int(a[15], &h0)) {
    Py_RETURN_FALSE;
  }
  if (a[16] == Py_None) nt = nq;
  else if (!as_int(a[16], &nt)) Py_RETURN_FALSE;
  Call c;
  c.need(n_kv == 1 && nq > 0 && nq % 16 == 0 && h0 >= 0 && h0 + nq <= nt && topk >= 1);
  Attention x{};
  take_attention(c, a[0], a[1], a[5], a[6], a[7], a[8], nt, topk, x);
  const at::Tensor *kn = c.take(a[2]), *kr = c.take(a[3]);
  if (!c.ok()) Py_RETURN_FALSE;
  const bool bf16 = kn->scalar_type() == kBf16;
  c.need((bf16 || kn->scalar_type() == kI8) && kn->dim() == 2 && kn->size(1) == 512 && x.max_blocks >= mb);
  const int64_t rows = kn->dim() == 2 ? kn->size(0) : 0;
  c.need(kr->scalar_type() == kBf16 && kr->dim() == 2 && kr->size(0) == rows && kr->size(1) == 64);
  const void* sc = nullptr;
  if (c.ok() && !bf16) {
    const at::Tensor* t = c.take(a[4]);
    if (!c.ok()) Py_RETURN_FALSE;
    c.need(t->scalar_type() == kF32 && t->dim() == 2 && t->size(0) == rows && t->size(1) == 4);
    sc = t->data_ptr();
  }
  if (!c.ok()) Py_RETURN_FALSE;
  const void *knp = kn->data_ptr(), *krp = kr->data_ptr();
  return launch(c, pto_sfa_workspace_bytes(x.t, static_cast<int>(nq)) + pto_sfa_extra_bytes(x.t, static_cast<int>(nq)), [&](void* ws, size_t have, pto_stream_t s) {
    const auto *ti = static_cast<const int32_t*>(x.ti), *bt = static_cast<const int32_t*>(x.bt), *act = static_cast<const int32_t*>(x.act);
    const int s1 = x.t / x.b, inq = static_cast<int>(nq), ik = static_cast<int>(topk), ibs = static_cast<int>(bs),
              int_ = static_cast<int>(nt), ih = static_cast<int>(h0);
    if (bf16) {
      return pto_sfa_bf16(x.qn, x.qr, knp, krp, ti, bt, act, x.out, x.b, s1, inq, 1, static_cast<float>(scale), ik, ibs, rows,
                          x.max_blocks, int_, ih, ws, have, s);
    }
    return pto_sfa_quant(x.qn, x.qr, static_cast<const int8_t*>(knp), krp, static_cast<const float*>(sc), ti, bt, act, x.out, x.b,
                         s1, inq, 1, static_cast<float>(scale), ik, ibs, rows, x.max_blocks, int_, ih, ws, have, s);
  });
  PTO_GUARD_END
}

// query_nope, query_rope, nope_cache, topk_indices, block_table, kv_act_seqs, attention_out, nq, n_kv, softmax_scale, topk, block_size
PyObject* sfa_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  int64_t nq = 0, n_kv = 0, topk = 0, bs = 0;
  double scale = 0;
  if (n != 12 || !as_int(a[7], &nq) || !as_int(a[8], &n_kv) || !as_float(a[9], &scale) || !as_int(a[10], &topk) ||
      !as_int(a[11], &bs)) {
    Py_RETURN_FALSE;
  }
  Call c;
  c.need(n_kv == 1 && nq > 0 && topk >= 1);
  Attention x{};
  take_attention(c, a[0], a[1], a[3], a[4], a[5], a[6], nq, topk, x);
  const at::Tensor* cache = c.take(a[2]);
  if (!c.ok()) Py_RETURN_FALSE;
  c.need(cache->scalar_type() == kI8 && cache->dim() == 2 && cache->size(1) == 656);
  if (!c.ok()) Py_RETURN_FALSE;
  const int64_t rows = cache->size(0);
  const auto* p = static_cast<const int8_t*>(cache->data_ptr());
  return launch(c, pto_sfa_workspace_bytes(x.t, static_cast<int>(nq)) + pto_sfa_extra_bytes(x.t, static_cast<int>(nq)), [&](void* ws, size_t have, pto_stream_t s) {
    return pto_sfa_packed(x.qn, x.qr, p, static_cast<const int32_t*>(x.ti), static_cast<const int32_t*>(x.bt),
                          static_cast<const int32_t*>(x.act), x.out, x.b, x.t / x.b, static_cast<int>(nq), 1,
                          static_cast<float>(scale), static_cast<int>(topk), static_cast<int>(bs), rows, x.max_blocks,
                          static_cast<int>(nq), 0, ws, have, s);
  });
  PTO_GUARD_END
}

// idx_query, idx_query_scale, idx_key_cache, idx_key_scale, idx_weight, query_nope, query_rope, key_nope_2d, key_rope_2d, k_nope_scales,
// act_seq, block_table, topk_res, attention_out, nq, softmax_scale, selected_count, flags
PyObject* fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  int64_t nq = 0, k = 0, flags = 0;
  double scale = 0;
  if (n != 18 || !as_int(a[14], &nq) || !as_float(a[15], &scale) || !as_int(a[16], &k) || !as_int(a[17], &flags) || k < 1) {
    Py_RETURN_FALSE;
  }
  Call c;
  Indexer x{};
  PyObject* const ia[7] = {a[0], a[1], a[2], a[3], a[4], a[10], a[11]};
  take_indexer(c, ia, x);
  Attention y{};
  take_attention(c, a[5], a[6], a[12], a[11], a[10], a[13], nq, k, y);
  const at::Tensor *kn = c.take(a[7]), *kr = c.take(a[8]), *sc = c.take(a[9]);
  if (!c.ok()) Py_RETURN_FALSE;
  const int64_t rows = static_cast<int64_t>(x.block_num) * 128;
  c.need(x.t == y.t && kn->scalar_type() == kI8 && kn->dim() == 2 && kn->size(0) == rows && kn->size(1) == 512);
  c.need(kr->scalar_type() == kBf16 && kr->dim() == 2 && kr->size(0) == rows && kr->size(1) == 64);
  c.need(sc->scalar_type() == kF32 && sc->dim() == 2 && sc->size(0) == rows && sc->size(1) == 4);
  if (!c.ok()) Py_RETURN_FALSE;
  const void *knp = kn->data_ptr(), *krp = kr->data_ptr(), *scp = sc->data_ptr();
  return launch(c, pto_decode_workspace_bytes(x.t, x.max_blocks, 128, static_cast<int>(nq)) + pto_sfa_extra_bytes(x.t, static_cast<int>(nq)), [&](void* ws, size_t have, pto_stream_t s) {
    return pto_decode_fused(static_cast<const int8_t*>(x.q), x.qs, static_cast<const int8_t*>(x.kc), x.ks, x.w, x.scale_dtype,
                            y.qn, y.qr, static_cast<const int8_t*>(knp), krp, static_cast<const float*>(scp),
                            static_cast<const int32_t*>(x.act), static_cast<const int32_t*>(x.bt), static_cast<int32_t*>(y.ti),
                            y.out, x.b, x.t / x.b, x.block_num, x.max_blocks, static_cast<int>(k), static_cast<int>(nq),
                            static_cast<float>(scale), static_cast<int>(flags), ws, have, s);
  });
  PTO_GUARD_END
}

// idx_query, idx_key_cache, idx_weight, query_nope, query_rope, key_nope_2d, key_rope_2d, act_seq, block_table, topk_res, attention_out,
// nq, softmax_scale, selected_count, flags
PyObject* fused_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  int64_t nq = 0, k = 0, flags = 0;
  double scale = 0;
  if (n != 15 || !as_int(a[11], &nq) || !as_float(a[12], &scale) || !as_int(a[13], &k) || !as_int(a[14], &flags) || k < 1) {
    Py_RETURN_FALSE;
  }
  Call c;
  IndexerBf16 x{};
  PyObject* const ia[5] = {a[0], a[1], a[2], a[7], a[8]};
  take_indexer_bf16(c, ia, x);
  Attention y{};
  take_attention(c, a[3], a[4], a[9], a[8], a[7], a[10], nq, k, y);
  const at::Tensor *kn = c.take(a[5]), *kr = c.take(a[6]);
  if (!c.ok()) Py_RETURN_FALSE;
  const int64_t rows = static_cast<int64_t>(x.block_num) * 128;
  c.need(nq == 128 && x.t == y.t && kn->scalar_type() == kBf16 && kn->dim() == 2 && kn->size(0) == rows && kn->size(1) == 512);
  c.need(kr->scalar_type() == kBf16 && kr->dim() == 2 && kr->size(0) == rows && kr->size(1) == 64);
  if (!c.ok()) Py_RETURN_FALSE;
  const void *knp = kn->data_ptr(), *krp = kr->data_ptr();
  return launch(c, pto_decode_workspace_bytes(x.t, x.max_blocks, 128, static_cast<int>(nq)) + pto_sfa_extra_bytes(x.t, static_cast<int>(nq)), [&](void* ws, size_t have, pto_stream_t s) {
    return pto_decode_fused_bf16(x.q, x.kc, x.w, y.qn, y.qr, knp, krp, static_cast<const int32_t*>(x.act),
                                 static_cast<const int32_t*>(x.bt), static_cast<int32_t*>(y.ti), y.out, x.b, x.t / x.b, x.block_num,
                                 x.max_blocks, static_cast<int>(k), static_cast<int>(nq), static_cast<float>(scale),
                                 static_cast<int>(flags), ws, have, s);
  });
  PTO_GUARD_END
}

// the 24 inputs and 10 outputs of the quantised prolog, the packed cache or None, eps_cq, eps_ckv, ln_eps
PyObject* prolog_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  double e0 = 0, e1 = 0, e2 = 0;
  if (n != 38 || !as_float(a[35], &e0) || !as_float(a[36], &e1) || !as_float(a[37], &e2)) Py_RETURN_FALSE;
  Call c;
  const at::Tensor *x = c.take(a[0]), *w_dq = c.take(a[1]), *kv = c.take(a[11]);
  if (!c.ok()) Py_RETURN_FALSE;
  c.need(x->scalar_type() == kBf16 && x->dim() == 2 && w_dq->scalar_type() == kBf16 && w_dq->dim() == 2 && kv->scalar_type() == kI8 &&
         kv->numel() % 512 == 0);
  if (!c.ok()) Py_RETURN_FALSE;
  const int64_t t = x->size(0), h = x->size(1), r = w_dq->size(1), rows = kv->numel() / 512;
  c.need(w_dq->size(0) == h && t <= INT32_MAX && h <= INT32_MAX && r <= INT32_MAX);
  void *w_uqqr = c.flat(a[2], kI8, r * 128 * 192), *w_sc = c.flat(a[3], kF32, 128 * 192), *w_uk = c.flat(a[4], kBf16, 128 * 128 * 512),
       *w_dkv = c.flat(a[5], kBf16, h * 576), *g_cq = c.flat(a[6], kBf16, r), *g_ckv = c.flat(a[7], kBf16, 512),
       *cos = c.flat(a[8], kBf16, t * 64), *sin = c.flat(a[9], kBf16, t * 64), *ci = c.flat(a[10], kI64, t),
       *kr = c.flat(a[12], kBf16, rows * 64), *ks = c.flat(a[13], kF32, rows * 4), *w_qb = c.flat(a[14], kI8, r * 64 * 128),
       *w_qbs = c.flat(a[15], kF32, 64 * 128), *w_k = c.flat(a[16], kBf16, h * 128), *w_p = c.flat(a[17], kBf16, h * 64),
       *lg = c.flat(a[18], kBf16, 128), *lb = c.flat(a[19], kBf16, 128), *hq = c.flat(a[20], kBf16, 128 * 128),
       *hk = c.flat(a[21], kBf16, 128 * 128), *ik = c.flat(a[22], kI8, rows * 128), *iks = c.flat(a[23], kF16, rows),
       *q_nope = c.flat(a[24], kBf16, t * 128 * 512), *q_rope = c.flat(a[25], kBf16, t * 128 * 64),
       *q_i8 = c.flat(a[29], kI8, t * 64 * 128), *q_sc = c.flat(a[30], kF16, t * 64), *w_out = c.flat(a[33], kF16, t * 64);
  if (!c.ok()) Py_RETURN_FALSE;
  // the caches' outputs are the caches themselves (another tensor is filled from its input first: not here)
  const int in_place[5][2] = {{11, 26}, {12, 27}, {13, 28}, {22, 31}, {23, 32}};
  for (const auto& io : in_place) {
    if (a[io[0]] != a[io[1]]) {
      const at::Tensor *in = c.take(a[io[0]]), *out = c.take(a[io[1]]);
      if (!c.ok() || in->data_ptr() != out->data_ptr() || in->scalar_type() != out->scalar_type() || in->sizes() != out->sizes()) {
        Py_RETURN_FALSE;
      }
    }
  }
  void* packed = nullptr;
  if (a[34] != Py_None) packed = c.flat(a[34], kI8, rows * 656);
  if (!c.ok()) Py_RETURN_FALSE;
  void *xp = x->data_ptr(), *dqp = w_dq->data_ptr(), *kvp = kv->data_ptr();
  return launch(c, pto_prolog_workspace_bytes(static_cast<int>(t), static_cast<int>(h), static_cast<int>(r)),
                [&](void* ws, size_t have, pto_stream_t s) {
    return pto_mla_indexer_prolog_quant(
        xp, dqp, static_cast<const int8_t*>(w_uqqr), static_cast<const float*>(w_sc), w_uk, w_dkv, g_cq, g_ckv, cos, sin,
        static_cast<const int64_t*>(ci), static_cast<int8_t*>(kvp), kr, static_cast<float*>(ks), static_cast<const int8_t*>(w_qb),
        static_cast<const float*>(w_qbs), w_k, w_p, lg, lb, hq, hk, static_cast<int8_t*>(ik), iks, q_nope, q_rope,
        static_cast<int8_t*>(q_i8), q_sc, w_out, nullptr, static_cast<int8_t*>(packed), static_cast<int>(t), static_cast<int>(h),
        static_cast<int>(r), rows, static_cast<float>(e0), static_cast<float>(e1), static_cast<float>(e2), ws, have, s);
  });
  PTO_GUARD_END
}

// token_x, w_dq, w_uq_qr, w_uk, w_dkv_kr, gamma_cq, gamma_ckv, cos, sin, cache_index, kv_cache, kr_cache, idx_w_qb, idx_wk, idx_w_proj,
// idx_ln_gamma, idx_ln_beta, idx_k_cache, query_nope_out, query_rope_out, idx_query_out, idx_weights_out, q_norm_out or None, eps_cq,
// eps_ckv, ln_eps
PyObject* prolog(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PTO_GUARD_BEGIN
  double e0 = 0, e1 = 0, e2 = 0;
  if (n != 26 || !as_float(a[23], &e0) || !as_float(a[24], &e1) || !as_float(a[25], &e2)) Py_RETURN_FALSE;
  Call c;
  const at::Tensor *x = c.take(a[0]), *w_dq = c.take(a[1]), *kv = c.take(a[10]);
  if (!c.ok()) Py_RETURN_FALSE;
  c.need(x->scalar_type() == kBf16 && x->dim() == 2 && w_dq->scalar_type() == kBf16 && w_dq->dim() == 2 &&
         kv->scalar_type() == kBf16 && kv->numel() % 512 == 0);
  if (!c.ok()) Py_RETURN_FALSE;
  const int64_t t = x->size(0), h = x->size(1), r = w_dq->size(1), rows = kv->numel() / 512;
  c.need(w_dq->size(0) == h && t <= INT32_MAX && h <= INT32_MAX && r <= INT32_MAX);
  void *w_uqqr = c.flat(a[2], kBf16, r * 128 * 192), *w_uk = c.flat(a[3], kBf16, 128 * 128 * 512), *w_dkv = c.flat(a[4], kBf16, h * 576),
       *g_cq = c.flat(a[5], kBf16, r), *g_ckv = c.flat(a[6], kBf16, 512), *cos = c.flat(a[7], kBf16, t * 64),
       *sin = c.flat(a[8], kBf16, t * 64), *ci = c.flat(a[9], kI64, t), *kr = c.flat(a[11], kBf16, rows * 64),
       *w_qb = c.flat(a[12], kBf16, r * 64 * 128), *w_k = c.flat(a[13], kBf16, h * 128), *w_p = c.flat(a[14], kBf16, h * 64),
       *lg = c.flat(a[15], kBf16, 128), *lb = c.flat(a[16], kBf16, 128), *ik = c.flat(a[17], kBf16, rows * 128),
       *q_nope = c.flat(a[18], kBf16, t * 128 * 512), *q_rope = c.flat(a[19], kBf16, t * 128 * 64),
       *iq = c.flat(a[20], kBf16, t * 64 * 128), *w_out = c.flat(a[21], kBf16, t * 64);
  void* qn = nullptr;
  if (c.ok() && a[22] != Py_None) qn = c.flat(a[22], kBf16, t * r);
  if (!c.ok()) Py_RETURN_FALSE;
  void *xp = x->data_ptr(), *dqp = w_dq->data_ptr(), *kvp = kv->data_ptr();
  return launch(c, pto_prolog_nonquant_workspace_bytes(static_cast<int>(t), static_cast<int>(h), static_cast<int>(r)),
                [&](void* ws, size_t have, pto_stream_t s) {
    return pto_mla_indexer_prolog(xp, dqp, w_uqqr, w_uk, w_dkv, g_cq, g_ckv, cos, sin, static_cast<const int64_t*>(ci), kvp, kr, w_qb,
                                  w_k, w_p, lg, lb, ik, q_nope, q_rope, iq, w_out, qn, nullptr, static_cast<int>(t),
                                  static_cast<int>(h), static_cast<int>(r), rows, static_cast<float>(e0), static_cast<float>(e1),
                                  static_cast<float>(e2), ws, have, s);
  });
  PTO_GUARD_END
}

// handle type (compat.Tensor), workspace dict, _lib.check
PyObject* setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 3 || !PyDict_Check(a[1])) {
    PyErr_SetString(PyExc_TypeError, "setup(handle_type, workspaces, check)");
    return nullptr;
  }
  g_handle_type = Py_NewRef(a[0]);
  g_workspaces = Py_NewRef(a[1]);
  g_check = Py_NewRef(a[2]);
  if (g_handle_attr == nullptr) g_handle_attr = PyUnicode_InternFromString("_t");
  Py_RETURN_NONE;
}

#define PTO_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {PTO_METHOD(setup), PTO_METHOD(li_decode), PTO_METHOD(li_decode_bf16), PTO_METHOD(sfa), PTO_METHOD(sfa_packed),
                           PTO_METHOD(fused), PTO_METHOD(fused_bf16), PTO_METHOD(prolog_quant), PTO_METHOD(prolog),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&g_module); }
