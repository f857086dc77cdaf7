// Host path of one attention call, in native code: what lies between the Python entry points and the C ABI
// (argument checks, output and workspace allocation, the parameter block, the autograd node).
//
// A call on a short cache or a short sequence takes the GPU a few microseconds, and the same steps in
// Python (a call object, a ctypes structure filled field by field, torch.autograd.Function) took 40-50 us
// for a forward and about 200 us for a forward and backward, so such calls ran at the speed of the host.
// Here they take a few microseconds.  Decisions stay where they are: the Python layer traces and lowers
// the mods (modtrace.py) and registers the compiled module for a pair of callables; this file looks the
// pair up and calls fa_fwd / fa_decode / fa_bwd.  Whatever is not a plain call on CUDA tensors
// with registered mods is declined (None is returned) and taken by the Python layer, which also raises
// the errors of the reference for bad arguments (flaxattention/core/attention.py:119-198).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <cmath>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "../../include/flaxattn.h"

namespace {

// query blocks of at most this many rows over at least this many keys go to the split-KV kernels
// (the same constants as attention.py)
constexpr int64_t kDecodeMaxSq = 64, kDecodeMinSkv = 512;

// A module registered for a (score_mod, mask_mod) pair, with the tensors the mods capture.
struct Mods {
  fa_module* module = nullptr;
  std::vector<at::Tensor> buffers;
  PyObject* keep = nullptr;  // the Python module object (owns `module`)
  ~Mods() {
    if (keep != nullptr && Py_IsInitialized()) {
      PyGILState_STATE g = PyGILState_Ensure();
      Py_DECREF(keep);
      PyGILState_Release(g);
    }
  }
};
using ModsPtr = std::shared_ptr<Mods>;
struct PairHash {
  size_t operator()(const std::pair<PyObject*, PyObject*>& p) const {
    return ((size_t)p.first >> 4) * 1000003u ^ ((size_t)p.second >> 4);
  }
};
// All of these are read and written with the GIL held.
std::unordered_map<std::pair<PyObject*, PyObject*>, ModsPtr, PairHash>* g_mods = nullptr;
volatile int* g_status = nullptr;  // the process's status word (pinned host memory)
PyObject *g_identity = nullptr, *g_noop = nullptr, *g_error = nullptr, *g_check_status = nullptr;
// Launches of modules with captured buffers: the addresses are set and taken over by the launch under this
// lock, so that calls with other tensors on the same module from other threads do not come between.
std::mutex g_buffers_mu;

PyObject *s_mask_mod, *s_block_size, *s_mask_bits, *s_mask_bits_t, *s_bits_mod, *s_bits_sources, *s_bits_snapshot, *s_bits_at, *s_kv_tiles;
PyObject* s_tables[8];

// A reference that is dropped at the end of its scope.
struct Ref {
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};

// Everything a backward needs besides the saved tensors.
struct Call {
  ModsPtr mods;
  fa_attn_params p;          // shapes, scale, offsets, tables, flags; tensors are filled in per launch
  bool bshd = false;
  std::vector<at::Tensor> tables;  // keeps the BlockMask tensors alive
  // bit matrices over captured tensors: these tensors, and the copy of them the matrices belong to
  std::vector<at::Tensor> sources;
  at::Tensor snapshot;
};

fa_tensor describe(const at::Tensor& t, bool bshd) {
  TORCH_CHECK_VALUE(t.stride(3) == 1, "the head dimension must be contiguous");
  fa_tensor r;
  r.ptr = t.data_ptr();
  r.stride_b = t.stride(0);
  r.stride_h = t.stride(bshd ? 2 : 1);
  r.stride_s = t.stride(bshd ? 1 : 2);
  return r;
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dt, c10::Device dev) {
  return at::detail::empty_cuda(sizes, dt, dev, std::nullopt);
}
at::Tensor empty_as(const at::Tensor& t) {
  return t.is_contiguous() ? empty(t.sizes(), t.scalar_type(), t.device()) : at::empty_like(t);
}

// The scratch memory of a launch of `p`.  The fp32 kernels over bf16 parts need up to one and a half times the inputs;
// where that does not fit, the general kernels, which need next to none, are asked for instead.
at::Tensor workspace(fa_attn_params& p, size_t (*need)(const fa_attn_params*), c10::Device dev, size_t& bytes) {
  bytes = need(&p);
  try {
    return bytes > 0 ? empty({(int64_t)bytes}, at::kByte, dev) : at::Tensor();
  } catch (const c10::OutOfMemoryError&) {
    if (p.dtype != FA_F32 || (p.flags & FA_FLAG_GENERAL_KERNELS)) throw;
  }
  p.flags |= FA_FLAG_GENERAL_KERNELS;
  bytes = need(&p);
  return bytes > 0 ? empty({(int64_t)bytes}, at::kByte, dev) : at::Tensor();
}

// Holds the addresses of the captured buffers in the module for the duration of one launch.
struct BuffersLock {
  std::unique_lock<std::mutex> lk;
  int rc = FA_OK;
  explicit BuffersLock(const Mods& m) : BuffersLock(m.module, m.buffers) {}
  BuffersLock(fa_module* module, const std::vector<at::Tensor>& buffers) {
    if (buffers.empty()) return;
    lk = std::unique_lock<std::mutex>(g_buffers_mu);
    const void* ptrs[8];
    for (size_t i = 0; i < buffers.size(); ++i) ptrs[i] = buffers[i].const_data_ptr();
    rc = fa_module_set_buffers(module, ptrs, (int)buffers.size());
  }
};

// FlaxAttnError of the calling thread's last library error
[[noreturn]] void raise(int rc) {
  const std::string msg = fa_last_error();
  PyGILState_STATE g = PyGILState_Ensure();
  Ref exc(PyObject_CallFunction(g_error, "is", rc, msg.c_str()));
  if (exc.p != nullptr) PyErr_SetObject(g_error, exc.p);
  python_error err;
  err.persist();
  PyGILState_Release(g);
  throw err;
}

// What the Python layer raises when an earlier launch has reported an error in the status word
void check_status() {
  if (*g_status == 0) return;
  PyGILState_STATE g = PyGILState_Ensure();
  Ref r(PyObject_CallNoArgs(g_check_status));
  if (r.p == nullptr) {
    python_error err;
    err.persist();
    PyGILState_Release(g);
    throw err;
  }
  PyGILState_Release(g);
}

// The memory that tensors span, as fa_snapshot takes it (at most 8)
struct Ranges {
  const void* src[8];
  size_t bytes[8];
  int n;
  explicit Ranges(const std::vector<at::Tensor>& ts) : n((int)ts.size()) {
    for (int i = 0; i < n; ++i) {
      const at::Tensor& t = ts[i];
      int64_t span = 1;
      for (int64_t d = 0; d < t.dim(); ++d) span += (t.size(d) - 1) * t.stride(d);
      src[i] = t.const_data_ptr();
      bytes[i] = t.numel() == 0 ? 0 : (size_t)span * t.element_size();
    }
  }
};

// Queues the comparison of the tensors a mask captures with what they were when its bit matrices were built; the
// kernels launched next with `p` look at the word it writes (returned, to be kept until then).
at::Tensor check_snapshot(const Call& c, fa_attn_params& p, c10::Device dev, void* stream) {
  if (!c.snapshot.defined()) return {};
  const Ranges r(c.sources);
  if (fa_snapshot_bytes(r.bytes, r.n) != (size_t)c.snapshot.numel()) {
    p.tables.mask_bits = p.tables.mask_bits_t = nullptr;
    return {};
  }
  at::Tensor hold = empty({1}, at::kInt, dev);
  p.tables.mask_bits_hold = hold.mutable_data_ptr<int32_t>();
  const int rc = fa_snapshot_holds(r.src, r.bytes, r.n, c.snapshot.const_data_ptr(), hold.mutable_data_ptr<int32_t>(), stream);
  if (rc != FA_OK) raise(rc);
  return hold;
}

// q, k, v -> out, lse; throws FlaxAttnError
std::pair<at::Tensor, at::Tensor> forward(const Call& c, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
  const fa_attn_params& s = c.p;
  c10::cuda::OptionalCUDAGuard guard(q.device());
  at::Tensor out = c.bshd ? empty({s.B, s.Sq, s.Hq, s.Dv}, q.scalar_type(), q.device())
                          : empty({s.B, s.Hq, s.Sq, s.Dv}, q.scalar_type(), q.device());
  at::Tensor lse = empty({s.B, s.Hq, s.Sq}, at::kFloat, q.device());
  fa_attn_params p = s;
  p.q = describe(q, c.bshd);
  p.k = describe(k, c.bshd);
  p.v = describe(v, c.bshd);
  p.o = describe(out, c.bshd);
  p.lse = lse.mutable_data_ptr<float>();
  void* stream = (void*)c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  const at::Tensor hold = check_snapshot(c, p, q.device(), stream);
  int rc = FA_OK;
  if (p.Sq <= kDecodeMaxSq && p.Skv >= kDecodeMinSkv && p.dtype != FA_F32) {
    const int splits = fa_decode_num_splits(&p, 0);
    const size_t bytes = fa_decode_workspace_bytes(&p, splits);
    at::Tensor ws;
    if (bytes > 0) ws = empty({(int64_t)bytes}, at::kByte, q.device());
    BuffersLock buffers(*c.mods);
    rc = buffers.rc != FA_OK ? buffers.rc
                             : fa_decode(c.mods->module, &p, splits, bytes > 0 ? ws.mutable_data_ptr() : nullptr, bytes, stream);
  } else {
    size_t bytes = 0;
    const at::Tensor ws = workspace(p, fa_fwd_workspace_bytes, q.device(), bytes);
    BuffersLock buffers(*c.mods);
    rc = buffers.rc != FA_OK ? buffers.rc : fa_fwd_ws(c.mods->module, &p, bytes > 0 ? ws.mutable_data_ptr() : nullptr, bytes, stream);
  }
  if (rc != FA_OK) raise(rc);
  return {std::move(out), std::move(lse)};
}

// The residuals are those of the reference's custom_vjp (flaxattention/kernel/attention.py:335).
struct AttentionBackward : public torch::autograd::Node {
  Call call;
  torch::autograd::SavedVariable q_, k_, v_, out_, lse_;

  std::string name() const override { return "FlaxAttentionBackward"; }
  void release_variables() override {
    q_.reset_data();
    k_.reset_data();
    v_.reset_data();
    out_.reset_data();
    lse_.reset_data();
  }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    const at::Tensor q = q_.unpack(), k = k_.unpack(), v = v_.unpack(), out = out_.unpack(shared_from_this()), lse = lse_.unpack();
    at::NoGradGuard no_grad;
    check_status();
    {
      // (a saved-tensor hook may have given back something else than it was given)
      const fa_attn_params& p = call.p;
      const auto same = [&](const at::Tensor& t, int64_t H, int64_t S, int64_t D) {
        return t.device() == q.device() && t.scalar_type() == q.scalar_type() &&
               (call.bshd ? t.sizes() == at::IntArrayRef({p.B, S, H, D}) : t.sizes() == at::IntArrayRef({p.B, H, S, D}));
      };
      const auto type = p.dtype == FA_F16 ? at::kHalf : p.dtype == FA_BF16 ? at::kBFloat16 : at::kFloat;
      TORCH_CHECK(q.is_cuda() && q.scalar_type() == type && same(q, p.Hq, p.Sq, p.D) && same(k, p.Hkv, p.Skv, p.D) &&
                      same(v, p.Hkv, p.Skv, p.Dv) && same(out, p.Hq, p.Sq, p.Dv) && lse.device() == q.device() &&
                      lse.scalar_type() == at::kFloat && lse.is_contiguous() && lse.numel() == (int64_t)p.B * p.Hq * p.Sq,
                  "a saved tensor has come back with another shape, type or device");
    }
    c10::cuda::OptionalCUDAGuard guard(q.device());
    at::Tensor dout = grads[0].defined() ? grads[0] : at::zeros_like(out);
    if (dout.stride(-1) != 1) dout = dout.contiguous();
    at::Tensor dq = empty_as(q), dk = empty_as(k), dv = empty_as(v);
    fa_attn_params p = call.p;
    p.q = describe(q, call.bshd);
    p.k = describe(k, call.bshd);
    p.v = describe(v, call.bshd);
    p.o = describe(out, call.bshd);
    p.lse = (float*)lse.data_ptr();
    // dQ over bf16 parts is added up in no fixed order; the general fp32 kernels have one
    if (p.dtype == FA_F32 && at::globalContext().deterministicAlgorithms()) p.flags |= FA_FLAG_GENERAL_KERNELS;
    const fa_tensor gdo = describe(dout, call.bshd), gdq = describe(dq, call.bshd), gdk = describe(dk, call.bshd),
                    gdv = describe(dv, call.bshd);
    size_t bytes = 0;
    const at::Tensor ws = workspace(p, fa_bwd_workspace_bytes, q.device(), bytes);
    void* stream = (void*)c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    const at::Tensor hold = check_snapshot(call, p, q.device(), stream);
    int rc;
    {
      BuffersLock buffers(*call.mods);
      rc = buffers.rc != FA_OK ? buffers.rc
                               : fa_bwd(call.mods->module, &p, &gdo, &gdq, &gdk, &gdv, ws.mutable_data_ptr(), bytes, stream);
    }
    if (rc != FA_OK) raise(rc);
    return {dq, dk, dv};
  }
};

// ---- arguments -----------------------------------------------------------------------------
bool plain_tensor(PyObject* o, const at::Tensor** t) {
  if (!THPVariable_CheckExact(o)) return false;
  *t = &THPVariable_Unpack(o);
  return (*t)->defined() && (*t)->is_cuda() && (*t)->has_storage() && (*t)->layout() == at::kStrided;
}

// Calls that something looks on at: a tracer, a dispatch mode, a functorch transform.  This path makes its tensors
// and its autograd node without them, so such calls belong to the Python layer, which they see (or which refuses).
bool watched() {
  return at::tracer::impl::is_dispatch_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
         c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

// int32, contiguous, on `dev`: its address, with the tensor kept in `keep`; null on failure (None gives null with *none)
const int32_t* table(PyObject* o, c10::Device dev, std::vector<at::Tensor>& keep, bool* none) {
  *none = o == Py_None;
  const at::Tensor* t = nullptr;
  if (*none || !plain_tensor(o, &t)) return nullptr;
  if (t->scalar_type() != at::kInt || !t->is_contiguous() || t->device() != dev) return nullptr;
  keep.push_back(*t);
  return (const int32_t*)t->const_data_ptr();
}

// Fills c.p.tables from a BlockMask; false: declined.
bool read_block_mask(PyObject* bm, PyObject* mask_mod, c10::Device dev, Call& c) {
  fa_block_tables& t = c.p.tables;
  const int32_t** dst[8] = {&t.kv_num_blocks, &t.kv_indices, &t.full_kv_num_blocks, &t.full_kv_indices,
                            &t.q_num_blocks, &t.q_indices, &t.full_q_num_blocks, &t.full_q_indices};
  c.tables.reserve(10);
  for (int i = 0; i < 8; ++i) {
    Ref a(PyObject_GetAttr(bm, s_tables[i]));
    if (a.p == nullptr) return false;
    bool none = false;
    *dst[i] = table(a.p, dev, c.tables, &none);
    if (*dst[i] == nullptr && !none) return false;
    if (i == 1) {
      if (none) return false;
      const at::Tensor& idx = c.tables.back();
      if (idx.dim() != 4) return false;
      t.mask_B = (int)idx.size(0);
      t.mask_H = (int)idx.size(1);
      t.num_q_blocks = (int)idx.size(2);
      t.num_kv_blocks = (int)idx.size(3);
    }
  }
  Ref bs(PyObject_GetAttr(bm, s_block_size));
  if (bs.p == nullptr || !PyTuple_Check(bs.p) || PyTuple_GET_SIZE(bs.p) != 2) return false;
  const long qb = PyLong_AsLong(PyTuple_GET_ITEM(bs.p, 0)), kvb = PyLong_AsLong(PyTuple_GET_ITEM(bs.p, 1));
  if (qb <= 0 || kvb <= 0 || qb > INT32_MAX || kvb > INT32_MAX) return false;
  t.q_block_size = (int)qb;
  t.kv_block_size = (int)kvb;
  Ref listed(PyObject_GetAttr(bm, s_kv_tiles));  // (a hint)
  if (listed.p == nullptr) PyErr_Clear();
  const long n_tiles = listed.p != nullptr && PyLong_Check(listed.p) ? PyLong_AsLong(listed.p) : 0;
  if (n_tiles > 0 && n_tiles <= 65535) c.p.flags |= FA_FLAG_KV_TILES((int)n_tiles);
  // the bit matrices belong to the mask_mod they were built from, and to the contents its captured tensors had then
  Ref bits(PyObject_GetAttr(bm, s_mask_bits));
  if (bits.p == nullptr) return false;
  if (bits.p == Py_None) return true;
  Ref bm_mod(PyObject_GetAttr(bm, s_mask_mod)), bits_mod(PyObject_GetAttr(bm, s_bits_mod)), src(PyObject_GetAttr(bm, s_bits_sources));
  if (bm_mod.p == nullptr || bits_mod.p == nullptr || src.p == nullptr || !PyTuple_Check(src.p)) return false;
  if (mask_mod != bm_mod.p || mask_mod != bits_mod.p) return true;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(src.p); ++i) {
    PyObject* pair = PyTuple_GET_ITEM(src.p, i);  // (tensor, version)
    if (!PyTuple_Check(pair) || !THPVariable_Check(PyTuple_GET_ITEM(pair, 0))) return true;
    const at::Tensor& s = THPVariable_Unpack(PyTuple_GET_ITEM(pair, 0));
    if ((long)s._version() != PyLong_AsLong(PyTuple_GET_ITEM(pair, 1)) || s.device() != dev) return true;
    c.sources.push_back(s);
  }
  if (!c.sources.empty()) {
    Ref snap(PyObject_GetAttr(bm, s_bits_snapshot));
    const at::Tensor* t = nullptr;
    if (snap.p == nullptr) return false;
    if (c.sources.size() > 8 || !plain_tensor(snap.p, &t) || t->device() != dev) return true;
    c.snapshot = *t;
  }
  bool none = false;
  const int32_t* b = table(bits.p, dev, c.tables, &none);
  if (b == nullptr) return false;
  const at::Tensor& mb = c.tables.back();
  if (mb.dim() != 4 || mb.size(2) < c.p.Sq || mb.size(3) * 32 < c.p.Skv || !(mb.size(0) == 1 || mb.size(0) == c.p.B) ||
      !(mb.size(1) == 1 || mb.size(1) == c.p.Hq))
    return true;
  // (a mask that reads the batch or head index: entries of other indices than the call's are none, see BlockMask._bits_at)
  Ref at(PyObject_GetAttr(bm, s_bits_at));
  if (at.p == nullptr || !PyTuple_Check(at.p) || PyTuple_GET_SIZE(at.p) != 2) return false;
  for (int i = 0; i < 2; ++i) {
    PyObject* first = PyTuple_GET_ITEM(at.p, i);
    if (first == Py_None) continue;
    const long index = PyLong_AsLong(first);
    if (index == -1 && PyErr_Occurred()) return false;
    if (mb.size(i) != (i == 0 ? c.p.B : c.p.Hq) || index != (i == 0 ? c.p.b_offset : c.p.h_offset)) return true;
  }
  t.mask_bits = (const uint32_t*)b;
  t.mask_bits_stride = mb.size(3);
  t.mask_bits_rows = (int32_t)mb.size(2);
  t.mask_bits_B = (int32_t)mb.size(0);
  t.mask_bits_H = (int32_t)mb.size(1);
  Ref bits_t(PyObject_GetAttr(bm, s_mask_bits_t));
  if (bits_t.p == nullptr) return false;
  if (bits_t.p == Py_None) return true;
  const int32_t* bt = table(bits_t.p, dev, c.tables, &none);
  if (bt == nullptr) return false;
  const at::Tensor& mt = c.tables.back();
  if (mt.dim() == 4 && mt.size(0) == t.mask_bits_B && mt.size(1) == t.mask_bits_H && mt.size(2) >= c.p.Skv && mt.size(3) * 32 >= c.p.Sq) {
    t.mask_bits_t = (const uint32_t*)bt;
    t.mask_bits_t_stride = mt.size(3);
    t.mask_bits_t_rows = (int32_t)mt.size(2);
  }
  return true;
}

// attention(q, k, v, score_mod, mask_mod, block_mask, scale, enable_gqa, return_lse, bshd, round_scores, b_offset, h_offset)
// -> out or (out, lse); None: not a call this path takes
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 13) {
    PyErr_SetString(PyExc_TypeError, "attention takes 13 arguments");
    return nullptr;
  }
  const at::Tensor *q, *k, *v;
  if (g_status == nullptr || *g_status != 0) Py_RETURN_NONE;
  if (!plain_tensor(a[0], &q) || !plain_tensor(a[1], &k) || !plain_tensor(a[2], &v) || watched()) Py_RETURN_NONE;
  // forward-mode derivatives: there is no rule for them, which torch.autograd.Function says
  if (q->_fw_grad(0).defined() || k->_fw_grad(0).defined() || v->_fw_grad(0).defined()) Py_RETURN_NONE;
  const at::ScalarType dt = q->scalar_type();
  if (k->scalar_type() != dt || v->scalar_type() != dt || k->device() != q->device() || v->device() != q->device()) Py_RETURN_NONE;
  if (dt != at::kHalf && dt != at::kBFloat16 && dt != at::kFloat) Py_RETURN_NONE;
  if (q->dim() != 4 || k->dim() != 4 || v->dim() != 4) Py_RETURN_NONE;
  if (q->stride(3) != 1 || k->stride(3) != 1 || v->stride(3) != 1) Py_RETURN_NONE;
  Call c;
  c.bshd = a[9] == Py_True;
  const int ih = c.bshd ? 2 : 1, is = c.bshd ? 1 : 2;
  fa_attn_params& p = c.p;
  memset(&p, 0, sizeof p);
  const int64_t B = q->size(0), Hq = q->size(ih), Hkv = k->size(ih), Sq = q->size(is), Skv = k->size(is), D = q->size(3), Dv = v->size(3);
  if (k->size(0) != B || v->size(0) != B || v->size(ih) != Hkv || v->size(is) != Skv || k->size(3) != D || Dv > D) Py_RETURN_NONE;
  if (B <= 0 || Hq <= 0 || Hkv <= 0 || Sq <= 0 || Skv <= 0 || Dv <= 0) Py_RETURN_NONE;
  if (B > INT32_MAX || Hq > INT32_MAX || Sq > INT32_MAX || Skv > INT32_MAX || D > INT32_MAX) Py_RETURN_NONE;
  if (a[7] == Py_True ? Hq % Hkv != 0 : Hq != Hkv) Py_RETURN_NONE;
  p.dtype = dt == at::kHalf ? FA_F16 : dt == at::kBFloat16 ? FA_BF16 : FA_F32;
  p.B = (int)B; p.Hq = (int)Hq; p.Hkv = (int)Hkv; p.Sq = (int)Sq; p.Skv = (int)Skv; p.D = (int)D; p.Dv = (int)Dv;
  if (a[6] == Py_None) {
    p.scale = (float)(1.0 / std::sqrt((double)D));
  } else {
    if (!PyFloat_Check(a[6]) && !PyLong_Check(a[6])) Py_RETURN_NONE;
    p.scale = (float)PyFloat_AsDouble(a[6]);
  }
  if (!PyLong_Check(a[11]) || !PyLong_Check(a[12])) Py_RETURN_NONE;
  p.b_offset = (int)PyLong_AsLong(a[11]);
  p.h_offset = (int)PyLong_AsLong(a[12]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  p.flags = a[10] == Py_True ? FA_FLAG_ROUND_SCORES : 0;
  const int return_lse = PyObject_IsTrue(a[8]);  // (1 and numpy.True_ too)
  if (return_lse < 0) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  p.status = (int32_t*)g_status;

  // the mods: an explicit mask_mod, or the one of the BlockMask
  PyObject* block_mask = a[5];
  Ref bm_mod(block_mask != Py_None ? PyObject_GetAttr(block_mask, s_mask_mod) : nullptr);
  if (block_mask != Py_None && bm_mod.p == nullptr) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  PyObject* mask_mod = a[4] != Py_None ? a[4] : bm_mod.p;
  if (mask_mod == Py_None) mask_mod = nullptr;
  PyObject* score_key = (a[3] == Py_None || a[3] == g_identity) ? nullptr : a[3];
  PyObject* mask_key = mask_mod == g_noop ? nullptr : mask_mod;
  const auto hit = g_mods->find({score_key, mask_key});
  if (hit == g_mods->end()) Py_RETURN_NONE;
  c.mods = hit->second;
  for (const auto& t : c.mods->buffers)
    if (t.device() != q->device()) Py_RETURN_NONE;
  if (block_mask != Py_None && !read_block_mask(block_mask, mask_mod, q->device(), c)) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }

  at::Tensor out, lse;
  const bool need_grad = at::GradMode::is_enabled() && (q->requires_grad() || k->requires_grad() || v->requires_grad());
  const at::Tensor tq = *q, tk = *k, tv = *v;
  {
    pybind11::gil_scoped_release no_gil;
    std::tie(out, lse) = forward(c, tq, tk, tv);
    if (need_grad) {
      auto node = std::shared_ptr<AttentionBackward>(new AttentionBackward(), torch::autograd::deleteNode);
      node->set_next_edges(torch::autograd::collect_next_edges(tq, tk, tv));
      node->call = std::move(c);
      node->q_ = torch::autograd::SavedVariable(tq, false);
      node->k_ = torch::autograd::SavedVariable(tk, false);
      node->v_ = torch::autograd::SavedVariable(tv, false);
      torch::autograd::set_history(out, node);
      node->out_ = torch::autograd::SavedVariable(out, true);
      node->lse_ = torch::autograd::SavedVariable(lse, false);
    }
  }
  if (!return_lse) return THPVariable_Wrap(out);
  Ref o(THPVariable_Wrap(out)), l(THPVariable_Wrap(lse));
  if (o.p == nullptr || l.p == nullptr) return nullptr;
  return PyTuple_Pack(2, o.p, l.p);
  END_HANDLE_TH_ERRORS
}

// A tensor over a part of `base`'s storage, contiguous, starting `offset` elements in.
at::Tensor part(const at::Tensor& base, int64_t offset, at::IntArrayRef sizes) {
  auto impl = c10::make_intrusive<c10::TensorImpl>(c10::Storage(base.storage()), base.key_set(), base.dtype());
  impl->set_sizes_contiguous(sizes);
  impl->set_storage_offset(offset);
  return at::Tensor(std::move(impl));
}

// The tensors of a tuple (at most 8)
std::vector<at::Tensor> tensors(PyObject* o) {
  TORCH_CHECK(PyTuple_Check(o) && PyTuple_GET_SIZE(o) <= 8, "buffers: a tuple of at most 8 tensors");
  std::vector<at::Tensor> r;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(o); ++i) {
    TORCH_CHECK(THPVariable_Check(PyTuple_GET_ITEM(o, i)), "buffers: tensors");
    r.push_back(THPVariable_Unpack(PyTuple_GET_ITEM(o, i)));
  }
  return r;
}

// build_block_mask(module handle, buffers, device, B, H, distinct_B, distinct_H, Q_LEN, KV_LEN, q_block, kv_block, b_offset,
//                  h_offset, want_bits: 0, 1 or 2 matrices) -> the eight tables, mask_bits, mask_bits_t, copy of the buffers if
//                  there are matrices
// buffers: the tensors the mask_mod captures, on the device
PyObject* build_block_mask(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 14) {
    PyErr_SetString(PyExc_TypeError, "build_block_mask takes 14 arguments");
    return nullptr;
  }
  fa_module* module = (fa_module*)PyLong_AsVoidPtr(a[0]);
  if (PyErr_Occurred()) return nullptr;
  const std::vector<at::Tensor> captured = tensors(a[1]);
  long x[12];
  for (int i = 0; i < 12; ++i) x[i] = PyLong_AsLong(a[2 + i]);
  if (PyErr_Occurred()) return nullptr;
  const c10::Device dev(c10::kCUDA, (c10::DeviceIndex)x[0]);
  const int want_bits = (int)x[11];
  fa_mask_build mb{};
  mb.B = (int)x[1]; mb.H = (int)x[2]; mb.distinct_B = (int)x[3]; mb.distinct_H = (int)x[4];
  mb.Q_LEN = (int)x[5]; mb.KV_LEN = (int)x[6]; mb.q_block = (int)x[7]; mb.kv_block = (int)x[8];
  mb.b_offset = (int)x[9]; mb.h_offset = (int)x[10];
  for (const auto& t : captured) TORCH_CHECK(t.device() == dev, "a captured tensor is on another device");
  std::vector<at::Tensor> out;
  {
    pybind11::gil_scoped_release no_gil;
    c10::cuda::OptionalCUDAGuard guard(dev);
    const int64_t B = mb.B, H = mb.H, nq = mb.Q_LEN / mb.q_block, nkv = mb.KV_LEN / mb.kv_block;
    // one allocation for the tables (16-byte aligned parts), and the class grid behind them while it is small: an allocation less, but
    // it lives as long as they do; a large one is given back at once
    constexpr size_t kScratchInTables = 64 << 10;
    const auto up = [](int64_t v) { return (v + 3) / 4 * 4; };
    const int64_t idx = up(B * H * nq * nkv), num_q = up(B * H * nq), num_kv = up(B * H * nkv);
    const size_t ws = fa_block_mask_workspace_bytes(mb.distinct_B, mb.distinct_H, mb.Q_LEN, mb.KV_LEN, mb.q_block, mb.kv_block);
    const int64_t n_tables = 4 * idx + 2 * num_q + 2 * num_kv;
    const int64_t n_scratch = (int64_t)(std::max<size_t>(ws, 16) + 3) / 4;
    const bool own_scratch = ws > kScratchInTables;
    at::Tensor base = empty({n_tables + (own_scratch ? 0 : n_scratch)}, at::kInt, dev);
    at::Tensor scratch = own_scratch ? empty({n_scratch}, at::kInt, dev) : at::Tensor();
    int64_t off = 0;
    int32_t* ptr[8];
    for (int i = 0; i < 8; ++i) {
      const bool kv_side = i < 4, is_num = i % 2 == 0;
      out.push_back(is_num ? part(base, off, {B, H, kv_side ? nq : nkv})
                           : part(base, off, {B, H, kv_side ? nq : nkv, kv_side ? nkv : nq}));
      ptr[i] = (int32_t*)out.back().mutable_data_ptr();
      off += is_num ? (kv_side ? num_q : num_kv) : idx;
    }
    mb.kv_num_blocks = ptr[0]; mb.kv_indices = ptr[1]; mb.full_kv_num_blocks = ptr[2]; mb.full_kv_indices = ptr[3];
    mb.q_num_blocks = ptr[4]; mb.q_indices = ptr[5]; mb.full_q_num_blocks = ptr[6]; mb.full_q_indices = ptr[7];
    mb.workspace = own_scratch ? (int32_t*)scratch.mutable_data_ptr() : (int32_t*)base.mutable_data_ptr() + n_tables;
    mb.workspace_bytes = ws;
    // the matrices come out of the same evaluation where the blocks are whole words, else out of one of their own
    const bool apart = want_bits && ((nq > 1 && mb.q_block % 32) || (nkv > 1 && mb.kv_block % 32));
    fa_mask_build own = mb;
    own.kv_num_blocks = nullptr;
    own.q_block = own.kv_block = 128;
    fa_mask_build& with_bits = apart ? own : mb;
    if (want_bits) {
      // (rows of whole 16 bytes: the second matrix begins at such a boundary)
      const int64_t words = fa_mask_bits_row_words(mb.KV_LEN), words_t = fa_mask_bits_row_words(mb.Q_LEN);
      const int64_t n = (int64_t)mb.distinct_B * mb.distinct_H * mb.Q_LEN * words, n_t = want_bits > 1 ? (int64_t)mb.distinct_B * mb.distinct_H * mb.KV_LEN * words_t : 0;
      at::Tensor both = empty({n + n_t}, at::kInt, dev);
      out.push_back(part(both, 0, {mb.distinct_B, mb.distinct_H, mb.Q_LEN, words}));
      with_bits.bits = (uint32_t*)out[8].mutable_data_ptr();
      if (want_bits > 1) {
        out.push_back(part(both, n, {mb.distinct_B, mb.distinct_H, mb.KV_LEN, words_t}));
        with_bits.bits_t = (uint32_t*)out[9].mutable_data_ptr();
      }
    }
    void* stream = (void*)c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    out.resize(10);
    if (want_bits && !captured.empty()) {
      const Ranges r(captured);
      out.push_back(empty({(int64_t)fa_snapshot_bytes(r.bytes, r.n)}, at::kByte, dev));
      const int rc = fa_snapshot(r.src, r.bytes, r.n, out.back().mutable_data_ptr(), stream);
      if (rc != FA_OK) raise(rc);
    }
    BuffersLock buffers(module, captured);
    int rc = buffers.rc != FA_OK ? buffers.rc : fa_block_mask_build(module, &mb, stream);
    if (rc == FA_OK && apart) rc = fa_block_mask_build(module, &own, stream);
    if (rc != FA_OK) raise(rc);
  }
  PyObject* t = PyTuple_New(11);
  if (t == nullptr) return nullptr;
  for (int i = 0; i < 11; ++i) {
    PyObject* o = i < (int)out.size() && out[i].defined() ? THPVariable_Wrap(out[i]) : Py_NewRef(Py_None);
    if (o == nullptr) {
      Py_DECREF(t);
      return nullptr;
    }
    PyTuple_SET_ITEM(t, i, o);
  }
  return t;
  END_HANDLE_TH_ERRORS
}

// register(score_mod, mask_mod, module, handle, buffers): the module of a pair of mods (None: no mod).
// The pair is known by identity; the Python layer calls forget when one of the two goes away.
PyObject* register_mods(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "register takes 5 arguments");
    return nullptr;
  }
  auto m = std::make_shared<Mods>();
  m->module = (fa_module*)PyLong_AsVoidPtr(a[3]);
  if (PyErr_Occurred()) return nullptr;
  m->buffers = tensors(a[4]);
  m->keep = Py_NewRef(a[2]);
  (*g_mods)[{a[0] == Py_None ? nullptr : a[0], a[1] == Py_None ? nullptr : a[1]}] = std::move(m);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// forget(score_id, mask_id): ids as id() gives them, 0 for no mod
PyObject* forget(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "forget takes 2 arguments");
    return nullptr;
  }
  PyObject *s = (PyObject*)PyLong_AsVoidPtr(a[0]), *m = (PyObject*)PyLong_AsVoidPtr(a[1]);
  if (PyErr_Occurred()) return nullptr;
  g_mods->erase({s, m});
  Py_RETURN_NONE;
}

// setup(status_address, identity_score_mod, noop_mask, FlaxAttnError, check_status)
PyObject* setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "setup takes 5 arguments");
    return nullptr;
  }
  g_status = (volatile int*)PyLong_AsVoidPtr(a[0]);
  if (PyErr_Occurred()) return nullptr;
  g_identity = Py_NewRef(a[1]);
  g_noop = Py_NewRef(a[2]);
  g_error = Py_NewRef(a[3]);
  g_check_status = Py_NewRef(a[4]);
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"attention", (PyCFunction)(void*)attention, METH_FASTCALL, nullptr},
    {"build_block_mask", (PyCFunction)(void*)build_block_mask, METH_FASTCALL, nullptr},
    {"register", (PyCFunction)(void*)register_mods, METH_FASTCALL, nullptr},
    {"forget", (PyCFunction)(void*)forget, METH_FASTCALL, nullptr},
    {"setup", (PyCFunction)(void*)setup, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "native host path of the attention entry points", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  g_mods = new std::unordered_map<std::pair<PyObject*, PyObject*>, ModsPtr, PairHash>();
  const char* const names[8] = {"kv_num_blocks", "kv_indices", "full_kv_num_blocks", "full_kv_indices",
                                "q_num_blocks", "q_indices", "full_q_num_blocks", "full_q_indices"};
  for (int i = 0; i < 8; ++i) s_tables[i] = PyUnicode_InternFromString(names[i]);
  s_mask_mod = PyUnicode_InternFromString("mask_mod");
  s_block_size = PyUnicode_InternFromString("BLOCK_SIZE");
  s_mask_bits = PyUnicode_InternFromString("mask_bits");
  s_mask_bits_t = PyUnicode_InternFromString("mask_bits_t");
  s_bits_mod = PyUnicode_InternFromString("_bits_mod");
  s_bits_sources = PyUnicode_InternFromString("_bits_sources");
  s_bits_snapshot = PyUnicode_InternFromString("_bits_snapshot");
  s_bits_at = PyUnicode_InternFromString("_bits_at");
  s_kv_tiles = PyUnicode_InternFromString("_kv_tiles");
  return PyModule_Create(&kModule);
}
