// The launch path of a call, in C++: argument checks, output and scratch allocation, tensor descriptors and the
// libkfa call itself, for the torch ops of op.py and mask.py. In Python (a dozen ctypes structures, half a dozen
// allocations, the dispatch of a Python custom op) a small problem's call took several times its kernels: a forward
// of 1 x 8 heads x 64 rows 67 us, now 10; forward + backward of 2 x 4 heads x 512 rows 286 us, now 90, of which about 45
// are the autograd engine's own (a step through one view takes 35); with a boolean mask of 2048 x 2048 395 us, now 110.
//
// A plain CPython extension module (`_kfa_host`), for the torch and the Python it was built with only: the build leaves
// their names in it, and _lib.host() does not load it under others. It holds no state but the addresses of the libkfa
// entry points it was given (`bind`): which library is loaded, and every policy (status word, backward mode), stays in
// Python.
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <array>
#include <initializer_list>
#include <string>
#include <tuple>

#include "../../include/kfa.h"

namespace {

struct Api {
  decltype(&kfa_last_error) last_error = nullptr;
  decltype(&kfa_fwd) fwd = nullptr;
  decltype(&kfa_bwd) bwd = nullptr;
  decltype(&kfa_bwd_fused) bwd_fused = nullptr;
  decltype(&kfa_fwd_masked) fwd_masked = nullptr;
  decltype(&kfa_bwd_masked) bwd_masked = nullptr;
  decltype(&kfa_fwd_varlen) fwd_varlen = nullptr;
  decltype(&kfa_bwd_varlen) bwd_varlen = nullptr;
  decltype(&kfa_pack_mask) pack_mask = nullptr;
  decltype(&kfa_fwd_narrow) fwd_narrow = nullptr;
  decltype(&kfa_bwd_narrow) bwd_narrow = nullptr;
  decltype(&kfa_bwd_parts_bytes) bwd_parts_bytes = nullptr;
  decltype(&kfa_bwd_parts_count) bwd_parts_count = nullptr;
  decltype(&kfa_bwd_parts) bwd_parts = nullptr;
  decltype(&kfa_varlen_zero_rows) varlen_zero_rows = nullptr;
} api;

PyObject* g_error = nullptr;  // kohakufa_b200._lib.KfaError
PyObject* g_route = nullptr;  // route(head dim, batch * heads) -> what backward() is asked for, < 0: not to be called directly

struct PyError {};  // a Python exception is set

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "expected a tensor");
    throw PyError();
  }
  return THPVariable_Unpack(o);
}
double number(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyError();
  return v;
}
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyError();
  return v;
}

struct KfaFailure {  // becomes a KfaError once the GIL is held again
  int rc;
  std::string message;
};

void check(int rc) {
  if (rc != 0) throw KfaFailure{rc, api.last_error()};  // (the message is this thread's)
}

// Allocations and launches run without the GIL: an allocation may have to wait for the device, a launch for room in the
// stream's queue, and what they wait for may need another Python thread.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  NoGil() = default;
  NoGil(const NoGil&) = delete;
  ~NoGil() { PyEval_RestoreThread(state); }
};
template <typename F>
auto released(F run) -> decltype(run()) {
  const NoGil guard;
  return run();
}

KfaTensor4 desc(const at::Tensor& t) {
  TORCH_CHECK(t.dim() == 4 && t.is_cuda(), "a 4-D CUDA tensor");
  KfaTensor4 d;
  d.ptr = t.data_ptr();
  for (int i = 0; i < 4; ++i) {
    d.shape[i] = t.size(i);
    d.stride[i] = t.stride(i);
  }
  return d;
}
// [T, H, D] packed rows as the [1, H, T, D] view the library takes
KfaTensor4 desc_packed(const at::Tensor& t) {
  TORCH_CHECK(t.dim() == 3 && t.is_cuda(), "a 3-D CUDA tensor");
  KfaTensor4 d;
  d.ptr = t.data_ptr();
  const int64_t shape[4] = {1, t.size(1), t.size(0), t.size(2)};
  const int64_t stride[4] = {t.size(0) * t.stride(0), t.stride(1), t.stride(0), t.stride(2)};
  for (int i = 0; i < 4; ++i) {
    d.shape[i] = shape[i];
    d.stride[i] = stride[i];
  }
  return d;
}

// The kernels read these as they lie in memory: an address of another device is a fault, other strides wrong offsets.
void check_lengths(const at::Tensor& cu_q, const at::Tensor& cu_k, const at::Tensor& q) {
  for (const at::Tensor* cu : {&cu_q, &cu_k})
    TORCH_CHECK_VALUE(cu->device() == q.device() && cu->scalar_type() == at::kInt && cu->is_contiguous() && cu->numel() >= 2,
                      "attention_varlen: cu_seqlens: contiguous int32 offsets on the device of q");
  TORCH_CHECK_VALUE(cu_q.numel() == cu_k.numel(), "attention_varlen: cu_seqlens of different lengths");
}
void check_device(std::initializer_list<const at::Tensor*> others, const at::Tensor& q) {
  for (const at::Tensor* t : others) TORCH_CHECK_VALUE(t->device() == q.device(), "attention: tensors on different devices");
}

int dtype_code(const at::Tensor& t) {
  if (t.scalar_type() == at::kHalf) return KFA_F16;
  if (t.scalar_type() == at::kBFloat16) return KFA_BF16;
  TORCH_CHECK_TYPE(false, "libkfa: fp16 or bf16");
}

// [B, H, S, D] view of fresh [B, S, H, D] storage
at::Tensor bshd_like(const at::Tensor& t) {
  return at::empty({t.size(0), t.size(2), t.size(1), t.size(3)}, t.options()).transpose(1, 2);
}
// the same layout for a gradient, which need not be a view
at::Tensor grad_like(const at::Tensor& t) {
  const int64_t h = t.size(1), s = t.size(2), d = t.size(3);
  return at::empty_strided(t.sizes(), {h * s * d, d, h * d, 1}, t.options());
}
at::Tensor floats(const at::Tensor& like, at::IntArrayRef shape) {
  return at::empty(shape, like.options().dtype(at::kFloat));
}
// the backward's statistics, and room for so many floats behind them (384 a tile: on a 16-byte boundary)
int64_t stats_floats(int64_t batch, int64_t heads, int64_t seq) { return batch * heads * ((seq + 127) / 128) * 384; }
at::Tensor stats_scratch(const at::Tensor& like, int64_t batch, int64_t heads, int64_t seq, int64_t more = 0) {
  return floats(like, {stats_floats(batch, heads, seq) + more});
}
void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

bool strides_ok(const at::Tensor& t) {
  const int64_t n = t.dim();
  if (t.stride(n - 1) != 1) return false;
  for (int64_t i = 0; i + 1 < n; ++i)
    if (t.size(i) > 1 && (t.stride(i) <= 0 || t.stride(i) % 8 != 0)) return false;
  return true;
}

// Whether q, k, v are what the kernels take (the conditions of op.py's _check, which raises for the rest).
// step: the head dims taken are its multiples.
bool inputs_ok(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, int64_t dims, int64_t step) {
  if (q.dim() != dims || k.dim() != dims || v.dim() != dims) return false;
  if ((q.scalar_type() != at::kHalf && q.scalar_type() != at::kBFloat16) || k.scalar_type() != q.scalar_type() ||
      v.scalar_type() != q.scalar_type())
    return false;
  if (!q.is_cuda() || k.device() != q.device() || v.device() != q.device()) return false;
  if (q.layout() != at::kStrided || k.layout() != at::kStrided || v.layout() != at::kStrided) return false;
  const int64_t d = q.size(-1), heads = q.size(1), kv_heads = k.size(1);
  if (d < step || d > 128 || d % step || k.size(-1) != d) return false;
  if (k.sizes() != v.sizes() || (dims == 4 && k.size(0) != q.size(0))) return false;
  if (q.numel() == 0 || k.numel() == 0 || kv_heads == 0 || heads % kv_heads) return false;
  return strides_ok(q) && strides_ok(k) && strides_ok(v);
}

KfaMaskWords mask_words(const at::Tensor& w) {
  TORCH_CHECK(w.dim() == 4 && w.scalar_type() == at::kInt && w.stride(3) == 1, "packed mask words");
  return {w.data_ptr<int32_t>(), w.size(0) > 1 ? w.stride(0) : 0, w.size(1) > 1 ? w.stride(1) : 0, w.stride(2)};
}
KfaMaskTiles mask_tiles(const at::Tensor& t) {
  TORCH_CHECK(t.dim() == 4 && t.scalar_type() == at::kInt && t.is_contiguous(), "mask tile table");
  return {t.data_ptr<int32_t>(), t.size(0) > 1 ? t.stride(0) : 0, t.size(1) > 1 ? t.stride(1) : 0};
}

template <typename... T>
PyObject* pack(std::tuple<T...> results) {
  return std::apply(
      [](auto&... ts) {
        PyObject* items[] = {THPVariable_Wrap(std::move(ts))...};
        PyObject* tuple = PyTuple_New(sizeof...(ts));
        for (size_t i = 0; i < sizeof...(ts); ++i) PyTuple_SET_ITEM(tuple, i, items[i]);
        return tuple;
      },
      results);
}

void need(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    throw PyError();
  }
}

using Args = PyObject* const*;

// plain(*tensors) -> bool: whether an operator on these tensors would go straight to its kernel. That is, no dispatch or
// function mode, no torch.func transform and no tracer is active, and each is a torch.Tensor (no subclass) whose address
// points to its value: batched tensors (gradients of `is_grads_batched`), pending negations and zero tensors are
// torch.Tensor too, but only the dispatcher resolves them.
bool nothing_interposed() {
  using c10::DispatchKey;
  static const c10::DispatchKeySet interposed(
      {DispatchKey::FuncTorchDynamicLayerFrontMode, DispatchKey::FuncTorchDynamicLayerBackMode, DispatchKey::Tracer});
  return !c10::impl::tls_local_dispatch_key_set().included_.has_any(interposed) &&
         c10::impl::TorchDispatchModeTLS::stack_len() == 0 && at::impl::PythonTorchFunctionTLS::stack_len() == 0;
}
bool plain_tensor(PyObject* o) {
  using c10::DispatchKey;
  static const uint64_t plain =
      c10::DispatchKeySet({DispatchKey::CPU, DispatchKey::CUDA, DispatchKey::ADInplaceOrView, DispatchKey::AutogradCPU,
                           DispatchKey::AutogradCUDA, DispatchKey::AutocastCPU, DispatchKey::AutocastCUDA})
          .raw_repr();
  return Py_TYPE(o) == reinterpret_cast<PyTypeObject*>(THPVariableClass) &&
         !(THPVariable_Unpack(o).key_set().raw_repr() & ~plain);
}
PyObject* py_plain(Args a, Py_ssize_t n) {
  if (!nothing_interposed()) Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!plain_tensor(a[i])) Py_RETURN_FALSE;
  Py_RETURN_TRUE;
}

// inputs_ok(q, k, v) -> bool: head dims that are multiples of 16
PyObject* py_inputs_ok(Args a, Py_ssize_t n) {
  need(n, 3);
  const at::Tensor &q = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]);
  return PyBool_FromLong(inputs_ok(q, k, v, q.dim() == 3 ? 3 : 4, 16));
}

bool aligned16(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

// narrow_ok(q, k, v) -> bool: [B, H, S, D], head dims that are multiples of 8, 16-byte aligned
PyObject* py_narrow_ok(Args a, Py_ssize_t n) {
  need(n, 3);
  const at::Tensor &q = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]);
  // (a tensor that does not start on 16 bytes is copied when it is widened)
  return PyBool_FromLong(inputs_ok(q, k, v, 4, 8) && aligned16(q) && aligned16(k) && aligned16(v));
}

using Two = std::tuple<at::Tensor, at::Tensor>;                // out, lse
using Three = std::tuple<at::Tensor, at::Tensor, at::Tensor>;  // dq, dk, dv

// The bodies of the calls: they hold no reference to Python and run without the GIL.

Two run_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, float scale, int block, const at::Tensor& status) {
  check_device({&k, &v, &status}, q);
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor out = bshd_like(q), lse = floats(q, {q.size(0), q.size(1), 2, q.size(2)});
  const KfaTensor4 dq = desc(q), dk = desc(k), dv = desc(v), dout = desc(out);
  const auto call = q.size(3) % 16 ? api.fwd_narrow : api.fwd;
  check(call(&dq, &dk, &dv, &dout, lse.data_ptr<float>(), scale, block, dtype_code(q), status.data_ptr<int32_t>(), stream_of(q)));
  return {std::move(out), std::move(lse)};
}

// fused: 1 the fused kernels; 3 the split ones, one CTA per tile; 0 the split ones, which share out their steps where that
// helps (kfa_bwd_parts); 2 ("auto" at the head dims of the fused ones) those, unless the split ones share out their steps
// and are faster for it
Three run_backward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, at::Tensor g,
                   const at::Tensor& lse, float scale, int block, const at::Tensor& status, int64_t fused) {
  check_device({&k, &v, &o, &g, &lse, &status}, q);
  const c10::cuda::CUDAGuard guard(q.device());
  if (q.size(3) % 16 && !aligned16(g)) g = g.clone();  // (widening copied it)
  at::Tensor dq = grad_like(q), dk = grad_like(k), dv = grad_like(v);
  const KfaTensor4 d[8] = {desc(q), desc(k), desc(v), desc(o), desc(g), desc(dq), desc(dk), desc(dv)};
  const bool parts = (fused == 0 || fused == 2) && api.bwd_parts_count(d, d + 1, fused == 2) > 1;
  const bool one = !parts && (fused == 1 || fused == 2);
  const int64_t rows = q.size(0) * q.size(1) * ((q.size(2) + 127) / 128) * 128;
  const int64_t more = parts ? api.bwd_parts_bytes(d, d + 1) / 4 : (one ? rows * ((q.size(3) + 15) / 16 * 16) : 0);
  at::Tensor scratch = stats_scratch(q, q.size(0), q.size(1), q.size(2), more);
  float *l = lse.data_ptr<float>(), *st = scratch.data_ptr<float>(), *behind = st + stats_floats(q.size(0), q.size(1), q.size(2));
  int* word = status.data_ptr<int32_t>();
  if (parts) {
    check(api.bwd_parts(d, d + 1, d + 2, d + 3, d + 4, l, st, behind, d + 5, d + 6, d + 7, scale, block, dtype_code(q), word,
                        stream_of(q)));
  } else if (one) {
    check((q.size(3) % 16 ? api.bwd_narrow : api.bwd_fused)(d, d + 1, d + 2, d + 3, d + 4, l, st, behind, d + 5, d + 6, d + 7, scale,
                                                            block, dtype_code(q), word, stream_of(q)));
  } else if (q.size(3) % 16) {
    check(api.bwd_narrow(d, d + 1, d + 2, d + 3, d + 4, l, st, nullptr, d + 5, d + 6, d + 7, scale, block, dtype_code(q), word,
                         stream_of(q)));
  } else {
    check(api.bwd(d, d + 1, d + 2, d + 3, d + 4, l, st, d + 5, d + 6, d + 7, scale, block, dtype_code(q), word, stream_of(q)));
  }
  return {std::move(dq), std::move(dk), std::move(dv)};
}

Two run_forward_masked(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& words,
                       const at::Tensor& tiles, float scale, const at::Tensor& status) {
  check_device({&k, &v, &words, &tiles, &status}, q);
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor out = bshd_like(q), lse = floats(q, {q.size(0), q.size(1), 2, q.size(2)});
  const KfaTensor4 dq = desc(q), dk = desc(k), dv = desc(v), dout = desc(out);
  const KfaMaskWords w = mask_words(words);
  const KfaMaskTiles t = mask_tiles(tiles);
  check(api.fwd_masked(&dq, &dk, &dv, &dout, lse.data_ptr<float>(), &w, &t, scale, dtype_code(q), status.data_ptr<int32_t>(),
                       stream_of(q)));
  return {std::move(out), std::move(lse)};
}

Three run_backward_masked(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& g,
                          const at::Tensor& lse, const at::Tensor& words, const at::Tensor& words_t, const at::Tensor& tiles,
                          float scale, const at::Tensor& status) {
  check_device({&k, &v, &o, &g, &lse, &words, &words_t, &tiles, &status}, q);
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor dq = grad_like(q), dk = grad_like(k), dv = grad_like(v);
  at::Tensor stats = stats_scratch(q, q.size(0), q.size(1), q.size(2));
  const KfaTensor4 d[8] = {desc(q), desc(k), desc(v), desc(o), desc(g), desc(dq), desc(dk), desc(dv)};
  const KfaMaskWords w = mask_words(words), wt = mask_words(words_t);
  const KfaMaskTiles t = mask_tiles(tiles);
  check(api.bwd_masked(d, d + 1, d + 2, d + 3, d + 4, lse.data_ptr<float>(), stats.data_ptr<float>(), d + 5, d + 6, d + 7, &w, &wt,
                       &t, scale, dtype_code(q), status.data_ptr<int32_t>(), stream_of(q)));
  return {std::move(dq), std::move(dk), std::move(dv)};
}

Two run_forward_varlen(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& cu_q,
                       const at::Tensor& cu_k, int max_q, int max_k, float scale, int block, const at::Tensor& status) {
  check_device({&k, &v, &status}, q);
  check_lengths(cu_q, cu_k, q);
  const c10::cuda::CUDAGuard guard(q.device());
  const int32_t *cq = cu_q.data_ptr<int32_t>(), *ck = cu_k.data_ptr<int32_t>();
  const int n_seqs = static_cast<int>(cu_q.numel() - 1);
  at::Tensor out = at::empty_like(q), lse = floats(q, {1, q.size(1), 2, q.size(0)});
  const KfaTensor4 dq = desc_packed(q), dk = desc_packed(k), dv = desc_packed(v), dout = desc_packed(out);
  check(api.fwd_varlen(&dq, &dk, &dv, &dout, lse.data_ptr<float>(), cq, ck, n_seqs, max_q, max_k, scale, block, dtype_code(q),
                       status.data_ptr<int32_t>(), stream_of(q)));
  // rows no CTA writes (a sequence with queries but no keys, rows outside cu_seqlens) read as "no visible key":
  // output 0, statistics 0
  check(api.varlen_zero_rows(&dout, 1, cq, ck, n_seqs, max_q, max_k, lse.data_ptr<float>(), stream_of(q)));
  return {std::move(out), std::move(lse)};
}

Three run_backward_varlen(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& g,
                          const at::Tensor& lse, const at::Tensor& cu_q, const at::Tensor& cu_k, int max_q, int max_k, float scale,
                          int block, const at::Tensor& status) {
  check_device({&k, &v, &o, &g, &lse, &status}, q);
  check_lengths(cu_q, cu_k, q);
  const c10::cuda::CUDAGuard guard(q.device());
  const int32_t *cq = cu_q.data_ptr<int32_t>(), *ck = cu_k.data_ptr<int32_t>();
  const int n_seqs = static_cast<int>(cu_q.numel() - 1);
  at::Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  at::Tensor stats = stats_scratch(q, n_seqs, q.size(1), max_q);
  const KfaTensor4 d[8] = {desc_packed(q), desc_packed(k),  desc_packed(v),  desc_packed(o),
                           desc_packed(g), desc_packed(dq), desc_packed(dk), desc_packed(dv)};
  check(api.bwd_varlen(d, d + 1, d + 2, d + 3, d + 4, lse.data_ptr<float>(), stats.data_ptr<float>(), d + 5, d + 6, d + 7, cq, ck,
                       n_seqs, max_q, max_k, scale, block, dtype_code(q), status.data_ptr<int32_t>(), stream_of(q)));
  check(api.varlen_zero_rows(d + 5, 3, cq, ck, n_seqs, max_q, max_k, nullptr, stream_of(q)));  // the other rows: zero
  return {std::move(dq), std::move(dk), std::move(dv)};
}

// forward(q, k, v, scale, block, status) -> out, lse
PyObject* py_forward(Args a, Py_ssize_t n) {
  need(n, 6);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), status = tensor(a[5]);
  const float scale = static_cast<float>(number(a[3]));
  const int block = static_cast<int>(integer(a[4]));
  return pack(released([&] { return run_forward(q, k, v, scale, block, status); }));
}

// backward(q, k, v, out, dout, lse, scale, block, status, fused) -> dq, dk, dv
PyObject* py_backward(Args a, Py_ssize_t n) {
  need(n, 10);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), o = tensor(a[3]), g = tensor(a[4]), lse = tensor(a[5]),
                   status = tensor(a[8]);
  const float scale = static_cast<float>(number(a[6]));
  const int block = static_cast<int>(integer(a[7]));
  const int64_t fused = integer(a[9]);
  return pack(released([&] { return run_backward(q, k, v, o, g, lse, scale, block, status, fused); }));
}

// forward_masked(q, k, v, words, tiles, scale, status) -> out, lse
PyObject* py_forward_masked(Args a, Py_ssize_t n) {
  need(n, 7);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), words = tensor(a[3]), tiles = tensor(a[4]),
                   status = tensor(a[6]);
  const float scale = static_cast<float>(number(a[5]));
  return pack(released([&] { return run_forward_masked(q, k, v, words, tiles, scale, status); }));
}

// backward_masked(q, k, v, out, dout, lse, words, words_t, tiles, scale, status) -> dq, dk, dv
PyObject* py_backward_masked(Args a, Py_ssize_t n) {
  need(n, 11);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), o = tensor(a[3]), g = tensor(a[4]), lse = tensor(a[5]),
                   words = tensor(a[6]), words_t = tensor(a[7]), tiles = tensor(a[8]), status = tensor(a[10]);
  const float scale = static_cast<float>(number(a[9]));
  return pack(released([&] { return run_backward_masked(q, k, v, o, g, lse, words, words_t, tiles, scale, status); }));
}

// forward_varlen(q, k, v, cu_q, cu_k, max_q, max_k, scale, block, status) -> out, lse
PyObject* py_forward_varlen(Args a, Py_ssize_t n) {
  need(n, 10);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), cu_q = tensor(a[3]), cu_k = tensor(a[4]),
                   status = tensor(a[9]);
  const int max_q = static_cast<int>(integer(a[5])), max_k = static_cast<int>(integer(a[6]));
  const float scale = static_cast<float>(number(a[7]));
  const int block = static_cast<int>(integer(a[8]));
  return pack(released([&] { return run_forward_varlen(q, k, v, cu_q, cu_k, max_q, max_k, scale, block, status); }));
}

// backward_varlen(q, k, v, out, dout, lse, cu_q, cu_k, max_q, max_k, scale, block, status) -> dq, dk, dv
PyObject* py_backward_varlen(Args a, Py_ssize_t n) {
  need(n, 13);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), o = tensor(a[3]), g = tensor(a[4]), lse = tensor(a[5]),
                   cu_q = tensor(a[6]), cu_k = tensor(a[7]), status = tensor(a[12]);
  const int max_q = static_cast<int>(integer(a[8])), max_k = static_cast<int>(integer(a[9]));
  const float scale = static_cast<float>(number(a[10]));
  const int block = static_cast<int>(integer(a[11]));
  return pack(released([&] { return run_backward_varlen(q, k, v, o, g, lse, cu_q, cu_k, max_q, max_k, scale, block, status); }));
}

// ---------------------------------------------------------------------------------------------------------------------
// Calls that autograd records. The nodes are C++ ones: a torch.autograd.Function in Python took another 30 to 40 us a
// step, on a thread of the engine that has to wait for the GIL (forward + backward of 2 x 4 x 512 rows: 118 -> 90 us with call() below).
// Saved tensors go through torch's own SavedVariable (hooks, version checks, release).
// ---------------------------------------------------------------------------------------------------------------------
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Call {  // what a node keeps beside its tensors
  double scale;
  int64_t block, max_q, max_k;
  at::Tensor status;
};

void keep(AutogradContext* ctx, const Call& c, variable_list saved) {
  ctx->save_for_backward(std::move(saved));
  ctx->saved_data["scale"] = c.scale;
  ctx->saved_data["block"] = c.block;
  ctx->saved_data["max_q"] = c.max_q;
  ctx->saved_data["max_k"] = c.max_k;
  ctx->saved_data["status"] = c.status;
}
Call kept(AutogradContext* ctx) {
  auto& d = ctx->saved_data;
  return {d["scale"].toDouble(), d["block"].toInt(), d["max_q"].toInt(), d["max_k"].toInt(), d["status"].toTensor()};
}

struct Gil {
  PyGILState_STATE state = PyGILState_Ensure();
  Gil() = default;
  Gil(const Gil&) = delete;
  ~Gil() { PyGILState_Release(state); }
};

// What Python says about a backward that is about to run: the route (see run_backward), or less than 0 where the registered op
// has to run instead: it is itself recorded, something is interposed, or a tensor is not a plain one.
int64_t backward_route(const variable_list& saved, const at::Tensor& g) {
  if (at::GradMode::is_enabled() || !nothing_interposed()) return -1;
  const Gil held;
  auto plain = [](const at::Tensor& t) {
    PyObject* o = THPVariable_Wrap(t);
    const bool yes = o && plain_tensor(o);
    Py_XDECREF(o);
    return yes;
  };
  for (const at::Tensor& t : saved)
    if (!plain(t)) return -1;
  if (!plain(g)) return -1;
  const at::Tensor& q = saved[0];
  PyObject* r = PyObject_CallFunction(g_route, "LL", static_cast<long long>(q.size(-1)),
                                      static_cast<long long>(q.dim() == 4 ? q.size(0) * q.size(1) : 0));
  const long long route = r ? PyLong_AsLongLong(r) : -1;
  Py_XDECREF(r);
  if (PyErr_Occurred()) {
    python_error e;
    e.persist();
    throw e;
  }
  return route;
}

// A libkfa error on a thread of the engine: the exception that Python sees is the same as from a direct call.
template <typename F>
auto in_engine(F run) -> decltype(run()) {
  try {
    return run();
  } catch (const KfaFailure& f) {
    const Gil held;
    PyErr_Format(g_error ? g_error : PyExc_RuntimeError, "libkfa error %d: %s", f.rc, f.message.c_str());
    python_error e;
    e.persist();
    throw e;
  }
}

template <typename... T>
Three registered(const char* name, const T&... args) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").template typed<Three(T...)>().call(args...);
}

// e.g. an expanded gradient; while a compiler traces with symbolic sizes there are no strides to look at
at::Tensor usable(const at::Tensor& g) {
  return !g.unsafeGetTensorImpl()->has_symbolic_sizes_strides() && strides_ok(g) ? g : g.contiguous();
}

// The nodes are traceable (is_traceable): compiled autograd then puts the registered op, which is what a backward takes under
// its dispatch modes, into its graph, where it would otherwise break the graph at the node (an error with fullgraph=True).
struct Attention : torch::autograd::Function<Attention> {
  static constexpr bool is_traceable = true;
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const Call& c) {
    auto [out, lse] = released([&] { return run_forward(q, k, v, static_cast<float>(c.scale), static_cast<int>(c.block), c.status); });
    keep(ctx, c, {q, k, v, out, lse});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Call c = kept(ctx);
    const at::Tensor g = usable(grads[0]);
    const int64_t route = backward_route(s, g);
    auto [dq, dk, dv] =
        route < 0 ? registered<at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, double, int64_t>(
                        "kohakufa_b200::sm100_backward", s[0], s[1], s[2], s[3], g, s[4], c.scale, c.block)
                  : in_engine([&] {
                      return run_backward(s[0], s[1], s[2], s[3], g, s[4], static_cast<float>(c.scale), static_cast<int>(c.block),
                                          c.status, route);
                    });
    return {dq, dk, dv, at::Tensor()};
  }
};

struct MaskedAttention : torch::autograd::Function<MaskedAttention> {
  static constexpr bool is_traceable = true;
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                            const std::array<at::Tensor, 3>& mask, const Call& c) {
    auto [out, lse] = released([&] { return run_forward_masked(q, k, v, mask[0], mask[2], static_cast<float>(c.scale), c.status); });
    keep(ctx, c, {q, k, v, out, lse, mask[0], mask[1], mask[2]});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Call c = kept(ctx);
    const at::Tensor g = usable(grads[0]);
    auto [dq, dk, dv] =
        backward_route(s, g) < 0
            ? registered<at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor,
                         double>("kohakufa_b200::sm100_masked_backward", s[0], s[1], s[2], s[3], g, s[4], s[5], s[6], s[7], c.scale)
            : in_engine([&] {
                return run_backward_masked(s[0], s[1], s[2], s[3], g, s[4], s[5], s[6], s[7], static_cast<float>(c.scale), c.status);
              });
    return {dq, dk, dv, at::Tensor(), at::Tensor()};
  }
};

struct VarlenAttention : torch::autograd::Function<VarlenAttention> {
  static constexpr bool is_traceable = true;
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                            const std::array<at::Tensor, 2>& cu, const Call& c) {
    auto [out, lse] = released([&] {
      return run_forward_varlen(q, k, v, cu[0], cu[1], static_cast<int>(c.max_q), static_cast<int>(c.max_k),
                                static_cast<float>(c.scale), static_cast<int>(c.block), c.status);
    });
    keep(ctx, c, {q, k, v, out, lse, cu[0], cu[1]});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Call c = kept(ctx);
    const at::Tensor g = grads[0].contiguous();
    auto [dq, dk, dv] =
        backward_route(s, g) < 0
            ? registered<at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, int64_t,
                         int64_t, double, int64_t>("kohakufa_b200::sm100_varlen_backward", s[0], s[1], s[2], s[3], g, s[4], s[5],
                                                   s[6], c.max_q, c.max_k, c.scale, c.block)
            : in_engine([&] {
                return run_backward_varlen(s[0], s[1], s[2], s[3], g, s[4], s[5], s[6], static_cast<int>(c.max_q),
                                           static_cast<int>(c.max_k), static_cast<float>(c.scale), static_cast<int>(c.block), c.status);
              });
    return {dq, dk, dv, at::Tensor(), at::Tensor()};
  }
};

// attention(q, k, v, scale, block, status) -> out, with its gradient where autograd records
PyObject* py_attention(Args a, Py_ssize_t n) {
  need(n, 6);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]);
  const Call c{number(a[3]), integer(a[4]), 0, 0, tensor(a[5])};
  return THPVariable_Wrap(Attention::apply(q, k, v, c));
}
// call(q, k, v, scale, block, status) -> out, or None for [B, H, S, D] inputs that the kernels do not take as they are: the
// checks of the inputs, whether autograd records, and the call in one go.
PyObject* py_call(Args a, Py_ssize_t n) {
  need(n, 6);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]);
  if (!inputs_ok(q, k, v, 4, 16)) Py_RETURN_NONE;
  const Call c{number(a[3]), integer(a[4]), 0, 0, tensor(a[5])};
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad()))
    return THPVariable_Wrap(Attention::apply(q, k, v, c));
  return THPVariable_Wrap(std::get<0>(
      released([&] { return run_forward(q, k, v, static_cast<float>(c.scale), static_cast<int>(c.block), c.status); })));
}
// attention_masked(q, k, v, words, words_t, tiles, scale, status) -> out
PyObject* py_attention_masked(Args a, Py_ssize_t n) {
  need(n, 8);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]);
  const std::array<at::Tensor, 3> mask{tensor(a[3]), tensor(a[4]), tensor(a[5])};
  const Call c{number(a[6]), 0, 0, 0, tensor(a[7])};
  return THPVariable_Wrap(MaskedAttention::apply(q, k, v, mask, c));
}
// attention_varlen(q, k, v, cu_q, cu_k, max_q, max_k, scale, block, status) -> out
PyObject* py_attention_varlen(Args a, Py_ssize_t n) {
  need(n, 10);
  const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]);
  const std::array<at::Tensor, 2> cu{tensor(a[3]), tensor(a[4])};
  const Call c{number(a[7]), integer(a[8]), integer(a[5]), integer(a[6]), tensor(a[9])};
  return THPVariable_Wrap(VarlenAttention::apply(q, k, v, cu, c));
}

// pack_mask(mask [Bm, Hm, Sq, Skv] bool or bytes, any strides, s_q, s_kv) -> words, words_t, tiles
PyObject* py_pack_mask(Args a, Py_ssize_t n) {
  need(n, 3);
  const at::Tensor m = tensor(a[0]);
  const int64_t s_q = integer(a[1]), s_kv = integer(a[2]);
  return pack(released([&] {
    TORCH_CHECK(m.dim() == 4 && m.is_cuda() && m.element_size() == 1, "a 4-D mask of bytes on the GPU");
    const c10::cuda::CUDAGuard guard(m.device());
    const int64_t bm = m.size(0), hm = m.size(1), tq = (s_q + 127) / 128, tk = (s_kv + 127) / 128;
    const auto ints = m.options().dtype(at::kInt);
    at::Tensor words = at::empty({bm, hm, s_q, 4 * tk}, ints), words_t = at::empty({bm, hm, s_kv, 4 * tq}, ints);
    at::Tensor tiles = at::empty({bm, hm, tq, tk}, ints);
    const int64_t strides[4] = {m.stride(0), m.stride(1), m.stride(2), m.stride(3)};
    check(api.pack_mask(m.data_ptr(), strides, static_cast<int>(bm), static_cast<int>(hm), static_cast<int>(s_q),
                        static_cast<int>(s_kv), words.data_ptr<int32_t>(), words_t.data_ptr<int32_t>(),
                        tiles.data_ptr<int32_t>(), stream_of(m)));
    return std::make_tuple(std::move(words), std::move(words_t), std::move(tiles));
  }));
}

// bind(KfaError, {entry point: address}, route)
PyObject* py_bind(Args a, Py_ssize_t n) {
  need(n, 3);
  auto take = [&](const char* name, auto& slot) {
    PyObject* v = PyDict_GetItemString(a[1], name);
    if (!v) {
      PyErr_Format(PyExc_KeyError, "%s", name);
      throw PyError();
    }
    slot = reinterpret_cast<std::remove_reference_t<decltype(slot)>>(static_cast<uintptr_t>(integer(v)));
  };
  take("kfa_last_error", api.last_error);
  take("kfa_fwd", api.fwd);
  take("kfa_bwd", api.bwd);
  take("kfa_bwd_fused", api.bwd_fused);
  take("kfa_fwd_masked", api.fwd_masked);
  take("kfa_bwd_masked", api.bwd_masked);
  take("kfa_fwd_varlen", api.fwd_varlen);
  take("kfa_bwd_varlen", api.bwd_varlen);
  take("kfa_pack_mask", api.pack_mask);
  take("kfa_fwd_narrow", api.fwd_narrow);
  take("kfa_bwd_narrow", api.bwd_narrow);
  take("kfa_bwd_parts_bytes", api.bwd_parts_bytes);
  take("kfa_bwd_parts_count", api.bwd_parts_count);
  take("kfa_bwd_parts", api.bwd_parts);
  take("kfa_varlen_zero_rows", api.varlen_zero_rows);
  Py_INCREF(a[0]);
  Py_XDECREF(g_error);
  g_error = a[0];
  Py_INCREF(a[2]);
  Py_XDECREF(g_route);
  g_route = a[2];
  Py_RETURN_NONE;
}

// C++ exceptions end here: torch's become the Python exceptions they stand for.
template <PyObject* (*F)(Args, Py_ssize_t)>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    return F(args, n);
  } catch (const PyError&) {
    return nullptr;
  } catch (const KfaFailure& e) {
    PyErr_Format(g_error ? g_error : PyExc_RuntimeError, "libkfa error %d: %s", e.rc, e.message.c_str());
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define KFA_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(entry<py_##name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    KFA_METHOD(bind),
    KFA_METHOD(plain),
    KFA_METHOD(inputs_ok),
    KFA_METHOD(narrow_ok),
    KFA_METHOD(forward),
    KFA_METHOD(backward),
    KFA_METHOD(forward_masked),
    KFA_METHOD(backward_masked),
    KFA_METHOD(forward_varlen),
    KFA_METHOD(backward_varlen),
    KFA_METHOD(attention),
    KFA_METHOD(call),
    KFA_METHOD(attention_masked),
    KFA_METHOD(attention_varlen),
    KFA_METHOD(pack_mask),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_kfa_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__kfa_host(void) {
  PyObject* m = PyModule_Create(&module_def);
  if (m && PyModule_AddStringConstant(m, "built_for", KFA_HOST_STAMP) < 0) Py_CLEAR(m);
  return m;
}
