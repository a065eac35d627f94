// Host path of the operators as a CPython extension over libflyb200: one call from Python checks the tensors,
// allocates the outputs and launches, where the same steps as Python statements and ctypes calls took longer
// than the kernels of a small layer.  Nothing is kept between calls.
//
// Every function takes only the common form of its arguments.  For anything else it launches nothing and
// returns None: the caller's Python statements then take the call, or raise what they raise.  A library
// error comes back as its code (int).
//
// Host time of a pass, us, Python and ctypes / this (outputs allocated, launches included): per-token quantiser 16.2 / 5.3,
// linear layer 31.6 / 17.6, block-scaled layers MXFP8 46.0 / 22.6, MXFP4 43.8 / 22.2, MXFP6 66.3 / 27.4, mixture-of-experts
// layer 109.9 / 31.4, its stages called one by one 85.3 / 43.9.
#include "../../include/flyb200.h"

#include <ATen/ATen.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <initializer_list>

namespace {

// Arguments of a vectorcall: tensors and integers by position; `ok` goes false on anything unexpected.
struct Args {
  PyObject* const* v;
  Py_ssize_t n;
  Py_ssize_t i = 0;
  bool ok = true;
  const at::Tensor none;
  const at::Tensor& tensor() {
    if (i >= n || !THPVariable_Check(v[i])) {
      ++i;
      ok = false;
      return none;
    }
    return THPVariable_Unpack(v[i++]);
  }
  const at::Tensor& tensor_or_none() {
    if (i < n && v[i] == Py_None) {
      ++i;
      return none;
    }
    return tensor();
  }
  long long integer() {
    const long long x = i < n ? PyLong_AsLongLong(v[i]) : -1;
    ++i;
    if (x == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      ok = false;
    }
    return x;
  }
  int i32() {
    const long long x = integer();
    if (x < INT_MIN || x > INT_MAX) ok = false;
    return static_cast<int>(x);
  }
  bool done() const { return ok && i == n; }
};

// Launches may block on a full queue: other Python threads run meanwhile.
struct NoGil {
  PyThreadState* st = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(st); }
};

PyObject* none() { Py_RETURN_NONE; }
PyObject* code(int rc) { return PyLong_FromLong(rc); }
PyObject* tuple(std::initializer_list<at::Tensor> ts) {
  PyObject* t = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  if (!t) return nullptr;
  Py_ssize_t i = 0;
  for (const at::Tensor& x : ts) {
    PyObject* o = x.defined() ? THPVariable_Wrap(x) : (Py_INCREF(Py_None), Py_None);
    if (!o) {
      Py_DECREF(t);
      return nullptr;
    }
    PyTuple_SET_ITEM(t, i++, o);
  }
  return t;
}

bool plain(const at::Tensor& t) { return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous(); }
bool bytes(const at::Tensor& t, long long n) { return plain(t) && t.element_size() == 1 && t.numel() >= n; }
bool floats(const at::Tensor& t, long long n) { return plain(t) && t.scalar_type() == at::kFloat && t.numel() >= n; }
bool at16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
template <typename T>
T* as(const at::Tensor& t) {
  return static_cast<T*>(ptr(t));
}
void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
// Whether a kernel may stand for torch operations on the tensor `o`: a plain tensor (no subclass, fake,
// functionalised, functorch-wrapped, lazily negated or conjugated one), with no dispatch mode, trace or transform
// in force that has to see the operations.  `differentiable`: nor a gradient that they would carry.
bool runs_eagerly(PyObject* o, bool differentiable) {
  using K = c10::DispatchKey;
  constexpr c10::DispatchKeySet wrapped({K::Python, K::PythonTLSSnapshot, K::Functionalize, K::Negative, K::Conjugate, K::ZeroTensor,
                                         K::FuncTorchBatched, K::FuncTorchGradWrapper, K::BatchedNestedTensor, K::Batched});
  constexpr c10::DispatchKeySet watching({K::Python, K::PythonTLSSnapshot, K::Functionalize, K::FuncTorchDynamicLayerFrontMode,
                                          K::FuncTorchVmapMode, K::VmapMode, K::Tracer, K::PreDispatch, K::PythonDispatcher});
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (t.key_set().has_any(wrapped) || c10::impl::tls_local_dispatch_key_set().included_.has_any(watching)) return false;
  return !differentiable || !((c10::GradMode::is_enabled() && t.requires_grad()) || t._fw_grad(0).defined());
}
void* handle(long long s) { return reinterpret_cast<void*>(static_cast<uintptr_t>(s)); }
int input_code(const at::Tensor& x) {
  switch (x.scalar_type()) {
    case at::kFloat: return 0;
    case at::kHalf: return 1;
    case at::kBFloat16: return 2;
    default: return -1;
  }
}

// pertoken_quant(x, quant_dtype) -> (codes, scales)
PyObject* pertoken_quant(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const at::Tensor& x = a.tensor();
  const int qd = a.i32();
  if (!a.done() || (qd != FLYB200_DT_FP8 && qd != FLYB200_DT_INT8) || !plain(x) || x.dim() < 1) return none();
  const int in = input_code(x);
  const long long k = x.size(-1);
  if (in < 0 || k <= 0 || k % (in == 0 ? 4 : 8) != 0 || x.numel() >= (1ll << 31) || !at16(ptr(x))) return none();
  at::Tensor y, s;
  int rc;
  {
    NoGil g;
    const c10::cuda::CUDAGuard dev(x.device());
    y = at::empty(x.sizes(), x.options().dtype(qd == FLYB200_DT_FP8 ? at::kFloat8_e4m3fn : at::kChar));
    c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = 1;
    s = at::empty(shape, x.options().dtype(at::kFloat));
    rc = flyb200_pertoken_quant(ptr(y), as<float>(s), ptr(x), static_cast<int>(x.numel() / k), static_cast<int>(k), in, qd, stream_of(x));
  }
  return rc ? code(rc) : tuple({y, s});
  END_HANDLE_TH_ERRORS
}

// gemm_a8w8(c, a, b, scale_a | None, scale_b | None, bias | None, M, N, K, in, out, epilogue, hint, ws, ws_bytes, stream) -> code.
// No checks: the compiled launcher's, on the arguments it was compiled for.
PyObject* gemm_a8w8(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const at::Tensor &c = a.tensor(), &x = a.tensor(), &w = a.tensor(), &sa = a.tensor_or_none(), &sb = a.tensor_or_none(), &bias = a.tensor_or_none();
  const int M = a.i32(), N = a.i32(), K = a.i32(), in = a.i32(), out = a.i32(), epi = a.i32(), hint = a.i32();
  const long long ws = a.integer(), ws_bytes = a.integer(), s = a.integer();
  if (!a.done()) return none();
  void *cp = ptr(c), *xp = ptr(x), *wp = ptr(w);
  const float *sap = as<float>(sa), *sbp = as<float>(sb);
  const void* bp = ptr(bias);
  int rc;
  {
    NoGil g;
    rc = flyb200_gemm_a8w8(cp, xp, wp, sap, sbp, bp, M, N, K, in, out, epi, hint, handle(ws), static_cast<size_t>(ws_bytes), handle(s));
  }
  return code(rc);
  END_HANDLE_TH_ERRORS
}

// eager(x) -> bool
PyObject* eager(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return PyBool_FromLong(n == 1 && runs_eagerly(argv[0], false));
  END_HANDLE_TH_ERRORS
}

// mx_quant(x, format) -> (codes, scales, raw | None), shaped like x.  Only E4M3 codes are differentiable as torch
// operations; the others come out of integer arithmetic.
PyObject* mx_quant(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const at::Tensor& arg = a.tensor();
  const int fmt = a.i32();
  if (!a.done() || !runs_eagerly(argv[0], fmt == FLYB200_MXFMT_E4M3) || !arg.is_cuda() || arg.layout() != at::kStrided || arg.dim() < 1 || arg.numel() == 0 || arg.size(-1) % 32 != 0) return none();
  const int in = input_code(arg);
  if (in < 0 || (fmt != FLYB200_MXFMT_E4M3 && fmt != FLYB200_MXFMT_E2M3 && fmt != FLYB200_MXFMT_E2M1)) return none();
  at::Tensor x, codes, scale, raw;
  int rc;
  {
    NoGil g;
    const c10::cuda::CUDAGuard dev(arg.device());
    x = arg.contiguous();
    if (!at16(ptr(x))) {
      rc = -1;
    } else {
      const at::TensorOptions u8 = x.options().dtype(at::kByte);
      c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
      const int64_t k = shape.back();
      if (fmt == FLYB200_MXFMT_E2M1) shape.back() = k / 2;
      codes = at::empty(shape, fmt == FLYB200_MXFMT_E4M3 ? x.options().dtype(at::kFloat8_e4m3fn) : u8);
      shape.back() = k / 32;
      scale = at::empty(shape, u8);
      if (fmt == FLYB200_MXFMT_E2M3) raw = at::empty(x.sizes(), u8);
      rc = flyb200_mx_quant(ptr(codes), ptr(scale), ptr(raw), ptr(x), x.numel(), in, fmt, stream_of(x));
    }
  }
  if (rc < 0) return none();
  return rc ? code(rc) : tuple({codes, scale, raw});
  END_HANDLE_TH_ERRORS
}

// mx_scale_image(scale) -> image
PyObject* mx_scale_image(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const at::Tensor& arg = a.tensor();
  if (!a.done() || !arg.is_cuda() || arg.layout() != at::kStrided || arg.dim() != 2 || arg.element_size() != 1 || arg.size(1) % 4 != 0 ||
      arg.numel() == 0 || arg.numel() >= (1ll << 26))
    return none();
  const int rows = static_cast<int>(arg.size(0)), K = static_cast<int>(arg.size(1)) * 32;
  at::Tensor out;
  int rc;
  {
    NoGil g;
    const c10::cuda::CUDAGuard dev(arg.device());
    const at::Tensor src = arg.contiguous();
    out = at::empty({static_cast<int64_t>(flyb200_mx_scale_image_bytes(rows, K))}, src.options().dtype(at::kByte));
    rc = flyb200_mx_scale_image(ptr(out), ptr(src), rows, K, stream_of(src));
  }
  return rc ? code(rc) : THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// mx_gemm(a_format, w_format, c, a, b, scale_a, scale_b, M, N, K, out, stream) -> code.  Formats E4M3 x E4M3 and
// E2M1 x E2M1 (packed) are kinds of their own, the rest is mixed; E2M3 activations go through their byte containers.
PyObject* mx_gemm(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const int fa = a.i32(), fw = a.i32();
  const at::Tensor &c = a.tensor(), &x = a.tensor(), &w = a.tensor(), &sa = a.tensor(), &sb = a.tensor();
  const int M = a.i32(), N = a.i32(), K = a.i32(), out = a.i32();
  const long long s = a.integer();
  if (!a.done() || M <= 0 || N <= 0 || K <= 0) return none();
  const bool fp8 = fa == FLYB200_MXFMT_E4M3 && fw == FLYB200_MXFMT_E4M3, fp4 = fa == FLYB200_MXFMT_E2M1 && fw == FLYB200_MXFMT_E2M1;
  const long long per = fp4 ? 2 : 1, m = M, nn = N, k = K;
  if (!plain(c) || c.numel() < m * nn || c.scalar_type() != (out == FLYB200_OUT_FP16 ? at::kHalf : at::kBFloat16)) return none();
  if (!bytes(x, m * k / per) || !bytes(w, nn * k / per) || (!fp8 && !fp4 && w.numel() != nn * k)) return none();
  if (!bytes(sa, static_cast<long long>(flyb200_mx_scale_image_bytes(M, K))) || !bytes(sb, static_cast<long long>(flyb200_mx_scale_image_bytes(N, K))))
    return none();
  void *cp = ptr(c), *xp = ptr(x), *wp = ptr(w), *sap = ptr(sa), *sbp = ptr(sb);
  int rc = 0;
  {
    NoGil g;
    const c10::cuda::CUDAGuard dev(c.device());
    at::Tensor containers;  // in the memory pool of the launch stream, which has to be the current one
    if (fa == FLYB200_MXFMT_E2M3) {
      if (stream_of(x) != handle(s) || x.device() != c.device() || !at16(xp)) {
        rc = -1;
      } else {
        containers = at::empty({m, k}, x.options().dtype(at::kByte));
        rc = flyb200_mx_fp6_containers(ptr(containers), xp, m * k, handle(s));
        xp = ptr(containers);
      }
    }
    if (rc == 0)
      rc = fp8   ? flyb200_gemm_mxfp8(cp, xp, wp, sap, sbp, M, N, K, out, handle(s))
           : fp4 ? flyb200_gemm_mxfp4(cp, xp, wp, sap, sbp, M, N, K, out, handle(s))
                 : flyb200_gemm_mx_mixed(cp, xp, wp, sap, sbp, M, N, K, fa, fw, out, handle(s));
  }
  return rc < 0 ? none() : code(rc);
  END_HANDLE_TH_ERRORS
}

// Routing table of the experts [first, first + experts); false where the ids or weights are not of the common form.
struct Routing {
  at::Tensor ids, weights, experts, valid;
  int blocks = 0;
};
bool routing_takes(const at::Tensor& ids, const at::Tensor& wts, long long experts, long long block) {
  if (!ids.defined() || !wts.defined() || !ids.is_cuda() || ids.layout() != at::kStrided || ids.dim() != 2 || ids.numel() == 0) return false;
  if (wts.device() != ids.device() || wts.layout() != at::kStrided || wts.numel() != ids.numel() || experts <= 0 || block <= 0) return false;
  return ids.numel() + experts * block < (1ll << 31);
}
// Sorted rows that the table has room for, and the blocks that cover them.
int64_t routing_rows(int64_t pairs, int64_t topk, int64_t experts, int64_t block) { return pairs + experts * block - topk; }
int routing_blocks(int64_t pairs, int64_t topk, int64_t experts, int64_t block) {
  return static_cast<int>((routing_rows(pairs, topk, experts, block) + block - 1) / block);
}
int sort_routes(const at::Tensor& topk_ids, const at::Tensor& topk_weights, int experts, int block, long long first, void* s, Routing& r) {
  const at::ScalarType t = topk_ids.scalar_type();
  const at::Tensor ids = (t == at::kInt || t == at::kLong ? topk_ids : topk_ids.to(at::kInt)).contiguous();
  const at::Tensor w = topk_weights.to(at::kFloat).contiguous();
  const int tokens = static_cast<int>(ids.size(0)), topk = static_cast<int>(ids.size(1));
  const int64_t padded = routing_rows(ids.numel(), topk, experts, block);
  r.blocks = routing_blocks(ids.numel(), topk, experts, block);
  const at::TensorOptions i32 = ids.options().dtype(at::kInt);
  r.ids = at::empty({padded}, i32);
  r.weights = at::empty({padded}, ids.options().dtype(at::kFloat));
  r.experts = at::empty({r.blocks}, i32);
  r.valid = at::empty({2}, i32);
  return flyb200_moe_sorting_range(ptr(ids), static_cast<int>(ids.element_size()), as<float>(w), tokens, topk, experts, first, block,
                                   as<int>(r.ids), as<float>(r.weights), as<int>(r.experts), as<int>(r.valid), s);
}

// moe_sort(topk_ids, topk_weights, experts, block, first_expert) -> (ids, weights, experts, valid)
PyObject* moe_sort(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const at::Tensor &ids = a.tensor(), &wts = a.tensor();
  const int experts = a.i32(), block = a.i32();
  const long long first = a.integer();
  if (!a.done() || !routing_takes(ids, wts, experts, block)) return none();
  Routing r;
  int rc;
  {
    NoGil g;
    const c10::cuda::CUDAGuard dev(ids.device());
    rc = sort_routes(ids, wts, experts, block, first, stream_of(ids), r);
  }
  return rc ? code(rc) : tuple({r.ids, r.weights, r.experts, r.valid});
  END_HANDLE_TH_ERRORS
}

// moe_stage(out, x, w, scale_x, scale_w, ids, experts, weights | None, valid, a_sorted, sa_sorted, stage, tokens, topk, gather, k,
//           n_experts, model, inter, tile_m, blocks, in, out, doweight, accumulate, stream, all_experts) -> code: gather pass and
// grouped GEMM.  No checks: the launcher's own, or the compiled launcher's.
PyObject* moe_stage(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const at::Tensor &out = a.tensor(), &x = a.tensor(), &w = a.tensor(), &sx = a.tensor(), &sw = a.tensor(), &ids = a.tensor(),
                   &eids = a.tensor(), &wts = a.tensor_or_none(), &valid = a.tensor(), &a_s = a.tensor(), &sa_s = a.tensor();
  const int stage = a.i32(), tokens = a.i32(), topk = a.i32(), gather = a.i32(), k = a.i32(), experts = a.i32(), model = a.i32(),
            inter = a.i32(), tile_m = a.i32(), blocks = a.i32(), in = a.i32(), out_t = a.i32(), dow = a.i32(), acc = a.i32();
  const long long s = a.integer();
  const int all = a.i32();
  if (!a.done()) return none();
  void *op = ptr(out), *xp = ptr(x), *wp = ptr(w);
  const float *sxp = as<float>(sx), *swp = as<float>(sw), *tp = wts.defined() && wts.numel() ? as<float>(wts) : nullptr;
  const int *ip = as<int>(ids), *ep = as<int>(eids), *vp = as<int>(valid);
  int rc;
  {
    NoGil g;
    rc = flyb200_moe_gather_rows(ptr(a_s), as<float>(sa_s), xp, sxp, ip, vp, tokens, topk, gather, k, blocks * tile_m, handle(s));
    if (!rc)
      rc = flyb200_moe_gemm_shard(stage, op, ptr(a_s), wp, as<float>(sa_s), swp, ip, ep, tp, vp, tokens, topk, experts, all, model, inter,
                                  tile_m, blocks, in, out_t, dow, acc, 1, handle(s));
  }
  return code(rc);
  END_HANDLE_TH_ERRORS
}

// moe_layer(x, scale_x, topk_ids, topk_weights, w1, scale_w1, w2, scale_w2, mask, a1, sa1, a2, sa2, experts, first, all_experts,
//           model, inter, topk, tile_m, in) -> output [tokens, model] bf16.  Routing table, stage 1, quantiser, stage 2 (a row per
// route) and the masked top-k sum on the current stream; a1 ... sa2 is the scratch of the two stages.
PyObject* moe_layer(PyObject*, PyObject* const* argv, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{argv, n};
  const at::Tensor &x = a.tensor(), &sx = a.tensor(), &ids = a.tensor(), &wts = a.tensor(), &w1 = a.tensor(), &sw1 = a.tensor(),
                   &w2 = a.tensor(), &sw2 = a.tensor(), &mask = a.tensor(), &a1 = a.tensor(), &sa1 = a.tensor(), &a2 = a.tensor(),
                   &sa2 = a.tensor();
  const int experts = a.i32();
  const long long first = a.integer();
  const int all = a.i32(), model = a.i32(), inter = a.i32(), topk = a.i32(), tile_m = a.i32(), in = a.i32();
  if (!a.done() || !plain(x) || x.dim() != 2 || x.size(0) <= 0 || inter > FLYB200_MOE_QUANT_MAX_K) return none();
  const long long tokens = x.size(0), m = model, i = inter, e = experts;
  if (tokens >= (1 << 24) || !bytes(x, tokens * m) || !floats(sx, tokens) || !routing_takes(ids, wts, experts, tile_m)) return none();
  if (ids.size(0) != tokens || ids.size(1) != topk || ids.device() != x.device() || sx.device() != x.device()) return none();
  if (!bytes(w1, e * 2 * i * m) || !bytes(w2, e * m * i) || !floats(sw1, e * 2 * i) || !floats(sw2, e * m)) return none();
  for (const at::Tensor* t : {&w1, &w2, &sw1, &sw2, &mask, &a1, &sa1, &a2, &sa2})
    if (t->device() != x.device()) return none();
  const long long rows = static_cast<long long>(routing_blocks(ids.numel(), topk, experts, tile_m)) * tile_m;
  if (!bytes(a1, rows * m) || !bytes(a2, rows * i) || !floats(sa1, rows) || !floats(sa2, rows)) return none();
  at::Tensor y;
  int rc;
  {
    NoGil g;
    const c10::cuda::CUDAGuard dev(x.device());
    void* s = stream_of(x);
    Routing r;
    rc = sort_routes(ids, wts, experts, tile_m, first, s, r);
    if (!rc) {
      const int t = static_cast<int>(tokens), rn = static_cast<int>(rows);
      const int *ip = as<int>(r.ids), *ep = as<int>(r.experts), *vp = as<int>(r.valid);
      const float* tp = as<float>(r.weights);
      const at::TensorOptions bf16 = x.options().dtype(at::kBFloat16);
      // rows of routes that belong to other ranks are neither written nor read
      const at::Tensor out1 = at::empty({tokens * topk, i}, bf16);
      rc = flyb200_moe_gather_rows(ptr(a1), as<float>(sa1), ptr(x), as<float>(sx), ip, vp, t, topk, 0, model, rn, s);
      if (!rc)
        rc = flyb200_moe_gemm_shard(1, ptr(out1), ptr(a1), ptr(w1), as<float>(sa1), as<float>(sw1), ip, ep, tp, vp, t, topk, experts,
                                    all, model, inter, tile_m, r.blocks, in, FLYB200_OUT_BF16, 0, 0, 1, s);
      if (!rc) rc = flyb200_moe_quant_sorted(ptr(a2), as<float>(sa2), ptr(out1), ip, vp, t, topk, inter, rn, in, s);
      const at::Tensor out2 = at::empty({tokens * topk, m}, bf16);
      if (!rc)
        rc = flyb200_moe_gemm_shard(2, ptr(out2), ptr(a2), ptr(w2), as<float>(sa2), as<float>(sw2), ip, ep, tp, vp, t, topk, experts,
                                    all, model, inter, tile_m, r.blocks, in, FLYB200_OUT_BF16, 1, 0, 1, s);
      const at::Tensor ids32 = ids.to(at::kInt).contiguous();
      y = at::empty({tokens, m}, bf16);
      if (!rc) rc = flyb200_moe_reduce(ptr(y), ptr(out2), t, topk, model, FLYB200_OUT_BF16, as<int>(mask), as<int>(ids32), all, s);
    }
  }
  return rc ? code(rc) : THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(pertoken_quant), FAST(gemm_a8w8), FAST(eager), FAST(mx_quant), FAST(mx_scale_image), FAST(mx_gemm),
                         FAST(moe_sort),       FAST(moe_stage), FAST(moe_layer), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "flyb200_ops", "Host path of the operators.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_flyb200_ops() { return PyModule_Create(&module); }
