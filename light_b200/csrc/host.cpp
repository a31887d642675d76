// The common form of the hot operators as one call from Python into native code: checks, output allocation, current
// stream, C-ABI call.  A decode step's kernels run for 5 to 20 us; the same work in Python (ctypes argument boxing, tensor
// attribute look-ups, torch.empty) costs 12 to 20 us per operator and leaves the GPU idle between them, here 4 to 6 us.
//
// Every function returns None when its arguments are not the common form (another type, layout or device, an error of the
// library's, a workspace that has to grow first); the caller in ops.py / nn.py then takes the general path, which handles or
// rejects them with the reference's messages.  Nothing is checked less: a call that succeeds here satisfies what that path
// checks.  What torch throws on the way (no memory for the output, a tensor without storage) becomes the Python exception
// that the same call raises from Python.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>

#include "../../include/light_b200.h"

namespace {

std::atomic<unsigned long long> g_ws[64];  // bytes of workspace registered per device (set_workspace below)

struct Arg {
  const at::Tensor *t = nullptr;
  bool ok(PyObject *o) {
    if (!THPVariable_Check(o)) return false;
    t = &THPVariable_Unpack(o);
    return true;
  }
};

bool cuda_contig(const at::Tensor &t) { return t.is_cuda() && t.is_contiguous() && !t.requires_grad(); }
// Whether something beside the result is to come of an operator of torch's on this tensor (a forward-mode tangent), or somebody is to see it: function
// transforms, torch-function and dispatch modes, tracing.  For operators that stand in for one of torch's.
bool watched(const at::Tensor &t) {
  return t._fw_grad(0).defined() || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) ||
         at::impl::PythonTorchFunctionTLS::stack_len() > 0 || c10::impl::TorchDispatchModeTLS::any_modes_set() || torch::jit::tracer::isTracing();
}
bool long_of(PyObject *o, long long &v) {
  if (!PyLong_Check(o)) return false;
  int overflow;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);  // (no Python error is set: the caller answers None)
  return !overflow;
}
void *stream_of(int dev) { return (void *)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }
bool workspace_fits(int dev, long long M, long long K) {
  return dev >= 0 && dev < 64 && g_ws[dev].load(std::memory_order_relaxed) >= light_b200_matmul_q_workspace_bytes((int)M, (int)K);
}
at::Tensor out_like(const at::Tensor &x, int64_t cols) {  // x (..., K) -> (..., cols)
  auto s = x.sizes().vec();
  s.back() = cols;
  return at::empty(s, x.options());
}
PyObject *give(int rc, const at::Tensor &out) {
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(out);
}
int act_of(const at::Tensor &t) {
  switch (t.scalar_type()) {
    case at::kFloat: return LB200_F32;
    case at::kBFloat16: return LB200_BF16;
    case at::kHalf: return LB200_F16;
    default: return -1;
  }
}
#define ARGS(n) \
  if (nargs != n) { PyErr_SetString(PyExc_TypeError, "wrong number of arguments"); return nullptr; }
#define NEED(c) \
  if (!(c)) Py_RETURN_NONE

// The rows of x when it is a (..., K) activation this file takes: at least one row, fewer than 2^31 elements a side.
bool rows_of(const at::Tensor &x, long long K, long long &M) {
  if (!cuda_contig(x) || x.dim() < 1 || K <= 0 || x.size(-1) != K || x.numel() == 0) return false;
  M = x.numel() / K;
  return M < (1ll << 31);
}

PyObject *set_workspace(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(2)
  long long dev, n;
  if (!long_of(a[0], dev) || !long_of(a[1], n) || dev < 0 || dev >= 64) {
    PyErr_SetString(PyExc_ValueError, "set_workspace: a device of 0 .. 63 and a size in bytes");
    return nullptr;
  }
  g_ws[dev].store((unsigned long long)n, std::memory_order_relaxed);
  Py_RETURN_NONE;
}

// (x (..., K) F32, blocks uint8, ggml type, N, K) -> (..., N) F32
PyObject *linear_q(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(5)
  Arg x, w;
  long long type, N, K, M;
  NEED(x.ok(a[0]) && w.ok(a[1]) && long_of(a[2], type) && long_of(a[3], N) && long_of(a[4], K));
  NEED(rows_of(*x.t, K, M) && x.t->scalar_type() == at::kFloat && cuda_contig(*w.t) && w.t->get_device() == x.t->get_device());
  const int be = light_b200_block_elems((int)type), dev = x.t->get_device();
  NEED(be > 0 && N > 0 && K % be == 0 && w.t->scalar_type() == at::kByte && w.t->numel() == N * (K / be) * light_b200_block_bytes((int)type));
  NEED(M == 1 || workspace_fits(dev, M, K));
  at::Tensor out = out_like(*x.t, N), own;
  const auto own_bytes = light_b200_matmul_q_scratch_bytes((int)type, w.t->const_data_ptr(), M, N, (int)K);
  if (own_bytes) own = at::empty({(int64_t)own_bytes}, w.t->options());
  return give(light_b200_matmul_q_scratch((int)type, x.t->const_data_ptr<float>(), w.t->const_data_ptr(), out.data_ptr<float>(), (int)M, (int)N, (int)K,
                                          own_bytes ? own.data_ptr() : nullptr, own_bytes, dev, stream_of(dev)), out);
}

// (x (..., K) F32 / BF16, codes I32 (N, K/8), scales, zeros F32 (N, K/G), G) -> (..., N) at x's type
PyObject *linear_int4(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(5)
  Arg x, c, s, z;
  long long G, M;
  NEED(x.ok(a[0]) && c.ok(a[1]) && s.ok(a[2]) && z.ok(a[3]) && long_of(a[4], G));
  NEED(cuda_contig(*c.t) && cuda_contig(*s.t) && cuda_contig(*z.t) && c.t->dim() == 2 && c.t->scalar_type() == at::kInt);
  const long long N = c.t->size(0), K = c.t->size(1) * 8;
  NEED(rows_of(*x.t, K, M) && (x.t->scalar_type() == at::kFloat || x.t->scalar_type() == at::kBFloat16));
  const int dev = x.t->get_device();
  NEED(G > 0 && K % G == 0 && N > 0 && s.t->scalar_type() == at::kFloat && z.t->scalar_type() == at::kFloat && s.t->numel() == N * (K / G) &&
       z.t->numel() == N * (K / G) && c.t->get_device() == dev && s.t->get_device() == dev && z.t->get_device() == dev);
  NEED(M == 1 || workspace_fits(dev, M, K));
  at::Tensor out = out_like(*x.t, N);
  return give(light_b200_int4_gemv(x.t->const_data_ptr(), (const uint32_t *)c.t->const_data_ptr(), s.t->const_data_ptr<float>(), z.t->const_data_ptr<float>(), out.data_ptr(),
                                   act_of(*x.t), (int)M, (int)N, (int)K, (int)G, dev, stream_of(dev)), out);
}

// (x (..., K) F32 / BF16, e4m3 codes (N, K), scale F32 (N/bR, K/bC), bR, bC) -> (..., N) at x's type
PyObject *linear_f8(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(5)
  Arg x, w, s;
  long long bR, bC, M;
  NEED(x.ok(a[0]) && w.ok(a[1]) && s.ok(a[2]) && long_of(a[3], bR) && long_of(a[4], bC));
  NEED(cuda_contig(*w.t) && cuda_contig(*s.t) && w.t->dim() == 2 && w.t->element_size() == 1 && s.t->scalar_type() == at::kFloat);
  const long long N = w.t->size(0), K = w.t->size(1);
  NEED(rows_of(*x.t, K, M) && (x.t->scalar_type() == at::kFloat || x.t->scalar_type() == at::kBFloat16));
  const int dev = x.t->get_device();
  NEED(bR > 0 && bC > 0 && N > 0 && N % bR == 0 && K % bC == 0 && s.t->numel() == (N / bR) * (K / bC) && w.t->get_device() == dev && s.t->get_device() == dev);
  NEED(M == 1 || workspace_fits(dev, M, K));
  at::Tensor out = out_like(*x.t, N);
  return give(light_b200_fp8_block_gemv(x.t->const_data_ptr(), (const uint8_t *)w.t->const_data_ptr(), s.t->const_data_ptr<float>(), out.data_ptr(),
                                        act_of(*x.t), (int)M, (int)N, (int)K, (int)bR, (int)bC, dev, stream_of(dev)), out);
}

// (x (T, K) F32 / BF16, w (E, K) F32) -> (T, E) F32
PyObject *router_logits(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(2)
  Arg x, w;
  NEED(x.ok(a[0]) && w.ok(a[1]) && !watched(*x.t) && !watched(*w.t) && x.t->dim() == 2 && w.t->dim() == 2 && cuda_contig(*x.t) && cuda_contig(*w.t) && w.t->scalar_type() == at::kFloat);
  const auto dt = x.t->scalar_type();
  const long long T = x.t->size(0), E = w.t->size(0), K = x.t->size(1);
  NEED((dt == at::kBFloat16 || dt == at::kFloat) && T > 0 && T <= 1ll << 21 && E > 0 && E < 1ll << 31 && K > 0 && K < 1ll << 31 && K % 8 == 0 && w.t->size(1) == K &&
       w.t->get_device() == x.t->get_device());
  const void *const xp = x.t->const_data_ptr();
  const float *const wp = w.t->const_data_ptr<float>();
  NEED(!((uintptr_t)xp & 15) && !((uintptr_t)wp & 15));
  const int dev = x.t->get_device();
  at::Tensor out = at::empty({T, E}, w.t->options());
  return give(light_b200_router_logits(xp, act_of(*x.t), wp, out.data_ptr<float>(), (int)T, (int)E, (int)K, dev, stream_of(dev)), out);
}

// (h (M, 2 I), gelu) -> (M, I)
PyObject *gate_mul(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(2)
  Arg h;
  NEED(h.ok(a[0]) && h.t->dim() == 2 && cuda_contig(*h.t) && act_of(*h.t) >= 0 && h.t->size(1) % 16 == 0 && h.t->numel() > 0);
  const int gelu = PyObject_IsTrue(a[1]), dev = h.t->get_device();
  if (gelu < 0) return nullptr;
  at::Tensor out = at::empty({h.t->size(0), h.t->size(1) / 2}, h.t->options());
  return give(light_b200_moe_gate_mul(h.t->const_data_ptr(), out.data_ptr(), act_of(*h.t), h.t->size(0), (int)(h.t->size(1) / 2), gelu, dev, stream_of(dev)), out);
}

// (pair rows (M, N), topk) -> (M / topk, N)
PyObject *combine(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(2)
  Arg p;
  long long topk;
  NEED(p.ok(a[0]) && long_of(a[1], topk) && p.t->dim() == 2 && cuda_contig(*p.t) && act_of(*p.t) >= 0 && topk > 0 && p.t->size(0) % topk == 0 &&
       p.t->size(1) % 8 == 0 && p.t->numel() > 0);
  const int dev = p.t->get_device();
  at::Tensor out = at::empty({p.t->size(0) / topk, p.t->size(1)}, p.t->options());
  return give(light_b200_moe_combine(p.t->const_data_ptr(), out.data_ptr(), act_of(*p.t), p.t->size(0) / topk, (int)p.t->size(1), (int)topk, dev,
                                     stream_of(dev)), out);
}

// (q, kbuf, vbuf, pos, scale, window, k_new, v_new, rope_base) -> (B, NH, 1, D)
PyObject *decode_attention(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(9)
  Arg q, kb, vb, pos, kn, vn;
  long long window;
  NEED(q.ok(a[0]) && kb.ok(a[1]) && vb.ok(a[2]) && pos.ok(a[3]) && PyFloat_Check(a[4]) && long_of(a[5], window) && PyFloat_Check(a[8]));
  NEED(cuda_contig(*q.t) && cuda_contig(*kb.t) && cuda_contig(*vb.t) && cuda_contig(*pos.t) && q.t->dim() == 4 && q.t->size(2) == 1 && kb.t->dim() == 4 &&
       kb.t->sizes() == vb.t->sizes() && q.t->numel() > 0 && kb.t->numel() > 0);
  const auto dt = q.t->scalar_type();
  const int dev = q.t->get_device();
  const int64_t B = q.t->size(0), NH = q.t->size(1), D = q.t->size(3), KH = kb.t->size(1);
  NEED((dt == at::kFloat || dt == at::kBFloat16) && kb.t->scalar_type() == dt && vb.t->scalar_type() == dt && kb.t->size(0) == B && kb.t->size(3) == D &&
       NH % KH == 0 && kb.t->get_device() == dev && vb.t->get_device() == dev);
  NEED(pos.t->scalar_type() == at::kLong && pos.t->numel() == 1 && pos.t->get_device() == dev);
  const bool append = a[6] != Py_None && a[7] != Py_None;
  NEED(append || (a[6] == Py_None && a[7] == Py_None));
  if (append) {
    NEED(kn.ok(a[6]) && vn.ok(a[7]) && cuda_contig(*kn.t) && cuda_contig(*vn.t) && kn.t->scalar_type() == dt && vn.t->scalar_type() == dt &&
         kn.t->sizes() == vn.t->sizes() && kn.t->dim() == 4 && kn.t->size(0) == B && kn.t->size(1) == KH && kn.t->size(2) == 1 && kn.t->size(3) == D &&
         kn.t->get_device() == dev && vn.t->get_device() == dev);
  }
  at::Tensor out = at::empty({B, NH, 1, D}, q.t->options());
  lb200_decode_attn_args d{};
  d.q = q.t->const_data_ptr(), d.kbuf = kb.t->data_ptr(), d.vbuf = vb.t->data_ptr();
  d.k_new = append ? kn.t->const_data_ptr() : nullptr, d.v_new = append ? vn.t->const_data_ptr() : nullptr;
  d.pos = pos.t->const_data_ptr<int64_t>(), d.out = out.data_ptr(), d.dtype = act_of(*q.t);
  d.B = (int)B, d.NH = (int)NH, d.KH = (int)KH, d.Cap = (int)kb.t->size(2), d.D = (int)D, d.window = (int)window;
  d.scale = (float)PyFloat_AsDouble(a[4]), d.rope_base = (float)PyFloat_AsDouble(a[8]);
  return give(light_b200_decode_attn(&d, dev, stream_of(dev)), out);
}

// A route's expert sort: ids I64 (T, topk) and weights are the first two of the answer, then the sorted pairs and their experts.
PyObject *sorted_route(const at::Tensor &ids, const at::Tensor &w, long long E, int dev) {
  const int64_t M = ids.numel();
  const auto i32 = ids.options().dtype(at::kInt);
  at::Tensor sp = at::empty({M}, ids.options()), se = at::empty({M}, ids.options());
  at::Tensor scratch = at::empty({M + (M + 1023) / 1024 * E + 1 + 2 * E + 1}, i32);
  int *s = scratch.data_ptr<int>(), *counts = s, *offsets = s + E;
  if (light_b200_moe_sort_pairs(ids.const_data_ptr<int64_t>(), counts, offsets, sp.data_ptr<int64_t>(), se.data_ptr<int64_t>(), s + 2 * E + 1, M, (int)E, dev,
                                stream_of(dev)) != 0)
    Py_RETURN_NONE;
  PyObject *t = PyTuple_New(4);
  const at::Tensor flat = w.reshape({M});
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(ids)), PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(flat));
  PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(sp)), PyTuple_SET_ITEM(t, 3, THPVariable_Wrap(se));
  return t;
}

// (scores F32 (T, E), bias F32 (E) or None, topk, normalize, sigmoid) -> (ids, weights, sorted pairs, sorted experts)
PyObject *moe_route(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(5)
  Arg x, b;
  long long topk;
  NEED(x.ok(a[0]) && long_of(a[2], topk) && cuda_contig(*x.t) && x.t->dim() == 2 && x.t->scalar_type() == at::kFloat && x.t->numel() > 0);
  const int dev = x.t->get_device(), norm = PyObject_IsTrue(a[3]), sigmoid = PyObject_IsTrue(a[4]);
  if (norm < 0 || sigmoid < 0) return nullptr;
  const int64_t T = x.t->size(0), E = x.t->size(1);
  NEED(topk >= 1 && topk <= E && topk <= 32 && E <= 1024 && T * topk < (1ll << 31));
  if (a[1] != Py_None)
    NEED(sigmoid && b.ok(a[1]) && cuda_contig(*b.t) && b.t->scalar_type() == at::kFloat && b.t->numel() == E && b.t->get_device() == dev);
  at::Tensor ids = at::empty({T, topk}, x.t->options().dtype(at::kLong)), w = at::empty({T, topk}, x.t->options());
  const float *in = x.t->const_data_ptr<float>();
  const int rc = sigmoid ? light_b200_moe_route_sigmoid(in, b.t ? b.t->const_data_ptr<float>() : nullptr, ids.data_ptr<int64_t>(), w.data_ptr<float>(), (int)T, (int)E,
                                                        (int)topk, norm, dev, stream_of(dev))
                         : light_b200_moe_route_topk(in, ids.data_ptr<int64_t>(), w.data_ptr<float>(), (int)T, (int)E, (int)topk, norm, dev, stream_of(dev));
  if (rc != 0) Py_RETURN_NONE;
  return sorted_route(ids, w, E, dev);
}

// (input (rows, K), weights, scale or None, block rows, block columns, ggml type (-1: block FP8), E, N, K, sorted pairs, sorted
// experts, pair weights or None, topk) -> (M, N) at the input's type
PyObject *moe_gemm(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  ARGS(13)
  Arg x, w, s, sp, se, tw;
  long long bR, bC, type, E, N, K, topk;
  NEED(x.ok(a[0]) && w.ok(a[1]) && long_of(a[3], bR) && long_of(a[4], bC) && long_of(a[5], type) && long_of(a[6], E) && long_of(a[7], N) && long_of(a[8], K) &&
       sp.ok(a[9]) && se.ok(a[10]) && long_of(a[12], topk));
  NEED(cuda_contig(*x.t) && cuda_contig(*w.t) && cuda_contig(*sp.t) && cuda_contig(*se.t) && x.t->dim() == 2 && x.t->size(1) == K && x.t->numel() > 0);
  const int dev = x.t->get_device();
  const int64_t M = sp.t->numel(), rows = x.t->size(0);
  NEED(sp.t->scalar_type() == at::kLong && se.t->scalar_type() == at::kLong && sp.t->dim() == 1 && se.t->dim() == 1 && se.t->numel() == M && M > 0 && M < (1ll << 31) &&
       topk > 0 && E > 0 && N > 0 && N < (1ll << 31) && (rows == M || rows == M / topk));
  NEED(w.t->get_device() == dev && sp.t->get_device() == dev && se.t->get_device() == dev);
  const auto dt = x.t->scalar_type();
  if (type >= 0) {
    const int be = light_b200_block_elems((int)type);
    NEED(dt == at::kFloat && be > 0 && K % be == 0 && w.t->scalar_type() == at::kByte && w.t->numel() == E * N * (K / be) * light_b200_block_bytes((int)type));
  } else {
    NEED((dt == at::kFloat || dt == at::kBFloat16) && s.ok(a[2]) && cuda_contig(*s.t) && s.t->scalar_type() == at::kFloat && s.t->get_device() == dev && bR > 0 &&
         bC > 0 && N % bR == 0 && K % bC == 0 && w.t->element_size() == 1 && w.t->numel() == E * N * K &&
         s.t->sizes() == at::IntArrayRef({E, N / bR, K / bC}));
  }
  if (a[11] != Py_None) NEED(tw.ok(a[11]) && cuda_contig(*tw.t) && tw.t->scalar_type() == at::kFloat && tw.t->numel() == M && tw.t->get_device() == dev);
  // 256 pairs or more work in the device's workspace; fewer, of bf16 rows, in memory of this call alone, so that several streams may
  // have one each (the caching allocator hands it to this stream's later work only).
  const bool few = M < 256;
  NEED(few || workspace_fits(dev, M, K));
  // Rows that no pair writes are zero: cleared as a whole while that is cheaper than finding them.
  const int64_t row_bytes = N * (int64_t)x.t->element_size(), words = (M + 31) / 32;
  const bool find = M * row_bytes > (8 << 20);
  at::Tensor out = find ? at::empty({M, N}, x.t->options()) : at::zeros({M, N}, x.t->options());
  at::Tensor scratch = at::empty({2 * E + 1 + (find ? words : 0)}, sp.t->options().dtype(at::kInt));
  int *sc = scratch.data_ptr<int>();
  void *st = stream_of(dev);
  if (find && light_b200_moe_clear_unrouted(sp.t->const_data_ptr<int64_t>(), se.t->const_data_ptr<int64_t>(), (uint32_t *)(sc + 2 * E + 1), out.data_ptr(), M, M,
                                            row_bytes, (int)E, dev, st) != 0)
    Py_RETURN_NONE;
  lb200_moe_args m{};
  m.input = x.t->const_data_ptr(), m.weights = w.t->const_data_ptr(), m.sorted_pairs = sp.t->const_data_ptr<int64_t>();
  m.expert_ids = se.t->const_data_ptr<int64_t>(), m.counts = sc, m.offsets = sc + E, m.topk_weights = tw.t ? tw.t->const_data_ptr<float>() : nullptr;
  m.out = out.data_ptr(), m.M = M, m.size_m = M, m.E = (int)E, m.N = (int)N, m.K = (int)K, m.topk = (int)topk, m.row_per_pair = rows == M;
  m.dtype = type >= 0 ? (int)type : act_of(*x.t);
  at::Tensor own;
  if (type >= 0) {
    const auto q6k_bytes = light_b200_q6k_scratch_bytes((int)type, m.weights, M, (int)K, 1);
    if (q6k_bytes) own = at::empty({(int64_t)q6k_bytes}, w.t->options());
    return give(light_b200_moe_gemm_q_scratch(&m, q6k_bytes ? own.data_ptr() : nullptr, q6k_bytes, dev, st), out);
  }
  const int64_t own_bytes = few && dt == at::kBFloat16 ? (int64_t)light_b200_moe_scratch_bytes(M, (int)K) : 0;
  if (own_bytes) own = at::empty({own_bytes}, w.t->options().dtype(at::kByte));
  return give(light_b200_moe_gemm_scratch(&m, s.t->const_data_ptr<float>(), (int)bR, (int)bC, own_bytes ? own.data_ptr() : nullptr, own_bytes, dev, st), out);
}

template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
PyObject *guarded(PyObject *self, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  return F(self, a, nargs);
  END_HANDLE_TH_ERRORS
}
#define FN(f, doc) {#f, (PyCFunction)(void (*)(void))guarded<f>, METH_FASTCALL, doc}
PyMethodDef kMethods[] = {FN(set_workspace, "registers a device's workspace size"),
                          FN(linear_q, "x . W^T, GGUF blocks"),
                          FN(linear_int4, "x . W^T, 4-bit groups"),
                          FN(linear_f8, "x . W^T, block-scaled FP8"),
                          FN(router_logits, "x . W^T, F32"),
                          FN(gate_mul, "act(gate) * up"),
                          FN(combine, "sum of the top-k slot rows"),
                          FN(moe_route, "top-k experts of each token and the pairs sorted by expert"),
                          FN(moe_gemm, "grouped x . W^T"),
                          FN(decode_attention, "append + rotary embedding + attention"),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "native host path of light_b200", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&kModule); }
