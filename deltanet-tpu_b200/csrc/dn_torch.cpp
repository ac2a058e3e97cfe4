// The operators' host path in native code: a CPython extension that takes torch tensors, checks that a call is a plain one
// (CUDA tensors of one device, contiguous, one dtype for q/k/v and one for the gates, shapes as documented), allocates, and calls the
// C ABI.  A call that is not plain is answered with None: the Python layer then validates it, with its error messages,
// converts what has to be converted and comes back through `forward`, inside a Python autograd function unless nothing
// watches the call (`bare`).  What is left to that function: tangents (forward-mode AD), function transforms, tracing, and
// dispatch modes.  They see a Python autograd function and either follow it or raise their own error, whereas addresses handed
// over here would leave them with results that look like constants.
//
// Why: a decode step of one sequence takes 4.5 us on the GPU, its path through the interpreter (shape checks, seven
// conversions that change nothing, ctypes structures) took 25; a short prompt 25 of 50.
//
// Nothing of the CUDA library is linked: `bind` receives the addresses of the C-ABI functions from the module that has
// loaded it (which may be an instrumented build).
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>

#include "../../include/deltanet_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

struct Abi {
  decltype(&dn_decode_step) decode_step = nullptr;
  decltype(&dn_chunk_fwd) chunk_fwd = nullptr;
  decltype(&dn_chunk_bwd) chunk_bwd = nullptr;
  decltype(&dn_residual_bytes) residual_bytes = nullptr;
  decltype(&dn_residual_carve) residual_carve = nullptr;
  decltype(&dn_scratch_bytes) scratch_bytes = nullptr;
  decltype(&dn_canonical_segments) canonical_segments = nullptr;
  decltype(&dn_cu_seqlens_segments) cu_seqlens_segments = nullptr;
  decltype(&dn_status_string) status_string = nullptr;
} abi;

void check(int status, const char* what) {
  TORCH_CHECK(status == 0, "deltanet_b200: ", what, " failed: ", abi.status_string(status), " (status ", status, ")");
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
int code(at::ScalarType t) { return t == at::kBFloat16 ? DN_BF16 : (t == at::kFloat ? DN_F32 : -1); }
// A tensor with memory of its own behind it: not a wrapper of a function transform, a fake or a tensor that stands for
// something else than what its memory holds.
bool dense(const Tensor& t) {
  constexpr c10::DispatchKeySet wrappers({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                          c10::DispatchKey::Functionalize, c10::DispatchKey::Negative, c10::DispatchKey::Conjugate,
                                          c10::DispatchKey::ZeroTensor});
  return t.layout() == at::kStrided && !t.key_set().has_any(wrappers) && t.has_storage();
}
// Can a kernel take the tensor as it is, beside `q`?  (What is not on q's device the general path moves or refuses.)
bool plain(const Tensor& t, const Tensor& q) { return dense(t) && t.device() == q.device() && t.is_contiguous(); }
// The kernels read and write the operator's tensors 16 bytes at a time.  A view at an odd offset is copied first.
bool at16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(ptr(t)) & 15) == 0; }
Tensor aligned(const Tensor& t) { return !t.defined() || at16(t) ? t : t.clone(at::MemoryFormat::Contiguous); }
// Does something follow the calls of this thread that an address would escape?
bool watched() { return torch::jit::tracer::isTracing() || c10::impl::TorchDispatchModeTLS::any_modes_set(); }
bool tangent(const Tensor& t) { return t.defined() && t._fw_grad(0).defined(); }

// ------------------------------------------------------------------------------------------------ the chunked operator
void require_dense(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    TORCH_CHECK(!t->defined() || dense(*t),
                "deltanet_b200: a tensor of this call has no memory of its own (a fake tensor, or the wrapper of a function transform)");
}
Tensor bytes_on(const Tensor& like, size_t n) {
  return at::empty({(int64_t)(n < 256 ? 256 : n)}, like.options().dtype(at::kByte));
}

// the forward; keeps the residuals in *kept when asked
variable_list forward(const dn_shape& shape, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& g_in, const Tensor& b_in,
                      const Tensor& w_in, const Tensor& init, const Tensor& seg, bool want_final, Tensor* kept, Tensor out = Tensor()) {
  require_dense({&q_in, &k_in, &v_in, &g_in, &b_in, &w_in, &init, &seg});
  const Tensor q = aligned(q_in), k = aligned(k_in), v = aligned(v_in), g = aligned(g_in), b = aligned(b_in), w = aligned(w_in);
  if (!out.defined()) out = at::empty({shape.B, shape.L, shape.Hv, shape.V}, q.options().requires_grad(false));
  Tensor fin;
  if (want_final) fin = at::empty({shape.B, shape.Hv, shape.K, shape.V}, q.options().dtype(at::kFloat).requires_grad(false));
  dn_residuals res;
  dn_shape f = shape;
  if (kept) {
    *kept = bytes_on(q, abi.residual_bytes(&shape));
    require_dense({kept});
    check(abi.residual_carve(&shape, kept->mutable_data_ptr(), &res), "dn_residual_carve");
  } else {
    f.flags |= DN_INFERENCE;
  }
  Tensor scratch = bytes_on(q, abi.scratch_bytes(&f, 0, 0));
  require_dense({&out, &fin, &scratch});
  check(abi.chunk_fwd(&f, ptr(q), ptr(k), ptr(v), ptr(g), ptr(b), ptr(w), static_cast<const int32_t*>(ptr(seg)),
                      static_cast<const float*>(ptr(init)), out.mutable_data_ptr(), want_final ? fin.mutable_data_ptr<float>() : nullptr,
                      kept ? &res : nullptr, scratch.mutable_data_ptr(), scratch.numel(), stream()),
        "dn_chunk_fwd");
  if (want_final) return {out, fin};
  return {out};
}

// its adjoint: the gradients of q, k, v, g, b, w and the initial state
variable_list backward(const dn_shape& shape, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& g_in, const Tensor& b_in,
                       const Tensor& w_in, const Tensor& init, const Tensor& seg, const Tensor& kept, const Tensor& d_out_in, const Tensor& d_final_in) {
  require_dense({&q_in, &k_in, &v_in, &g_in, &b_in, &w_in, &init, &seg, &kept});
  const Tensor q = aligned(q_in), k = aligned(k_in), v = aligned(v_in), g = aligned(g_in), b = aligned(b_in), w = aligned(w_in);
  Tensor d_out = d_out_in.defined() ? aligned(d_out_in.to(q.scalar_type()).resolve_neg().contiguous())
                                    : at::zeros({shape.B, shape.L, shape.Hv, shape.V}, q.options().requires_grad(false));
  Tensor d_final;
  if (d_final_in.defined()) d_final = d_final_in.to(at::kFloat).resolve_neg().contiguous();
  auto like = [](const Tensor& t) { return at::empty(t.sizes(), t.options().requires_grad(false)); };
  Tensor dq = like(q), dk = like(k), dv = like(v), dg = like(g), db = like(b), dw = like(w), d_init;
  if (init.defined()) d_init = like(init);
  dn_residuals res;
  if (kept.defined()) check(abi.residual_carve(&shape, const_cast<void*>(kept.const_data_ptr()), &res), "dn_residual_carve");
  Tensor scratch = bytes_on(q, abi.scratch_bytes(&shape, 1, kept.defined() ? 0 : 1));
  require_dense({&d_out, &d_final, &dq, &scratch});
  check(abi.chunk_bwd(&shape, ptr(q), ptr(k), ptr(v), ptr(g), ptr(b), ptr(w), static_cast<const int32_t*>(ptr(seg)),
                      static_cast<const float*>(ptr(init)), kept.defined() ? &res : nullptr, ptr(d_out),
                      static_cast<const float*>(ptr(d_final)), dq.mutable_data_ptr(), dk.mutable_data_ptr(), dv.mutable_data_ptr(),
                      dg.mutable_data_ptr(), db.mutable_data_ptr(), dw.mutable_data_ptr(),
                      d_init.defined() ? d_init.mutable_data_ptr<float>() : nullptr, scratch.mutable_data_ptr(), scratch.numel(), stream()),
        "dn_chunk_bwd");
  return {dq, dk, dv, dg, db, dw, d_init};
}

// The differentiable operator boundary (reference: gdn2.py:1461-1766) of plain calls.
struct ChunkOp : public torch::autograd::Function<ChunkOp> {
  static variable_list forward(AutogradContext* ctx, Variable q, Variable k, Variable v, Variable g, Variable b, Variable w,
                               std::optional<Tensor> init_in, std::optional<Tensor> seg_in, std::string shape_bytes, bool want_final,
                               bool recompute, bool inference) {
    const Tensor init = init_in.value_or(Tensor()), seg = seg_in.value_or(Tensor());
    dn_shape shape;
    std::memcpy(&shape, shape_bytes.data(), sizeof(shape));
    Tensor kept;
    variable_list r = ::forward(shape, q, k, v, g, b, w, init, seg, want_final, inference || recompute ? nullptr : &kept);
    ctx->saved_data["shape"] = shape_bytes;
    ctx->saved_data["inference"] = inference;
    // The residuals are no tensor of the user's and do not pass through saved-tensor hooks: a hook that stores tensors in fewer
    // bits would turn the block of bytes into others.
    ctx->saved_data["kept"] = kept;
    ctx->save_for_backward({q, k, v, g, b, w, init, seg});
    ctx->set_materialize_grads(false);
    return r;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    TORCH_CHECK_VALUE(!ctx->saved_data["inference"].toBool(),
                      "chunk_gdn2: differentiation is not supported when is_inference=True; set is_inference=False for training.");
    dn_shape shape;
    const std::string bytes = ctx->saved_data["shape"].toStringRef();
    std::memcpy(&shape, bytes.data(), sizeof(shape));
    const variable_list s = ctx->get_saved_variables();
    variable_list d = ::backward(shape, s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], ctx->saved_data["kept"].toTensor(), grads[0],
                                 grads.size() > 1 ? grads[1] : Tensor());
    if (!torch::autograd::get_current_graph_task_keep_graph()) ctx->saved_data.erase("kept");      // goes when the saved tensors do
    d.resize(12);
    return d;
  }
};

bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

variable_list run(const dn_shape& shape, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& b, const Tensor& w,
                  const Tensor& init, const Tensor& seg, bool want_final, bool recompute, bool inference) {
  if (!wants_grad({&q, &k, &v, &g, &b, &w, &init})) return forward(shape, q, k, v, g, b, w, init, seg, want_final, nullptr);
  auto opt = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
  return ChunkOp::apply(q, k, v, g, b, w, opt(init), opt(seg), std::string(reinterpret_cast<const char*>(&shape), sizeof(shape)), want_final,
                        recompute, inference);
}

// Allocation and enqueueing go on without the interpreter's lock: a call that waits for room in the launch queue, or for
// cudaMalloc, does not hold up the other Python threads.
struct Free_gil {
  PyThreadState* state = PyEval_SaveThread();
  void back() {
    if (state) PyEval_RestoreThread(state);
    state = nullptr;
  }
  ~Free_gil() { back(); }
};

PyObject* wrap(const variable_list& r) {
  if (r.size() == 1) return THPVariable_Wrap(r[0]);
  return PyTuple_Pack(2, py::reinterpret_steal<py::object>(THPVariable_Wrap(r[0])).ptr(),
                      py::reinterpret_steal<py::object>(THPVariable_Wrap(r[1])).ptr());
}

// arguments
Tensor tensor_or_none(PyObject* o) { return o == Py_None ? Tensor() : THPVariable_Unpack(o); }
bool all_tensors(PyObject* const* a, int n) {
  for (int i = 0; i < n; ++i)
    if (!THPVariable_Check(a[i])) return false;
  return true;
}
// (heads, columns) of a gate whose leading `lead` dimensions are given; false if it is not a plain one
bool gate(const Tensor& x, int lead, int64_t d0, int64_t d1, int Hk, int Hv, int64_t width, int32_t& heads, int32_t& cols) {
  const int64_t nd = x.dim();
  if ((nd != lead + 1 && nd != lead + 2) || x.size(0) != d0 || (lead == 2 && x.size(1) != d1)) return false;
  heads = (int32_t)x.size(lead);
  cols = nd == lead + 1 ? 1 : (int32_t)x.size(lead + 1);
  return (heads == 1 || heads == Hk || heads == Hv) && (cols == 1 || cols == width);
}

// chunk(q, k, v, g, b, w, segment_ids, cu_seqlens, initial_state, want_final, chunk, precision, scale, flags, recompute,
//       inference) -> out | (out, final) | None.  scale: a float, or None for K^-1/2.
PyObject* py_chunk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 16 || !all_tensors(a, 6)) Py_RETURN_NONE;
  const Tensor q = THPVariable_Unpack(a[0]), k = THPVariable_Unpack(a[1]), v = THPVariable_Unpack(a[2]);
  const Tensor g = THPVariable_Unpack(a[3]), b = THPVariable_Unpack(a[4]), w = THPVariable_Unpack(a[5]);
  for (int i = 6; i < 9; ++i)
    if (a[i] != Py_None && !THPVariable_Check(a[i])) Py_RETURN_NONE;
  const Tensor ids = tensor_or_none(a[6]), cu = tensor_or_none(a[7]), init = tensor_or_none(a[8]);
  if (!q.is_cuda() || watched()) Py_RETURN_NONE;
  for (const Tensor* t : {&q, &k, &v, &g, &b, &w})
    if (!plain(*t, q)) Py_RETURN_NONE;
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || q.sizes() != k.sizes()) Py_RETURN_NONE;
  const int64_t B = q.size(0), Lq = q.size(1), Hk = q.size(2), K = q.size(3), Hv = v.size(2), V = v.size(3);
  if (v.size(0) != B || v.size(1) != Lq || B < 1 || Lq < 1 || Hk < 1 || Hv < 1 || Hv % Hk) Py_RETURN_NONE;
  if ((K != 64 && K != 128) || (V != 64 && V != 128)) Py_RETURN_NONE;
  const int qdt = code(q.scalar_type()), gdt = code(g.scalar_type());
  if (qdt < 0 || gdt < 0 || code(k.scalar_type()) != qdt || code(v.scalar_type()) != qdt || code(b.scalar_type()) != gdt ||
      code(w.scalar_type()) != gdt)
    Py_RETURN_NONE;
  for (const Tensor* t : {&q, &k, &v, &g, &b, &w, &init})
    if (tangent(*t)) Py_RETURN_NONE;
  dn_shape s{};
  if (!gate(g, 2, B, Lq, Hk, Hv, K, s.g_heads, s.g_cols) || !gate(b, 2, B, Lq, Hk, Hv, K, s.b_heads, s.b_cols) ||
      !gate(w, 2, B, Lq, Hk, Hv, V, s.w_heads, s.w_cols))
    Py_RETURN_NONE;
  if (init.defined() && (!plain(init, q) || init.scalar_type() != at::kFloat || init.dim() != 4 || init.size(0) != B || init.size(1) != Hv ||
                         init.size(2) != K || init.size(3) != V))
    Py_RETURN_NONE;
  if (ids.defined() && (cu.defined() || !plain(ids, q) || ids.scalar_type() != at::kInt || ids.numel() != B * Lq ||
                        !(ids.dim() == 2 ? ids.size(0) == B : ids.dim() == 1)))
    Py_RETURN_NONE;
  if (cu.defined() && (!plain(cu, q) || cu.scalar_type() != at::kInt || cu.dim() != 1 || cu.numel() < 2)) Py_RETURN_NONE;
  s.B = (int32_t)B; s.L = (int32_t)Lq; s.Hk = (int32_t)Hk; s.Hv = (int32_t)Hv; s.K = (int32_t)K; s.V = (int32_t)V;
  s.qkv_dtype = qdt;
  s.gate_dtype = gdt;
  s.chunk = (int32_t)PyLong_AsLong(a[10]);
  s.precision = (int32_t)PyLong_AsLong(a[11]);
  s.scale = a[12] == Py_None ? (float)(1.0 / std::sqrt((double)K)) : (float)PyFloat_AsDouble(a[12]);
  s.flags = (uint32_t)PyLong_AsUnsignedLong(a[13]) | (init.defined() ? DN_HAS_INIT : 0u);
  if (PyErr_Occurred()) return nullptr;
  const bool want_final = a[9] == Py_True, recompute = a[14] == Py_True, inference = a[15] == Py_True;
  variable_list r;
  Free_gil gil;
  Tensor seg;
  if (ids.defined() || cu.defined()) {
    seg = at::empty({B, Lq}, q.options().dtype(at::kInt).requires_grad(false));
    int32_t* out = seg.mutable_data_ptr<int32_t>();
    if (ids.defined())
      check(abi.canonical_segments(ids.const_data_ptr<int32_t>(), nullptr, out, s.B, s.L, stream()), "dn_canonical_segments");
    else
      check(abi.cu_seqlens_segments(cu.const_data_ptr<int32_t>(), (int32_t)cu.numel(), nullptr, out, s.B, s.L, stream()), "dn_cu_seqlens_segments");
  }
  r = run(s, q, k, v, g, b, w, init, seg, want_final, recompute, inference);
  gil.back();
  return wrap(r);
  END_HANDLE_TH_ERRORS
}

std::vector<Tensor> tensors(PyObject* const* a, int n) {
  std::vector<Tensor> t;
  for (int i = 0; i < n; ++i) t.push_back(tensor_or_none(a[i]));
  return t;
}
// The two directions on prepared tensors and canonical ids, without autograd.
bool shape_of(PyObject* o, dn_shape* s) {
  if (!PyBytes_Check(o) || PyBytes_GET_SIZE(o) != (Py_ssize_t)sizeof(dn_shape)) return false;
  std::memcpy(s, PyBytes_AS_STRING(o), sizeof(dn_shape));
  return true;
}
PyObject* tuple_of(const variable_list& r) {                                     // (an undefined tensor is None)
  PyObject* t = PyTuple_New((Py_ssize_t)r.size());
  for (size_t i = 0; i < r.size(); ++i) PyTuple_SET_ITEM(t, (Py_ssize_t)i, THPVariable_Wrap(r[i]));
  return t;
}
// forward(q, k, v, g, b, w, initial_state, seg, shape bytes, want_final, keep, out) -> (out, final | None, residuals | None);
// out: a contiguous tensor for the outputs, or None
PyObject* py_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  dn_shape s;
  TORCH_CHECK_VALUE(n == 12 && all_tensors(a, 6) && shape_of(a[8], &s), "forward: bad arguments");
  const std::vector<Tensor> t = tensors(a, 8);
  const Tensor out = tensor_or_none(a[11]);
  const bool want_final = a[9] == Py_True, keep = a[10] == Py_True;
  Tensor kept;
  Free_gil gil;
  const variable_list r = forward(s, t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], want_final, keep ? &kept : nullptr, out);
  gil.back();
  return tuple_of({r[0], r.size() > 1 ? r[1] : Tensor(), kept});
  END_HANDLE_TH_ERRORS
}
// backward(q, k, v, g, b, w, initial_state, seg, residuals, d_out, d_final, shape bytes) -> the seven gradients
PyObject* py_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  dn_shape s;
  TORCH_CHECK_VALUE(n == 12 && all_tensors(a, 6) && shape_of(a[11], &s), "backward: bad arguments");
  const std::vector<Tensor> t = tensors(a, 11);
  Free_gil gil;
  const variable_list r = backward(s, t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], t[10]);
  gil.back();
  return tuple_of(r);
  END_HANDLE_TH_ERRORS
}
// bare(*tensors): may a call on them pass autograd by?  No gradient is wanted, and nothing follows it.
PyObject* py_bare(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (watched()) Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const Tensor t = tensor_or_none(a[i]);
    if (t.defined() && (!dense(t) || tangent(t) || wants_grad({&t}))) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------------ decode
// decode(q, k, v, g, b, w, state, reset, scale, flags, bf16_state, tau, out_state) -> (out, state) | None
PyObject* py_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 13 || !all_tensors(a, 7)) Py_RETURN_NONE;
  if ((a[7] != Py_None && !THPVariable_Check(a[7])) || (a[12] != Py_None && !THPVariable_Check(a[12]))) Py_RETURN_NONE;
  const Tensor q = THPVariable_Unpack(a[0]), k = THPVariable_Unpack(a[1]), v = THPVariable_Unpack(a[2]);
  const Tensor g = THPVariable_Unpack(a[3]), b = THPVariable_Unpack(a[4]), w = THPVariable_Unpack(a[5]);
  Tensor state = THPVariable_Unpack(a[6]);
  const Tensor reset = tensor_or_none(a[7]);
  Tensor next = tensor_or_none(a[12]);
  if (!q.is_cuda() || watched()) Py_RETURN_NONE;
  for (const Tensor* t : std::initializer_list<const Tensor*>{&q, &k, &v, &g, &b, &w, &state})
    if (!plain(*t, q)) Py_RETURN_NONE;
  if (q.dim() != 3 || k.dim() != 3 || v.dim() != 3 || q.sizes() != k.sizes() || state.dim() != 4) Py_RETURN_NONE;
  const int64_t B = q.size(0), Hk = q.size(1), K = q.size(2), Hv = v.size(1), V = v.size(2);
  if (v.size(0) != B || B < 1 || Hk < 1 || Hv < 1 || Hv % Hk || (K != 64 && K != 128) || (V != 64 && V != 128)) Py_RETURN_NONE;
  if (state.size(0) != B || state.size(1) != Hv || state.size(2) != K || state.size(3) != V) Py_RETURN_NONE;
  const int qdt = code(q.scalar_type()), gdt = code(g.scalar_type()), sdt = code(state.scalar_type());
  if (qdt < 0 || gdt < 0 || sdt < 0 || code(k.scalar_type()) != qdt || code(v.scalar_type()) != qdt || code(b.scalar_type()) != gdt ||
      code(w.scalar_type()) != gdt)
    Py_RETURN_NONE;
  dn_decode_shape s{};
  if (!gate(g, 1, B, 0, Hk, Hv, K, s.g_heads, s.g_cols) || !gate(b, 1, B, 0, Hk, Hv, K, s.b_heads, s.b_cols) ||
      !gate(w, 1, B, 0, Hk, Hv, V, s.w_heads, s.w_cols))
    Py_RETURN_NONE;
  for (const Tensor* t : {&g, &b, &w})               // (B, 1, H): a gate with a token dimension
    if (t->dim() == 3 && t->size(1) == 1 && (t->size(2) == 1 || t->size(2) == Hk || t->size(2) == Hv)) Py_RETURN_NONE;
  s.flags = (uint32_t)PyLong_AsUnsignedLong(a[9]);
  if (reset.defined()) {
    if (!plain(reset, q) || (reset.scalar_type() != at::kBool && reset.scalar_type() != at::kByte)) Py_RETURN_NONE;
    if (reset.dim() == 2 && reset.size(0) == B && reset.size(1) == Hv && Hv > 1) s.flags |= DN_RESET_PER_HEAD;
    else if (reset.dim() != 1 || reset.size(0) != B) Py_RETURN_NONE;
  }
  s.B = (int32_t)B; s.Hk = (int32_t)Hk; s.Hv = (int32_t)Hv; s.K = (int32_t)K; s.V = (int32_t)V;
  s.qkv_dtype = qdt;
  s.gate_dtype = gdt;
  s.state_in_dtype = sdt;
  s.state_out_dtype = a[10] == Py_True ? DN_BF16 : DN_F32;
  s.scale = a[8] == Py_None ? (float)(1.0 / std::sqrt((double)K)) : (float)PyFloat_AsDouble(a[8]);
  s.stability_tau = (float)PyFloat_AsDouble(a[11]);
  if (PyErr_Occurred()) return nullptr;
  const at::ScalarType st = s.state_out_dtype == DN_BF16 ? at::kBFloat16 : at::kFloat;
  PyObject* next_py = next.defined() ? a[12] : nullptr;
  if (next_py && (!plain(next, q) || !at16(next) || next.scalar_type() != st || next.sizes() != state.sizes())) Py_RETURN_NONE;
  Free_gil gil;
  state = aligned(state);
  if (!next_py) next = at::empty({B, Hv, K, V}, state.options().dtype(st).requires_grad(false));
  Tensor o = at::empty({B, Hv, V}, q.options().requires_grad(false));
  check(abi.decode_step(&s, ptr(q), ptr(k), ptr(v), ptr(g), ptr(b), ptr(w), ptr(state), static_cast<const uint8_t*>(ptr(reset)),
                        o.mutable_data_ptr(), const_cast<void*>(next.const_data_ptr()), stream()),
        "dn_decode_step");
  gil.back();
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(o));
  PyTuple_SET_ITEM(r, 1, next_py ? Py_NewRef(next_py) : THPVariable_Wrap(next));
  return r;
  END_HANDLE_TH_ERRORS
}

// plain(t, q): the test that every tensor of a call has to pass
PyObject* py_plain(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_VALUE(n == 2 && all_tensors(a, 2), "plain: two tensors");
  return PyBool_FromLong(plain(THPVariable_Unpack(a[0]), THPVariable_Unpack(a[1])));
  END_HANDLE_TH_ERRORS
}

// aligned(t): t itself, or a copy of it that starts at a multiple of 16 bytes
PyObject* py_aligned(PyObject*, PyObject* o) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_VALUE(THPVariable_Check(o), "aligned: a tensor");
  const Tensor& t = THPVariable_Unpack(o);
  return at16(t) ? Py_NewRef(o) : THPVariable_Wrap(aligned(t));
  END_HANDLE_TH_ERRORS
}

// bind({name: address of the C-ABI function})
PyObject* py_bind(PyObject*, PyObject* d) {
  HANDLE_TH_ERRORS
  auto get = [&](const char* name, auto& f) {
    PyObject* v = PyDict_GetItemString(d, name);
    TORCH_CHECK_VALUE(v, "bind: no ", name);
    f = reinterpret_cast<std::decay_t<decltype(f)>>(PyLong_AsVoidPtr(v));
  };
  get("dn_decode_step", abi.decode_step);
  get("dn_chunk_fwd", abi.chunk_fwd);
  get("dn_chunk_bwd", abi.chunk_bwd);
  get("dn_residual_bytes", abi.residual_bytes);
  get("dn_residual_carve", abi.residual_carve);
  get("dn_scratch_bytes", abi.scratch_bytes);
  get("dn_canonical_segments", abi.canonical_segments);
  get("dn_cu_seqlens_segments", abi.cu_seqlens_segments);
  get("dn_status_string", abi.status_string);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"chunk", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_chunk)), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_forward)), METH_FASTCALL, nullptr},
    {"backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_backward)), METH_FASTCALL, nullptr},
    {"bare", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_bare)), METH_FASTCALL, nullptr},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_decode)), METH_FASTCALL, nullptr},
    {"plain", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_plain)), METH_FASTCALL, nullptr},
    {"aligned", py_aligned, METH_O, nullptr},
    {"bind", py_bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
