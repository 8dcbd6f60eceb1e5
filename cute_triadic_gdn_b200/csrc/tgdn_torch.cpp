// Host path of the Python package: operator registrations, autograd, argument checks, output allocation and kernel launches
// in C++, so that a call costs the launches and little else.
//
// Through Python (torch.library.custom_op, autograd.Function, one ctypes call per kernel) the host needed 550 to 750 us for
// one forward + backward of the smallest configuration, whose kernels take 48 us, and 40 us for a decode step of 6 us: every
// small call was host-bound.
//
//   * TORCH_LIBRARY(tgdn_b200): joint_fwd / joint_bwd / joint_metadata / conv_split_act_fwd / _bwd / conv_split_norm_fwd / _bwd,
//     with autograd kernels built on torch::autograd::Function (saved tensors are read exactly once in a backward, auxiliary
//     outputs are not differentiable and get no materialised gradients: what activation checkpointing needs); the fake
//     implementations live in Python beside the calls (joint_torch_ops.py, conv_split_act.py, joint_packing.py).
//   * Python functions: what chunk_gdn_joint, gdn_joint_call, gdn_joint_decode and the convolution calls run when they are
//     not being traced, and the single stages (run_masks, ...) that the tests and the benchmark time one by one.
//
// The device work is libtgdn_b200, with which this file is linked: the entry points of include/tgdn.h in the forms of tgdn_host.h (token
// ranges of longer rows, rows of any alignment, the glue's backward in one pass).
#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <torch/library.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <optional>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "tgdn_host.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int64_t CHUNK = 64, HEAD_DIM = 128;

// ---- errors -----------------------------------------------------------------------------------------------------------
// The package raises AssertionError from the argument checks of the core (as the reference does), ValueError for
// packed-row and device / E problems, and TgdnError (_lib.py) when the library rejects a call.
struct AssertFail : std::runtime_error { using std::runtime_error::runtime_error; };
struct LibraryFail : std::runtime_error { using std::runtime_error::runtime_error; };

py::handle library_error;                                  // TgdnError, set by _lib.py
void set_python_error(const AssertFail& e) { PyErr_SetString(PyExc_AssertionError, e.what()); }
void set_python_error(const LibraryFail& e) { PyErr_SetString(library_error ? library_error.ptr() : PyExc_RuntimeError, e.what()); }

// Impl::forward and Impl::backward as an autograd function.  A backward runs under torch's engine, which keeps the class of a Python
// error only: the two above are turned into one there (elsewhere the module's translator does it).
template <typename Impl>
struct Differentiable : public torch::autograd::Function<Differentiable<Impl>> {
  template <typename... Args>
  static auto forward(AutogradContext* ctx, Args&&... args) { return Impl::forward(ctx, std::forward<Args>(args)...); }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    try {
      return Impl::backward(ctx, std::move(grads));
    } catch (const AssertFail& e) {
      rethrow(e);
    } catch (const LibraryFail& e) {
      rethrow(e);
    }
  }
  template <typename Fail>
  [[noreturn]] static void rethrow(const Fail& e) {
    py::gil_scoped_acquire gil;
    set_python_error(e);
    python_error error;
    error.persist();
    throw error;
  }
};

void check_rc(int rc, const char* what) {
  if (rc != 0) throw LibraryFail(std::string(what) + ": " + tgdn_error_string(rc) + " (code " + std::to_string(rc) + ")");
}

std::string shape_of(const Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + ")";
}

#define TGDN_ASSERT(cond, ...) do { if (!(cond)) throw AssertFail(c10::str(__VA_ARGS__)); } while (0)

// Shapes, dtypes, contiguity and device of the seven inputs; names the first thing that is off (same conditions as
// ops/gdn_joint.py:235-249 of the reference).
void check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2, const Tensor& g,
                  const Tensor& beta, bool packed) {
  TGDN_ASSERT(q.dim() == 4, "q: expected (B, T, H, 128), got ", shape_of(q));
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2);
  TGDN_ASSERT(q.size(3) == HEAD_DIM, "q: the head dimension must be ", HEAD_DIM, ", got ", q.size(3));
  const Tensor* heads[2] = {&k, &v};
  for (int i = 0; i < 2; ++i)
    TGDN_ASSERT(heads[i]->sizes() == q.sizes(), i ? "v" : "k", ": expected ", shape_of(q), " like q, got ", shape_of(*heads[i]));
  TGDN_ASSERT(T >= 1, "the sequence is empty");
  TGDN_ASSERT(packed || T % CHUNK == 0, "T = ", T, ": rows without cu_seqlens must hold whole chunks of ", CHUNK, " tokens");
  const int64_t E = k2.dim() == 4 ? k2.size(3) : 0;
  TGDN_ASSERT(E >= 1, "k2: expected (B, T, H, E) with E >= 1, got ", shape_of(k2));
  const Tensor* gates[3] = {&k2, &q2, &g};
  static const char* gate_names[3] = {"k2", "q2", "g"};
  for (int i = 0; i < 3; ++i) {
    const Tensor& t = *gates[i];
    TGDN_ASSERT(t.dim() == 4 && t.size(0) == B && t.size(1) == T && t.size(2) == H && t.size(3) == E, gate_names[i], ": expected (", B,
                ", ", T, ", ", H, ", ", E, "), got ", shape_of(t));
  }
  TGDN_ASSERT(beta.dim() == 3 && beta.size(0) == B && beta.size(1) == T && beta.size(2) == H, "beta: expected (", B, ", ", T, ", ", H,
              ") (one write strength per head), got ", shape_of(beta));
  const Tensor* all[7] = {&q, &k, &v, &k2, &q2, &g, &beta};
  static const char* names[7] = {"q", "k", "v", "k2", "q2", "g", "beta"};
  for (int i = 0; i < 7; ++i) {
    const auto want = i < 3 ? at::kBFloat16 : at::kFloat;
    TGDN_ASSERT(all[i]->scalar_type() == want, names[i], ": dtype ", all[i]->scalar_type(), ", expected ", want);
    TGDN_ASSERT(all[i]->is_cuda() && all[i]->device() == q.device(), names[i], ": every input must live on q's CUDA device");
    TGDN_ASSERT(all[i]->is_contiguous(), names[i], ": not contiguous");
  }
}

void check_device_and_e(const Tensor& q, int64_t E) {
  const bool ok = E == 1 || E == 2 || E == 4 || E == 8 || E == 12 || E == 16;
  TORCH_CHECK_VALUE(ok && at::cuda::getDeviceProperties(q.device().index())->major == 10,
                    "the Triadic GDN kernels require an sm_100 device and E=1/2/4/8/12/16");
}

// GJ_SAVE_MASKS=1 (default) keeps the chunk operators of the forward for the backward; anything else drops them and lets the
// backward form them again with the same kernel (bitwise identical).  Read at forward time, like the reference
// (ops/gdn_joint.py:167-173), and under the interpreter's lock: os.environ of another thread writes the same table, and getenv is
// not safe beside that.
bool save_masks() {
  py::gil_scoped_acquire gil;
  const char* s = std::getenv("GJ_SAVE_MASKS");
  return s == nullptr || std::strcmp(s, "1") == 0;
}

// ---- the stages -------------------------------------------------------------------------------------------------------
template <typename T = void>
T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }
template <typename T = void>
T* ptr(const OptTensor& t) { return t.has_value() ? ptr<T>(*t) : nullptr; }
const float* fptr(const Tensor& t) { return ptr<float>(t); }
bool has(const OptTensor& t) { return t.has_value() && t->defined(); }

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

struct Dims {
  int B, T, H, E, NC, row_tokens, n_docs;
  int64_t blocks() const { return 128 / tgdn_value_block(E); }      // value blocks of the reverse recurrence
};

// `row_tokens`: q may be a token range of longer rows, (B, T, H, 128) with the batch stride of the whole rows.
Dims dims(const Tensor& q, const Tensor& k2, const OptTensor& token_map, const OptTensor& chunk_starts = std::nullopt) {
  Dims d;
  d.B = static_cast<int>(q.size(0)); d.T = static_cast<int>(q.size(1)); d.H = static_cast<int>(q.size(2));
  d.E = static_cast<int>(k2.size(3));
  d.NC = has(token_map) ? static_cast<int>(token_map->size(1)) : static_cast<int>(q.size(1) / CHUNK);
  d.row_tokens = d.B > 1 && d.H > 0 ? static_cast<int>(q.stride(0) / (q.size(2) * HEAD_DIM)) : d.T;
  d.n_docs = has(chunk_starts) ? static_cast<int>(chunk_starts->numel() - 1) : 0;
  return d;
}

Tensor empty(at::IntArrayRef sizes, const Tensor& like, at::ScalarType dtype) { return at::empty(sizes, like.options().dtype(dtype)); }

struct Masks { Tensor gc, AP, Pm; };

// gc (cumulative log gate and gate factors), AP = [A; Pm A] operand image, Pm image of every chunk; see include/tgdn.h.
Masks run_masks(const Tensor& q, const Tensor& k, const Tensor& k2, const Tensor& q2, const Tensor& g, const Tensor& beta, double scale,
                const OptTensor& token_map) {
  const c10::cuda::CUDAGuard guard(q.device());
  const Dims d = dims(q, k2, token_map);
  Masks m{empty({d.B, d.NC, d.H, tgdn_gate_item_floats(d.E)}, q, at::kFloat), empty({d.B, d.NC, d.H, 128 * 64}, q, at::kBFloat16),
          empty({d.B, d.NC, d.H, 64 * 64}, q, at::kBFloat16)};
  check_rc(tgdn_masks_rows(ptr(q), ptr(k), fptr(k2), fptr(q2), fptr(g), fptr(beta), static_cast<float>(scale), ptr<int32_t>(token_map), d.B,
                           d.T, d.H, d.E, d.NC, d.row_tokens, ptr<float>(m.gc), ptr(m.AP), ptr(m.Pm), stream_of(q)),
           "tgdn_masks");
  return m;
}

struct Forward { Tensor o, h, W, U; };

// Forward recurrence; h, W, U stay undefined unless `save`.  `o`: where the output goes (a token range of a longer output), or
// undefined: a new tensor.  state_in / state_out: optional f32 (sequences, H, E, 128, 128).
Forward run_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2, const Tensor& beta,
                    const Tensor& gc, const Tensor& AP, double scale, bool save, const OptTensor& chunk_starts, const OptTensor& token_map,
                    const OptTensor& state_in, const OptTensor& state_out, Tensor o = Tensor()) {
  const c10::cuda::CUDAGuard guard(q.device());
  const Dims d = dims(q, k2, token_map, chunk_starts);
  Forward f;
  f.o = o.defined() ? o : empty(v.sizes(), v, at::kBFloat16);
  if (save) {
    f.h = empty({d.B, d.NC, d.H, d.E, 16, 128, 8}, q, at::kBFloat16);
    f.W = empty({d.B, d.NC, d.H, CHUNK, 128}, q, at::kBFloat16);
    f.U = empty({d.B, d.NC, d.H, CHUNK, 128}, q, at::kBFloat16);
  }
  check_rc(tgdn_fwd_rows(ptr(q), ptr(k), ptr(v), fptr(k2), fptr(q2), fptr(beta), fptr(gc), ptr(AP), static_cast<float>(scale),
                         ptr<int32_t>(chunk_starts), ptr<int32_t>(token_map), d.n_docs, d.B, d.T, d.H, d.E, d.NC, d.row_tokens, ptr(f.o),
                         ptr(f.W), ptr(f.U), ptr(f.h), ptr<float>(state_in), ptr<float>(state_out), stream_of(q)),
           "tgdn_fwd");
  return f;
}

// Gradients of the seven inputs, in their order.
struct Grads {
  Tensor q, k, v, k2, q2, g, beta;
  std::vector<Tensor> list() const { return {q, k, v, k2, q2, g, beta}; }
  static Grads like(const Tensor& q, const Tensor& k2, const Tensor& beta) {
    return {empty(q.sizes(), q, at::kBFloat16), empty(q.sizes(), q, at::kBFloat16), empty(q.sizes(), q, at::kBFloat16),
            empty(k2.sizes(), q, at::kFloat),   empty(k2.sizes(), q, at::kFloat),   empty(k2.sizes(), q, at::kFloat),
            empty(beta.sizes(), q, at::kFloat)};
  }
  Grads tokens(int64_t lo, int64_t n) const {           // views of a token range
    return {q.narrow(1, lo, n), k.narrow(1, lo, n), v.narrow(1, lo, n), k2.narrow(1, lo, n), q2.narrow(1, lo, n), g.narrow(1, lo, n),
            beta.narrow(1, lo, n)};
  }
};

// What travels between the kernels of the backward: from the reverse recurrence to the gradients; dkq, da, dc, dd between the two stages that
// the gradients also exist as.
struct Between {
  void *dU, *ds, *dkg, *dkq;
  float *dr, *da, *dc, *dd;
  int* next_item = nullptr;
};

// Reverse recurrence: dV, and dU, ds, dkg, dr of `x`.  ds is written only for slices whose chunk decay matters to dg.  Entries of a
// packed row's chunk map that no document uses are neither written here nor read by the later stages.
void launch_reverse(const Dims& d, const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& k2, const Tensor& q2,
                    const Tensor& beta, const Tensor& gc, const Tensor& AP, const Tensor& Pm, const Tensor& U, double scale,
                    const OptTensor& chunk_starts, const OptTensor& token_map, const OptTensor& grad_state_in,
                    const OptTensor& grad_state_out, const Tensor& dV, const Between& x) {
  check_rc(tgdn_bwd_recurrent_rows(ptr(q), ptr(k), ptr(dO), fptr(k2), fptr(q2), fptr(beta), fptr(gc), ptr(AP), ptr(Pm), ptr(U),
                                   static_cast<float>(scale), ptr<int32_t>(chunk_starts), ptr<int32_t>(token_map), d.n_docs, d.B, d.T, d.H,
                                   d.E, d.NC, d.row_tokens, ptr(dV), x.dU, x.ds, x.dkg, x.dr, ptr<float>(grad_state_in),
                                   ptr<float>(grad_state_out), stream_of(q), x.next_item),
           "tgdn_bwd_recurrent");
}

// State gradients: dkq, da, dc, dd of `x`.
void launch_state_grads(const Dims& d, const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& dV, const Tensor& h,
                        const Tensor& k2, const Tensor& q2, const Tensor& gc, double scale, const OptTensor& token_map, const Between& x) {
  check_rc(tgdn_bwd_state_grads_rows(ptr(q), ptr(k), ptr(dO), ptr(dV), ptr(h), x.ds, x.dkg, fptr(k2), fptr(q2), fptr(gc),
                                     static_cast<float>(scale), ptr<int32_t>(token_map), d.B, d.T, d.H, d.E, d.NC, d.row_tokens, x.dkq,
                                     x.da, x.dc, x.dd, stream_of(q)),
           "tgdn_bwd_state_grads");
}

// Matrix gradients, mask gradients and final assembly, into out's dq, dk, dk2, dq2, dg, dbeta.
void launch_matrix(const Dims& d, const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& W, const Tensor& U, const Tensor& AP,
                   const Tensor& k2, const Tensor& q2, const Tensor& beta, const Tensor& gc, double scale, const OptTensor& token_map,
                   const Between& x, const Grads& out) {
  check_rc(tgdn_bwd_matrix_rows(ptr(q), ptr(k), ptr(dO), x.dU, ptr(W), ptr(U), ptr(AP), fptr(k2), fptr(q2), fptr(beta), fptr(gc), x.dkq,
                                x.da, x.dc, x.dd, x.dr, static_cast<float>(scale), ptr<int32_t>(token_map), d.B, d.T, d.H, d.E, d.NC,
                                d.row_tokens, ptr(out.q), ptr(out.k), ptr<float>(out.k2), ptr<float>(out.q2), ptr<float>(out.g),
                                ptr<float>(out.beta), stream_of(q)),
           "tgdn_bwd_matrix");
}

// State gradients and matrix gradients in one kernel: all gradients but dV, into `out` (out.v: the dV of the reverse recurrence).
void launch_grads(const Dims& d, const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& h, const Tensor& W, const Tensor& U,
                  const Tensor& AP, const Tensor& k2, const Tensor& q2, const Tensor& beta, const Tensor& gc, double scale,
                  const OptTensor& token_map, const Between& x, const Grads& out) {
  check_rc(tgdn_bwd_grads_rows(ptr(q), ptr(k), ptr(dO), ptr(out.v), x.dU, ptr(W), ptr(U), ptr(AP), ptr(h), x.ds, x.dkg, fptr(k2), fptr(q2),
                               fptr(beta), fptr(gc), x.dr, static_cast<float>(scale), ptr<int32_t>(token_map), d.B, d.T, d.H, d.E, d.NC,
                               d.row_tokens, x.next_item, ptr(out.q), ptr(out.k), ptr<float>(out.k2), ptr<float>(out.q2),
                               ptr<float>(out.g), ptr<float>(out.beta), stream_of(q)),
           "tgdn_bwd_grads");
}

// The stages one by one on tensors of their own, for the tests and the benchmark.
struct Reverse { Tensor dV, dU, ds, dkg, dr; };

Reverse run_reverse(const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& k2, const Tensor& q2, const Tensor& beta,
                    const Tensor& gc, const Tensor& AP, const Tensor& Pm, const Tensor& U, double scale, const OptTensor& chunk_starts,
                    const OptTensor& token_map, const OptTensor& grad_state_in, const OptTensor& grad_state_out) {
  const c10::cuda::CUDAGuard guard(q.device());
  const Dims d = dims(q, k2, token_map, chunk_starts);
  const int64_t NV = d.blocks();
  Reverse r;
  r.dV = empty(dO.sizes(), dO, at::kBFloat16);
  r.dU = empty({d.B, d.NC, d.H, CHUNK, 128}, q, at::kBFloat16);
  r.ds = empty({d.B, d.NC, d.H, d.E, 16, 128, 8}, q, at::kBFloat16);
  r.dkg = empty({d.B, d.NC, d.H, NV, 8, 128, 8}, q, at::kBFloat16);    // image [token / 8][key row][token % 8] per value block
  r.dr = empty({d.B, d.NC, d.H, NV, CHUNK, d.E}, q, at::kFloat);
  launch_reverse(d, q, k, dO, k2, q2, beta, gc, AP, Pm, U, scale, chunk_starts, token_map, grad_state_in, grad_state_out, r.dV,
                 Between{ptr(r.dU), ptr(r.ds), ptr(r.dkg), nullptr, ptr<float>(r.dr), nullptr, nullptr, nullptr});
  return r;
}

struct StateGrads { Tensor dkq, da, dc, dd; };

StateGrads run_state_grads(const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& dV, const Tensor& h, const Tensor& ds,
                           const Tensor& dkg, const Tensor& k2, const Tensor& q2, const Tensor& gc, double scale,
                           const OptTensor& token_map) {
  const c10::cuda::CUDAGuard guard(q.device());
  const Dims d = dims(q, k2, token_map);
  StateGrads s;
  s.dkq = empty({d.B, d.NC, d.H, 16, 128, 8}, q, at::kBFloat16);       // image [column / 8][row][column % 8]
  s.da = empty({d.B, d.NC, d.H, CHUNK, d.E}, q, at::kFloat);
  s.dc = empty({d.B, d.NC, d.H, CHUNK, d.E}, q, at::kFloat);
  s.dd = empty({d.B, d.NC, d.H, d.E}, q, at::kFloat);
  launch_state_grads(d, q, k, dO, dV, h, k2, q2, gc, scale, token_map,
                     Between{nullptr, ptr(ds), ptr(dkg), ptr(s.dkq), nullptr, ptr<float>(s.da), ptr<float>(s.dc), ptr<float>(s.dd)});
  return s;
}

void run_matrix(const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& dU, const Tensor& W, const Tensor& U, const Tensor& AP,
                const Tensor& k2, const Tensor& q2, const Tensor& beta, const Tensor& gc, const StateGrads& s, const Tensor& dr,
                double scale, const OptTensor& token_map, const Grads& out) {
  const c10::cuda::CUDAGuard guard(q.device());
  launch_matrix(dims(q, k2, token_map), q, k, dO, W, U, AP, k2, q2, beta, gc, scale, token_map,
                Between{ptr(dU), nullptr, nullptr, ptr(s.dkq), ptr<float>(dr), ptr<float>(s.da), ptr<float>(s.dc), ptr<float>(s.dd)}, out);
}

void run_grads(const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& dU, const Tensor& ds, const Tensor& dkg, const Tensor& dr,
               const Tensor& h, const Tensor& W, const Tensor& U, const Tensor& AP, const Tensor& k2, const Tensor& q2, const Tensor& beta,
               const Tensor& gc, double scale, const OptTensor& token_map, Tensor next_item, const Grads& out) {
  const c10::cuda::CUDAGuard guard(q.device());
  launch_grads(dims(q, k2, token_map), q, k, dO, h, W, U, AP, k2, q2, beta, gc, scale, token_map,
               Between{ptr(dU), ptr(ds), ptr(dkg), nullptr, ptr<float>(dr), nullptr, nullptr, nullptr, ptr<int>(next_item)}, out);
}

// reverse recurrence -> state and matrix gradients, into `out`.  AP, Pm undefined: GJ_SAVE_MASKS=0, the forward's own
// kernel forms them again.
void run_backward(const Tensor& q, const Tensor& k, const Tensor& k2, const Tensor& q2, const Tensor& g, const Tensor& beta,
                  const Tensor& gc, Tensor AP, Tensor Pm, const Tensor& h, const Tensor& W, const Tensor& U, const Tensor& dO, double scale,
                  const OptTensor& chunk_starts, const OptTensor& token_map, const OptTensor& grad_state_in,
                  const OptTensor& grad_state_out, const Grads& out) {
  if (!AP.defined()) {
    Masks m = run_masks(q, k, k2, q2, g, beta, scale, token_map);
    AP = m.AP;
    Pm = m.Pm;
  }
  const c10::cuda::CUDAGuard guard(q.device());
  const Dims d = dims(q, k2, token_map, chunk_starts);
  const int64_t items = static_cast<int64_t>(d.B) * d.NC * d.H, NV = d.blocks();
  Tensor between = empty({items * (d.E * 32768 + NV * 16384 + 16384 + NV * 64 * d.E * 4) + 16}, q, at::kByte);   // ds, dkg, dU, dr, the item counter
  uint8_t *ds = ptr<uint8_t>(between), *dkg = ds + items * d.E * 32768, *dU = dkg + items * NV * 16384;
  uint8_t *dr = dU + items * 16384, *counter = dr + items * NV * 64 * d.E * 4;
  const Between x{dU, ds, dkg, nullptr, reinterpret_cast<float*>(dr), nullptr, nullptr, nullptr, reinterpret_cast<int*>(counter)};
  launch_reverse(d, q, k, dO, k2, q2, beta, gc, AP, Pm, U, scale, chunk_starts, token_map, grad_state_in, grad_state_out, out.v, x);
  launch_grads(d, q, k, dO, h, W, U, AP, k2, q2, beta, gc, scale, token_map, x, out);
}

// ---- operators of the core --------------------------------------------------------------------------------------------
// `covered`: the documents of the chunk map hold every token of the row, as those of prepare_documents do.  Otherwise rows of o and of
// dV that no document holds are zero; with it nothing has to be filled.
std::vector<Tensor> joint_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2, const Tensor& g,
                              const Tensor& beta, double scale, const OptTensor& chunk_starts, const OptTensor& token_map, bool covered) {
  check_inputs(q, k, v, k2, q2, g, beta, has(token_map));
  check_device_and_e(q, k2.size(3));
  Masks m = run_masks(q, k, k2, q2, g, beta, scale, token_map);
  Forward f = run_forward(q, k, v, k2, q2, beta, m.gc, m.AP, scale, true, chunk_starts, token_map, std::nullopt, std::nullopt,
                          has(token_map) && !covered ? at::zeros(v.sizes(), v.options()) : Tensor());
  return {f.o, m.gc, m.AP, m.Pm, f.h, f.W, f.U};
}

// saved: q, k, k2, q2, g, beta, gc, [AP, Pm,] h, W, U
std::vector<Tensor> joint_bwd(std::vector<Tensor> saved, const Tensor& dO, double scale, const OptTensor& chunk_starts,
                              const OptTensor& token_map, bool covered) {
  TORCH_CHECK_VALUE(saved.size() == 12 || saved.size() == 10, "joint_bwd: 12 saved tensors, or 10 without the chunk operators");
  const bool with_masks = saved.size() == 12;
  const int64_t o = with_masks ? 2 : 0;
  Grads out = Grads::like(saved[0], saved[2], saved[5]);
  if (has(token_map) && !covered) out.v.zero_();
  run_backward(saved[0], saved[1], saved[2], saved[3], saved[4], saved[5], saved[6], with_masks ? saved[7] : Tensor(),
               with_masks ? saved[8] : Tensor(), saved[7 + o], saved[8 + o], saved[9 + o], dO.contiguous(), scale, chunk_starts, token_map,
               std::nullopt, std::nullopt, out);
  return out.list();
}

int64_t chunk_capacity(int64_t tokens, int64_t documents) {
  const int64_t worst = (tokens + CHUNK - 1) / CHUNK + documents - 1;
  return (worst + 15) / 16 * 16;
}

std::tuple<Tensor, Tensor, Tensor> joint_metadata(const Tensor& cu, int64_t tokens) {
  const c10::cuda::CUDAGuard guard(cu.device());
  const int64_t n = cu.numel() - 1, capacity = chunk_capacity(tokens, n);
  Tensor offsets = empty({n + 1}, cu, at::kInt), mapping = empty({3, capacity}, cu, at::kInt), valid = empty({1}, cu, at::kBool);
  check_rc(tgdn_metadata(ptr(cu), cu.scalar_type() == at::kLong ? 1 : 0, static_cast<int>(n), static_cast<int>(tokens),
                         ptr<int32_t>(offsets), ptr<int32_t>(mapping), static_cast<int>(capacity), ptr<uint8_t>(valid), stream_of(cu)),
           "tgdn_metadata");
  return {offsets, mapping, valid};
}

std::vector<Tensor> call_joint_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2, const Tensor& g,
                                   const Tensor& beta, double scale, const OptTensor& chunk_starts, const OptTensor& token_map,
                                   bool covered) {
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("tgdn_b200::joint_fwd", "").typed<decltype(joint_fwd)>();
  return op.call(q, k, v, k2, q2, g, beta, scale, chunk_starts, token_map, covered);
}
std::vector<Tensor> call_joint_bwd(at::TensorList saved, const Tensor& dO, double scale, const OptTensor& chunk_starts,
                                   const OptTensor& token_map, bool covered) {
  using Sig = std::vector<Tensor>(at::TensorList, const Tensor&, double, const OptTensor&, const OptTensor&, bool);
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("tgdn_b200::joint_bwd", "").typed<Sig>();
  return op.call(saved, dO, scale, chunk_starts, token_map, covered);
}
std::vector<Tensor> joint_bwd_entry(at::TensorList saved, const Tensor& dO, double scale, const OptTensor& chunk_starts,
                                    const OptTensor& token_map, bool covered) {
  return joint_bwd(saved.vec(), dO, scale, chunk_starts, token_map, covered);
}

Tensor or_undefined(const OptTensor& t) { return has(t) ? *t : Tensor(); }
OptTensor or_nullopt(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }

bool any_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->requires_grad()) return true;
  return false;
}

// Differentiates joint_fwd (reference: ops/joint_torch_ops.py:50-80, ops/gdn_joint.py:201-232).
struct JointSteps {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2,
                               const Tensor& g, const Tensor& beta, double scale, const OptTensor& chunk_starts,
                               const OptTensor& token_map, bool covered) {
    at::AutoDispatchBelowADInplaceOrView below;
    std::vector<Tensor> out = call_joint_fwd(q, k, v, k2, q2, g, beta, scale, chunk_starts, token_map, covered);
    variable_list keep{q, k, k2, q2, g, beta, out[1]};
    if (save_masks()) {
      keep.push_back(out[2]);
      keep.push_back(out[3]);
    }
    for (int i = 4; i < 7; ++i) keep.push_back(out[i]);
    keep.push_back(or_undefined(chunk_starts));
    keep.push_back(or_undefined(token_map));
    ctx->save_for_backward(std::move(keep));
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["covered"] = covered;
    ctx->mark_non_differentiable(variable_list(out.begin() + 1, out.end()));
    ctx->set_materialize_grads(false);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list res(11);
    if (!grads[0].defined()) return res;                 // the output was not used
    variable_list kept = ctx->get_saved_variables();      // read exactly once: under activation checkpointing every read unpacks
    const OptTensor token_map = or_nullopt(kept.back());
    kept.pop_back();
    const OptTensor chunk_starts = or_nullopt(kept.back());
    kept.pop_back();
    std::vector<Tensor> seven = call_joint_bwd(kept, grads[0].contiguous(), ctx->saved_data["scale"].toDouble(), chunk_starts, token_map,
                                               ctx->saved_data["covered"].toBool());
    for (int i = 0; i < 7; ++i) res[i] = std::move(seven[i]);
    return res;
  }
};
using JointFunction = Differentiable<JointSteps>;

std::vector<Tensor> joint_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2,
                                       const Tensor& g, const Tensor& beta, double scale, const OptTensor& chunk_starts,
                                       const OptTensor& token_map, bool covered) {
  // Nothing to differentiate: no autograd function, which would refuse inputs that carry a tangent (forward-mode differentiation),
  // whatever the caller means to do with it.
  if (!any_grad({&q, &k, &v, &k2, &q2, &g, &beta})) {
    at::AutoDispatchBelowADInplaceOrView below;
    return call_joint_fwd(q, k, v, k2, q2, g, beta, scale, chunk_starts, token_map, covered);
  }
  return JointFunction::apply(q, k, v, k2, q2, g, beta, scale, chunk_starts, token_map, covered);
}

double scale_or_default(std::optional<double> scale, const Tensor& q) {
  return scale.has_value() ? *scale : 1.0 / std::sqrt(static_cast<double>(q.size(-1)));
}

// What can be checked about a packed row without reading the offsets (ops/joint_packing.py:38-49 of the reference), then the
// chunk metadata, built on the device; offsets that do not start at 0, end at T and strictly increase trip a device-side
// assertion, as there (ops/joint_packing.py:52-62).
std::tuple<Tensor, Tensor> prepare_documents(const Tensor& row, const Tensor& cu) {
  TORCH_CHECK_VALUE(row.dim() >= 2 && row.size(0) == 1 && row.size(1) >= 1, "a packed row has shape (1, T, ...) with T >= 1; got ",
                    shape_of(row));
  TORCH_CHECK_VALUE(cu.dim() == 1 && cu.numel() >= 2, "cu_seqlens: a vector of document offsets, at least [0, T]");
  TORCH_CHECK_VALUE(cu.scalar_type() == at::kInt || cu.scalar_type() == at::kLong, "cu_seqlens: int32 or int64 offsets, got ",
                    cu.scalar_type());
  TORCH_CHECK_VALUE(cu.is_contiguous() && cu.device() == row.device(),
                    "cu_seqlens: must be contiguous and live on the device of the inputs");
  TORCH_CHECK_VALUE(row.size(1) < (int64_t{1} << 31), "a packed row is limited to 2^31 - 1 tokens (offsets are 32-bit on the device)");
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("tgdn_b200::joint_metadata", "").typed<decltype(joint_metadata)>();
  auto [offsets, mapping, valid] = op.call(cu, row.size(1));
  at::_assert_async(valid, "cu_seqlens must start at 0, end at T, and strictly increase");
  return {offsets, mapping};
}

Tensor joint_call(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2, const Tensor& g,
                  const Tensor& beta, std::optional<double> scale, const OptTensor& cu) {
  const Tensor qc = q.contiguous();
  OptTensor chunk_starts, token_map;
  if (has(cu)) std::tie(chunk_starts, token_map) = prepare_documents(qc, *cu);
  return call_joint_fwd(qc, k.contiguous(), v.contiguous(), k2.contiguous(), q2.contiguous(), g.contiguous(), beta.contiguous(),
                        scale_or_default(scale, qc), chunk_starts, token_map, true)[0];
}

void check_state(const Tensor& s, at::IntArrayRef shape, const Tensor& q, const char* name) {
  TORCH_CHECK_VALUE(s.sizes() == shape && s.scalar_type() == at::kFloat && s.device() == q.device(), name,
                    " must be an f32 tensor of shape ", shape, " on the inputs' device");
}

// ---- segments and recomputation ---------------------------------------------------------------------------------------
// The pipeline on ONE SEGMENT of longer sequences: the recurrent state comes in and goes out, and so does its gradient in the
// backward (f32 (B, H, E, 128, 128) each).  Dense rows only.
struct SegmentSteps {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2,
                               const Tensor& g, const Tensor& beta, const OptTensor& state_in, double scale) {
    at::AutoDispatchBelowADInplaceOrView below;
    Masks m = run_masks(q, k, k2, q2, g, beta, scale, std::nullopt);
    Tensor state_out = empty({q.size(0), q.size(2), k2.size(3), 128, 128}, q, at::kFloat);
    Forward f = run_forward(q, k, v, k2, q2, beta, m.gc, m.AP, scale, true, std::nullopt, std::nullopt,
                            has(state_in) ? OptTensor(state_in->contiguous()) : OptTensor(), state_out);
    ctx->save_for_backward({q, k, k2, q2, g, beta, m.gc, m.AP, m.Pm, f.h, f.W, f.U});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["has_state"] = has(state_in);
    ctx->set_materialize_grads(false);                   // an unused state_out arrives undefined, not as a tensor of zeros
    return {f.o, state_out};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list s = ctx->get_saved_variables();
    const Tensor& q = s[0];
    const bool has_state = ctx->saved_data["has_state"].toBool();
    Tensor dstate_in;
    if (has_state) dstate_in = empty({q.size(0), q.size(2), s[2].size(3), 128, 128}, q, at::kFloat);
    const OptTensor g_in = grads[1].defined() ? OptTensor(grads[1].to(at::kFloat).contiguous()) : OptTensor();
    const Tensor dO = grads[0].defined() ? grads[0].contiguous() : at::zeros(q.sizes(), q.options());
    Grads out = Grads::like(q, s[2], s[5]);
    run_backward(q, s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8], s[9], s[10], s[11], dO, ctx->saved_data["scale"].toDouble(),
                 std::nullopt, std::nullopt, g_in, or_nullopt(dstate_in), out);
    variable_list res = out.list();
    res.push_back(dstate_in);
    res.push_back(Tensor());
    return res;
  }
};
using SegmentFunction = Differentiable<SegmentSteps>;

// Backward state recomputation: the forward keeps only the inputs and the f32 state at every segment boundary instead of the
// per-chunk tensors; the backward walks the segments from the last to the first, runs each segment's forward again with
// everything saved, then its backward, and hands the gradient of the state to the segment before.  Bitwise the results of the
// plain function; the price is one more masks + forward pass.  Dense rows only.
// The kernels read a segment in place (row_tokens: the batch stride of the whole rows) and write its part of o and of the
// gradients in place; copying the segments out and the results back was a third of the step (1.0 of 3.0 ms at B=4, T=4096,
// H=16, E=2 in four segments).
struct CheckpointedSteps {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2,
                        const Tensor& g, const Tensor& beta, double scale, int64_t seg) {
    at::AutoDispatchBelowADInplaceOrView below;
    const int64_t T = q.size(1);
    Tensor o = empty(v.sizes(), v, at::kBFloat16), state;
    variable_list keep{q, k, v, k2, q2, g, beta};
    for (int64_t lo = 0; lo < T; lo += seg) {
      const int64_t n = std::min(seg, T - lo);
      auto cut = [&](const Tensor& t) { return t.narrow(1, lo, n); };
      const Tensor sq = cut(q), sk = cut(k), sk2 = cut(k2), sq2 = cut(q2), sb = cut(beta);
      Masks m = run_masks(sq, sk, sk2, sq2, cut(g), sb, scale, std::nullopt);
      Tensor next;
      if (lo + n < T) next = empty({q.size(0), q.size(2), k2.size(3), 128, 128}, q, at::kFloat);
      run_forward(sq, sk, cut(v), sk2, sq2, sb, m.gc, m.AP, scale, false, std::nullopt, std::nullopt, or_nullopt(state), or_nullopt(next),
                  cut(o));
      if (next.defined()) keep.push_back(next);
      state = next;
    }
    ctx->save_for_backward(std::move(keep));
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["seg"] = seg;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k2 = s[3];
    const int64_t T = q.size(1), seg = ctx->saved_data["seg"].toInt();
    const double scale = ctx->saved_data["scale"].toDouble();
    const Tensor dO = grads[0].contiguous();
    Grads out = Grads::like(q, k2, s[6]);
    Tensor g_state;                                      // dL/dS at the end of the segment at hand
    for (int64_t i = (T + seg - 1) / seg - 1; i >= 0; --i) {
      const int64_t lo = i * seg, n = std::min(seg, T - lo);
      auto cut = [&](const Tensor& t) { return t.narrow(1, lo, n); };
      const Tensor sq = cut(q), sk = cut(s[1]), sv = cut(s[2]), sk2 = cut(k2), sq2 = cut(s[4]), sg = cut(s[5]), sb = cut(s[6]);
      Masks m = run_masks(sq, sk, sk2, sq2, sg, sb, scale, std::nullopt);
      // the output of the segment is formed again with the rest; it goes where the segment's dV will go after it
      Grads part = out.tokens(lo, n);
      Forward f = run_forward(sq, sk, sv, sk2, sq2, sb, m.gc, m.AP, scale, true, std::nullopt, std::nullopt,
                              i > 0 ? OptTensor(s[7 + i - 1]) : OptTensor(), std::nullopt, part.v);
      Tensor g_prev;
      if (i > 0) g_prev = empty({q.size(0), q.size(2), k2.size(3), 128, 128}, q, at::kFloat);
      run_backward(sq, sk, sk2, sq2, sg, sb, m.gc, m.AP, m.Pm, f.h, f.W, f.U, cut(dO), scale, std::nullopt, std::nullopt,
                   or_nullopt(g_state), or_nullopt(g_prev), part);
      g_state = g_prev;
    }
    variable_list res = out.list();
    res.resize(9);
    return res;
  }
};
using CheckpointedFunction = Differentiable<CheckpointedSteps>;

// chunk_gdn_joint: training, recomputation, or inference with the state handed in and out.  Returns (o, final state or None).
std::tuple<Tensor, OptTensor> chunk_joint(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2,
                                          const Tensor& g, const Tensor& beta, std::optional<double> scale_in, const OptTensor& cu,
                                          const OptTensor& initial_state, bool output_final_state,
                                          std::optional<int64_t> checkpoint_tokens) {
  check_inputs(q, k, v, k2, q2, g, beta, has(cu));
  const int64_t B = q.size(0), H = q.size(2), E = k2.size(3);
  check_device_and_e(q, E);
  OptTensor chunk_starts, token_map;
  if (has(cu)) std::tie(chunk_starts, token_map) = prepare_documents(q, *cu);
  const double scale = scale_or_default(scale_in, q);
  const bool needs_grad = any_grad({&q, &k, &v, &k2, &q2, &g, &beta});
  if (needs_grad) {
    TORCH_CHECK_VALUE(!has(initial_state) && !output_final_state,
                      "initial_state / output_final_state are forward-only: run them under torch.no_grad()");
    if (checkpoint_tokens.has_value()) {
      TORCH_CHECK_VALUE(!has(cu), "checkpoint_tokens: dense rows only (a packed row is already cut at its documents)");
      TORCH_CHECK_VALUE(*checkpoint_tokens > 0 && *checkpoint_tokens % CHUNK == 0, "checkpoint_tokens must be a positive multiple of ",
                        CHUNK);
      if (*checkpoint_tokens < q.size(1))
        return {CheckpointedFunction::apply(q, k, v, k2, q2, g, beta, scale, *checkpoint_tokens), std::nullopt};
    }
    return {call_joint_fwd(q, k, v, k2, q2, g, beta, scale, chunk_starts, token_map, true)[0], std::nullopt};
  }
  const int64_t n_seq = has(cu) ? cu->numel() - 1 : B;
  OptTensor s_in, s_out;
  if (has(initial_state)) {
    check_state(*initial_state, {n_seq, H, E, 128, 128}, q, "initial_state");
    s_in = initial_state->contiguous();
  }
  if (output_final_state) s_out = empty({n_seq, H, E, 128, 128}, q, at::kFloat);
  at::AutoDispatchBelowADInplaceOrView below;
  Masks m = run_masks(q, k, k2, q2, g, beta, scale, token_map);
  Forward f = run_forward(q, k, v, k2, q2, beta, m.gc, m.AP, scale, false, chunk_starts, token_map, s_in, s_out);
  return {f.o, s_out};
}

std::tuple<Tensor, Tensor> joint_segment(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2,
                                         const Tensor& g, const Tensor& beta, const OptTensor& state_in, std::optional<double> scale) {
  check_inputs(q, k, v, k2, q2, g, beta, false);
  check_device_and_e(q, k2.size(3));
  if (has(state_in)) check_state(*state_in, {q.size(0), q.size(2), k2.size(3), 128, 128}, q, "state_in");
  variable_list out = SegmentFunction::apply(q, k, v, k2, q2, g, beta, state_in, scale_or_default(scale, q));
  return {out[0], out[1]};
}

// One token per sequence on a resident state, which is updated in place.
Tensor decode(Tensor q, Tensor k, Tensor v, Tensor k2, Tensor q2, Tensor g, Tensor beta, const Tensor& state, std::optional<double> scale) {
  TORCH_CHECK_VALUE(!any_grad({&q, &k, &v, &k2, &q2, &g, &beta, &state}), "gdn_joint_decode is forward-only: run it under torch.no_grad()");
  at::AutoDispatchBelowADInplaceOrView below;
  const bool squeeze = q.dim() == 4;
  int64_t t = squeeze ? q.size(1) : 1;
  TORCH_CHECK_VALUE(t == 1, "gdn_joint_decode takes one token per sequence: T must be 1");
  if (squeeze)                                            // the token axis of the others is dropped at its first token, however long it is
    for (Tensor* x : {&k, &v, &k2, &q2, &g, &beta})
      if (x->dim() > 1 && x->size(1) > 1) *x = x->narrow(1, 0, 1);
  // (B, 1, H, X) and (B, H, X) hold the same elements in the same order: shapes are compared with the token axis dropped
  auto sizes3 = [&](const Tensor& x, int64_t b, int64_t h, int64_t w) {
    return squeeze ? x.dim() == 4 && x.size(0) == b && x.size(1) == 1 && x.size(2) == h && x.size(3) == w
                   : x.dim() == 3 && x.size(0) == b && x.size(1) == h && x.size(2) == w;
  };
  const int64_t B = q.dim() > 0 ? q.size(0) : 0, H = q.dim() >= 3 ? q.size(-2) : 0;
  TORCH_CHECK_VALUE((squeeze || q.dim() == 3) && q.size(-1) == HEAD_DIM && k.sizes() == q.sizes() && v.sizes() == q.sizes(),
                    "q, k, v must be (B, H, 128) (or (B, 1, H, 128)) and agree");
  const int64_t E = k2.dim() > 0 ? k2.size(-1) : 0;
  const bool beta_ok = squeeze ? beta.dim() == 3 && beta.size(0) == B && beta.size(1) == 1 && beta.size(2) == H
                               : beta.dim() == 2 && beta.size(0) == B && beta.size(1) == H;
  TORCH_CHECK_VALUE(sizes3(k2, B, H, E) && sizes3(q2, B, H, E) && sizes3(g, B, H, E) && beta_ok,
                    "k2, q2, g must be (B, H, E) and beta (B, H)");
  TORCH_CHECK_VALUE(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16 &&
                        k2.scalar_type() == at::kFloat && q2.scalar_type() == at::kFloat && g.scalar_type() == at::kFloat &&
                        beta.scalar_type() == at::kFloat,
                    "q, k, v must be bfloat16 and k2, q2, g, beta float32");
  for (const Tensor* x : {&q, &k, &v, &k2, &q2, &g, &beta})
    TORCH_CHECK_VALUE(x->is_cuda() && x->device() == q.device(), "every input must live on q's CUDA device");
  check_device_and_e(q, E);
  TORCH_CHECK_VALUE(state.dim() == 5 && state.size(0) == B && state.size(1) == H && state.size(2) == E && state.size(3) == 128 &&
                        state.size(4) == 128 && state.scalar_type() == at::kFloat && state.device() == q.device() && state.is_contiguous(),
                    "state must be a contiguous f32 tensor of shape (", B, ", ", H, ", ", E, ", 128, 128) on the inputs' device");
  const c10::cuda::CUDAGuard guard(q.device());
  q = q.contiguous(); k = k.contiguous(); v = v.contiguous(); k2 = k2.contiguous(); q2 = q2.contiguous(); g = g.contiguous();
  beta = beta.contiguous();
  Tensor o = empty(v.sizes(), v, at::kBFloat16);
  check_rc(tgdn_decode_step(ptr(q), ptr(k), ptr(v), fptr(k2), fptr(q2), fptr(g), fptr(beta), static_cast<float>(scale_or_default(scale, q)),
                            static_cast<int>(B), static_cast<int>(H), static_cast<int>(E), ptr<float>(state), ptr(o), stream_of(q)),
           "tgdn_decode_step");
  return o;
}

// ---- convolution pre-pass ---------------------------------------------------------------------------------------------
struct ConvInput {
  Tensor x, weight, cu;
  int n_docs = 0;
};

bool aligned(const Tensor& t, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % bytes == 0; }
// Strides of the token and the batch axis.  An axis of size one may carry any stride, and contiguous() leaves it: it counts as dense.
int64_t token_stride(const Tensor& t) { return t.size(1) == 1 ? t.size(2) : t.stride(1); }
int64_t batch_stride(const Tensor& t) { return t.size(0) == 1 ? t.size(1) * token_stride(t) : t.stride(0); }
bool rows_aligned(const Tensor& t) { return token_stride(t) % 8 == 0 && batch_stride(t) % 8 == 0 && aligned(t, 16); }
// Rows of consecutive channels that do not overlap: what the kernels read in place.
bool rows_readable(const Tensor& t) { return (t.size(2) == 1 || t.stride(2) == 1) && token_stride(t) >= t.size(2); }

// `pieces`: the rows must be whole 16-byte pieces (the fused kernels); otherwise any readable row will do.
ConvInput conv_prep(const Tensor& x, const Tensor& weight, const OptTensor& cu, bool pieces = false) {
  TORCH_CHECK_VALUE(x.dim() == 3 && weight.dim() == 2 && weight.size(0) == x.size(2) && weight.size(1) == 4,
                    "x must be (B, T, C) and weight (C, 4)");
  TORCH_CHECK_VALUE(x.scalar_type() == at::kBFloat16, "x must be bf16");
  TORCH_CHECK_VALUE(x.is_cuda() && weight.device() == x.device(), "x and weight must be on the same CUDA device");
  ConvInput c;
  c.x = x;
  if (!rows_readable(c.x)) c.x = c.x.contiguous();
  if (pieces && !rows_aligned(c.x)) c.x = c.x.clone(at::MemoryFormat::Contiguous);
  c.weight = weight.to(at::kBFloat16).contiguous();
  if (!aligned(c.weight, 16)) c.weight = c.weight.clone();
  if (has(cu)) {
    TORCH_CHECK_VALUE(c.x.size(0) == 1, "cu_seqlens requires a packed row: B=1");
    TORCH_CHECK_VALUE(cu->dim() == 1 && cu->numel() >= 2 && cu->device() == x.device(),
                      "cu_seqlens must be a vector of at least two offsets on the input device");
    c.cu = cu->to(at::kInt).contiguous();
    c.n_docs = static_cast<int>(c.cu.numel() - 1);
  }
  return c;
}

Tensor conv_fwd(const Tensor& x, const Tensor& weight, int64_t act_channels, const OptTensor& cu) {
  const c10::cuda::OptionalCUDAGuard guard(x.is_cuda() ? std::optional<c10::Device>(x.device()) : std::nullopt);
  ConvInput c = conv_prep(x, weight, cu);
  const int64_t B = c.x.size(0), T = c.x.size(1), C = c.x.size(2);
  Tensor y = empty({B, T, C}, c.x, at::kBFloat16);
  check_rc(tgdn_conv_fwd_any(ptr(c.x), ptr(c.weight), ptr(y), ptr<int32_t>(c.cu), c.n_docs, static_cast<int>(B), static_cast<int>(T),
                             static_cast<int>(C), batch_stride(c.x), token_stride(c.x), static_cast<int>(act_channels), stream_of(c.x)),
           "tgdn_conv_fwd");
  return y;
}

std::tuple<Tensor, Tensor> conv_bwd(const Tensor& x, const Tensor& dy_in, const Tensor& weight, int64_t act_channels, const OptTensor& cu) {
  const c10::cuda::OptionalCUDAGuard guard(x.is_cuda() ? std::optional<c10::Device>(x.device()) : std::nullopt);
  ConvInput c = conv_prep(x, weight, cu);
  const Tensor dy = rows_readable(dy_in) ? dy_in : dy_in.contiguous();
  const int64_t B = c.x.size(0), T = c.x.size(1), C = c.x.size(2);
  Tensor dx = empty({B, T, C}, c.x, at::kBFloat16), dw = empty({C, 4}, c.x, at::kBFloat16);
  const int64_t nbytes = tgdn_conv_bwd_best_scratch(static_cast<int>(B), static_cast<int>(T), static_cast<int>(C));
  Tensor scratch = empty({nbytes / 4}, c.x, at::kFloat);
  check_rc(tgdn_conv_bwd_any(ptr(c.x), ptr(c.weight), ptr(dy), ptr(dx), ptr(dw), ptr<int32_t>(c.cu), c.n_docs, static_cast<int>(B),
                             static_cast<int>(T), static_cast<int>(C), batch_stride(c.x), token_stride(c.x), batch_stride(dy), token_stride(dy),
                             static_cast<int>(act_channels), ptr(scratch), nbytes, stream_of(c.x)),
           "tgdn_conv_bwd");
  return {dx, dw.to(weight.scalar_type())};
}

using Five = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>;

void glue_dims(const Tensor& x, int64_t H, int64_t E) {
  const bool e_ok = E == 1 || E == 2 || E == 4 || E == 8 || E == 12 || E == 16;
  TORCH_CHECK_VALUE(x.dim() == 3 && H > 0 && x.size(2) == H * (3 * 128 + 2 * E) && e_ok, "conv_split_norm: C=", x.dim() == 3 ? x.size(2) : -1,
                    " is not H*(3*128 + 2*E) for H=", H, ", E=", E, " (E in 1, 2, 4, 8, 12, 16)");
  TORCH_CHECK_VALUE(x.size(2) % 8 == 0, "conv_split_norm: the channel count must be a multiple of 8");
}

Five norm_fwd(const Tensor& x, const Tensor& weight, int64_t heads, int64_t slices, double eps, const OptTensor& cu) {
  const c10::cuda::OptionalCUDAGuard guard(x.is_cuda() ? std::optional<c10::Device>(x.device()) : std::nullopt);
  glue_dims(x, heads, slices);
  ConvInput c = conv_prep(x, weight, cu, true);
  const int64_t B = c.x.size(0), T = c.x.size(1), C = c.x.size(2);
  Tensor q = empty({B, T, heads, 128}, x, at::kBFloat16), k = empty({B, T, heads, 128}, x, at::kBFloat16),
         v = empty({B, T, heads, 128}, x, at::kBFloat16), k2 = empty({B, T, heads, slices}, x, at::kFloat),
         q2 = empty({B, T, heads, slices}, x, at::kFloat);
  check_rc(tgdn_glue_fwd(ptr(c.x), ptr(c.weight), ptr<int32_t>(c.cu), c.n_docs, static_cast<int>(B), static_cast<int>(T), static_cast<int>(C),
                         batch_stride(c.x), token_stride(c.x), static_cast<int>(heads), static_cast<int>(slices), static_cast<float>(eps), ptr(q),
                         ptr(k), ptr(v), ptr<float>(k2), ptr<float>(q2), stream_of(c.x)),
           "tgdn_glue_fwd");
  return {q, k, v, k2, q2};
}

std::tuple<Tensor, Tensor> norm_bwd(const Tensor& x, const Tensor& weight, const Tensor& dq, const Tensor& dk, const Tensor& dv,
                                    const Tensor& dk2, const Tensor& dq2, int64_t heads, int64_t slices, double eps, const OptTensor& cu) {
  const c10::cuda::OptionalCUDAGuard guard(x.is_cuda() ? std::optional<c10::Device>(x.device()) : std::nullopt);
  glue_dims(x, heads, slices);
  ConvInput c = conv_prep(x, weight, cu, true);
  const int64_t B = c.x.size(0), T = c.x.size(1), C = c.x.size(2);
  auto bf = [](const Tensor& t) { return t.to(at::kBFloat16).contiguous(); };
  auto f32 = [](const Tensor& t) { return t.to(at::kFloat).contiguous(); };
  const Tensor q = bf(dq), k = bf(dk), v = bf(dv), k2 = f32(dk2), q2 = f32(dq2);
  Tensor dx = empty({B, T, C}, c.x, at::kBFloat16), dw = empty({C, 4}, c.x, at::kBFloat16);
  Tensor dy_gates = empty({B, T, 2 * heads * slices}, c.x, at::kBFloat16);
  const int64_t nbytes = tgdn_conv_bwd_best_scratch(static_cast<int>(B), static_cast<int>(T), static_cast<int>(C));
  Tensor scratch = empty({nbytes / 4}, c.x, at::kFloat);
  check_rc(tgdn_glue_bwd(ptr(c.x), ptr(c.weight), ptr<int32_t>(c.cu), c.n_docs, static_cast<int>(B), static_cast<int>(T), static_cast<int>(C),
                         batch_stride(c.x), token_stride(c.x), static_cast<int>(heads), static_cast<int>(slices), static_cast<float>(eps), ptr(q),
                         ptr(k), ptr(v), fptr(k2), fptr(q2), ptr(dx), ptr(dw), ptr(dy_gates), ptr(scratch), nbytes, stream_of(c.x)),
           "tgdn_glue_bwd");
  return {dx, dw.to(weight.scalar_type())};
}

Tensor call_conv_fwd(const Tensor& x, const Tensor& weight, int64_t act_channels, const OptTensor& cu) {
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("tgdn_b200::conv_split_act_fwd", "").typed<decltype(conv_fwd)>();
  return op.call(x, weight, act_channels, cu);
}
Five call_norm_fwd(const Tensor& x, const Tensor& weight, int64_t heads, int64_t slices, double eps, const OptTensor& cu) {
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("tgdn_b200::conv_split_norm_fwd", "").typed<decltype(norm_fwd)>();
  return op.call(x, weight, heads, slices, eps, cu);
}

struct ConvSteps {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, int64_t act_channels, const OptTensor& cu) {
    at::AutoDispatchBelowADInplaceOrView below;
    Tensor y = call_conv_fwd(x, weight, act_channels, cu);
    ctx->save_for_backward({x, weight, or_undefined(cu)});
    ctx->saved_data["act"] = act_channels;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list s = ctx->get_saved_variables();
    static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("tgdn_b200::conv_split_act_bwd", "").typed<decltype(conv_bwd)>();
    auto [dx, dw] = op.call(s[0], grads[0], s[1], ctx->saved_data["act"].toInt(), or_nullopt(s[2]));
    return {dx, dw, Tensor(), Tensor()};
  }
};
using ConvFunction = Differentiable<ConvSteps>;
Tensor conv_fwd_autograd(const Tensor& x, const Tensor& weight, int64_t act_channels, const OptTensor& cu) {
  if (!any_grad({&x, &weight})) {
    at::AutoDispatchBelowADInplaceOrView below;
    return call_conv_fwd(x, weight, act_channels, cu);
  }
  return ConvFunction::apply(x, weight, act_channels, cu);
}

struct NormSteps {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, int64_t heads, int64_t slices, double eps,
                               const OptTensor& cu) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [q, k, v, k2, q2] = call_norm_fwd(x, weight, heads, slices, eps, cu);
    ctx->save_for_backward({x, weight, or_undefined(cu)});
    ctx->saved_data["heads"] = heads;
    ctx->saved_data["slices"] = slices;
    ctx->saved_data["eps"] = eps;
    return {q, k, v, k2, q2};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list s = ctx->get_saved_variables();
    static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("tgdn_b200::conv_split_norm_bwd", "").typed<decltype(norm_bwd)>();
    auto [dx, dw] = op.call(s[0], s[1], g[0], g[1], g[2], g[3], g[4], ctx->saved_data["heads"].toInt(), ctx->saved_data["slices"].toInt(),
                            ctx->saved_data["eps"].toDouble(), or_nullopt(s[2]));
    return {dx, dw, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
using NormFunction = Differentiable<NormSteps>;
Five norm_fwd_autograd(const Tensor& x, const Tensor& weight, int64_t heads, int64_t slices, double eps, const OptTensor& cu) {
  if (!any_grad({&x, &weight})) {
    at::AutoDispatchBelowADInplaceOrView below;
    return call_norm_fwd(x, weight, heads, slices, eps, cu);
  }
  variable_list o = NormFunction::apply(x, weight, heads, slices, eps, cu);
  return {o[0], o[1], o[2], o[3], o[4]};
}

}  // namespace

TORCH_LIBRARY(tgdn_b200, m) {
  m.def("joint_fwd(Tensor q, Tensor k, Tensor v, Tensor k2, Tensor q2, Tensor g, Tensor beta, float scale, Tensor? chunk_starts=None, "
        "Tensor? token_map=None, bool covered=False) -> Tensor[]");
  m.def("joint_bwd(Tensor[] saved, Tensor do, float scale, Tensor? chunk_starts=None, Tensor? token_map=None, bool covered=False) -> "
        "Tensor[]");
  m.def("joint_metadata(Tensor cu_seqlens, SymInt tokens) -> (Tensor, Tensor, Tensor)");
  m.def("conv_split_act_fwd(Tensor x, Tensor weight, SymInt act_channels, Tensor? cu_seqlens=None) -> Tensor");
  m.def("conv_split_act_bwd(Tensor x, Tensor dy, Tensor weight, SymInt act_channels, Tensor? cu_seqlens=None) -> (Tensor, Tensor)");
  m.def("conv_split_norm_fwd(Tensor x, Tensor weight, SymInt heads, SymInt slices, float eps, Tensor? cu_seqlens=None) -> "
        "(Tensor, Tensor, Tensor, Tensor, Tensor)");
  m.def("conv_split_norm_bwd(Tensor x, Tensor weight, Tensor dq, Tensor dk, Tensor dv, Tensor dk2, Tensor dq2, SymInt heads, SymInt slices, "
        "float eps, Tensor? cu_seqlens=None) -> (Tensor, Tensor)");
}

TORCH_LIBRARY_IMPL(tgdn_b200, CUDA, m) {
  m.impl("joint_fwd", TORCH_FN(joint_fwd));
  m.impl("joint_bwd", TORCH_FN(joint_bwd_entry));
  m.impl("joint_metadata", TORCH_FN(joint_metadata));
  m.impl("conv_split_act_fwd", TORCH_FN(conv_fwd));
  m.impl("conv_split_act_bwd", TORCH_FN(conv_bwd));
  m.impl("conv_split_norm_fwd", TORCH_FN(norm_fwd));
  m.impl("conv_split_norm_bwd", TORCH_FN(norm_bwd));
}

TORCH_LIBRARY_IMPL(tgdn_b200, Autograd, m) {
  m.impl("joint_fwd", TORCH_FN(joint_fwd_autograd));
  m.impl("conv_split_act_fwd", TORCH_FN(conv_fwd_autograd));
  m.impl("conv_split_norm_fwd", TORCH_FN(norm_fwd_autograd));
  m.impl("joint_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("conv_split_act_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("conv_split_norm_bwd", torch::autograd::autogradNotImplementedFallback());
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const AssertFail& e) {
      set_python_error(e);
    } catch (const LibraryFail& e) {
      set_python_error(e);
    }
  });
  m.def("set_library_error", [](py::object cls) { library_error = cls.release(); });
  const py::call_guard<py::gil_scoped_release> nogil;     // nothing below touches Python objects
  m.def("joint_call", &joint_call, nogil);
  m.def("chunk_joint", &chunk_joint, nogil);
  m.def("joint_segment", &joint_segment, nogil);
  m.def("decode", &decode, nogil);
  m.def("conv_call", &call_conv_fwd, nogil);
  m.def("conv_norm_call", &call_norm_fwd, nogil);
  m.def("prepare_documents", &prepare_documents, nogil);
  // the stages one by one, with every optional argument given
  m.def("run_masks", [](const Tensor& q, const Tensor& k, const Tensor& k2, const Tensor& q2, const Tensor& g, const Tensor& beta,
                        double scale, const OptTensor& token_map) {
    Masks r = run_masks(q, k, k2, q2, g, beta, scale, token_map);
    return std::make_tuple(r.gc, r.AP, r.Pm);
  }, nogil);
  m.def("run_forward", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k2, const Tensor& q2, const Tensor& beta,
                          const Tensor& gc, const Tensor& AP, double scale, bool save, const OptTensor& chunk_starts,
                          const OptTensor& token_map, const OptTensor& state_in, const OptTensor& state_out) {
    Forward r = run_forward(q, k, v, k2, q2, beta, gc, AP, scale, save, chunk_starts, token_map, state_in, state_out);
    return std::make_tuple(r.o, or_nullopt(r.h), or_nullopt(r.W), or_nullopt(r.U));
  }, nogil);
  m.def("run_reverse", [](const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& k2, const Tensor& q2, const Tensor& beta,
                          const Tensor& gc, const Tensor& AP, const Tensor& Pm, const Tensor& U, double scale,
                          const OptTensor& chunk_starts, const OptTensor& token_map, const OptTensor& g_in, const OptTensor& g_out) {
    Reverse r = run_reverse(q, k, dO, k2, q2, beta, gc, AP, Pm, U, scale, chunk_starts, token_map, g_in, g_out);
    return std::make_tuple(r.dV, r.dU, r.ds, r.dkg, r.dr);
  }, nogil);
  m.def("run_state_grads", [](const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& dV, const Tensor& h, const Tensor& ds,
                              const Tensor& dkg, const Tensor& k2, const Tensor& q2, const Tensor& gc, double scale,
                              const OptTensor& token_map) {
    StateGrads r = run_state_grads(q, k, dO, dV, h, ds, dkg, k2, q2, gc, scale, token_map);
    return std::make_tuple(r.dkq, r.da, r.dc, r.dd);
  }, nogil);
  m.def("run_matrix", [](const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& dU, const Tensor& W, const Tensor& U,
                         const Tensor& AP, const Tensor& k2, const Tensor& q2, const Tensor& beta, const Tensor& gc, const Tensor& dkq,
                         const Tensor& da, const Tensor& dc, const Tensor& dd, const Tensor& dr, double scale, const OptTensor& token_map) {
    Grads out = Grads::like(q, k2, beta);
    run_matrix(q, k, dO, dU, W, U, AP, k2, q2, beta, gc, StateGrads{dkq, da, dc, dd}, dr, scale, token_map, out);
    return std::make_tuple(out.q, out.k, out.k2, out.q2, out.g, out.beta);
  }, nogil);
  m.def("run_grads", [](const Tensor& q, const Tensor& k, const Tensor& dO, const Tensor& dV, const Tensor& dU, const Tensor& ds,
                        const Tensor& dkg, const Tensor& dr, const Tensor& h, const Tensor& W, const Tensor& U, const Tensor& AP,
                        const Tensor& k2, const Tensor& q2, const Tensor& beta, const Tensor& gc, double scale, const OptTensor& token_map,
                        const OptTensor& next_item) {
    Grads out = Grads::like(q, k2, beta);
    out.v = dV;
    run_grads(q, k, dO, dU, ds, dkg, dr, h, W, U, AP, k2, q2, beta, gc, scale, token_map,
              next_item.has_value() ? *next_item : at::zeros({1}, q.options().dtype(at::kInt)), out);
    return std::make_tuple(out.q, out.k, out.k2, out.q2, out.g, out.beta);
  }, nogil);
}
