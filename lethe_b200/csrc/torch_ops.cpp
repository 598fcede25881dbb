// The PyTorch side of the op in native code: argument preparation, allocation, the autograd node and the calls of the
// C library (include/lethe_gdn.h).  ops.py keeps the public functions; each of them is one call into this module.
//
// Why native: a forward + backward through Python (argument checks, some fifteen tensor allocations, two ctypes structs,
// the autograd function's own bookkeeping, a status word copied back to the host per call) cost about 0.4 ms of host
// time per step, against 0.14 ms of kernels at B=2, H=8, L=2048; a decode step 24 us against 3 us.  Here the backward
// also runs on the autograd engine's thread without the interpreter lock.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/extension.h>

#include <mutex>
#include <string>
#include <vector>

#include "../../include/lethe_gdn.h"

namespace {

using at::Tensor;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

constexpr int kMaxDevices = 64;

// ---------------------------------------------------------------------------------------------
// errors: lethe_b200.ops.GdnError, from threads with and without the interpreter lock
// ---------------------------------------------------------------------------------------------
PyObject* g_error_type = nullptr;

[[noreturn]] void fail(const std::string& msg, PyObject* type = g_error_type) {
  python_error e;
  {
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(type ? type : PyExc_RuntimeError, ("lethe_gdn: " + msg).c_str());
    e.persist();
  }
  throw e;
}
void check(int rc) {
  if (rc != 0) fail(std::string(lethe_gdn_strerror(rc)) + " (code " + std::to_string(rc) + ")");
}
// what a bound function throws has to be a Python error while the interpreter lock is held
template <typename F>
auto guarded(F&& f) -> decltype(f()) {
  try {
    return f();
  } catch (python_error& e) {
    e.restore();
    throw pybind11::error_already_set();
  }
}

// ---------------------------------------------------------------------------------------------
// Status words.  A device-side wait that gives up writes its code through `status` (host memory the GPU can write to,
// one word per device): nothing is copied, no event is recorded, and the host reads it at every later call.  An error
// therefore surfaces at a later call, as any asynchronous error does; the word is cleared when it has been reported.
// ---------------------------------------------------------------------------------------------
struct HostWords {
  volatile int32_t* status = nullptr;      // [kMaxDevices]
};
HostWords& host_words() {
  static HostWords w = [] {
    HostWords h;
    void* p = nullptr;
    if (cudaHostAlloc(&p, kMaxDevices * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess)
      fail("no pinned host memory for the status words");
    memset(p, 0, kMaxDevices * sizeof(int32_t));
    h.status = static_cast<volatile int32_t*>(p);
    return h;
  }();
  return w;
}
int32_t* status_word(int dev) {
  TORCH_CHECK(dev >= 0 && dev < kMaxDevices);
  volatile int32_t* w = host_words().status + dev;
  const int32_t code = *w;
  if (code != 0) {
    *w = 0;
    fail("a device-side wait of an earlier call timed out at site " + std::to_string(code) +
         "; the results of that call are invalid");
  }
  return const_cast<int32_t*>(w);
}

// ---------------------------------------------------------------------------------------------
// tensors
// ---------------------------------------------------------------------------------------------
// memory that does not hold the values: a negated view, a tensor of zeros without storage
bool lazy(const Tensor& t) { return t.is_neg() || t._is_zerotensor(); }
Tensor as(const Tensor& t, at::ScalarType dt) {
  if (t.scalar_type() != dt) return t.to(dt).contiguous();      // (writes them out)
  return lazy(t) ? t.clone().contiguous() : t.contiguous();
}
Tensor as32(const Tensor& t) { return t.defined() ? as(t, at::kFloat) : t; }
// a gate per channel is read through a tensor map, which wants its start on a 16-byte boundary
Tensor as_gate(const Tensor& t) {
  const Tensor r = as32(t);
  return r.defined() && (reinterpret_cast<uintptr_t>(r.data_ptr()) & 15) ? r.clone() : r;
}
Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
Tensor cast_back(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }
template <typename T = void>
T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

// Byte buffer for a workspace.  The library wants its start on a 1024-byte boundary, the allocator gives 512: the tensor
// is cut to the part that begins there.
constexpr int64_t kWorkspaceAlign = 1024;
bool workspace_aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % kWorkspaceAlign == 0; }
Tensor workspace(size_t bytes, const at::TensorOptions& o) {
  const int64_t n = static_cast<int64_t>(bytes);
  Tensor t = at::empty({n + kWorkspaceAlign}, o.dtype(at::kByte));
  const auto past = static_cast<int64_t>(reinterpret_cast<uintptr_t>(t.data_ptr()) % kWorkspaceAlign);
  t.unsafeGetTensorImpl()->set_storage_offset(past ? kWorkspaceAlign - past : 0);
  t.unsafeGetTensorImpl()->set_sizes_contiguous({n});
  return t;
}

// q and k as the normalisation kernels read them: as they are when both are bf16, fp32 or fp16, else both as fp32.
int l2_inputs(const Tensor& q, const Tensor& k, Tensor* qc, Tensor* kc) {
  const auto dt = q.scalar_type();
  const bool same = k.scalar_type() == dt && (dt == at::kBFloat16 || dt == at::kHalf || dt == at::kFloat);
  *qc = as(q, same ? dt : at::kFloat);
  *kc = as(k, same ? dt : at::kFloat);
  const auto in = qc->scalar_type();
  return in == at::kFloat ? LETHE_L2_IN_F32 : in == at::kHalf ? LETHE_L2_IN_F16 : 0;
}
constexpr float kL2Eps = 1e-6f;

cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// bf16 <-> fp32 by a kernel of the library, where `t` is that in one piece (Tensor::to costs the host three times a launch)
bool converts(const Tensor& t, at::ScalarType from) {
  return t.scalar_type() == from && t.is_contiguous() && !lazy(t) && t.numel() > 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}
Tensor to_f32(const Tensor& t) {
  Tensor r = at::empty(t.sizes(), t.options().dtype(at::kFloat));
  check(lethe_gdn_convert(t.data_ptr(), r.data_ptr(), t.numel(), 1, stream_of(t)));
  return r;
}

// ---------------------------------------------------------------------------------------------
// The chunked op.  One description serves every surface: g per row, per channel or absent; beta, or the erase / write
// gates b, w of the full op; L2 normalisation of q, k inside; and the six-input surface, whose per-channel gates have
// been compacted to one value per row and whose gradients are spread back.
// ---------------------------------------------------------------------------------------------
enum Slot { kQ, kKey, kV, kG, kBeta, kH0, kB, kW, kSlots };

struct Problem {
  int64_t B = 0, L = 0, H = 0, K = 0, V = 0;
  int gate = LETHE_GATE_NONE, delta = 0;
  float scale = 1.f;
  bool l2 = false;
  LetheGdnDims dims() const {
    LetheGdnDims d;
    d.B = static_cast<int32_t>(B); d.H = static_cast<int32_t>(H); d.L = static_cast<int32_t>((L + 63) / 64 * 64);
    d.K = 128; d.V = static_cast<int32_t>(V); d.gate = gate; d.delta = delta;
    return d;
  }
};

// What both directions hand to the library.
struct Operands {
  Tensor q, k, v, g, beta, h0, b, w;      // q, k bf16 or fp16; v bf16; the rest fp32
  bool raw = false;                       // q, k are still to be normalised, by the forward's first kernel
};

LetheGdnArgs base_args(const Problem& p, const Operands& x, void* saved, size_t saved_bytes) {
  LetheGdnArgs a;
  memset(&a, 0, sizeof(a));
  a.dims = p.dims();
  a.l_tokens = static_cast<uint32_t>(p.L);
  a.k_channels = static_cast<uint32_t>(p.K);
  a.scale = p.scale;
  a.q = ptr(x.q); a.k = ptr(x.k); a.v = ptr(x.v);
  a.g = ptr<float>(x.g); a.beta = ptr<float>(x.beta); a.h0 = ptr<float>(x.h0);
  a.b_gate = ptr<float>(x.b); a.w_gate = ptr<float>(x.w);
  a.saved = saved;
  a.saved_bytes = saved_bytes;
  a.status = status_word(x.q.device().index());
  a.lean = 1u;
  a.qk_f16 = x.q.scalar_type() == at::kHalf ? 1u : 0u;
  return a;
}

// What a backward needs for itself, by how long: the library's scratch and the converted gradient of o until its kernels are launched,
// the gradients of normalised rows until their VJP is, the rest until the results are made.  One allocation for all of it where that is
// small (an allocation costs the host a microsecond), one for each otherwise, given back when it is done with: a call of hundreds
// of megabytes then peaks no higher than its scratch and its results ask for.  Pieces on 1024-byte boundaries.
class Slab {
 public:
  enum Until { kKernels, kRows, kEnd, kGroups };
  struct Piece {
    Until until = kEnd;
    size_t at = 0;
  };
  Piece piece(Until until, size_t n) {
    const Piece p{until, bytes_[until]};
    bytes_[until] += (n + 1023) / 1024 * 1024;
    return p;
  }
  void make(const at::TensorOptions& o) {
    const size_t all = bytes_[kKernels] + bytes_[kRows] + bytes_[kEnd];
    if (all <= kOne) {
      t_[kKernels] = workspace(all, o);
      char* base = static_cast<char*>(t_[kKernels].data_ptr());
      for (int i = 0; i < kGroups; base += bytes_[i++]) base_[i] = base;
      return;
    }
    for (int i = 0; i < kGroups; ++i) {
      if (!bytes_[i]) continue;
      t_[i] = workspace(bytes_[i], o);
      base_[i] = static_cast<char*>(t_[i].data_ptr());
      own_ = true;
    }
  }
  void* at(const Piece& p) const { return base_[p.until] + p.at; }
  // what was for `until` is done with: on this stream, whose later kernels write it behind those that read it
  void drop(Until until) {
    if (own_) t_[until].reset();
  }

 private:
  static constexpr size_t kOne = 16u << 20;
  size_t bytes_[kGroups] = {};
  char* base_[kGroups] = {};
  Tensor t_[kGroups];
  bool own_ = false;
};

struct Forward {
  Tensor o, hT;
  Operands x;
  Tensor saved;
};

// `keep`: a backward follows, which reads the normalised rows.  `state`: the final state is wanted
Forward run_forward(const Problem& p, Operands x, bool keep, bool state) {
  Forward f;
  const LetheGdnDims d = p.dims();
  const size_t need = lethe_gdn_saved_bytes(&d);
  if (need == 0)
    fail("unsupported sizes B=" + std::to_string(p.B) + " H=" + std::to_string(p.H) + " L=" + std::to_string(p.L) +
         " K=" + std::to_string(p.K) + " V=" + std::to_string(p.V) + " (need V = 64 or 128, and at least one of B, H, L)");
  const auto o16 = x.v.options();
  const auto o32 = o16.dtype(at::kFloat);
  f.saved = workspace(need, o16);
  f.o = at::empty({p.B, p.L, p.H, p.V}, o16);
  if (state) f.hT = at::empty({p.B, p.H, p.K, p.V}, o32);
  LetheGdnArgs a = base_args(p, x, f.saved.data_ptr(), need);
  a.o = ptr(f.o);
  a.hT = ptr<float>(f.hT);
  if (!keep) a.lean = 2u;
  Tensor qn, kn;
  if (x.raw) {
    a.l2_eps = kL2Eps;
    if (keep || p.gate != LETHE_GATE_CHANNEL) {      // (with one decay or none the output kernel reads q, too)
      qn = at::empty(x.q.sizes(), o16.dtype(at::kHalf));
      a.q_norm = ptr(qn);
    }
    if (keep) {
      kn = at::empty(x.k.sizes(), o16.dtype(at::kHalf));
      a.k_norm = ptr(kn);
    }
  }
  check(lethe_gdn_forward(&a, stream_of(x.q)));
  if (keep && qn.defined()) {
    x.q = qn;
    x.k = kn;
    x.raw = false;
  }
  f.x = std::move(x);
  return f;
}

// Tensors for what the caller gets; pointers into `slab` for what is worked on further (or to the tensors).
struct Grads {
  Tensor dq, dk, dv, dg, dbeta, dh0, db, dw;
  Slab slab;
  void *p_dq = nullptr, *p_dk = nullptr, *p_dv = nullptr;
  float *p_dg = nullptr, *p_dbeta = nullptr, *p_dbeta_w = nullptr;
};

// `spread`: gate gradients per row are to be spread over the channels.  `dv32`: dv is to be fp32
Grads run_backward(const Problem& p, const Operands& x, const Tensor& saved, const Tensor& d_o_in, const Tensor& dhT, bool spread,
                   bool dv32) {
  Grads r;
  const LetheGdnDims d = p.dims();
  const auto bytes = [](const Tensor& t) { return static_cast<size_t>(t.numel()) * t.element_size(); };
  const size_t need = lethe_gdn_scratch_bytes(&d), o_bytes = bytes(x.v);
  const bool cast_do = d_o_in.defined() && converts(d_o_in, at::kFloat), one = x.beta.defined() && p.delta == 1;
  const bool row_g = spread && p.gate == LETHE_GATE_SCALAR;
  Slab& s = r.slab;
  using P = Slab::Piece;
  const P scratch = s.piece(Slab::kKernels, need);
  const P at_do = cast_do ? s.piece(Slab::kKernels, o_bytes) : P();
  const P at_dq = p.l2 ? s.piece(Slab::kRows, bytes(x.q)) : P(), at_dk = p.l2 ? s.piece(Slab::kRows, bytes(x.k)) : P();
  const P at_dv = dv32 ? s.piece(Slab::kEnd, o_bytes) : P(), at_dg = row_g ? s.piece(Slab::kEnd, bytes(x.g)) : P();
  const bool rows_b = spread && one;
  const P at_db = rows_b ? s.piece(Slab::kEnd, bytes(x.beta)) : P(), at_dw = rows_b ? s.piece(Slab::kEnd, bytes(x.beta)) : P();
  s.make(x.v.options());
  auto place = [&](Tensor& t, const Tensor& like, bool inside, const P& at) -> void* {
    if (inside) return s.at(at);
    t = at::empty_like(like);
    return t.data_ptr();
  };
  r.p_dq = place(r.dq, x.q, p.l2, at_dq);
  r.p_dk = place(r.dk, x.k, p.l2, at_dk);
  r.p_dv = place(r.dv, x.v, dv32, at_dv);
  if (x.g.defined()) r.p_dg = static_cast<float*>(place(r.dg, x.g, row_g, at_dg));
  if (one) r.p_dbeta = static_cast<float*>(place(r.dbeta, x.beta, spread, at_db));
  if (one && spread) r.p_dbeta_w = static_cast<float*>(s.at(at_dw));
  if (x.h0.defined()) r.dh0 = at::empty_like(x.h0);
  LetheGdnArgs a = base_args(p, x, saved.data_ptr(), static_cast<size_t>(saved.numel()));
  if (p.delta == 2) {
    r.db = at::empty_like(x.b);
    r.dw = at::empty_like(x.w);
  }
  Tensor d_o;
  if (cast_do) {
    check(lethe_gdn_convert(d_o_in.data_ptr(), s.at(at_do), d_o_in.numel(), 0, stream_of(x.q)));
    a.d_o = s.at(at_do);
  } else {
    d_o = d_o_in.defined() ? as(d_o_in, at::kBFloat16) : at::zeros({p.B, p.L, p.H, p.V}, x.v.options());
    a.d_o = ptr(d_o);
  }
  a.dhT = ptr<float>(dhT);
  a.dq = r.p_dq; a.dk = r.p_dk; a.dv = r.p_dv; a.dg = r.p_dg; a.dh0 = ptr<float>(r.dh0);
  a.dbeta = r.p_dbeta; a.dbeta_write = r.p_dbeta_w;
  a.db_gate = ptr<float>(r.db); a.dw_gate = ptr<float>(r.dw);
  a.scratch = s.at(scratch);
  a.scratch_bytes = need;
  check(lethe_gdn_backward(&a, stream_of(x.q)));
  s.drop(Slab::kKernels);
  return r;
}

// The autograd node.  First order only: a second derivative runs into the error node that wraps the gradients.
struct GdnBackward : public torch::autograd::Node {
  Problem p;
  bool six = false;                        // gates came per channel: gradients go back per channel
  torch::autograd::SavedVariable q_in, k_in;            // inputs of the normalisation
  torch::autograd::SavedVariable q, k, v, g, beta, h0, b, w;
  torch::autograd::SavedVariable saved;    // the workspace, most of what is kept: hooks that move or recompute it see it
  at::ScalarType dtypes[kSlots];
  bool released = false;

  std::string name() const override { return "GdnBackward"; }
  void release_variables() override {
    for (auto* s : {&q_in, &k_in, &q, &k, &v, &g, &beta, &h0, &b, &w, &saved}) s->reset_data();
    released = true;
  }
  variable_list apply(variable_list&& grads) override {
    const bool second = torch::autograd::GradMode::is_enabled() &&
                        ((grads[0].defined() && grads[0].requires_grad()) ||
                         (grads.size() > 1 && grads[1].defined() && grads[1].requires_grad()));
    variable_list out;
    {
      at::NoGradGuard no_grad;
      out = first_order(grads[0], grads.size() > 1 ? grads[1] : Tensor());
    }
    if (!second) return out;
    for (auto& t : out)
      if (t.defined()) t = t.detach().requires_grad_(true);
    auto err = std::make_shared<torch::autograd::DelayedError>(
        "trying to differentiate twice a function that was marked with @once_differentiable", static_cast<int64_t>(out.size()));
    return (*err)(std::move(out));
  }

  variable_list first_order(const Tensor& d_o_in, const Tensor& dhT_in) {
    variable_list out(kSlots);
    if (!d_o_in.defined() && !dhT_in.defined()) return out;
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    auto self = getptr();
    Operands x{q.unpack(self), k.unpack(self), v.unpack(self), g.unpack(self), beta.unpack(self), h0.unpack(self),
               b.unpack(self), w.unpack(self)};
    c10::cuda::CUDAGuard guard(x.q.device());
    Tensor ws = saved.unpack(self);
    if (!workspace_aligned(ws)) {            // a hook brought it back somewhere else
      Tensor t = workspace(static_cast<size_t>(ws.numel()), ws.options());
      ws = t.copy_(ws);
    }
    const Tensor dhT = as32(dhT_in);
    // the raw rows come back before the backward is launched: older than its last kernel, unless they are converted below
    const Tensor q_raw = p.l2 ? q_in.unpack(self) : Tensor(), k_raw = p.l2 ? k_in.unpack(self) : Tensor();
    const bool rows = six && p.delta != 2, dv32 = dtypes[kV] == at::kFloat && task_should_compute_output(kV);
    Grads r = run_backward(p, x, ws, d_o_in, dhT, rows, dv32);
    if (p.l2) {     // VJP of x / sqrt(|x|^2 + eps) (the reference gets it by autograd, gdn2_assemble.py:300-312)
      Tensor qc, kc;
      int flags = l2_inputs(q_raw, k_raw, &qc, &kc) | LETHE_L2_NORM_F16;
      if (qc.data_ptr() == q_raw.data_ptr() && kc.data_ptr() == k_raw.data_ptr()) flags |= LETHE_L2_EARLY;
      Tensor dq = at::empty_like(qc), dk = at::empty_like(kc);
      check(lethe_gdn_l2norm_qk_vjp(qc.data_ptr(), kc.data_ptr(), r.p_dq, r.p_dk, dq.data_ptr(), dk.data_ptr(),
                                     qc.numel() / p.K, static_cast<int32_t>(p.K), flags, kL2Eps, stream_of(qc)));
      r.slab.drop(Slab::kRows);
      r.dq = dq;
      r.dk = dk;
    }
    if (rows) spread(x, &r);
    if (dv32) {
      r.dv = at::empty(x.v.sizes(), x.v.options().dtype(at::kFloat));
      check(lethe_gdn_convert(r.p_dv, r.dv.data_ptr(), r.dv.numel(), 1, stream_of(x.v)));
    }
    const Tensor got[kSlots] = {r.dq, r.dk, r.dv, r.dg, r.dbeta, r.dh0, r.db, r.dw};
    for (int i = 0; i < kSlots; ++i)
      if (got[i].defined() && task_should_compute_output(i)) out[i] = cast_back(got[i], dtypes[i]);
    return out;
  }

  // per-row gate gradients of the six-input surface, spread evenly over the channels
  void spread(const Operands& x, Grads* r) {
    const auto o32 = x.v.options().dtype(at::kFloat);
    Tensor dg, db, dw;
    if (p.gate == LETHE_GATE_SCALAR && task_should_compute_output(kG)) dg = at::empty({p.B, p.L, p.H, p.K}, o32);
    if (task_should_compute_output(kB)) db = at::empty({p.B, p.L, p.H, p.K}, o32);
    if (task_should_compute_output(kW)) dw = at::empty({p.B, p.L, p.H, p.V}, o32);
    if (dg.defined() || db.defined() || dw.defined())
      check(lethe_gdn_gate_spread(p.gate == LETHE_GATE_SCALAR ? r->p_dg : nullptr, r->p_dbeta, r->p_dbeta_w, p.B * p.L * p.H,
                                  static_cast<int32_t>(p.K), static_cast<int32_t>(p.V), ptr<float>(dg), ptr<float>(db),
                                  ptr<float>(dw), stream_of(x.q)));
    if (p.gate == LETHE_GATE_SCALAR) r->dg = dg;
    r->db = db;
    r->dw = dw;
    r->dbeta = Tensor();
  }
};

// Runs the forward and, when something asks for gradients, hangs the node on the results.
std::pair<Tensor, Tensor> apply(const Problem& p, const Tensor (&in)[kSlots], Operands x, bool six) {
  for (const Tensor& t : in)      // (the kernels would return the value without its tangent)
    if (t.defined() && t._fw_grad(/*level=*/0).defined())
      fail("forward-mode differentiation is not implemented", PyExc_NotImplementedError);
  bool need = false;
  if (torch::autograd::GradMode::is_enabled())
    for (const Tensor& t : in) need = need || (t.defined() && t.requires_grad());
  Forward f;
  {
    at::NoGradGuard no_grad;
    f = run_forward(p, std::move(x), need, !six);
    f.o = in[kV].scalar_type() == at::kFloat ? to_f32(f.o) : cast_back(f.o, in[kV].scalar_type());
  }
  if (need) {
    std::shared_ptr<GdnBackward> node(new GdnBackward(), torch::autograd::deleteNode);
    node->p = p;
    node->six = six;
    node->set_next_edges(torch::autograd::collect_next_edges(in[0], in[1], in[2], in[3], in[4], in[5], in[6], in[7]));
    for (int i = 0; i < kSlots; ++i) node->dtypes[i] = in[i].defined() ? in[i].scalar_type() : at::kFloat;
    using torch::autograd::SavedVariable;
    if (p.l2) {
      node->q_in = SavedVariable(in[kQ], false);
      node->k_in = SavedVariable(in[kKey], false);
    }
    node->q = SavedVariable(f.x.q, false);
    node->k = SavedVariable(f.x.k, false);
    node->v = SavedVariable(f.x.v, false);
    node->g = SavedVariable(f.x.g, false);
    node->beta = SavedVariable(f.x.beta, false);
    node->h0 = SavedVariable(f.x.h0, false);
    node->b = SavedVariable(f.x.b, false);
    node->w = SavedVariable(f.x.w, false);
    node->saved = SavedVariable(f.saved, false);
    torch::autograd::set_history(f.o, node);
    if (f.hT.defined()) torch::autograd::set_history(f.hT, node);
  }
  return {f.o, f.hT};
}

void need_shape(bool ok, const char* what) {
  if (!ok) fail(std::string("shapes do not match: ") + what);
}
// a pointer from somewhere else would fault in a kernel
template <typename... T>
void need_device(const Tensor& like, const T&... ts) {
  auto one = [&](const Tensor& t) {
    if (t.defined() && t.device() != like.device())
      fail("all inputs must live on one CUDA device (" + like.device().str() + " and " + t.device().str() + ")");
  };
  (one(ts), ...);
}

Problem describe(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool l2) {
  if (!q.is_cuda()) fail("inputs must live on a CUDA device (there is no CPU path)");
  need_shape(q.dim() == 4 && v.dim() == 4 && k.sizes() == q.sizes() && v.sizes().slice(0, 3) == q.sizes().slice(0, 3),
             "q, k [B, L, H, K], v [B, L, H, V]");
  Problem p;
  p.B = q.size(0); p.L = q.size(1); p.H = q.size(2); p.K = q.size(3); p.V = v.size(3);
  p.scale = static_cast<float>(scale);
  p.l2 = l2;
  if (p.K != 64 && p.K != 128) fail("unsupported sizes K=" + std::to_string(p.K) + " (need K = 64 or 128)");
  return p;
}

// q and k as the kernels read them: normalised rows in fp16 (rounded once from fp32), fp16 when both came as fp16,
// bf16 otherwise
// `fuse`: the prepare kernel may normalise 16-bit rows itself
void prepare_qk(const Problem& p, const Tensor& q, const Tensor& k, Operands* x, bool fuse = false) {
  if (p.l2) {
    Tensor qc, kc;
    const int flags = l2_inputs(q, k, &qc, &kc) | LETHE_L2_NORM_F16;
    if (fuse && !(flags & LETHE_L2_IN_F32)) {
      x->q = qc;
      x->k = kc;
      x->raw = true;
      return;
    }
    x->q = at::empty(qc.sizes(), qc.options().dtype(at::kHalf));
    x->k = at::empty(kc.sizes(), kc.options().dtype(at::kHalf));
    check(lethe_gdn_l2norm_qk(qc.data_ptr(), kc.data_ptr(), x->q.data_ptr(), x->k.data_ptr(), qc.numel() / p.K,
                              static_cast<int32_t>(p.K), flags, kL2Eps, stream_of(qc)));
  } else if (q.scalar_type() == at::kHalf && k.scalar_type() == at::kHalf) {
    x->q = as(q, at::kHalf);
    x->k = as(k, at::kHalf);
  } else {
    x->q = as(q, at::kBFloat16);
    x->k = as(k, at::kBFloat16);
  }
}

void check_gate(const Problem& p, const Tensor& g) {
  if (!g.defined()) return;
  need_shape((g.dim() == 3 || (g.dim() == 4 && g.size(3) == p.K)) && g.size(0) == p.B && g.size(1) == p.L && g.size(2) == p.H,
             "g [B, L, H] or [B, L, H, K]");
}
void check_state(const Problem& p, const Tensor& h0) {
  if (h0.defined()) need_shape(h0.sizes() == at::IntArrayRef({p.B, p.H, p.K, p.V}), "h0 [B, H, K, V]");
}

std::pair<Tensor, Tensor> chunk(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& g_, const OptTensor& beta_,
                                const OptTensor& h0_, double scale, bool l2) {
  return guarded([&] {
    const Tensor g = opt(g_), beta = opt(beta_), h0 = opt(h0_);
    Problem p = describe(q, k, v, scale, l2);
    need_device(q, k, v, g, beta, h0);
    check_gate(p, g);
    check_state(p, h0);
    if (beta.defined()) need_shape(beta.sizes() == q.sizes().slice(0, 3), "beta [B, L, H]");
    c10::cuda::CUDAGuard guard(q.device());
    p.gate = !g.defined() ? LETHE_GATE_NONE : g.dim() == 3 ? LETHE_GATE_SCALAR : LETHE_GATE_CHANNEL;
    p.delta = beta.defined() ? 1 : 0;
    Operands x;
    {
      at::NoGradGuard no_grad;
      prepare_qk(p, q, k, &x, true);
      x.v = as(v, at::kBFloat16);
      x.g = as_gate(g); x.beta = as32(beta); x.h0 = as32(h0);
    }
    return apply(p, {q, k, v, g, beta, h0, Tensor(), Tensor()}, std::move(x), false);
  });
}

// independent per-channel erase and write gates
std::pair<Tensor, Tensor> full_with(Problem p, Operands x, const Tensor (&in)[kSlots], bool six) {
  if (p.K != 128 || p.L % 64) fail("the full-gate op needs d_k = 128 and L a multiple of 64");
  p.gate = LETHE_GATE_CHANNEL;
  p.delta = 2;
  {
    at::NoGradGuard no_grad;
    if (!x.q.defined()) prepare_qk(p, in[kQ], in[kKey], &x, true);
    x.v = as(in[kV], at::kBFloat16);
    x.g = as_gate(in[kG]); x.b = as32(in[kB]); x.w = as32(in[kW]); x.h0 = as32(in[kH0]);
  }
  return apply(p, in, std::move(x), six);
}
void check_channel_gates(const Problem& p, const Tensor& q, const Tensor& v, const Tensor& g, const Tensor& b, const Tensor& w) {
  need_shape(g.sizes() == q.sizes() && b.sizes() == q.sizes() && w.sizes() == v.sizes(), "g, b [B, L, H, K], w [B, L, H, V]");
}
std::pair<Tensor, Tensor> chunk_full(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& b,
                                     const Tensor& w, const OptTensor& h0_, double scale, bool l2) {
  return guarded([&] {
    const Tensor h0 = opt(h0_);
    const Problem p = describe(q, k, v, scale, l2);
    need_device(q, k, v, g, b, w, h0);
    check_channel_gates(p, q, v, g, b, w);
    check_state(p, h0);
    c10::cuda::CUDAGuard guard(q.device());
    return full_with(p, Operands(), {q, k, v, g, Tensor(), h0, b, w}, false);
  });
}

// ---------------------------------------------------------------------------------------------
// Which kernels a six-input call needs.  The verdict has to reach the host, because it decides what is launched; it
// comes through a mapped host word that the test kernel writes, so the host waits for that kernel only and what else
// the call can enqueue meanwhile (the normalisation) runs behind it.  A slot (host word + 8 bytes of device memory) is
// taken for the time of one call and given back: there are never more slots than calls that were in flight at once.
// ---------------------------------------------------------------------------------------------
struct RegimeSlot {
  volatile uint32_t* word = nullptr;
  uint32_t* work = nullptr;
};
struct RegimePool {
  std::mutex mu;
  std::vector<RegimeSlot> free[kMaxDevices];
  int made = 0;
  RegimeSlot take(int dev) {
    {
      std::lock_guard<std::mutex> lock(mu);
      if (!free[dev].empty()) {
        RegimeSlot s = free[dev].back();
        free[dev].pop_back();
        return s;
      }
    }
    RegimeSlot s;
    void *h = nullptr, *d = nullptr;
    if (cudaHostAlloc(&h, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess ||
        cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) {
      cudaFree(d);
      cudaFreeHost(h);
      fail("no memory for the gate test");
    }
    s.word = static_cast<volatile uint32_t*>(h);
    s.work = static_cast<uint32_t*>(d);
    std::lock_guard<std::mutex> lock(mu);
    ++made;
    return s;
  }
  void give(int dev, RegimeSlot s) {
    std::lock_guard<std::mutex> lock(mu);
    free[dev].push_back(s);
  }
  std::pair<int, int> count() {      // slots made, slots free
    std::lock_guard<std::mutex> lock(mu);
    size_t n = 0;
    for (const auto& f : free) n += f.size();
    return {made, static_cast<int>(n)};
  }
};
RegimePool& regime_pool() {
  static RegimePool* pool = new RegimePool();     // outlives the interpreter's own teardown
  return *pool;
}

// The gate test of one call: enqueue, then wait.  A call that fails in between waits as well: the slot goes back when the
// kernel that uses it is done.
struct RegimeTest {
  int dev;
  cudaStream_t st;
  RegimeSlot slot;
  bool pending = false;
  Tensor g0, b0;
  RegimeTest(const Tensor& g, const Tensor& b, const Tensor& w) : dev(g.device().index()), st(stream_of(g)) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
      fail("the gate test of a six-input call reads its result on the host and cannot be captured into a graph");
    g0 = at::empty(g.sizes().slice(0, 3), g.options());
    b0 = at::empty_like(g0);
    slot = regime_pool().take(dev);
    *slot.word = 0;
    const int rc = lethe_gdn_gate_regime(ptr<float>(g), ptr<float>(b), ptr<float>(w), g0.numel(), static_cast<int32_t>(g.size(3)),
                                         static_cast<int32_t>(w.size(3)), ptr<float>(g0), ptr<float>(b0),
                                         const_cast<uint32_t*>(slot.word), slot.work, st);
    if (rc != 0) regime_pool().give(dev, slot);      // nothing was launched
    check(rc);
    pending = true;
  }
  ~RegimeTest() {
    if (pending) finish();
  }
  uint32_t wait() {
    const uint32_t v = finish();
    if (!(v & LETHE_REGIME_DONE)) fail("the gate test did not complete");
    return v;
  }

 private:
  // the verdict, or 0 after a failed kernel, whose slot is not used again
  uint32_t finish() {
    uint32_t v = 0;
    pending = false;
    {
      pybind11::gil_scoped_release nogil;
      for (uint32_t n = 1; !((v = *slot.word) & LETHE_REGIME_DONE); ++n) {
        if (n % 4096) continue;
        const cudaError_t e = cudaStreamQuery(st);      // a failed kernel never writes the word
        if (e == cudaErrorNotReady) continue;
        if (e == cudaSuccess && (*slot.word & LETHE_REGIME_DONE)) continue;
        v = 0;
        break;
      }
    }
    if (v & LETHE_REGIME_DONE) regime_pool().give(dev, slot);
    return v;
  }
};

bool plain32(const Tensor& t) {
  return t.scalar_type() == at::kFloat && t.is_contiguous() && !lazy(t) && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}

// the same tests with library operations, for gates of other types or layouts
uint32_t regime_by_ops(const Tensor& g, const Tensor& b, const Tensor& w) {
  const Tensor bf = b.slice(3, 0, 1), wf = w.slice(3, 0, 1);
  const Tensor flags = at::stack({(g == g.slice(3, 0, 1)).all(),
                                  ((b == bf).all()).logical_and((w == wf).all()).logical_and((bf == wf).all()),
                                  (b == 0).all().logical_and((w == 1).all())}).cpu();
  const bool* f = flags.const_data_ptr<bool>();
  return (f[0] ? LETHE_REGIME_SCALAR_GATE : 0u) | (f[1] ? LETHE_REGIME_ONE_BETA : 0u) | (f[2] ? LETHE_REGIME_NO_DELTA : 0u);
}

uint32_t gate_regime(const Tensor& g, const Tensor& b, const Tensor& w) {
  return guarded([&]() -> uint32_t {
    at::NoGradGuard no_grad;
    need_device(g, b, w);
    const int64_t V = w.size(-1);
    if (!(g.is_cuda() && g.dim() == 4 && b.dim() == 4 && w.dim() == 4 && g.size(3) == 128 && (V == 64 || V == 128) &&
          g.sizes() == b.sizes() && plain32(g) && plain32(b) && plain32(w)))
      return regime_by_ops(g, b, w);
    c10::cuda::CUDAGuard guard(g.device());
    return RegimeTest(g, b, w).wait();
  });
}

Tensor six_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& b, const Tensor& w,
                  double scale, bool l2) {
  return guarded([&]() -> Tensor {
    Problem p = describe(q, k, v, scale, l2);
    if (p.K != 128) fail("gdn2_op needs d_k = 128 (use gdn_chunk for d_k = 64)");
    need_device(q, k, v, g, b, w);
    check_channel_gates(p, q, v, g, b, w);
    c10::cuda::CUDAGuard guard(q.device());
    const Tensor in[kSlots] = {q, k, v, g, Tensor(), Tensor(), b, w};
    Operands x;
    uint32_t regime;
    bool full = false;
    {
      at::NoGradGuard no_grad;
      if (plain32(g) && plain32(b) && plain32(w) && (p.V == 64 || p.V == 128)) {
        RegimeTest test(g, b, w);
        prepare_qk(p, q, k, &x);
        x.v = as(v, at::kBFloat16);
        regime = test.wait();
        x.g = test.g0;
        x.beta = test.b0;
      } else {
        regime = regime_by_ops(g, b, w);
        prepare_qk(p, q, k, &x);
        x.v = as(v, at::kBFloat16);
        x.g = as32(g.select(3, 0));
        x.beta = as32(b.select(3, 0));
      }
      const bool one_beta = regime & LETHE_REGIME_ONE_BETA;
      full = !one_beta && !(regime & LETHE_REGIME_NO_DELTA);
      if (full) x.g = x.beta = Tensor();
      p.delta = one_beta ? 1 : 0;
      if (!one_beta) x.beta = Tensor();
      p.gate = (regime & LETHE_REGIME_SCALAR_GATE) ? LETHE_GATE_SCALAR : LETHE_GATE_CHANNEL;
      if (!full && p.gate == LETHE_GATE_CHANNEL) x.g = as_gate(g);
    }
    return (full ? full_with(p, std::move(x), in, true) : apply(p, in, std::move(x), true)).first;
  });
}

// ---------------------------------------------------------------------------------------------
// One token
// ---------------------------------------------------------------------------------------------
Tensor decode_step(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& g_, const OptTensor& beta_,
                   const Tensor& state, double scale) {
  return guarded([&] {
    if (!state.is_cuda()) fail("inputs must live on a CUDA device (there is no CPU path)");
    if (state.scalar_type() != at::kFloat || !state.is_contiguous() || state.dim() != 4)
      fail("the decode state must be a contiguous fp32 tensor (it is updated in place)");
    at::NoGradGuard no_grad;
    const int64_t B = state.size(0), H = state.size(1), K = state.size(2), V = state.size(3);
    if (q.sizes() != at::IntArrayRef({B, H, K}) || k.sizes() != q.sizes() || v.sizes() != at::IntArrayRef({B, H, V}))
      fail("decode step expects q, k [B,H,K] and v [B,H,V] matching the state");
    const Tensor g_in = opt(g_), beta_in = opt(beta_);
    need_device(state, q, k, v, g_in, beta_in);
    const Tensor g = as32(g_in), beta = as32(beta_in);
    if (g.defined() && g.sizes() != at::IntArrayRef({B, H}) && g.sizes() != q.sizes())
      fail("decode step expects g [B,H] or [B,H,K]");
    if (beta.defined() && beta.sizes() != at::IntArrayRef({B, H})) fail("decode step expects beta [B,H]");
    c10::cuda::CUDAGuard guard(state.device());
    const bool f32 = q.scalar_type() == at::kFloat && k.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat;
    const at::ScalarType dt = f32 ? at::kFloat : at::kBFloat16;
    const Tensor qc = as(q, dt), kc = as(k, dt), vc = as(v, dt);
    Tensor o = at::empty({B, H, V}, state.options().dtype(at::kBFloat16));
    LetheGdnDecodeArgs a;
    memset(&a, 0, sizeof(a));
    a.B = static_cast<int32_t>(B); a.H = static_cast<int32_t>(H); a.K = static_cast<int32_t>(K); a.V = static_cast<int32_t>(V);
    a.gate = !g.defined() ? LETHE_GATE_NONE : g.dim() == 2 ? LETHE_GATE_SCALAR : LETHE_GATE_CHANNEL;
    a.delta = beta.defined() ? 1 : 0;
    a.scale = static_cast<float>(scale);
    a.q = ptr(qc); a.k = ptr(kc); a.v = ptr(vc);
    a.g = ptr<float>(g); a.beta = ptr<float>(beta);
    a.state = ptr<float>(state);
    a.o = ptr(o);
    a.in_f32 = f32 ? 1u : 0u;
    check(lethe_gdn_decode_step(&a, stream_of(state)));
    return o;
  });
}

}  // namespace

PYBIND11_MODULE(lethe_gdn_torch, m) {
  m.def("set_error_type", [](pybind11::object t) { g_error_type = t.release().ptr(); });
  m.def("chunk", &chunk);
  m.def("chunk_full", &chunk_full);
  m.def("six_inputs", &six_inputs);
  m.def("gate_regime", &gate_regime);
  m.def("status_address", [](int dev) {      // of a GPU's status word, for tests of what an expired wait leads to
    TORCH_CHECK(dev >= 0 && dev < kMaxDevices);
    return reinterpret_cast<uintptr_t>(host_words().status + dev);
  });
  m.def("gate_test_slots", [] { return regime_pool().count(); });
  m.def("decode_step", &decode_step);
}
