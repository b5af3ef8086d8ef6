// Host path of the operators as a CPython extension (b200gdn/_host*.so): argument checks, output and workspace tensors,
// autograd nodes and the calls into the C ABI of libb200gdn.so.  The kernels of a decoding step run for a few
// microseconds, so what such a call costs is this path: in Python (attribute look-ups, torch.autograd.Function, ctypes
// structures) it took 45-70 us a call and 180-300 us a forward + backward step, more than the kernels of every small
// problem; here a call costs about as much as its allocations and launches.
//
// Every entry point takes its arguments by position.  An argument combination that is not served (a shape error, an
// input that asks for the gradient of a forward-only operator, ...) returns NotImplemented BEFORE anything is launched;
// the Python wrapper then runs the checks that name the mistake.  Failures of a library call raise the package's error
// class, from the backward pass as well.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/custom_class.h>

#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/b200gdn.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

std::atomic<long long> g_launches{0};
PyObject* g_error_class = nullptr;   // B200GDNError

[[noreturn]] void raise(const std::string& msg) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(g_error_class ? g_error_class : PyExc_RuntimeError, msg.c_str());
  python_error e;
  e.persist();
  throw e;
}

template <typename Args>
void call(const char* name, int (*fn)(const Args*, void*), Args& a) {
  a.struct_bytes = (int32_t)sizeof(Args);
  const int rc = fn(&a, c10::cuda::getCurrentCUDAStream().stream());
  if (rc != 0) raise(std::string(name) + " failed (" + std::to_string(rc) + "): " + b200gdn_last_error());
  g_launches.fetch_add(b200gdn_last_launch_count(), std::memory_order_relaxed);
}

// ---- tensors ---------------------------------------------------------------------------------------------------
Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType t, const at::Device& dev) {
  return at::detail::empty_cuda(sizes, t, dev, std::nullopt);
}
Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType t, const at::Device& dev, bool zero) {
  Tensor x = new_tensor(sizes, t, dev);
  if (zero) x.zero_();
  return x;
}
// the tensor itself when it has that type, is contiguous and starts on the 16-byte boundary the kernels' copies need
Tensor dense(const Tensor& x) {
  if (!x.defined()) return x;
  const Tensor y = x.is_contiguous() ? x : x.contiguous();
  return (reinterpret_cast<uintptr_t>(y.data_ptr()) & 15) ? y.clone() : y;
}
Tensor dense(const Tensor& x, at::ScalarType t) { return !x.defined() || x.scalar_type() == t ? dense(x) : dense(x.to(t)); }
// a state that may be updated in place is never moved (the kernels take a slower path, or say that they do not serve it)
Tensor dense_state(const Tensor& x, at::ScalarType t) { return !x.defined() ? x : x.to(t).contiguous(); }
Tensor cast(const Tensor& x, at::ScalarType t) { return !x.defined() || x.scalar_type() == t ? x : x.to(t); }
void* ptr(const Tensor& x) { return x.defined() ? x.data_ptr() : nullptr; }
float* fptr(const Tensor& x) { return static_cast<float*>(ptr(x)); }
const int32_t* iptr(const Tensor& x) { return static_cast<const int32_t*>(ptr(x)); }

// element codes of activations (-1: not served) and of small parameter tensors
int act_code(at::ScalarType t) { return t == at::kBFloat16 ? 0 : t == at::kHalf ? 1 : t == at::kFloat ? 2 : -1; }
int param_code(at::ScalarType t) {
  return t == at::kFloat ? B200GDN_F32 : t == at::kBFloat16 ? B200GDN_BF16 : t == at::kHalf ? B200GDN_F16 : -1;
}
// g and beta (either may be absent) in one element type the kernels read: their own when it is common, else fp32
int gate_types(Tensor& g, Tensor& beta) {
  int code = param_code((g.defined() ? g : beta).scalar_type());
  if (g.defined() && beta.defined() && g.scalar_type() != beta.scalar_type()) code = -1;
  if (code < 0) {
    g = cast(g, at::kFloat);
    beta = cast(beta, at::kFloat);
    code = B200GDN_F32;
  }
  g = dense(g);
  beta = dense(beta);
  return code;
}
// whether the call has to go through its autograd node: for gradients, and for forward-mode tangents, which no node here
// serves and which it therefore refuses (without it they would be dropped in silence)
bool wants_grad(std::initializer_list<const Tensor*> xs) {
  for (const Tensor* x : xs) {
    if (!x->defined() || x->unsafeGetTensorImpl()->autograd_meta() == nullptr) continue;   // neither
    const auto& mode = c10::AutogradState::get_tls_state();
    if ((mode.get_grad_mode() && x->requires_grad()) || (mode.get_fw_grad_mode() && x->_fw_grad(0).defined())) return true;
  }
  return false;
}
// a tensor (or none) of which the kernels read `n` elements on `dev`: nothing on the device would notice that it is shorter
void check(const char* what, const Tensor& x, int64_t n, const at::Device& dev) {
  if (!x.defined()) return;
  if (x.device() != dev) raise(std::string(what) + " is on " + x.device().str() + " where " + dev.str() + " is expected");
  if (x.numel() < n)
    raise(std::string(what) + " has " + std::to_string(x.numel()) + " elements where " + std::to_string(n) + " are expected");
}
bool holds(const Tensor& x, int64_t n) { return !x.defined() || x.numel() >= n; }
// autograd's apply() takes an absent tensor as an empty optional
std::optional<Tensor> opt(const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; }
Tensor val(const std::optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }

// One workspace allocation, its pieces known as addresses on 256-byte boundaries (0 bytes: null).
struct Slab {
  int64_t total = 0;
  int64_t add(int64_t bytes) {
    if (bytes <= 0) return -1;
    const int64_t off = total;
    total += (bytes + 255) / 256 * 256;
    return off;
  }
  int64_t bytes() const { return total > 256 ? total : 256; }   // never an empty allocation
  Tensor make(const at::Device& dev, bool zero) const { return new_tensor({bytes()}, at::kByte, dev, zero); }
};
void* piece(const Tensor& buf, int64_t off) { return off < 0 ? nullptr : static_cast<char*>(buf.data_ptr()) + off; }

// ---- chunk tables and the split plan of a shape, built once by b200gdn/index.py ----------------------------------
struct Plan : torch::CustomClassHolder {
  Tensor chunk_meta, seq_meta, seq_order;
  int32_t n_chunks = 0, n_seq = 0;   // n_seq counts pieces under a split
  bool covered = true, split = false;
  bool empty_seqs = false;           // some sequence has no token
  Tensor chains, pre_fwd, pre_bwd, first_piece, last_piece;
  int32_t n_chains = 0, n_pre = 0;
  cudaStream_t made_on = nullptr;    // the stream whose memory the tables are
  static std::atomic<long> alive;
  Plan() { alive.fetch_add(1, std::memory_order_relaxed); }
  ~Plan() override { alive.fetch_sub(1, std::memory_order_relaxed); }
};
std::atomic<long> Plan::alive{0};
using PlanPtr = c10::intrusive_ptr<Plan>;
constexpr const char* kPlanName = "b200gdn.plan";

PlanPtr plan_of(PyObject* o) {
  auto* p = static_cast<Plan*>(PyCapsule_GetPointer(o, kPlanName));
  if (p == nullptr) throw python_error();
  return PlanPtr::reclaim_copy(p);
}

// References that captured graphs held on plans: the end of a graph may come on a thread that must not call CUDA, so they wait
// here until the next plan is made.  Never destroyed, since graphs may outlive this module.
struct Released {
  std::mutex lock;
  std::vector<PlanPtr> plans;
  void add(PlanPtr p) {
    std::lock_guard<std::mutex> g(lock);
    plans.push_back(std::move(p));
  }
  void drop() {
    std::vector<PlanPtr> old;
    std::lock_guard<std::mutex> g(lock);
    old.swap(plans);
  }
};
Released& released() {
  static Released* r = new Released;
  return *r;
}

// Called before kernels that read a plan's tables are launched on the current stream.  The tables are kept in a bounded cache
// and may leave it at any time: their memory must not be handed on before kernels on another stream than their own are done
// with it, and a graph that captures the kernels holds the plan for as long as it can be replayed.
void in_use(const PlanPtr& plan) {
  if (!plan->chunk_meta.defined() || !plan->chunk_meta.is_cuda()) return;
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
  if (stream.stream() != plan->made_on)
    for (const Tensor* t : {&plan->chunk_meta, &plan->seq_meta, &plan->seq_order, &plan->chains, &plan->pre_fwd, &plan->pre_bwd,
                            &plan->first_piece, &plan->last_piece})
      if (t->defined()) c10::cuda::CUDACachingAllocator::recordStream(t->storage().data_ptr(), stream);
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo(stream.stream(), &status, nullptr, &graph) != cudaSuccess) {
    (void)cudaGetLastError();   // the legacy stream while another one is being captured
    return;
  }
  if (status != cudaStreamCaptureStatusActive) return;
  auto* held = new PlanPtr(plan);
  auto end = [](void* p) {
    auto* h = static_cast<PlanPtr*>(p);
    released().add(std::move(*h));
    delete h;
  };
  cudaUserObject_t obj = nullptr;
  if (cudaUserObjectCreate(&obj, held, end, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
    delete held;
    raise(std::string("cudaUserObjectCreate: ") + cudaGetErrorString(cudaGetLastError()));
  }
  if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
    const std::string what = cudaGetErrorString(cudaGetLastError());
    cudaUserObjectRelease(obj, 1);
    raise("cudaGraphRetainUserObject: " + what);
  }
}

// ---- recurrent (decode) --------------------------------------------------------------------------------------
std::pair<Tensor, Tensor> recurrent(Tensor q, Tensor k, Tensor v, Tensor g, Tensor beta, const Tensor& A_log, const Tensor& dt_bias,
                                    double scale, const Tensor& initial_state, bool output_final_state, int64_t flags,
                                    const Tensor& cu_seqlens, bool inplace_state, const Tensor& state_indices) {
  const at::Device dev = q.device();
  c10::cuda::CUDAGuard guard(dev);
  const at::ScalarType out_t = q.scalar_type();
  const at::ScalarType t = act_code(out_t) >= 0 ? out_t : at::kFloat;
  q = dense(q, t);
  k = dense(k, t);
  v = dense(v, t);
  b200gdn_recurrent_args a{};
  a.B = (int32_t)q.size(0);
  a.T = (int32_t)q.size(1);
  a.H = (int32_t)q.size(2);
  a.K = (int32_t)q.size(3);
  a.HV = (int32_t)v.size(2);
  a.V = (int32_t)v.size(3);
  a.n_seq = cu_seqlens.defined() ? (int32_t)cu_seqlens.numel() - 1 : a.B;
  a.scale = (float)scale;
  a.flags = (uint32_t)flags;
  a.qkv_dtype = act_code(t);
  Tensor cu = cu_seqlens;
  if (cu.defined()) cu = cu.to(dev, at::kInt).contiguous();
  a.gb_dtype = gate_types(g, beta);
  const Tensor A = dense(A_log, at::kFloat), bias = dense(dt_bias, at::kFloat), h0 = dense_state(initial_state, at::kFloat);
  a.cu_seqlens = iptr(cu);
  a.q = ptr(q);
  a.k = ptr(k);
  a.v = ptr(v);
  a.g = ptr(g);
  a.beta = ptr(beta);
  a.A_log = fptr(A);
  a.dt_bias = fptr(bias);
  a.h0 = fptr(h0);
  Tensor o = new_tensor(v.sizes(), t, dev), ht, idx;
  bool own_state = false;
  if (state_indices.defined()) {
    idx = dense(state_indices.to(dev, at::kInt));
    a.state_indices = iptr(idx);
    a.n_slots = (int32_t)initial_state.size(0);
    ht = initial_state;
    own_state = true;
  } else if (output_final_state) {
    if (inplace_state && h0.defined() && h0.data_ptr() == initial_state.data_ptr()) {
      ht = initial_state;
      own_state = true;
    } else if (flags & B200GDN_REC_STATE_V_FIRST) {
      ht = new_tensor({a.n_seq, a.HV, a.V, a.K}, at::kFloat, dev);
    } else {
      ht = new_tensor({a.n_seq, a.HV, a.K, a.V}, at::kFloat, dev);
    }
  }
  a.o = ptr(o);
  a.ht = fptr(ht);
  call("b200gdn_recurrent_fwd", b200gdn_recurrent_fwd, a);
  if (own_state && !ht.is_inference()) torch::autograd::impl::bump_version(ht);
  return {cast(o, out_t), ht};
}

// ---- chunked rule --------------------------------------------------------------------------------------------
struct ChunkSaved : torch::CustomClassHolder {
  PlanPtr plan;
  int64_t off_gamma, off_A, off_qk, off_w, off_vnew, off_h;
  double scale;
  uint32_t options;
  int32_t gb_dtype;
  bool has_h0, transpose_states;
  at::ScalarType qt, kt, vt, gt, bt, At, dtt;
};

b200gdn_chunk_args chunk_args(const Tensor& q, const Tensor& k, const Tensor& v, double scale, const Plan& plan) {
  b200gdn_chunk_args a{};
  a.rows = (int32_t)(q.size(0) * q.size(1));
  a.H = (int32_t)q.size(2);
  a.HV = (int32_t)v.size(2);
  a.K = (int32_t)q.size(3);
  a.V = (int32_t)v.size(3);
  a.n_seq = plan.n_seq;
  a.n_chunks = plan.n_chunks;
  a.scale = (float)scale;
  a.chunk_meta = iptr(plan.chunk_meta);
  a.seq_meta = iptr(plan.seq_meta);
  a.seq_order = iptr(plan.seq_order);
  a.q = ptr(q);
  a.k = ptr(k);
  a.v = ptr(v);
  return a;
}

// the start state (reverse: the end gradient) of every piece of a split plan
void prefix_chains(const Plan& plan, int HV, int K, int V, float* M, float* h, float* x0, float* out, bool reverse) {
  b200gdn_prefix_args a{};
  a.HV = HV;
  a.K = K;
  a.V = V;
  a.n_chains = plan.n_chains;
  a.reverse = reverse;
  a.table = iptr(plan.chains);
  a.M = M;
  a.h = h;
  a.x0 = x0;
  a.out = out;
  call("b200gdn_cp_prefix", b200gdn_cp_prefix, a);
}

struct ChunkForward {
  Tensor o, ht;
  // kept for the backward pass
  Tensor q, k, v, beta, slab, g, A_log, dt_bias, rstd_q, rstd_k;
  c10::intrusive_ptr<ChunkSaved> saved;
};

ChunkForward chunk_forward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, Tensor g, Tensor beta, const Tensor& initial_state,
                           const Tensor& A_log_in, const Tensor& dt_bias_in, double scale, bool output_final_state, uint32_t options,
                           const PlanPtr& plan, bool need_grad) {
  ChunkForward r;
  const at::Device dev = q_in.device();
  c10::cuda::CUDAGuard guard(dev);
  in_use(plan);
  auto s = c10::make_intrusive<ChunkSaved>();
  s->qt = q_in.scalar_type();
  s->kt = k_in.scalar_type();
  s->vt = v_in.scalar_type();
  s->gt = g.scalar_type();
  s->bt = beta.scalar_type();
  s->plan = plan;
  s->scale = scale;
  s->has_h0 = initial_state.defined();
  const bool zero = !plan->covered;
  r.v = dense(v_in, at::kBFloat16);
  // q / k L2 norm (fla/modules/l2norm.py:84-144): for bf16 tensors the first forward kernel normalises the tiles it loads
  // and writes them for the others; other types are normalised to bf16 by a pass of their own.  The reciprocal norms go to
  // the backward kernels, which finish dq and dk with the norm's backward themselves.
  const bool l2_fused = (options & B200GDN_PREP_L2NORM) && s->qt == at::kBFloat16 && s->kt == at::kBFloat16;
  Tensor q_raw, k_raw;
  if (l2_fused) {
    q_raw = dense(q_in);
    k_raw = dense(k_in);
    r.q = new_tensor(q_raw.sizes(), at::kBFloat16, dev, zero);
    r.k = new_tensor(k_raw.sizes(), at::kBFloat16, dev, zero);
    if (need_grad) {
      r.rstd_q = new_tensor(q_raw.sizes().slice(0, 3), at::kFloat, dev, zero);
      r.rstd_k = new_tensor(q_raw.sizes().slice(0, 3), at::kFloat, dev, zero);
    }
  } else if (options & B200GDN_PREP_L2NORM) {
    const Tensor q = dense(q_in), k = dense(k_in);
    b200gdn_prep_args p{};
    p.rows = (int32_t)(q.size(0) * q.size(1));
    p.H = (int32_t)q.size(2);
    p.K = (int32_t)q.size(3);
    p.HV = (int32_t)v_in.size(2);
    p.flags = B200GDN_PREP_L2NORM;
    p.qk_dtype = act_code(q.scalar_type());
    r.q = new_tensor(q.sizes(), at::kBFloat16, dev);
    r.k = new_tensor(k.sizes(), at::kBFloat16, dev);
    r.rstd_q = new_tensor(q.sizes().slice(0, 3), at::kFloat, dev);
    r.rstd_k = new_tensor(q.sizes().slice(0, 3), at::kFloat, dev);
    p.q = ptr(q);
    p.k = ptr(k);
    p.qn = ptr(r.q);
    p.kn = ptr(r.k);
    p.rstd_q = fptr(r.rstd_q);
    p.rstd_k = fptr(r.rstd_k);
    call("b200gdn_prep_fwd", b200gdn_prep_fwd, p);
    options &= ~B200GDN_PREP_L2NORM;
  } else {
    r.q = dense(q_in, at::kBFloat16);
    r.k = dense(k_in, at::kBFloat16);
  }
  s->gb_dtype = gate_types(g, beta);
  r.beta = beta;
  Tensor h0 = dense(initial_state, at::kFloat);
  // states stored [V,K]: the scans read and write that layout themselves; only the split path, which composes states as
  // [K,V] matrices, transposes at its boundary
  s->transpose_states = (options & B200GDN_STATE_V_FIRST) && plan->split;
  if (s->transpose_states) {
    options &= ~B200GDN_STATE_V_FIRST;
    if (h0.defined()) h0 = h0.transpose(-1, -2).contiguous();
  }
  b200gdn_chunk_args a = chunk_args(l2_fused ? q_raw : r.q, l2_fused ? k_raw : r.k, r.v, scale, *plan);
  const int64_t rows = a.rows, HV = a.HV, K = a.K, V = a.V, C = a.n_chunks, N = a.n_seq;
  r.o = new_tensor(r.v.sizes(), at::kBFloat16, dev, zero);
  if (output_final_state)
    r.ht = (options & B200GDN_STATE_V_FIRST) ? new_tensor({N, HV, V, K}, at::kFloat, dev) : new_tensor({N, HV, K, V}, at::kFloat, dev);
  // h and v_new are only read by the backward pass: without one they are not even written.  u is read by the forward scan
  // only: an allocation of its own, returned to the pool when this pass ends.
  Slab slab;
  // Bounds of the chunks' transitions, for the pre-scans: they cost the first kernel 3 %, which heads that forget make good and heads
  // that remember do not, so not where pieces are short.  Forward pass without / with them, gates of logsigmoid(N(0,1)) | of -1e-4,
  // pieces of 3 chunks (2000 tokens, 4 heads of 64) 30.6 / 30.7 | 31.0 / 31.4 us, of 7 (4000, 4 of 128) 51.6 / 47.3 | 51.8 / 52.3, of 15
  // (8192, 8 of 128) 102 / 87 | 102 / 103, of 22 (12288, 8 of 128) 131 / 107 | 131 / 134: at 16 the loss is down to 2 % and the gain 15.
  const bool bounds = plan->split && C >= 16 * N;
  if (bounds) options |= B200GDN_TRANSITION_BOUNDS;
  s->options = options & ~B200GDN_PREP_L2NORM;
  s->off_gamma = slab.add(C * HV * (64 + (bounds ? 1 : 0)) * 4);
  s->off_A = slab.add(need_grad ? rows * HV * 64 * 2 : 0);
  s->off_qk = slab.add(rows * HV * 64 * 2);
  s->off_w = slab.add(rows * HV * K * 2);
  s->off_vnew = slab.add(need_grad ? rows * HV * V * 2 : 0);
  s->off_h = slab.add(need_grad ? C * HV * K * V * 2 : 0);
  r.slab = slab.make(dev, zero);
  const Tensor u = new_tensor({rows * HV * V}, at::kBFloat16, dev, zero);
  if (options & B200GDN_PREP_GATE) {
    s->At = A_log_in.scalar_type();
    s->dtt = dt_bias_in.defined() ? dt_bias_in.scalar_type() : at::kFloat;
    r.g = g;
    r.A_log = dense(A_log_in, at::kFloat);
    r.dt_bias = dense(dt_bias_in, at::kFloat);
  }
  a.options = options | (need_grad ? 0u : B200GDN_FORWARD_ONLY);
  a.gb_dtype = s->gb_dtype;
  a.g = ptr(g);
  a.beta = ptr(beta);
  a.h0 = fptr(h0);
  a.A_log = fptr(r.A_log);
  a.dt_bias = fptr(r.dt_bias);
  a.o = ptr(r.o);
  a.ht = fptr(r.ht);
  a.gamma = static_cast<float*>(piece(r.slab, s->off_gamma));
  a.A = piece(r.slab, s->off_A);
  a.qk = piece(r.slab, s->off_qk);
  a.w = piece(r.slab, s->off_w);
  a.u = ptr(u);
  if (l2_fused) {
    a.qn = ptr(r.q);
    a.kn = ptr(r.k);
    a.rstd_q = fptr(r.rstd_q);
    a.rstd_k = fptr(r.rstd_k);
  }
  a.v_new = piece(r.slab, s->off_vnew);
  a.h = piece(r.slab, s->off_h);
  if (!plan->split) {
    call("b200gdn_chunk_fwd", b200gdn_chunk_fwd, a);
  } else {
    a.stage_mask = B200GDN_FWD_INTRA;
    call("b200gdn_chunk_fwd", b200gdn_chunk_fwd, a);
    // the affine map (M, h) of every piece but the last of its sequence, from a zero start state
    const int64_t P = plan->n_pre, kv = HV * K * V;
    const Tensor ws = new_tensor({P * kv + P * HV * K * K + N * kv}, at::kFloat, dev);
    float* h_pre = fptr(ws);
    float* M_pre = h_pre + P * kv;
    float* h0_v = M_pre + P * HV * K * K;
    b200gdn_chunk_args p = chunk_args(l2_fused ? q_raw : r.q, l2_fused ? k_raw : r.k, r.v, scale, *plan);
    p.options = a.options;
    p.qn = a.qn;
    p.kn = a.kn;
    p.seq_meta = iptr(plan->pre_fwd);
    p.seq_order = nullptr;
    p.n_seq = plan->n_pre;
    p.gamma = a.gamma;
    p.w = a.w;
    p.u = a.u;
    p.ht = h_pre;
    p.cp_M = M_pre;
    p.stage_mask = B200GDN_FWD_SCAN;
    call("b200gdn_chunk_fwd", b200gdn_chunk_fwd, p);
    prefix_chains(*plan, a.HV, a.K, a.V, M_pre, h_pre, fptr(h0), h0_v, false);
    a.h0 = h0_v;
    a.stage_mask = B200GDN_FWD_SCAN | B200GDN_FWD_OUT;
    call("b200gdn_chunk_fwd", b200gdn_chunk_fwd, a);
    if (r.ht.defined()) r.ht = r.ht.index_select(0, plan->last_piece);
  }
  if (s->transpose_states && r.ht.defined()) r.ht = r.ht.transpose(-1, -2).contiguous();
  r.o = cast(r.o, s->qt);
  r.saved = std::move(s);
  return r;
}

class ChunkFunction : public torch::autograd::Function<ChunkFunction> {
 public:
  // role of fla/ops/gated_delta_rule/chunk.py:253-392
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                               const std::optional<Tensor>& h0, const std::optional<Tensor>& A_log, const std::optional<Tensor>& dt_bias,
                               double scale, bool output_final_state, int64_t options, const PlanPtr& plan) {
    ChunkForward r = chunk_forward(q, k, v, g, beta, val(h0), val(A_log), val(dt_bias), scale, output_final_state, (uint32_t)options,
                                   plan, true);
    ctx->save_for_backward({r.q, r.k, r.v, r.beta, r.slab, r.g, r.A_log, r.dt_bias, r.rstd_q, r.rstd_k});
    ctx->saved_data["s"] = at::IValue::make_capsule(r.saved);
    ctx->set_materialize_grads(false);
    if (!r.ht.defined()) return {r.o};
    return {r.o, r.ht};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &beta = saved[3], &slab = saved[4], &g = saved[5], &A_log = saved[6],
                 &dt_bias = saved[7], &rstd_q = saved[8], &rstd_k = saved[9];
    const auto capsule = ctx->saved_data["s"].toCapsule();
    const ChunkSaved& s = *static_cast<const ChunkSaved*>(capsule.get());
    const Plan& plan = *s.plan;
    const at::Device dev = q.device();
    c10::cuda::CUDAGuard guard(dev);
    in_use(s.plan);
    const bool zero = !plan.covered, gate = s.options & B200GDN_PREP_GATE;
    b200gdn_chunk_args a = chunk_args(q, k, v, s.scale, plan);
    const int64_t rows = a.rows, HV = a.HV, K = a.K, V = a.V, C = a.n_chunks, N = a.n_seq;
    const Tensor d_o = grads[0].defined() ? dense(grads[0], at::kBFloat16) : new_tensor(v.sizes(), at::kBFloat16, dev, true);
    Tensor dht = grads.size() > 1 ? dense(grads[1], at::kFloat) : Tensor();
    if (s.transpose_states && dht.defined()) dht = dht.transpose(-1, -2).contiguous();
    // the results are tensors of their own (they outlive the call); the workspace is one allocation
    const at::ScalarType gb_t = s.gb_dtype == B200GDN_F32 ? at::kFloat : s.gb_dtype == B200GDN_BF16 ? at::kBFloat16 : at::kHalf;
    Tensor dq = new_tensor(q.sizes(), at::kBFloat16, dev, zero), dk = new_tensor(k.sizes(), at::kBFloat16, dev, zero);
    Tensor dv = new_tensor(v.sizes(), at::kBFloat16, dev, zero);
    Tensor dg = new_tensor(beta.sizes(), gb_t, dev, zero), dbeta = new_tensor(beta.sizes(), gb_t, dev, zero);
    Tensor dh0, dA_log, ddt_bias;
    if (s.has_h0)
      dh0 = (s.options & B200GDN_STATE_V_FIRST) ? new_tensor({N, HV, V, K}, at::kFloat, dev) : new_tensor({N, HV, K, V}, at::kFloat, dev);
    if (gate) {
      dA_log = new_tensor({HV}, at::kFloat, dev);
      if (dt_bias.defined()) ddt_bias = new_tensor({HV}, at::kFloat, dev);
    }
    Slab slots;
    const int64_t o_dh = slots.add(C * HV * K * V * 2), o_dv2 = slots.add(rows * HV * V * 2);
    const int64_t o_gp = slots.add(gate ? C * HV * 2 * 4 : 0);
    const Tensor ws = slots.make(dev, zero);
    a.options = s.options;
    a.gb_dtype = s.gb_dtype;
    a.beta = ptr(beta);
    a.gamma = static_cast<float*>(piece(slab, s.off_gamma));
    a.A = piece(slab, s.off_A);
    a.qk = piece(slab, s.off_qk);
    a.w = piece(slab, s.off_w);
    a.v_new = piece(slab, s.off_vnew);
    a.h = piece(slab, s.off_h);
    a.d_o = ptr(d_o);
    a.dht = fptr(dht);
    a.rstd_q = fptr(rstd_q);   // given: dq, dk come out w.r.t. the un-normalised q, k
    a.rstd_k = fptr(rstd_k);
    a.dq = ptr(dq);
    a.dk = ptr(dk);
    a.dv = ptr(dv);
    a.dg = ptr(dg);
    a.dbeta = ptr(dbeta);
    a.dh0 = fptr(dh0);
    a.dh = piece(ws, o_dh);
    a.dv2 = piece(ws, o_dv2);
    if (gate) {
      a.g = ptr(g);
      a.A_log = fptr(A_log);
      a.dt_bias = fptr(dt_bias);
      a.gate_partials = static_cast<float*>(piece(ws, o_gp));
      a.dA_log = fptr(dA_log);
      a.ddt_bias = fptr(ddt_bias);
    }
    if (!plan.split) {
      call("b200gdn_chunk_bwd", b200gdn_chunk_bwd, a);
    } else {
      // the backward affine map (dM, dh) of every piece but the first of its sequence, from a zero end gradient; the
      // pre-scan forms dv_local on chip and stores neither dv2 nor dh
      const int64_t P = plan.n_pre, kv = HV * K * V;
      const Tensor pre = new_tensor({P * kv + P * HV * K * K + N * kv}, at::kFloat, dev);
      float* dh_pre = fptr(pre);
      float* dM_pre = dh_pre + P * kv;
      float* dht_v = dM_pre + P * HV * K * K;
      b200gdn_chunk_args p = chunk_args(q, k, v, s.scale, plan);
      p.options = s.options & B200GDN_TRANSITION_BOUNDS;
      p.seq_meta = iptr(plan.pre_bwd);
      p.seq_order = nullptr;
      p.n_seq = plan.n_pre;
      p.gamma = a.gamma;
      p.w = a.w;
      p.qk = a.qk;
      p.d_o = a.d_o;
      p.dh0 = dh_pre;
      p.cp_dM = dM_pre;
      p.stage_mask = B200GDN_BWD_DVLOCAL | B200GDN_BWD_SCAN;
      call("b200gdn_chunk_bwd", b200gdn_chunk_bwd, p);
      prefix_chains(plan, a.HV, a.K, a.V, dM_pre, dh_pre, fptr(dht), dht_v, true);
      a.dht = dht_v;
      call("b200gdn_chunk_bwd", b200gdn_chunk_bwd, a);
      if (dh0.defined()) dh0 = dh0.index_select(0, plan.first_piece);
    }
    if (s.transpose_states && dh0.defined()) dh0 = dh0.transpose(-1, -2).contiguous();
    if (gate) {
      dA_log = cast(dA_log, s.At);
      ddt_bias = cast(ddt_bias, s.dtt);
    }
    return {cast(dq, s.qt), cast(dk, s.kt), cast(dv, s.vt), cast(dg, s.gt), cast(dbeta, s.bt), dh0, dA_log, ddt_bias,
            Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- short convolution -----------------------------------------------------------------------------------------
struct ConvSaved : torch::CustomClassHolder {
  PlanPtr plan;
  uint32_t flags;
  int32_t W, param_dtype;
  bool has_res;
  at::ScalarType wt, bt, rt, ht;
  std::vector<int64_t> w_sizes;
};

struct ConvForward {
  Tensor y, final_state, x, w, b, h0;
  bool in_place = false;
  c10::intrusive_ptr<ConvSaved> saved;
};

ConvForward conv_forward(const Tensor& x, const Tensor& weight, const Tensor& bias, const Tensor& residual, const Tensor& initial_state,
                         bool silu, bool output_final_state, bool inplace_state, const PlanPtr& plan, bool need_grad) {
  ConvForward r;
  const at::Device dev = x.device();
  c10::cuda::CUDAGuard guard(dev);
  const at::ScalarType t = x.scalar_type();
  if (act_code(t) < 0) raise(std::string("causal_conv1d: dtype ") + c10::toString(t) + " is not supported");
  auto s = c10::make_intrusive<ConvSaved>();
  s->plan = plan;
  s->flags = silu ? B200GDN_CONV_SILU : 0;
  s->W = (int32_t)weight.size(-1);
  s->wt = weight.scalar_type();
  s->w_sizes = weight.sizes().vec();
  s->bt = bias.defined() ? bias.scalar_type() : s->wt;
  s->has_res = residual.defined();
  if (s->has_res) s->rt = residual.scalar_type();
  r.x = dense(x);
  r.w = weight;
  r.b = bias;
  s->param_dtype = gate_types(r.w, r.b);   // weight and bias in one element type the kernels read
  const Tensor res = dense(residual, t);
  r.h0 = dense_state(initial_state, t);
  if (initial_state.defined()) s->ht = initial_state.scalar_type();
  const int64_t D = x.size(2);
  r.y = new_tensor(r.x.sizes(), t, dev, !plan->covered);
  if (output_final_state) {
    if (inplace_state && r.h0.defined() && r.h0.data_ptr() == initial_state.data_ptr()) {
      r.final_state = initial_state;   // the decode step updates the cache in place
      r.in_place = true;
    } else {
      // no tile, and so no thread, visits a sequence without tokens: its cache stays as it is
      r.final_state = new_tensor({plan->n_seq, D, s->W}, t, dev, plan->empty_seqs && !r.h0.defined());
      if (plan->empty_seqs && r.h0.defined()) r.final_state.copy_(r.h0);
    }
  }
  b200gdn_conv_args a{};
  a.rows = (int32_t)(x.size(0) * x.size(1));
  a.D = (int32_t)D;
  a.W = s->W;
  a.n_seq = plan->n_seq;
  a.n_tiles = plan->n_chunks;
  a.flags = s->flags;
  a.dtype = act_code(t);
  a.param_dtype = s->param_dtype;
  a.tile_meta = iptr(plan->chunk_meta);
  a.seq_meta = iptr(plan->seq_meta);
  a.x = ptr(r.x);
  a.weight = ptr(r.w);
  a.bias = ptr(r.b);
  a.residual = ptr(res);
  a.initial_state = ptr(r.h0);
  a.y = ptr(r.y);
  a.final_state = ptr(r.final_state);
  if (a.rows != a.n_tiles || a.n_seq != a.n_tiles || a.n_seq > 65535) in_use(plan);   // a decoding step reads no table
  // the backward pass reads the cache as it was
  const Tensor before = need_grad && r.in_place ? r.h0.clone() : r.h0;
  call("b200gdn_conv_fwd", b200gdn_conv_fwd, a);
  r.h0 = before;
  r.saved = std::move(s);
  return r;
}

class ConvFunction : public torch::autograd::Function<ConvFunction> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias,
                               const std::optional<Tensor>& residual, const std::optional<Tensor>& initial_state, bool silu,
                               bool output_final_state, bool inplace_state, const PlanPtr& plan) {
    ConvForward r = conv_forward(x, weight, val(bias), val(residual), val(initial_state), silu, output_final_state, inplace_state, plan, true);
    ctx->save_for_backward({r.x, r.w, r.b, r.h0});
    ctx->saved_data["s"] = at::IValue::make_capsule(r.saved);
    ctx->set_materialize_grads(false);
    if (!r.final_state.defined()) return {r.y};
    if (r.in_place) ctx->mark_dirty({r.final_state});
    else ctx->mark_non_differentiable({r.final_state});
    return {r.y, r.final_state};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &b = saved[2], &h0 = saved[3];
    const auto capsule = ctx->saved_data["s"].toCapsule();
    const ConvSaved& s = *static_cast<const ConvSaved*>(capsule.get());
    const Plan& plan = *s.plan;
    const at::Device dev = x.device();
    c10::cuda::CUDAGuard guard(dev);
    in_use(s.plan);
    const at::ScalarType t = x.scalar_type(), pt = w.scalar_type();
    const int64_t D = x.size(2), tiles = plan.n_chunks;
    const Tensor dy = grads[0].defined() ? dense(grads[0], t) : new_tensor(x.sizes(), t, dev, true);
    Tensor dx = new_tensor(x.sizes(), t, dev, !plan.covered);
    Tensor dw = new_tensor(s.w_sizes, pt, dev), db, dh0;
    if (b.defined()) db = new_tensor({D}, pt, dev);
    if (h0.defined()) dh0 = new_tensor({plan.n_seq, D, s.W}, t, dev, plan.empty_seqs);   // zero where no tile visits
    const Tensor partials = new_tensor({2 * tiles * D * (s.W + 1)}, at::kFloat, dev);
    b200gdn_conv_args a{};
    a.rows = (int32_t)(x.size(0) * x.size(1));
    a.D = (int32_t)D;
    a.W = s.W;
    a.n_seq = plan.n_seq;
    a.n_tiles = plan.n_chunks;
    a.flags = s.flags;
    a.dtype = act_code(t);
    a.param_dtype = s.param_dtype;
    a.tile_meta = iptr(plan.chunk_meta);
    a.seq_meta = iptr(plan.seq_meta);
    a.x = ptr(x);
    a.weight = ptr(w);
    a.bias = ptr(b);
    a.initial_state = ptr(h0);
    a.dy = ptr(dy);
    a.dx = ptr(dx);
    a.dweight = ptr(dw);
    a.dbias = ptr(db);
    a.dinitial_state = ptr(dh0);
    a.partials = fptr(partials);
    call("b200gdn_conv_bwd", b200gdn_conv_bwd, a);
    return {dx, cast(dw, s.wt), cast(db, s.bt), s.has_res ? cast(grads[0].defined() ? grads[0] : dy, s.rt) : Tensor(),
            dh0.defined() ? cast(dh0, s.ht) : Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- gated RMS norm --------------------------------------------------------------------------------------------
struct NormForward {
  Tensor y, x, g, w, b, rstd;
  int32_t param_dtype = 0;
};

NormForward norm_forward(const Tensor& x, const Tensor& g, const Tensor& weight, const Tensor& bias, bool sigmoid, double eps,
                         bool need_grad) {
  NormForward r;
  const at::Device dev = x.device();
  c10::cuda::CUDAGuard guard(dev);
  const at::ScalarType t = x.scalar_type();
  if (act_code(t) < 0) raise(std::string("rms_norm_gated: dtype ") + c10::toString(t) + " is not supported");
  if (x.size(-1) == 0) raise("rms_norm_gated: rows without elements");
  r.x = dense(x);
  r.g = dense(g, t);
  r.w = weight;
  r.b = bias;
  if (weight.defined() || bias.defined()) r.param_dtype = gate_types(r.w, r.b);
  const int64_t D = x.size(-1), rows = x.numel() / D;
  r.y = new_tensor(r.x.sizes(), t, dev);
  if (need_grad) r.rstd = new_tensor({rows}, at::kFloat, dev);
  b200gdn_norm_gate_args a{};
  a.D = (int32_t)D;
  a.rows = rows;
  a.eps = (float)eps;
  a.flags = sigmoid ? B200GDN_NORM_GATE_SIGMOID : 0;
  a.dtype = act_code(t);
  a.param_dtype = r.param_dtype;
  a.x = ptr(r.x);
  a.g = ptr(r.g);
  a.weight = ptr(r.w);
  a.bias = ptr(r.b);
  a.y = ptr(r.y);
  a.rstd = fptr(r.rstd);
  call("b200gdn_norm_gate_fwd", b200gdn_norm_gate_fwd, a);
  return r;
}

class NormFunction : public torch::autograd::Function<NormFunction> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& g, const std::optional<Tensor>& weight,
                        const std::optional<Tensor>& bias, bool sigmoid, double eps) {
    NormForward r = norm_forward(x, g, val(weight), val(bias), sigmoid, eps, true);
    ctx->save_for_backward({r.x, r.g, r.w, r.b, r.rstd});
    auto ty = [](const Tensor& z) { return (int64_t)(z.defined() ? z.scalar_type() : at::kFloat); };
    ctx->saved_data["s"] = std::vector<int64_t>{sigmoid, r.param_dtype, ty(g), ty(val(weight)), ty(val(bias))};
    ctx->saved_data["eps"] = eps;
    return r.y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &g = saved[1], &w = saved[2], &b = saved[3], &rstd = saved[4];
    const auto s = ctx->saved_data["s"].toIntVector();
    const at::Device dev = x.device();
    c10::cuda::CUDAGuard guard(dev);
    const at::ScalarType t = x.scalar_type();
    const int64_t D = x.size(-1), rows = x.numel() / D;
    const Tensor dy = dense(grads[0], t);
    Tensor dx = new_tensor(x.sizes(), t, dev), dg = new_tensor(g.sizes(), t, dev), dw, db;
    const Tensor partials = new_tensor({(int64_t)b200gdn_norm_gate_ctas(rows) * 2 * D}, at::kFloat, dev);
    if (w.defined()) dw = new_tensor({D}, w.scalar_type(), dev);
    if (b.defined()) db = new_tensor({D}, b.scalar_type(), dev);
    b200gdn_norm_gate_args a{};
    a.D = (int32_t)D;
    a.rows = rows;
    a.eps = (float)ctx->saved_data["eps"].toDouble();
    a.flags = s[0] ? B200GDN_NORM_GATE_SIGMOID : 0;
    a.dtype = act_code(t);
    a.param_dtype = (int32_t)s[1];
    a.x = ptr(x);
    a.g = ptr(g);
    a.weight = ptr(w);
    a.bias = ptr(b);
    a.rstd = fptr(rstd);
    a.dy = ptr(dy);
    a.dx = ptr(dx);
    a.dg = ptr(dg);
    a.dweight = ptr(dw);
    a.dbias = ptr(db);
    a.partials = fptr(partials);
    call("b200gdn_norm_gate_bwd", b200gdn_norm_gate_bwd, a);
    return {dx, cast(dg, (at::ScalarType)s[2]), cast(dw, (at::ScalarType)s[3]), cast(db, (at::ScalarType)s[4]), Tensor(), Tensor()};
  }
};

// ---- Python side -----------------------------------------------------------------------------------------------
struct NoGil {
  PyThreadState* st = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(st); }
};

bool get(PyObject* o, Tensor& t) {   // None: an undefined tensor; false: neither None nor a tensor
  if (o == Py_None) return true;
  if (!THPVariable_Check(o)) return false;
  t = THPVariable_Unpack(o);
  return true;
}
PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* wrap_pair(const Tensor& a, const Tensor& b) {
  PyObject* x = wrap(a);
  PyObject* y = x ? wrap(b) : nullptr;
  PyObject* r = y ? PyTuple_New(2) : nullptr;
  if (r == nullptr) {
    Py_XDECREF(x);
    Py_XDECREF(y);
    return nullptr;
  }
  PyTuple_SET_ITEM(r, 0, x);
  PyTuple_SET_ITEM(r, 1, y);
  return r;
}
bool on_device(const Tensor& t, const at::Device& dev) { return !t.defined() || t.device() == dev; }
// while torch.jit.trace records, a call is left to the Python wrapper, which makes an operation of it
bool tracing() { return at::tracer::impl::is_dispatch_enabled(); }
bool truth(PyObject* o) { return o == Py_True || (o != Py_False && o != Py_None && PyObject_IsTrue(o) > 0); }

#define NEED_ARGS(n)                                                                                            \
  if (nargs != (n)) {                                                                                           \
    PyErr_Format(PyExc_TypeError, "%d positional arguments expected, got %zd", (n), nargs);                     \
    return nullptr;                                                                                             \
  }

// recurrent(q, k, v, g, beta, A_log, dt_bias, scale, initial_state, output_final_state, flags, cu_seqlens, inplace_state,
//           state_indices) -> (o, ht) or NotImplemented
PyObject* py_recurrent(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(14);
  if (tracing()) Py_RETURN_NOTIMPLEMENTED;
  Tensor q, k, v, g, beta, A, bias, h0, cu, idx;
  if (!get(args[0], q) || !get(args[1], k) || !get(args[2], v) || !get(args[3], g) || !get(args[4], beta) || !get(args[5], A) ||
      !get(args[6], bias) || !get(args[8], h0) || !get(args[11], cu) || !get(args[13], idx))
    Py_RETURN_NOTIMPLEMENTED;
  const bool out_state = truth(args[9]), inplace = truth(args[12]);
  const int64_t flags = PyLong_AsLongLong(args[10]);
  // what is not served here is named by the checks of the Python wrapper
  if (!q.defined() || !k.defined() || !v.defined() || !beta.defined() || !q.is_cuda() || q.dim() != 4 || k.dim() != 4 || v.dim() != 4 ||
      beta.dim() != 3 || (cu.defined() && q.size(0) != 1))
    Py_RETURN_NOTIMPLEMENTED;
  const double scale = args[7] == Py_None ? 1.0 / std::sqrt((double)k.size(3)) : PyFloat_AsDouble(args[7]);
  if (PyErr_Occurred()) return nullptr;
  const at::Device dev = q.device();
  if (!on_device(k, dev) || !on_device(v, dev) || !on_device(g, dev) || !on_device(beta, dev) || !on_device(A, dev) ||
      !on_device(bias, dev) || !on_device(h0, dev))
    Py_RETURN_NOTIMPLEMENTED;
  if ((flags & B200GDN_REC_GATE) && (!A.defined() || !g.defined())) Py_RETURN_NOTIMPLEMENTED;
  if ((flags & B200GDN_REC_NEG_EIGVAL) && !(flags & B200GDN_REC_BETA_SIGMOID)) Py_RETURN_NOTIMPLEMENTED;
  const int64_t n_seq = cu.defined() ? cu.numel() - 1 : q.size(0);
  if (idx.defined()) {
    if (!h0.defined() || h0.scalar_type() != at::kFloat || !h0.is_contiguous() || idx.numel() != n_seq) Py_RETURN_NOTIMPLEMENTED;
  } else if (cu.defined() && h0.defined() && h0.size(0) != n_seq) {
    Py_RETURN_NOTIMPLEMENTED;
  }
  const at::IntArrayRef qs = q.sizes(), vs = v.sizes();
  const int64_t tokens = qs[0] * qs[1], HV = vs[2], states = idx.defined() ? h0.size(0) : n_seq;
  if (!holds(k, q.numel()) || !holds(v, tokens * HV * vs[3]) || !holds(g, tokens * HV) || !holds(beta, tokens * HV) ||
      ((flags & B200GDN_REC_GATE) && (!holds(A, HV) || !holds(bias, HV))) || !holds(h0, states * HV * qs[3] * vs[3]))
    Py_RETURN_NOTIMPLEMENTED;
  if (wants_grad({&q, &k, &v, &g, &beta, &A, &bias, &h0})) Py_RETURN_NOTIMPLEMENTED;
  std::pair<Tensor, Tensor> r;
  {
    NoGil nogil;
    r = recurrent(q, k, v, g, beta, A, bias, scale, h0, out_state, flags, cu, inplace, idx);
  }
  return wrap_pair(r.first, r.second);
  END_HANDLE_TH_ERRORS
}

// chunk(q, k, v, g, beta, initial_state, A_log, dt_bias, scale, output_final_state, options, plan) -> (o, ht)
PyObject* py_chunk(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(12);
  Tensor q, k, v, g, beta, h0, A, bias;
  if (!get(args[0], q) || !get(args[1], k) || !get(args[2], v) || !get(args[3], g) || !get(args[4], beta) || !get(args[5], h0) ||
      !get(args[6], A) || !get(args[7], bias)) {
    PyErr_SetString(PyExc_TypeError, "chunk_gated_delta_rule: a tensor or None is expected");
    return nullptr;
  }
  const double scale = PyFloat_AsDouble(args[8]);
  const bool out_state = truth(args[9]);
  const int64_t options = PyLong_AsLongLong(args[10]);
  if (PyErr_Occurred()) return nullptr;
  const PlanPtr plan = plan_of(args[11]);
  variable_list out;
  {
    NoGil nogil;
    if (options & B200GDN_PREP_L2NORM)
      if (act_code(q.scalar_type()) < 0 || k.scalar_type() != q.scalar_type())
        raise(std::string("q/k dtypes ") + c10::toString(q.scalar_type()) + "/" + c10::toString(k.scalar_type()) +
              " are not supported by the L2-norm option");
    const at::Device dev = q.device();
    const int64_t tokens = q.size(0) * q.size(1), HV = v.size(2), seqs = plan->split ? plan->n_chains : plan->n_seq;
    check("k", k, q.numel(), dev);
    check("v", v, tokens * HV * v.size(3), dev);
    check("g", g, tokens * HV, dev);
    check("beta", beta, tokens * HV, dev);
    check("initial_state", h0, seqs * HV * q.size(3) * v.size(3), dev);
    check("A_log", A, HV, dev);
    check("dt_bias", bias, HV, dev);
    if (wants_grad({&q, &k, &v, &g, &beta, &h0, &A, &bias})) {
      out = ChunkFunction::apply(q, k, v, g, beta, opt(h0), opt(A), opt(bias), scale, out_state, options, plan);
    } else {
      ChunkForward r = chunk_forward(q, k, v, g, beta, h0, A, bias, scale, out_state, (uint32_t)options, plan, false);
      out = {r.o, r.ht};
    }
  }
  return wrap_pair(out[0], out.size() > 1 ? out[1] : Tensor());
  END_HANDLE_TH_ERRORS
}

// conv(x, weight, bias, residual, initial_state, silu, output_final_state, inplace_state, plan) -> (y, final_state)
PyObject* py_conv(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(9);
  Tensor x, w, b, res, h0;
  if (!get(args[0], x) || !get(args[1], w) || !get(args[2], b) || !get(args[3], res) || !get(args[4], h0)) {
    PyErr_SetString(PyExc_TypeError, "causal_conv1d: a tensor or None is expected");
    return nullptr;
  }
  const bool silu = truth(args[5]), out_state = truth(args[6]), inplace = truth(args[7]);
  if (PyErr_Occurred()) return nullptr;
  const PlanPtr plan = plan_of(args[8]);
  Tensor y, fin;
  {
    NoGil nogil;
    const at::Device dev = x.device();
    const int64_t D = x.size(2), W = w.size(-1);
    check("weight", w, D * W, dev);
    check("bias", b, D, dev);
    check("residual", res, x.numel(), dev);
    check("initial_state", h0, plan->n_seq * D * W, dev);
    if (wants_grad({&x, &w, &b, &res, &h0})) {
      variable_list out = ConvFunction::apply(x, w, opt(b), opt(res), opt(h0), silu, out_state, inplace, plan);
      y = out[0];
      if (out.size() > 1) fin = out[1];
    } else {
      ConvForward r = conv_forward(x, w, b, res, h0, silu, out_state, inplace, plan, false);
      if (r.in_place && !r.final_state.is_inference()) torch::autograd::impl::bump_version(r.final_state);
      y = r.y;
      fin = r.final_state;
    }
  }
  return wrap_pair(y, fin);
  END_HANDLE_TH_ERRORS
}

// norm_gate(x, g, weight, bias, sigmoid, eps) -> y or NotImplemented (while a trace is recorded)
PyObject* py_norm_gate(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  NEED_ARGS(6);
  if (tracing()) Py_RETURN_NOTIMPLEMENTED;
  Tensor x, g, w, b;
  if (!get(args[0], x) || !get(args[1], g) || !get(args[2], w) || !get(args[3], b) || !x.defined() || !g.defined()) {
    PyErr_SetString(PyExc_TypeError, "rms_norm_gated: a tensor is expected");
    return nullptr;
  }
  const bool sigmoid = truth(args[4]);
  const double eps = PyFloat_AsDouble(args[5]);
  if (PyErr_Occurred()) return nullptr;
  Tensor y;
  {
    NoGil nogil;
    check("g", g, x.numel(), x.device());
    check("weight", w, x.size(-1), x.device());
    check("bias", b, x.size(-1), x.device());
    y = wants_grad({&x, &g, &w, &b}) ? NormFunction::apply(x, g, opt(w), opt(b), sigmoid, eps) : norm_forward(x, g, w, b, sigmoid, eps, false).y;
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// plan(chunk_meta, seq_meta, n_chunks, n_seq, covered, empty_seqs, stream, seq_order or None
//      [, chains, pre_fwd, pre_bwd, first_piece, last_piece, n_chains, n_pre])
PyObject* py_plan(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 8) NEED_ARGS(15);
  released().drop();
  auto p = c10::make_intrusive<Plan>();
  bool ok = get(args[0], p->chunk_meta) && get(args[1], p->seq_meta) && get(args[7], p->seq_order);
  p->n_chunks = (int32_t)PyLong_AsLong(args[2]);
  p->n_seq = (int32_t)PyLong_AsLong(args[3]);
  p->covered = truth(args[4]);
  p->empty_seqs = truth(args[5]);
  p->made_on = static_cast<cudaStream_t>(PyLong_AsVoidPtr(args[6]));
  if (nargs == 15) {
    p->split = true;
    ok = ok && get(args[8], p->chains) && get(args[9], p->pre_fwd) && get(args[10], p->pre_bwd) && get(args[11], p->first_piece) &&
         get(args[12], p->last_piece);
    p->n_chains = (int32_t)PyLong_AsLong(args[13]);
    p->n_pre = (int32_t)PyLong_AsLong(args[14]);
  }
  if (!ok && !PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "plan: tensors expected");
  if (PyErr_Occurred()) return nullptr;
  return PyCapsule_New(p.release(), kPlanName, [](PyObject* c) {
    PlanPtr::reclaim(static_cast<Plan*>(PyCapsule_GetPointer(c, kPlanName)));
  });
  END_HANDLE_TH_ERRORS
}

// slab(bytes, bytes, ...) -> (bytes in all, offset, offset, ...): where the pieces of a workspace lie (-1: no such piece)
PyObject* py_slab(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  Slab slab;
  PyObject* r = PyTuple_New(nargs + 1);
  if (r == nullptr) return nullptr;
  for (Py_ssize_t i = 0; i < nargs; ++i) PyTuple_SET_ITEM(r, i + 1, PyLong_FromLongLong(slab.add(PyLong_AsLongLong(args[i]))));
  PyTuple_SET_ITEM(r, 0, PyLong_FromLongLong(slab.bytes()));
  if (!PyErr_Occurred()) return r;
  Py_DECREF(r);
  return nullptr;
}

// the streams and graphs of callers that launch kernels on a plan's tables themselves
PyObject* py_in_use(PyObject*, PyObject* plan) {
  HANDLE_TH_ERRORS
  const PlanPtr p = plan_of(plan);
  if (p->chunk_meta.defined() && p->chunk_meta.is_cuda()) {
    c10::cuda::CUDAGuard guard(p->chunk_meta.device());
    in_use(p);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* py_plans_alive(PyObject*, PyObject*) { return PyLong_FromLong(Plan::alive.load(std::memory_order_relaxed)); }

PyObject* py_launch_count(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches.load(std::memory_order_relaxed)); }

PyObject* py_set_error_class(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  Py_XSETREF(g_error_class, cls);
  Py_RETURN_NONE;
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL
PyMethodDef methods[] = {
    {"recurrent", FAST(py_recurrent), "token-by-token rule, forward only"},
    {"chunk", FAST(py_chunk), "chunked rule, differentiable"},
    {"conv", FAST(py_conv), "short causal convolution, differentiable"},
    {"norm_gate", FAST(py_norm_gate), "gated RMS norm, differentiable"},
    {"plan", FAST(py_plan), "chunk tables (and split plan) of a shape as one handle"},
    {"in_use", py_in_use, METH_O, "the tables of a plan are about to be read on the current stream"},
    {"plans_alive", py_plans_alive, METH_NOARGS, "plans that are cached, saved for a backward pass or held by a graph"},
    {"slab", FAST(py_slab), "layout of a workspace"},
    {"launch_count", py_launch_count, METH_NOARGS, "kernels enqueued through this module"},
    {"set_error_class", py_set_error_class, METH_O, "class raised when a library call fails"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "native host path of b200gdn", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
