// The package's own operator surface (ssm_b200.ops) over the C ABI: forward passes, and the autograd nodes whose backward
// passes call the backward entry points.  Everything between a Python call and its kernel launches happens here, once per
// call and without Python: a small operator is bound by exactly this work (a Python implementation of the same steps, with
// a ctypes struct per call and torch.autograd.Function, took 40 to 90 us a call; these take 6 to 15 us).
#include <ATen/SavedTensorHooks.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/autocast_mode.h>
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <utility>

#include "../decode_parts.h"
#include "../seq_table.h"
#include "operands.h"

namespace ssm_ext {
namespace {

namespace py = pybind11;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ---------------------------------------------------------------------------------------------
// one differentiable call
// ---------------------------------------------------------------------------------------------
// Gradients that a graph is recorded through (create_graph).  The kernels' backward passes have no derivative of their own, so the values are
// right, but differentiated again they would be constants: that raises.  They hang on all they depend on, because the engine walks only
// paths that lead to what it is asked for.
struct OnceFn : torch::autograd::Function<OnceFn> {
  static variable_list forward(AutogradContext*, const variable_list& values, at::TensorList sources) {
    (void)sources;
    return values;
  }
  static variable_list backward(AutogradContext*, const variable_list&) {
    TORCH_CHECK(false, "ssm_b200 operators are differentiable once: a gradient formed with create_graph=True cannot be differentiated through them");
  }
};
variable_list differentiable_once(const variable_list& grads, const variable_list& sources) {
  variable_list values, res;
  for (const Tensor& t : grads)
    if (t.defined()) values.push_back(t.detach());
  if (!values.empty()) values = OnceFn::apply(values, at::TensorList(sources));
  size_t next = 0;
  for (const Tensor& t : grads) res.push_back(t.defined() ? values[next++] : Tensor());
  return res;
}

// The operands of a call, kept by its autograd node.  `guarded` holds the tensors that the backward pass reads again with
// their version counters at the time of the forward pass: an in-place edit in between is an error, as for any saved tensor.  `unread` holds the
// others, which may be edited.
struct Call : torch::CustomClassHolder {
  std::vector<std::pair<Tensor, uint32_t>> guarded, unread;
  variable_list inputs;  // the defined tensor arguments, in the order backward() answers for them
  void input(const Tensor& t) { inputs.push_back(t); }
  void input(const OptTensor& t) {
    if (t.has_value() && t->defined()) inputs.push_back(*t);
  }
  // A call without a node would drop tangents in silence, so they are looked for first.
  bool needs_grad() const {
    for (const Tensor& t : inputs)
      TORCH_CHECK_NOT_IMPLEMENTED(!t._fw_grad(0).defined(), "ssm_b200 operators have no forward-mode derivative");
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor& t : inputs)
      if (t.requires_grad()) return true;
    return false;
  }
  virtual bool reads(size_t) const { return true; }  // whether backward() reads this input again
  virtual variable_list forward(bool train) = 0;
  // One gradient (or an undefined tensor) per input.  An incoming gradient is undefined where nothing flowed back to that output, and all
  // of them can be (a node downstream that returns none).
  virtual variable_list backward(const variable_list& grads) = 0;
  // Whether backward() may run again after a walk that does not retain the graph.  A whole mixer's tensors go with that walk, as those of the
  // products that it stands for would.
  virtual bool survives_its_walk() const { return true; }
  // backward() where a graph is recorded through the gradients.
  virtual variable_list backward_recorded(const variable_list& grads) {
    variable_list res, sources;
    {
      at::NoGradGuard values_only;
      res = backward(grads);
    }
    for (const auto& kept : guarded) sources.push_back(kept.first);
    for (const auto& kept : unread) sources.push_back(kept.first);
    for (const Tensor& g : grads)
      if (g.defined()) sources.push_back(g);
    return differentiable_once(res, sources);
  }
};

struct CallFn : torch::autograd::Function<CallFn> {
  static variable_list forward(AutogradContext* ctx, const c10::intrusive_ptr<Call>& call, at::TensorList inputs) {
    for (size_t i = 0; i < inputs.size(); ++i)
      if (!inputs[i].is_inference()) (call->reads(i) ? call->guarded : call->unread).emplace_back(inputs[i], inputs[i]._version());
    ctx->saved_data["call"] = c10::IValue::make_capsule(call);
    ctx->set_materialize_grads(false);
    return call->forward(true);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto saved = ctx->saved_data.find("call");
    TORCH_CHECK(saved != ctx->saved_data.end(), torch::autograd::ERR_BACKWARD_TWICE);
    auto holder = saved->second.toCapsule();
    Call* call = static_cast<Call*>(holder.get());
    for (const auto& kept : call->guarded) {
      if (kept.first._version() == kept.second) continue;
      std::string shape;
      for (int64_t d : kept.first.sizes()) shape += (shape.empty() ? "" : ", ") + std::to_string(d);
      TORCH_CHECK(false, "one of the tensors needed for the backward pass of an ssm_b200 operator has been modified in place (shape (" + shape + "), version " +
                             std::to_string(kept.first._version()) + ", expected " + std::to_string(kept.second) + ")");
    }
    ValueErrors scope;
    const bool last_walk = !call->survives_its_walk() && !torch::autograd::get_current_graph_task_keep_graph();
    variable_list res = at::GradMode::is_enabled() ? call->backward_recorded(grads) : call->backward(grads);
    if (last_walk) ctx->saved_data.clear();
    res.insert(res.begin(), Tensor());  // the slot of `call`
    return res;
  }
};

variable_list invoke_call(const c10::intrusive_ptr<Call>& call) {
  if (!call->needs_grad()) return call->forward(false);
  const variable_list inputs = call->inputs;
  call->inputs.clear();
  return CallFn::apply(call, at::TensorList(inputs));
}

Tensor cast(const Tensor& grad, at::ScalarType t) { return grad.scalar_type() == t ? grad : grad.to(t); }

// Several fp32 buffers that the kernels add into, zeroed by one launch; each starts on a 256-byte line.  They share one piece of memory,
// which lives as long as any of them, and autograd keeps a gradient it is given without a copy: gradients go into one pool only
// with others of their size class, and never with work buffers.
struct ZeroPool {
  std::vector<std::pair<Tensor*, std::vector<int64_t>>> want;
  int64_t total = 0;
  Tensor all;
  void add(Tensor& t, at::IntArrayRef shape) { want.emplace_back(&t, shape.vec()), total += padded(shape); }
  static int64_t padded(at::IntArrayRef shape) { return (c10::multiply_integers(shape) + 63) / 64 * 64; }
  void make(const at::TensorOptions& f32) {
    if (want.empty()) return;
    all = at::zeros({total}, f32);
    share();
  }
  // all of them in another type, by one conversion
  void cast_all(at::ScalarType type) {
    all = all.to(type);
    share();
  }
  void share() {
    int64_t at = 0;
    for (auto& [t, shape] : want) {
      *t = all.narrow(0, at, c10::multiply_integers(shape)).view(shape);
      at += padded(shape);
    }
  }
};

float* out_ptr(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }

// ---------------------------------------------------------------------------------------------
// selective scan
// ---------------------------------------------------------------------------------------------
struct ScanCall final : Call {
  ScanCtx c;
  bool want_last, has_init, init_grad;
  at::ScalarType last_type, t_delta, t_A, t_B, t_C, t_D{}, t_z{}, t_bias{}, t_init{};
  std::vector<int64_t> shape_B, shape_C;
  Tensor ck;

  ScanCall(const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D, const OptTensor& z,
           const OptTensor& dt_bias, bool softplus, bool return_last, const OptTensor& init, bool keep_fp32)
      : c(u, delta, A, B, C, D, z, dt_bias, softplus, init, true), want_last(return_last), has_init(init.has_value()) {
    for (const Tensor* t : {&u, &delta, &A, &B, &C}) input(*t);
    input(D), input(z), input(dt_bias), input(init);
    last_type = keep_fp32 ? at::kFloat : u.scalar_type();
    t_delta = delta.scalar_type(), t_A = A.scalar_type(), t_B = B.scalar_type(), t_C = C.scalar_type();
    if (D.has_value()) t_D = D->scalar_type();
    if (z.has_value()) t_z = z->scalar_type();
    if (dt_bias.has_value()) t_bias = dt_bias->scalar_type();
    if (has_init) t_init = init->scalar_type();
    init_grad = has_init && init->requires_grad();
    shape_B = B.sizes().vec(), shape_C = C.sizes().vec();
  }

  variable_list forward(bool train) override {
    c10::cuda::CUDAGuard guard(c.u.device());
    Tensor out = at::empty_like(c.u), last, split;
    ssm_scan_fwd_args a{};
    c.fill(a);
    a.out = out.data_ptr();
    if (want_last) {
      last = at::empty({c.nb, c.nd, c.nn}, c.u.options().dtype(last_type));
      a.last_state = last.data_ptr(), a.last_dtype = dtype_code(last, "selective_scan");
    }
    if (train) ck = scan_checkpoints(c), a.checkpoints = ck.data_ptr<float>();
    const int nseg = ssm_scan_split_segments((int)c.nb, (int)c.nd, (int)c.nl, (int)c.nn);  // > 1: the sequence is cut into parallel segments
    if (nseg > 1) {
      split = at::empty({2 * c.nb * c.nd * nseg * c.nn}, c.u.options().dtype(at::kFloat));
      a.split_scratch = split.data_ptr<float>(), a.split_segments = nseg;
    }
    run(ssm_selective_scan_fwd(&a, stream_of(c.u)));
    if (want_last) return {out, last};
    return {out};
  }

  variable_list backward(const variable_list& grads) override {
    c10::cuda::CUDAGuard guard(c.u.device());
    const auto f32 = c.u.options().dtype(at::kFloat);
    Tensor go = grads[0].defined() ? rows_like(grads[0], c.u) : at::zeros_like(c.u);
    OptTensor gl;
    if (grads.size() > 1 && grads[1].defined()) gl = f32c(grads[1]);
    Tensor du = at::empty_like(c.u), dd = at::empty_like(c.u), dz, dA, dB, dC, dD, db, dinit;
    if (c.z.has_value()) dz = at::empty_like(c.u);
    ZeroPool params, coeffs;
    params.add(dA, {c.nd, c.nn});
    if (c.D.has_value()) params.add(dD, {c.nd});
    if (c.bias.has_value()) params.add(db, {c.nd});
    // rows of dB and dC on 16-byte boundaries, so that the kernel's additions go out four steps at a time whatever the length
    const int64_t lp = (c.nl + 3) / 4 * 4;
    auto row_pitch = [&](const auto& k) { return k.st == 1 && k.t.dim() == 4 && k.t.size(3) == c.nl && k.sn == c.nl ? lp : c.nl; };
    auto grad_shape = [&](const auto& k) {
      std::vector<int64_t> shape = k.t.sizes().vec();
      if (row_pitch(k) != c.nl) shape.back() = lp;
      return shape;
    };
    coeffs.add(dB, grad_shape(c.B)), coeffs.add(dC, grad_shape(c.C));
    params.make(f32), coeffs.make(f32);
    if (init_grad) {  // an empty sequence hands the gradient of the last state straight to the initial state
      if (c.nl == 0) dinit = gl.has_value() ? gl->clone() : at::zeros({c.nb, c.nd, c.nn}, f32);
      else dinit = at::empty({c.nb, c.nd, c.nn}, f32);
    }
    ssm_scan_bwd_args g{};
    c.fill(g.fwd);
    g.fwd.checkpoints = ck.data_ptr<float>();
    g.dout = go.data_ptr(), g.dlast_state = fptr(gl);
    g.du = du.data_ptr(), g.ddelta = dd.data_ptr(), g.dz = dz.defined() ? dz.data_ptr() : nullptr;
    g.dA = out_ptr(dA), g.dB = out_ptr(dB), g.dC = out_ptr(dC), g.dD = out_ptr(dD), g.ddt_bias = out_ptr(db);
    auto scaled = [&](const auto& k, int64_t stride) { return row_pitch(k) != c.nl ? stride / c.nl * lp : stride; };
    g.db_sb = scaled(c.B, c.B.sb), g.db_sg = scaled(c.B, c.B.sg), g.db_sn = scaled(c.B, c.B.sn), g.db_st = c.B.st;
    g.dc_sb = scaled(c.C, c.C.sb), g.dc_sg = scaled(c.C, c.C.sg), g.dc_sn = scaled(c.C, c.C.sn), g.dc_st = c.C.st;
    g.dinitial_state = out_ptr(dinit);
    const int nseg = ssm_scan_bwd_split_segments((int)c.nb, (int)c.nd, (int)c.nl, (int)c.nn);
    Tensor split;
    if (nseg > 1) {
      split = at::empty({2 * c.nb * c.nd * nseg * c.nn}, f32);
      g.fwd.split_scratch = split.data_ptr<float>(), g.fwd.split_segments = nseg;
    }
    run(ssm_selective_scan_bwd(&g, stream_of(c.u)));
    auto fold = [&](Tensor grad, at::IntArrayRef shape, at::ScalarType t) {
      if (grad.dim() == 4 && grad.size(3) != shape.back()) {
        grad = grad.narrow(3, 0, shape.back());
        if (t == at::kFloat || grad.sizes() != shape) grad = grad.contiguous();
      }
      if (grad.sizes() != shape)  // the coefficient had been regrouped: sum the repeats back
        grad = grad.view({shape[0], shape[1], grad.size(1) / shape[1], shape[2], shape[3]}).sum(2);
      return cast(grad, t);
    };
    variable_list res = {du, cast(dd, t_delta), cast(dA, t_A), fold(dB, shape_B, t_B), fold(dC, shape_C, t_C)};
    if (c.D.has_value()) res.push_back(cast(dD, t_D));
    if (c.z.has_value()) res.push_back(cast(dz, t_z));
    if (c.bias.has_value()) res.push_back(cast(db, t_bias));
    if (has_init) res.push_back(init_grad ? cast(dinit, t_init) : Tensor());
    return res;
  }
};

py::object selective_scan(const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D, const OptTensor& z,
                          const OptTensor& dt_bias, bool softplus, bool return_last, const OptTensor& init, bool keep_fp32) {
  ValueErrors scope;
  variable_list r = invoke_call(c10::make_intrusive<ScanCall>(u, delta, A, B, C, D, z, dt_bias, softplus, return_last, init, keep_fp32));
  if (return_last) return py::make_tuple(r[0], r[1]);
  return py::cast(r[0]);
}

// ---------------------------------------------------------------------------------------------
// single-token state steps (no gradients)
// ---------------------------------------------------------------------------------------------
Tensor state_step(const Tensor& state, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D,
                  const OptTensor& z, const OptTensor& dt_bias, bool softplus, bool a_log) {
  ValueErrors scope;
  StepCtx c(state, x, dt, A, B, C, D, z, dt_bias, softplus, true);
  c10::cuda::CUDAGuard guard(state.device());
  const bool direct = state.scalar_type() == at::kFloat && state.is_contiguous();
  Tensor work = direct ? state.detach() : f32c(state);
  Tensor out = at::empty_like(c.x);
  ssm_step_args a{};
  c.fill(a, work);
  a.out = out.data_ptr(), a.a_log = a_log;
  run(ssm_selective_state_step(&a, stream_of(state)));
  if (!direct) state.detach().copy_(work);
  return out;
}

Tensor state_step_heads(const Tensor& state, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D,
                        const OptTensor& z, const OptTensor& dt_bias, bool softplus, bool a_log) {
  ValueErrors scope;
  SSM_ARG(state.dim() == 4 && x.dim() == 3, "state must be (B, H, P, N) and x (B, H, P).");
  const int64_t nb = state.size(0), nh = state.size(1), np = state.size(2), nn = state.size(3);
  SSM_ARG(x.size(0) == nb && x.size(1) == nh && x.size(2) == np && dt.dim() == 2 && dt.size(0) == nb && dt.size(1) == nh && A.dim() == 1 && A.size(0) == nh,
          "x must be (B, H, P), dt (B, H) and A (H,).");
  SSM_ARG(B.dim() == 3 && B.sizes() == C.sizes() && B.size(0) == nb && B.size(2) == nn && B.size(1) > 0 && nh % B.size(1) == 0,
          "B and C must have shape (B, G, N) with G dividing H.");
  same_device(state, {&x, &dt, &A, &B, &C});
  need_cuda(state, {&D, &z, &dt_bias});
  SSM_ARG((!D.has_value() || D->numel() == nh) && (!dt_bias.has_value() || dt_bias->numel() == nh), "D and dt_bias must have shape (H,).");
  if (z.has_value()) SSM_ARG(z->numel() == x.numel(), "z must have shape (B, H, P).");
  SSM_ARG(state.scalar_type() == at::kFloat && state.is_contiguous(), "state must be a contiguous float32 tensor.");
  c10::cuda::CUDAGuard guard(state.device());
  Tensor xs = x.detach().contiguous(), dts = like(dt, xs), Bt = B.detach().contiguous(), Ct = C.detach().contiguous();
  OptTensor zs;
  if (z.has_value()) zs = like(*z, xs);
  if (Bt.scalar_type() != Ct.scalar_type() || !io_dtype_ok(Bt)) Bt = f32c(Bt), Ct = f32c(Ct);
  Tensor A32 = f32c(A), out = at::empty_like(xs);
  OptTensor D32 = f32c(D), b32 = f32c(dt_bias);
  const int64_t g = Bt.size(1);
  ssm_step_args a{};
  a.batch = (int)nb, a.dim = (int)(nh * np), a.nstate = (int)nn, a.io_dtype = dtype_code(xs, "selective_state_step_heads");
  a.bc_dtype = dtype_code(Bt, "selective_state_step_heads B/C"), a.bc_groups = (int)g, a.dt_softplus = softplus, a.param_heads = (int)nh;
  a.state = state.data_ptr<float>(), a.x = xs.data_ptr(), a.dt = dts.data_ptr(), a.z = ptr(zs), a.A = A32.data_ptr<float>();
  a.Bm = Bt.data_ptr(), a.Cm = Ct.data_ptr();
  a.b_sb = a.c_sb = g * nn, a.b_sg = a.c_sg = nn, a.b_sn = a.c_sn = 1;
  a.D = fptr(D32), a.dt_bias = fptr(b32), a.out = out.data_ptr(), a.a_log = a_log;
  run(ssm_selective_state_step(&a, stream_of(state)));
  return out;
}

// ---------------------------------------------------------------------------------------------
// element-wise chunked recurrence
// ---------------------------------------------------------------------------------------------
struct ChunkCall final : Call {
  ChunkCtx c;
  at::ScalarType t_dt, t_A, t_B, t_C, t_D{}, t_z{}, t_init{};

  ChunkCall(const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk, const OptTensor& D, const OptTensor& z,
            const OptTensor& seq_lens, const OptTensor& cu_seqlens, const OptTensor& init)
      : c(X, dt, A, B, C, chunk, D, z, seq_lens, cu_seqlens, init) {
    for (const Tensor* t : {&X, &dt, &A, &B, &C}) input(*t);
    input(D), input(z), input(init);
    t_dt = dt.scalar_type(), t_A = A.scalar_type(), t_B = B.scalar_type(), t_C = C.scalar_type();
    if (D.has_value()) t_D = D->scalar_type();
    if (z.has_value()) t_z = z->scalar_type();
    if (init.has_value()) t_init = init->scalar_type();
  }

  Tensor kept;  // the forward call's scratch: the states entering every piece

  variable_list forward(bool train) override {
    c10::cuda::CUDAGuard guard(c.X.device());
    Tensor Y = at::empty_like(c.X);
    const int64_t n = ssm_chunk_scan_scratch_floats((int)c.nb, (int)c.nl, (int)c.nh, (int)c.np, c.chunk);
    Tensor scratch = at::empty({std::max<int64_t>(n, 1)}, c.X.options().dtype(at::kFloat));
    ssm_chunk_args a{};
    c.fill(a);
    a.Y = Y.data_ptr(), a.scratch = scratch.data_ptr<float>();
    run(ssm_chunk_scan_fwd(&a, stream_of(c.X)));
    if (train) kept = scratch;
    return {Y};
  }

  variable_list backward(const variable_list& grads) override {
    c10::cuda::CUDAGuard guard(c.X.device());
    const auto f32 = c.X.options().dtype(at::kFloat);
    Tensor gy = grads[0].defined() ? like(grads[0], c.X) : at::zeros_like(c.X);
    Tensor dX = at::empty_like(c.X), ddt, dA, dB, dC, dD, dz, dI, hist;
    ZeroPool params, per_row, per_step;
    int typed = 0;
    // per-token B / C / z: their gradients are written by the kernel in the tensor's own type (no zero-fill, no fp32 copy)
    auto own = [&](Tensor& grad, const OptTensor& t, Kind k, int bit) {
      if (!t.has_value()) return;
      if (k == Kind::BLHP) grad = at::empty_like(*t), typed |= bit;
      else (k == Kind::HP ? params : k == Kind::BHP ? per_row : per_step).add(grad, t->sizes());
    };
    own(dB, c.B, c.kB, 1), own(dC, c.C, c.kC, 2), own(dz, c.z, c.kz, 4);
    Tensor scratch = at::empty({std::max<int64_t>(1, ssm_chunk_scan_bwd_scratch_floats((int)c.nb, (int)c.nl, (int)c.nh, (int)c.np, c.chunk))}, f32);
    ssm_chunk_bwd_args g{};
    c.fill(g.fwd);
    g.dY = gy.data_ptr(), g.dX = dX.data_ptr(), g.scratch = scratch.data_ptr<float>(), g.fwd_scratch = kept.data_ptr<float>();
    auto grad_of = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
    auto set_bcz = [&]() { set_bc4(g.dB, grad_of(dB), c.kB), set_bc4(g.dC, grad_of(dC), c.kC), set_bc4(g.dz, grad_of(dz), c.kz); };
    bool fused = typed == (3 | (c.z.has_value() ? 4 : 0));
    if (fused) {
      set_bcz();
      g.fwd.typed_grads = typed;
      fused = ssm_chunk_scan_bwd_fused(&g) != 0;
    }
    if (fused) ddt = at::empty({c.nb, c.nl, c.nh}, c.X.options()), typed |= 8;
    else per_step.add(ddt, {c.nb, c.nl, c.nh}), hist = at::empty({c.nb, std::max<int64_t>(c.nl, 1), c.nh, c.np}, f32);
    params.add(dA, c.A->sizes());
    if (c.D.has_value()) params.add(dD, c.D->sizes());
    if (c.init.has_value()) per_row.add(dI, c.init->sizes());
    params.make(f32), per_row.make(f32), per_step.make(f32);
    set_bcz();
    g.fwd.typed_grads = typed, g.ddt = ddt.data_ptr(), g.history = out_ptr(hist);
    set_bc4(g.dA, grad_of(dA), c.kA), set_bc4(g.dD, grad_of(dD), c.kD), set_bc4(g.dinitial, grad_of(dI), Kind::BHP);
    run(ssm_chunk_scan_bwd(&g, stream_of(c.X)));
    variable_list res = {dX, cast(ddt, t_dt), cast(dA, t_A), cast(dB, t_B), cast(dC, t_C)};
    if (c.D.has_value()) res.push_back(cast(dD, t_D));
    if (c.z.has_value()) res.push_back(cast(dz, t_z));
    if (c.init.has_value()) res.push_back(cast(dI, t_init));
    return res;
  }
};

Tensor ssd_chunk_scan(const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk, const OptTensor& D,
                      const OptTensor& z, const OptTensor& seq_lens, const OptTensor& cu_seqlens, const OptTensor& init) {
  ValueErrors scope;
  return invoke_call(c10::make_intrusive<ChunkCall>(X, dt, A, B, C, chunk, D, z, seq_lens, cu_seqlens, init))[0];
}

// ---------------------------------------------------------------------------------------------
// depthwise causal conv
// ---------------------------------------------------------------------------------------------
struct ConvCall final : Call {
  ConvCtx c;
  at::ScalarType t_w, t_b{};
  std::vector<int64_t> shape_w;

  ConvCall(const Tensor& x, const Tensor& weight, const OptTensor& bias, const std::string& activation, const OptTensor& halo)
      : c(x, weight, bias, activation, halo, true) {
    input(x), input(weight), input(bias);
    t_w = weight.scalar_type(), shape_w = weight.sizes().vec();
    if (bias.has_value()) t_b = bias->scalar_type();
  }
  variable_list forward(bool) override {
    c10::cuda::CUDAGuard guard(c.x.device());
    Tensor y = at::empty_like(c.x);
    ssm_conv_args a{};
    c.fill(a);
    a.y = y.data_ptr();
    run(ssm_dw_causal_conv_fwd(&a, stream_of(c.x)));
    return {y};
  }
  variable_list backward(const variable_list& grads) override {
    c10::cuda::CUDAGuard guard(c.x.device());
    Tensor go = grads[0].defined() ? rows_like(grads[0], c.x) : at::zeros_like(c.x), dx = at::empty_like(c.x), dw, db;
    ZeroPool pool;
    pool.add(dw, {c.nc, c.k});
    if (c.b.has_value()) pool.add(db, {c.nc});
    pool.make(c.x.options().dtype(at::kFloat));
    ssm_conv_bwd_args g{};
    c.fill(g.fwd);
    g.dy = go.data_ptr(), g.dx = dx.data_ptr(), g.dweight = out_ptr(dw), g.dbias = out_ptr(db);
    run(ssm_dw_causal_conv_bwd(&g, stream_of(c.x)));
    if (t_w != at::kFloat && (!c.b.has_value() || t_b == t_w)) pool.cast_all(t_w);
    variable_list res = {dx, cast(dw.view(shape_w), t_w)};
    if (c.b.has_value()) res.push_back(cast(db, t_b));
    return res;
  }
};

Tensor dw_causal_conv(const Tensor& x, const Tensor& weight, const OptTensor& bias, const std::string& activation, const OptTensor& halo) {
  ValueErrors scope;
  return invoke_call(c10::make_intrusive<ConvCall>(x, weight, bias, activation, halo))[0];
}

Tensor dw_causal_conv_update(const Tensor& conv_state, const Tensor& x, const Tensor& weight, const OptTensor& bias, const std::string& activation) {
  ValueErrors scope;
  SSM_ARG(conv_state.dim() == 3 && x.dim() == 2 && conv_state.size(0) == x.size(0) && conv_state.size(1) == x.size(1),
          "conv_state must be (B, C, K) and x (B, C).");
  Tensor w2 = weight.dim() == 3 ? weight.select(1, 0) : weight;
  SSM_ARG(w2.dim() == 2 && w2.size(0) == x.size(1) && w2.size(1) == conv_state.size(2), "weight must have shape (C, K).");
  same_device(conv_state, {&x, &weight});
  need_cuda(conv_state, {&bias});
  if (bias.has_value()) SSM_ARG(bias->numel() == x.size(1), "bias must have shape (C,).");
  SSM_ARG(conv_state.scalar_type() == at::kFloat && conv_state.is_contiguous(), "conv_state must be a contiguous float32 tensor.");
  const bool silu = is_silu(activation);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor xs = x.detach().contiguous(), w = w2.detach().contiguous(), out = at::empty_like(xs);
  OptTensor b = bias.has_value() ? OptTensor(bias->detach().contiguous()) : OptTensor();
  if (!io_dtype_ok(w) || (b.has_value() && b->scalar_type() != w.scalar_type())) w = f32c(w), b = f32c(b);
  if (reinterpret_cast<uintptr_t>(w.data_ptr()) % 16) w = w.clone();  // a view into another tensor
  ssm_conv_update_args a{};
  a.batch = (int)x.size(0), a.channels = (int)x.size(1), a.width = (int)conv_state.size(2), a.io_dtype = dtype_code(xs, "dw_causal_conv_update");
  a.silu = silu;
  a.conv_state = conv_state.data_ptr<float>(), a.x = xs.data_ptr(), a.weight = w.data_ptr(), a.bias = ptr(b), a.out = out.data_ptr();
  a.param_dtype = dtype_code(w, "dw_causal_conv_update");
  run(ssm_dw_causal_conv_update(&a, stream_of(xs)));
  return out;
}

// ---------------------------------------------------------------------------------------------
// fused residual add + LayerNorm / RMSNorm
// ---------------------------------------------------------------------------------------------
struct NormCall final : Call {
  NormCtx c;
  bool want_res;
  at::ScalarType res_type, t_w, t_b{}, t_r{};

  NormCall(const Tensor& x, const Tensor& weight, const OptTensor& bias, const OptTensor& residual, bool is_rms, double eps, bool prenorm, bool return_residual,
           bool residual_in_fp32)
      : c(x, weight, bias, residual, is_rms, eps, prenorm), want_res(return_residual) {
    input(x), input(weight), input(bias), input(residual);
    res_type = residual_in_fp32 ? at::kFloat : x.scalar_type();
    t_w = weight.scalar_type();
    if (bias.has_value()) t_b = bias->scalar_type();
    if (residual.has_value()) t_r = residual->scalar_type();
  }
  variable_list forward(bool) override {
    c10::cuda::CUDAGuard guard(c.x.device());
    Tensor y = at::empty_like(c.x), ro;
    ssm_norm_args a{};
    c.fill(a);
    a.y = y.data_ptr();
    if (want_res) {
      ro = at::empty(c.x.sizes(), c.x.options().dtype(res_type));
      a.residual_out = ro.data_ptr(), a.resout_dtype = dtype_code(ro, "fused_layer_norm");
    }
    run(ssm_fused_add_norm_fwd(&a, stream_of(c.x)));
    if (want_res) return {y, ro};
    return {y};
  }
  variable_list backward(const variable_list& grads) override {
    c10::cuda::CUDAGuard guard(c.x.device());
    const auto f32 = c.x.options().dtype(at::kFloat);
    const int64_t rows = c.x.size(0) * c.x.size(1), hidden = c.x.size(2);
    Tensor go = grads[0].defined() ? like(grads[0], c.x) : at::zeros_like(c.x), gr;
    Tensor dx = at::empty_like(c.x), dres, dw = at::empty({hidden}, c.w.options()), db;
    if (c.res.has_value()) dres = at::empty_like(*c.res);
    if (c.b.has_value()) db = at::empty({hidden}, c.w.options());
    Tensor partial = at::empty({ssm_norm_bwd_scratch_floats(rows, (int)hidden)}, f32);
    ssm_norm_bwd_args g{};
    c.fill(g.fwd);
    g.dy = go.data_ptr(), g.dx = dx.data_ptr(), g.dresidual = dres.defined() ? dres.data_ptr() : nullptr;
    g.fwd.dparam_dtype = g.fwd.param_dtype;
    g.dweight = dw.data_ptr(), g.dbias = db.defined() ? db.data_ptr() : nullptr, g.partial = partial.data_ptr<float>();
    if (grads.size() > 1 && grads[1].defined()) {  // the gradient arriving through x + residual: added to dx and dresidual inside the kernel
      gr = grads[1].detach().to(res_type).contiguous();
      g.fwd.resout_dtype = dtype_code(gr, "fused_layer_norm"), g.dresidual_out = gr.data_ptr();
    }
    run(ssm_fused_add_norm_bwd(&g, stream_of(c.x)));
    variable_list res = {dx, cast(dw, t_w)};
    if (c.b.has_value()) res.push_back(cast(db, t_b));
    if (c.res.has_value()) res.push_back(cast(dres, t_r));
    return res;
  }
};

py::object fused_layer_norm(const Tensor& x, const Tensor& weight, const OptTensor& bias, const OptTensor& residual, bool is_rms, double eps, bool prenorm,
                            bool residual_in_fp32, bool return_residual) {
  ValueErrors scope;
  variable_list r = invoke_call(c10::make_intrusive<NormCall>(x, weight, bias, residual, is_rms, eps, prenorm, return_residual, residual_in_fp32));
  if (return_residual) return py::make_tuple(r[0], r[1]);
  return py::cast(r[0]);
}

// ---------------------------------------------------------------------------------------------
// one decode token through a whole mixer (no gradients)
// ---------------------------------------------------------------------------------------------
Tensor ssd_status(int64_t device);
void ssd_poll(int64_t device);

bool plain(const Tensor& t, at::ScalarType type) {
  return t.scalar_type() == type && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}
bool plain(const OptTensor& t, at::ScalarType type) { return !t.has_value() || plain(*t, type); }

// The outcome of a one-launch step: false when the kernel cannot run here (too few SMs for all of its CTAs at once).  Nothing has been
// launched then and the states are untouched, so the separate calls can serve the step.
bool launched(int rc) {
  if (rc == SSM_ERR_UNSUPPORTED) return false;
  run(rc);
  return true;
}

// A step of up to 256 sequences as five to seven launches of this library on one piece of scratch, each starting while the one before it
// drains.  The callers have checked types, sizes and alignment.
struct Parts {
  Tensor scratch;
  char* at;
  int io;
  int32_t* status;
  ssm_stream_t st;
  Parts(const Tensor& tok, int64_t elements, int pieces)
      : scratch(at::empty({(elements + 64 * pieces) * 2}, tok.options().dtype(at::kByte))), at(static_cast<char*>(scratch.data_ptr())), io(dtype_code(tok, "decode step")),
        status(ssd_status(tok.get_device()).data_ptr<int32_t>()), st(stream_of(tok)) {}
  char* take(int64_t elements) {  // 16-bit elements, from a 128-byte line
    char* p = at;
    at += (elements + 63) / 64 * 128;
    return p;
  }
  // out_i = x w_i^T, x (nb, k) with ldx elements from row to row
  void product(int64_t nb, const void* x, int64_t k, int64_t ldx, bool weights_ahead, std::initializer_list<std::pair<const Tensor*, void*>> mats) const {
    ssmb_rows_gemm_args a{};
    a.batch = (int)nb, a.k = (int)k, a.ldx = ldx, a.io_dtype = io, a.x = x, a.status = status, a.weights_ahead = weights_ahead;
    for (const auto& m : mats) {
      a.w[a.mats] = m.first->data_ptr(), a.rows[a.mats] = (int)m.first->size(0), a.out[a.mats] = m.second, a.ldo[a.mats] = m.first->size(0);
      ++a.mats;
    }
    run(ssmb_rows_gemm(&a, st));
  }
};
Tensor rows_of(void* p, int64_t rows, int64_t cols, int64_t ld, const Tensor& like) { return at::from_blob(p, {rows, cols}, {ld, 1}, like.options()); }
// The library's product of many token rows with one large matrix keeps more of the GPU busy than the kernel of Parts (us of products back to back, own
// and library: 2560 x 5120 at 256 rows 14.9 and 9.7, at 192 11.7 and 8.8, at 160 10.5 and 10.8, at 128 9.3 and 8.9; 1536 x 3072 at 256 8.1 and 6.7,
// at 128 6.4 and 6.3; 768 x 1536 at 256 5.6 and 4.4, for which the host's 10 us more are too many).  The projections in front are one launch here for
// two to five of the library's: 2 x (5120 x 2560) at 256 rows 19.2 and 16.6, at 192 15.1 and 15.5, at 128 11.5 and 13.1, at 32 8.5 and 14.8; 2 x
// (3072 x 1536) at 256 8.7 and 10.0.
bool library_product(int64_t nb, const Tensor& w) { return nb > 128 && w.size(0) >= 1024 && w.size(1) >= 2048; }

// What the separate calls refuse, or answer in another type, goes to them: shapes that agree in their number of elements only, tangents, autocast
// to another type.
bool by_parts(const Tensor& tok, std::initializer_list<std::pair<const Tensor*, std::initializer_list<int64_t>>> shapes, std::initializer_list<const Tensor*> tangents) {
  if (tok.size(1) % 8 != 0 || tok.size(0) > SSMB_GEMM_MAX_ROWS) return false;
  if (at::autocast::is_autocast_enabled(at::kCUDA) && at::autocast::get_autocast_dtype(at::kCUDA) != tok.scalar_type()) return false;
  for (const auto& [t, shape] : shapes)
    if (t->sizes() != at::IntArrayRef(shape)) return false;
  for (const Tensor* t : tangents)
    if (t && t->_fw_grad(0).defined()) return false;
  return true;
}
// conv weights (C, K), or (C, 1, K)
bool conv_weight(const Tensor& w, int64_t c, int64_t k) { return w.size(0) == c && w.size(-1) == k && (w.dim() == 2 || (w.dim() == 3 && w.size(1) == 1)); }

py::object mamba1_parts(const Tensor& tok, const OptTensor& residual, const Tensor& conv_state, const Tensor& ssm_state, const Tensor& in_x, const Tensor& in_z,
                        const Tensor& conv_w, const OptTensor& conv_b, const Tensor& x_proj, const Tensor& dt_proj, const Tensor& dt_bias, const Tensor& A, bool a_log,
                        const Tensor& D, const Tensor& out_proj, const OptTensor& norm_w, double eps) {
  c10::cuda::CUDAGuard guard(tok.device());
  ssd_poll(tok.get_device());
  const int64_t nb = tok.size(0), dm = tok.size(1), di = in_x.size(0), n = ssm_state.size(-1), r = dt_proj.size(1), xw = r + 2 * n;
  Parts p(tok, nb * (5 * di + xw + dm), 7);
  char *x = p.take(nb * di), *z = p.take(nb * di), *u = p.take(nb * di), *xd = p.take(nb * xw), *dt = p.take(nb * di), *y = p.take(nb * di), *o = p.take(nb * dm);
  Tensor out = at::empty_like(tok), res;
  p.product(nb, tok.data_ptr(), dm, dm, false, {{&in_x, x}, {&in_z, z}});
  ssm_conv_update_args c{};
  c.batch = (int)nb, c.channels = (int)di, c.width = (int)conv_w.size(-1), c.io_dtype = c.param_dtype = p.io, c.silu = 1;
  c.conv_state = conv_state.data_ptr<float>(), c.x = x, c.weight = conv_w.data_ptr(), c.bias = ptr(conv_b), c.out = u;
  run(ssmb_conv_update_many(&c, 1, p.st));
  p.product(nb, u, di, di, true, {{&x_proj, xd}});
  if (ssmb_rows_gemm_supported((int)nb, (int)r, xw, p.io)) {
    p.product(nb, xd, r, xw, true, {{&dt_proj, dt}});
  } else {  // rows of dt_proj that do not start on 16-byte boundaries
    Tensor to = rows_of(dt, nb, di, di, tok);
    at::mm_out(to, rows_of(xd, nb, r, xw, tok), dt_proj.t());
  }
  ssm_step_args s{};
  s.batch = (int)nb, s.dim = (int)di, s.nstate = (int)n, s.io_dtype = s.bc_dtype = p.io, s.bc_groups = 1, s.dt_softplus = 1, s.a_log = a_log;
  s.state = ssm_state.data_ptr<float>(), s.x = u, s.dt = dt, s.z = z, s.A = A.data_ptr<float>(), s.D = D.data_ptr<float>(), s.dt_bias = dt_bias.data_ptr<float>();
  s.Bm = xd + r * 2, s.Cm = xd + (r + n) * 2, s.b_sb = s.c_sb = xw, s.b_sn = s.c_sn = 1, s.out = y;
  run(ssm_selective_state_step(&s, p.st));
  void* mixed = norm_w.has_value() ? (void*)o : out.data_ptr();
  if (library_product(nb, out_proj)) {
    Tensor to = norm_w.has_value() ? rows_of(o, nb, dm, dm, tok) : out;
    at::mm_out(to, rows_of(y, nb, di, di, tok), out_proj.t());
  } else {
    p.product(nb, y, di, di, true, {{&out_proj, mixed}});
  }
  if (!norm_w.has_value()) return py::cast(out);
  res = at::empty({nb, dm}, tok.options().dtype(at::kFloat));
  ssm_norm_args a{};
  a.rows = nb, a.hidden = (int)dm, a.io_dtype = a.param_dtype = p.io, a.is_rms = 1, a.prenorm = 1, a.eps = (float)eps;
  a.x = o, a.weight = norm_w->data_ptr(), a.y = out.data_ptr(), a.residual_out = res.data_ptr(), a.resout_dtype = SSM_F32;
  if (residual.has_value()) a.residual = residual->data_ptr(), a.res_dtype = dtype_code(*residual, "mamba1_step residual");
  run(ssm_fused_add_norm_fwd(&a, p.st));
  return py::make_tuple(out, res);
}

Tensor mamba2_parts(const Tensor& tok, const Tensor& conv_x, const Tensor& conv_B, const Tensor& conv_C, const Tensor& ssm_state, const Tensor& in_z, const Tensor& in_x,
                    const Tensor& in_B, const Tensor& in_C, const Tensor& in_dt, const Tensor& wx, const OptTensor& bx, const Tensor& wB, const OptTensor& bB,
                    const Tensor& wC, const OptTensor& bC, const Tensor& dt_bias, const Tensor& A, bool a_log, const Tensor& D, const Tensor& norm_w,
                    const Tensor& out_proj, double eps) {
  c10::cuda::CUDAGuard guard(tok.device());
  ssd_poll(tok.get_device());
  const int64_t nb = tok.size(0), dm = tok.size(1), nh = ssm_state.size(1), n = ssm_state.size(3), di = in_x.size(0), gn = in_B.size(0);
  Parts p(tok, nb * (5 * di + 4 * gn + nh), 10);
  char *x = p.take(nb * di), *z = p.take(nb * di), *u = p.take(nb * di), *y = p.take(nb * di), *yn = p.take(nb * di), *B = p.take(nb * gn), *C = p.take(nb * gn),
       *uB = p.take(nb * gn), *uC = p.take(nb * gn), *dt = p.take(nb * nh);
  Tensor out = at::empty_like(tok);
  p.product(nb, tok.data_ptr(), dm, dm, false, {{&in_x, x}, {&in_z, z}, {&in_B, B}, {&in_C, C}, {&in_dt, dt}});
  ssm_conv_update_args c[3] = {};
  const Tensor* states[3] = {&conv_x, &conv_B, &conv_C};
  const Tensor* weights[3] = {&wx, &wB, &wC};
  const OptTensor* biases[3] = {&bx, &bB, &bC};
  const char* from[3] = {x, B, C};
  char* to[3] = {u, uB, uC};
  for (int i = 0; i < 3; ++i) {
    c[i].batch = (int)nb, c[i].channels = (int)(i ? gn : di), c[i].width = (int)wx.size(-1), c[i].io_dtype = c[i].param_dtype = p.io, c[i].silu = 1;
    c[i].conv_state = states[i]->data_ptr<float>(), c[i].x = from[i], c[i].weight = weights[i]->data_ptr(), c[i].bias = ptr(*biases[i]), c[i].out = to[i];
  }
  run(ssmb_conv_update_many(c, 3, p.st));
  ssm_step_args s{};
  s.batch = (int)nb, s.dim = (int)di, s.nstate = (int)n, s.io_dtype = s.bc_dtype = p.io, s.bc_groups = (int)(gn / n), s.dt_softplus = 1, s.param_heads = (int)nh, s.a_log = a_log;
  s.state = ssm_state.data_ptr<float>(), s.x = u, s.dt = dt, s.z = z, s.A = A.data_ptr<float>(), s.D = D.data_ptr<float>(), s.dt_bias = dt_bias.data_ptr<float>();
  s.Bm = uB, s.Cm = uC, s.b_sb = s.c_sb = gn, s.b_sg = s.c_sg = n, s.b_sn = s.c_sn = 1, s.out = y;
  run(ssm_selective_state_step(&s, p.st));
  ssm_norm_args a{};
  a.rows = nb, a.hidden = (int)di, a.io_dtype = a.param_dtype = p.io, a.is_rms = 1, a.prenorm = 1, a.eps = (float)eps;
  a.x = y, a.weight = norm_w.data_ptr(), a.y = yn;
  run(ssm_fused_add_norm_fwd(&a, p.st));
  if (library_product(nb, out_proj)) at::mm_out(out, rows_of(yn, nb, di, di, tok), out_proj.t());
  else p.product(nb, yn, di, di, true, {{&out_proj, out.data_ptr()}});
  return out;
}

// Up to 16 sequences: one launch (ssm_mamba1_decode).  Up to 256: the launches above.  More, or other types and layouts: library GEMMs around the conv and state kernels.  With norm_w the
// residual add and RMSNorm behind the mixer are included and the result is (normed, residual stream in fp32).
py::object mamba1_step(const Tensor& tok, const OptTensor& residual, const Tensor& conv_state, const Tensor& ssm_state, const Tensor& in_x, const Tensor& in_z,
                       const Tensor& conv_w, const OptTensor& conv_b, const Tensor& x_proj, const Tensor& dt_proj, const Tensor& dt_bias, const Tensor& A,
                       bool a_log, const Tensor& D, const Tensor& out_proj, const OptTensor& norm_w, double eps) {
  ValueErrors scope;
  at::NoGradGuard no_grad;
  SSM_ARG(tok.dim() == 2 && tok.is_cuda(), "mamba1_step: tok must be a (B, d_model) CUDA tensor.");
  same_device(tok, {&conv_state, &ssm_state, &in_x, &in_z, &conv_w, &x_proj, &dt_proj, &dt_bias, &A, &D, &out_proj});
  need_cuda(tok, {&residual, &conv_b, &norm_w});
  const int64_t nb = tok.size(0), dm = tok.size(1), di = in_x.size(0), n = ssm_state.size(-1), r = dt_proj.size(1), k = conv_w.size(-1);
  const auto T = tok.scalar_type();
  const bool half = T == at::kBFloat16 || T == at::kHalf;
  bool fused = half && plain(tok, T) && plain(conv_state, at::kFloat) && plain(ssm_state, at::kFloat) && plain(A, at::kFloat) && plain(D, at::kFloat) &&
               plain(dt_bias, at::kFloat) && plain(conv_b, T) && plain(norm_w, T) && (!residual.has_value() || (residual->is_contiguous() && io_dtype_ok(*residual)));
  for (const Tensor* w : {&in_x, &in_z, &conv_w, &x_proj, &dt_proj, &out_proj}) fused = fused && plain(*w, T);
  fused = fused && in_x.sizes() == in_z.sizes() && in_x.size(1) == dm && conv_w.size(0) == di && x_proj.size(0) == r + 2 * n && x_proj.size(1) == di &&
          dt_proj.size(0) == di && out_proj.size(0) == dm && out_proj.size(1) == di && conv_state.dim() == 3 && conv_state.size(0) == nb && conv_state.size(1) == di &&
          conv_state.size(2) == k && ssm_state.dim() == 3 && ssm_state.size(0) == nb && ssm_state.size(1) == di && A.dim() == 2 && A.size(0) == di && A.size(1) == n &&
          D.numel() == di && dt_bias.numel() == di && conv_w.numel() == di * k && (!conv_b.has_value() || conv_b->numel() == di) &&
          (!norm_w.has_value() || norm_w->numel() == dm) && (!residual.has_value() || residual->numel() == nb * dm) && nb > 0;
  if (fused && ssm_mamba1_decode_supported((int)nb, (int)dm, (int)di, (int)n, (int)r, (int)k, dtype_code(tok, "mamba1_step"))) {
    c10::cuda::CUDAGuard guard(tok.device());
    Tensor out = at::empty_like(tok), res;
    Tensor scratch = at::empty({ssm_mamba1_decode_scratch_bytes((int)nb, (int)dm, (int)di, (int)n, (int)r)}, tok.options().dtype(at::kByte));
    ssm_mamba1_decode_args a{};
    a.batch = (int)nb, a.d_model = (int)dm, a.d_inner = (int)di, a.nstate = (int)n, a.dt_rank = (int)r, a.width = (int)k;
    a.io_dtype = dtype_code(tok, "mamba1_step"), a.a_log = a_log, a.eps = (float)eps;
    a.hidden = tok.data_ptr(), a.in_x = in_x.data_ptr(), a.in_z = in_z.data_ptr(), a.conv_w = conv_w.data_ptr(), a.conv_b = ptr(conv_b);
    a.x_proj = x_proj.data_ptr(), a.dt_proj = dt_proj.data_ptr(), a.dt_bias = dt_bias.data_ptr<float>(), a.A = A.data_ptr<float>(), a.D = D.data_ptr<float>();
    a.out_proj = out_proj.data_ptr(), a.norm_w = ptr(norm_w);
    a.conv_state = conv_state.data_ptr<float>(), a.ssm_state = ssm_state.data_ptr<float>(), a.out = out.data_ptr(), a.scratch = scratch.data_ptr();
    if (norm_w.has_value()) {
      res = at::empty({nb, dm}, tok.options().dtype(at::kFloat));
      a.residual_out = res.data_ptr(), a.resout_dtype = SSM_F32;
      if (residual.has_value()) a.residual = residual->data_ptr(), a.res_dtype = dtype_code(*residual, "mamba1_step residual");
    }
    if (launched(ssm_mamba1_decode(&a, stream_of(tok)))) {
      if (norm_w.has_value()) return py::make_tuple(out, res);
      return py::cast(out);
    }
  }
  if (fused && di % 8 == 0 && conv_weight(conv_w, di, k) &&
      by_parts(tok, {{&D, {di}}, {&dt_bias, {di}}, {norm_w.has_value() ? &*norm_w : &D, {norm_w.has_value() ? dm : di}}},
               {residual.has_value() ? &*residual : nullptr, norm_w.has_value() ? &*norm_w : nullptr, &out_proj}))
    return mamba1_parts(tok, residual, conv_state, ssm_state, in_x, in_z, conv_w, conv_b, x_proj, dt_proj, dt_bias, A, a_log, D, out_proj, norm_w, eps);
  Tensor x = at::matmul(tok, in_x.t()), z = at::matmul(tok, in_z.t());
  Tensor u = dw_causal_conv_update(conv_state, x, conv_w, conv_b, "silu");
  Tensor xd = at::matmul(u, x_proj.t());
  Tensor delta = at::matmul(xd.narrow(1, 0, r), dt_proj.t());
  Tensor y = state_step(ssm_state, u, delta, A, xd.narrow(1, r, n).unsqueeze(1), xd.narrow(1, r + n, n).unsqueeze(1), D, z, dt_bias, true, a_log);
  Tensor out = at::matmul(y, out_proj.t());
  if (!norm_w.has_value()) return py::cast(out);
  OptTensor res = residual.has_value() ? OptTensor(residual->reshape({1, nb, dm})) : OptTensor();
  variable_list rr = invoke_call(c10::make_intrusive<NormCall>(out.unsqueeze(0), *norm_w, OptTensor(), res, true, eps, true, true, true));
  return py::make_tuple(rr[0].view({nb, dm}), rr[1].view({nb, dm}));
}

// The same for Mamba-2 (the gated norm is part of the mixer).
Tensor mamba2_step(const Tensor& tok, const Tensor& conv_x, const Tensor& conv_B, const Tensor& conv_C, const Tensor& ssm_state, const Tensor& in_z,
                   const Tensor& in_x, const Tensor& in_B, const Tensor& in_C, const Tensor& in_dt, const Tensor& wx, const OptTensor& bx, const Tensor& wB,
                   const OptTensor& bB, const Tensor& wC, const OptTensor& bC, const Tensor& dt_bias, const Tensor& A, bool a_log, const Tensor& D,
                   const Tensor& norm_w, const Tensor& out_proj, double eps) {
  ValueErrors scope;
  at::NoGradGuard no_grad;
  SSM_ARG(tok.dim() == 2 && tok.is_cuda() && ssm_state.dim() == 4, "mamba2_step: tok must be a (B, d_model) CUDA tensor and the state (B, H, P, N).");
  same_device(tok, {&conv_x, &conv_B, &conv_C, &ssm_state, &in_z, &in_x, &in_B, &in_C, &in_dt, &wx, &wB, &wC, &dt_bias, &A, &D, &norm_w, &out_proj});
  need_cuda(tok, {&bx, &bB, &bC});
  const int64_t nb = tok.size(0), dm = tok.size(1), nh = ssm_state.size(1), hp = ssm_state.size(2), n = ssm_state.size(3), di = nh * hp;
  SSM_ARG(in_B.size(0) % n == 0, "mamba2_step: in_B must have groups * d_state rows.");
  const int64_t g = in_B.size(0) / n, k = wx.size(-1);
  SSM_ARG(g > 0 && nh % g == 0, "B and C must have shape (B, G, N) with G dividing H.");  // before any window is written
  const auto T = tok.scalar_type();
  bool fused = (T == at::kBFloat16 || T == at::kHalf) && plain(tok, T) && plain(dt_bias, at::kFloat) && plain(A, at::kFloat) && plain(D, at::kFloat) &&
               plain(bx, T) && plain(bB, T) && plain(bC, T);
  for (const Tensor* t : {&conv_x, &conv_B, &conv_C, &ssm_state}) fused = fused && plain(*t, at::kFloat);
  for (const Tensor* w : {&in_z, &in_x, &in_B, &in_C, &in_dt, &wx, &wB, &wC, &norm_w, &out_proj}) fused = fused && plain(*w, T);
  for (const Tensor* w : {&in_z, &in_x, &in_B, &in_C, &in_dt}) fused = fused && w->dim() == 2 && w->size(1) == dm;
  fused = fused && in_x.size(0) == di && in_z.size(0) == di && in_C.size(0) == g * n && in_dt.size(0) == nh && wx.numel() == di * k && wB.numel() == g * n * k &&
          wC.numel() == g * n * k && (!bx.has_value() || bx->numel() == di) && (!bB.has_value() || bB->numel() == g * n) &&
          (!bC.has_value() || bC->numel() == g * n) && conv_x.numel() == nb * di * k && conv_B.numel() == nb * g * n * k && conv_C.numel() == nb * g * n * k &&
          ssm_state.size(0) == nb && dt_bias.numel() == nh && A.numel() == nh && D.numel() == nh && norm_w.numel() == di && out_proj.dim() == 2 &&
          out_proj.size(0) == dm && out_proj.size(1) == di && nb > 0;
  if (fused && ssm_mamba2_decode_supported((int)nb, (int)dm, (int)nh, (int)hp, (int)n, (int)g, (int)k, dtype_code(tok, "mamba2_step"))) {
    c10::cuda::CUDAGuard guard(tok.device());
    Tensor out = at::empty_like(tok);
    Tensor scratch = at::empty({ssm_mamba2_decode_scratch_bytes((int)nb, (int)nh, (int)g)}, tok.options().dtype(at::kByte));
    ssm_mamba2_decode_args a{};
    a.batch = (int)nb, a.d_model = (int)dm, a.heads = (int)nh, a.headdim = (int)hp, a.nstate = (int)n, a.groups = (int)g, a.width = (int)k;
    a.io_dtype = dtype_code(tok, "mamba2_step"), a.a_log = a_log, a.eps = (float)eps;
    a.hidden = tok.data_ptr(), a.in_z = in_z.data_ptr(), a.in_x = in_x.data_ptr(), a.in_B = in_B.data_ptr(), a.in_C = in_C.data_ptr(), a.in_dt = in_dt.data_ptr();
    a.conv_x_w = wx.data_ptr(), a.conv_x_b = ptr(bx), a.conv_B_w = wB.data_ptr(), a.conv_B_b = ptr(bB), a.conv_C_w = wC.data_ptr(), a.conv_C_b = ptr(bC);
    a.dt_bias = dt_bias.data_ptr<float>(), a.A = A.data_ptr<float>(), a.D = D.data_ptr<float>(), a.norm_w = norm_w.data_ptr(), a.out_proj = out_proj.data_ptr();
    a.conv_state_x = conv_x.data_ptr<float>(), a.conv_state_B = conv_B.data_ptr<float>(), a.conv_state_C = conv_C.data_ptr<float>();
    a.ssm_state = ssm_state.data_ptr<float>(), a.out = out.data_ptr(), a.scratch = scratch.data_ptr();
    if (launched(ssm_mamba2_decode(&a, stream_of(tok)))) return out;
  }
  if (fused && di % 8 == 0 && conv_weight(wx, di, k) && conv_weight(wB, g * n, k) && conv_weight(wC, g * n, k) &&
      by_parts(tok, {{&conv_x, {nb, di, k}}, {&conv_B, {nb, g * n, k}}, {&conv_C, {nb, g * n, k}}, {&A, {nh}}, {&norm_w, {di}}}, {&norm_w, &out_proj}))
    return mamba2_parts(tok, conv_x, conv_B, conv_C, ssm_state, in_z, in_x, in_B, in_C, in_dt, wx, bx, wB, bB, wC, bC, dt_bias, A, a_log, D, norm_w, out_proj, eps);
  Tensor z = at::matmul(tok, in_z.t());
  Tensor x = dw_causal_conv_update(conv_x, at::matmul(tok, in_x.t()), wx, bx, "silu");
  Tensor Bm = dw_causal_conv_update(conv_B, at::matmul(tok, in_B.t()), wB, bB, "silu").view({nb, g, n});
  Tensor Cm = dw_causal_conv_update(conv_C, at::matmul(tok, in_C.t()), wC, bC, "silu").view({nb, g, n});
  Tensor dt = at::matmul(tok, in_dt.t());
  Tensor y = state_step_heads(ssm_state, x.view({nb, nh, hp}), dt, A, Bm, Cm, D, z.view({nb, nh, hp}), dt_bias, true, a_log);
  variable_list rr = invoke_call(c10::make_intrusive<NormCall>(y.view({1, nb, di}), norm_w, OptTensor(), OptTensor(), true, eps, true, false, true));
  return at::matmul(rr[0].view({nb, di}), out_proj.t());
}

// ---------------------------------------------------------------------------------------------
// state-space-dual scan, forward on the tensor cores
// ---------------------------------------------------------------------------------------------
// The word a kernel sets when one of its bounded waits runs out, one per device, in pinned host memory that the kernels write
// directly: a failure is visible to the next call without a copy, an event or a synchronisation per launch.
Tensor ssd_status(int64_t device) {
  static std::mutex lock;
  static std::vector<Tensor> words(64);
  TORCH_CHECK(device >= 0 && device < (int64_t)words.size(), "ssd_scan: device index out of range");
  std::lock_guard<std::mutex> hold(lock);
  Tensor& w = words[device];
  if (!w.defined()) w = at::zeros({1}, at::TensorOptions().dtype(at::kInt)).pin_memory();
  return w;
}
// Raise if a launch since the last report ran out of a wait.
void ssd_poll(int64_t device) {
  volatile int32_t* word = ssd_status(device).data_ptr<int32_t>();
  const int32_t code = *word;
  if (code == 0) return;
  *word = 0;
  TORCH_CHECK(false, std::string() + "ssd_scan: a bounded device-side wait ran out in an earlier launch (status " + std::to_string(code) + "); its outputs are invalid");
}

struct SsdShape {
  int64_t nb, nl, nh, np, ng, nn;
};
SsdShape ssd_check(const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D, const OptTensor& z,
                   const OptTensor& dt_bias, const OptTensor& init) {
  SSM_ARG(X.dim() == 4 && dt.dim() == 3, "X must be (B, L, H, P) and dt (B, L, H).");
  SsdShape s{X.size(0), X.size(1), X.size(2), X.size(3), 0, 0};
  SSM_ARG(dt.size(0) == s.nb && dt.size(1) == s.nl && dt.size(2) == s.nh, "dt must align with (B, L, H).");
  SSM_ARG(A.dim() == 1 && A.size(0) == s.nh, "A must have shape (H,).");
  SSM_ARG(B.dim() == 4 && B.size(0) == s.nb && B.size(1) == s.nl && B.sizes() == C.sizes(), "B and C must have shape (B, L, G, N).");
  s.ng = B.size(2), s.nn = B.size(3);
  SSM_ARG(s.ng > 0 && s.nh % s.ng == 0, "Group dimension must divide H.");
  if (D.has_value())
    SSM_ARG((D->dim() == 1 && D->size(0) == s.nh) || (D->dim() == 2 && D->size(0) == s.nh && D->size(1) == s.np), "D must have shape (H,) or (H, P).");
  if (z.has_value()) SSM_ARG(z->sizes() == X.sizes(), "z must have shape (B, L, H, P).");
  if (dt_bias.has_value()) SSM_ARG(dt_bias->dim() == 1 && dt_bias->size(0) == s.nh, "dt_bias must have shape (H,).");
  if (init.has_value())
    SSM_ARG(init->dim() == 4 && init->size(0) == s.nb && init->size(1) == s.nh && init->size(2) == s.np && init->size(3) == s.nn,
            "initial_states must have shape (B, H, P, N).");
  same_device(X, {&dt, &A, &B, &C});
  need_cuda(X, {&D, &z, &dt_bias, &init});
  return s;
}

// Boundaries of packed sequences as host integers (one read of cu_seqlens), checked.  Called from Python; other threads of the
// interpreter run while this one waits for the device.
std::vector<int64_t> seq_bounds(const Tensor& cu, int64_t len) {
  Tensor host;
  {
    py::gil_scoped_release unlocked;
    host = cu.to(at::kCPU, at::kLong).contiguous();
  }
  std::vector<int64_t> v(host.data_ptr<int64_t>(), host.data_ptr<int64_t>() + host.numel());
  bool ok = v.size() >= 2 && v.front() == 0 && v.back() == len;
  for (size_t i = 1; i < v.size(); ++i) ok = ok && v[i] >= v[i - 1];
  SSM_ARG(ok, "cu_seqlens must rise from 0 to L.");
  return v;
}

// (Y, final states fp32); the caller has checked ssm_ssd_supported().  With `cu` the sequences packed along L of a batch of one are
// scanned each from a zero state and the states are per sequence (S, H, P, N); want_y false: states only.
std::tuple<Tensor, Tensor> ssd_run(const Tensor& X_, const Tensor& dt_, const Tensor& A_, const Tensor& B_, const Tensor& C_, const OptTensor& D_,
                                   const OptTensor& z_, const OptTensor& bias_, bool softplus, const OptTensor& init_, int64_t chunk,
                                   const std::vector<int64_t>* cu, bool want_y, const Tensor& cu_device = Tensor()) {
  const SsdShape s = ssd_check(X_, dt_, A_, B_, C_, D_, z_, bias_, init_);
  c10::cuda::CUDAGuard guard(X_.device());
  ssd_poll(X_.get_device());
  Tensor X = X_.detach().contiguous(), dt = like(dt_, X), B = like(B_, X), C = like(C_, X), A = f32c(A_), table;
  OptTensor D = f32c(D_), bias = f32c(bias_), init = f32c(init_), z;
  if (z_.has_value()) z = like(*z_, X);
  const auto f32 = X.options().dtype(at::kFloat);
  int64_t walks = s.nb, nchunks = s.nb * ((s.nl + chunk - 1) / chunk), bytes, state_bytes;
  ssm_ssd_args a{};
  if (cu) {
    walks = (int64_t)cu->size() - 1;
    std::vector<int32_t> t, first;
    for (int64_t q = 0; q < walks; ++q) {
      first.push_back((int32_t)(t.size() / 2));
      for (int64_t c = (*cu)[q]; c < (*cu)[q + 1]; c += chunk) t.push_back((int32_t)c), t.push_back((int32_t)(*cu)[q + 1]);
    }
    nchunks = (int64_t)t.size() / 2;
    first.push_back((int32_t)nchunks);
    t.insert(t.end(), first.begin(), first.end());
    table = at::empty({(int64_t)t.size()}, at::TensorOptions().dtype(at::kInt));
    std::copy(t.begin(), t.end(), table.data_ptr<int32_t>());
    table = table.to(X.device(), true);
    a.seq_table = table.data_ptr<int32_t>(), a.num_seqs = (int)walks, a.num_chunks = (int)nchunks;
    bytes = ssm_ssd_packed_scratch_bytes((int)walks, (int)nchunks, (int)s.nh, &state_bytes);
  } else if (cu_device.defined()) {  // the table is formed where the boundaries are; every sequence may end inside a chunk
    walks = cu_device.numel() - 1, nchunks = s.nl / chunk + walks;
    table = at::empty({2 * nchunks + walks + 1}, X.options().dtype(at::kInt));
    run(ssmb_seq_table(cu_device.data_ptr(), cu_device.scalar_type() == at::kLong, (int)walks, (int)s.nl, (int)nchunks, table.data_ptr<int32_t>(), stream_of(X)));
    a.seq_table = table.data_ptr<int32_t>(), a.num_seqs = (int)walks, a.num_chunks = (int)nchunks;
    bytes = ssm_ssd_packed_scratch_bytes((int)walks, (int)nchunks, (int)s.nh, &state_bytes);
  } else {
    bytes = ssm_ssd_scratch_bytes((int)s.nb, (int)s.nl, (int)s.nh), state_bytes = ssm_ssd_state_scratch_bytes((int)s.nb, (int)s.nl, (int)s.nh);
  }
  Tensor Y, fin;
  if (want_y) Y = at::empty_like(X);
  if (s.nl == 0) return {Y, init.has_value() ? init->clone() : at::zeros({walks, s.nh, s.np, s.nn}, f32)};  // no step: the state stays what it was
  fin = at::empty({walks, s.nh, s.np, s.nn}, f32);
  Tensor ws = at::empty({bytes}, X.options().dtype(at::kByte));
  const int64_t vec = s.nh * nchunks * chunk * 4;
  char* base = reinterpret_cast<char*>(ws.data_ptr());
  a.batch = (int)s.nb, a.len = (int)s.nl, a.heads = (int)s.nh, a.headdim = (int)s.np, a.nstate = (int)s.nn, a.groups = (int)s.ng;
  a.chunk_size = (int)chunk, a.io_dtype = dtype_code(X, "ssd_scan"), a.dt_softplus = softplus, a.d_has_p = D.has_value() && D->dim() == 2;
  a.phase = want_y ? 0 : 1;
  a.X = X.data_ptr(), a.dt = dt.data_ptr(), a.A = A.data_ptr<float>(), a.Bm = B.data_ptr(), a.Cm = C.data_ptr();
  a.D = fptr(D), a.z = ptr(z), a.dt_bias = fptr(bias), a.initial_states = fptr(init), a.Y = want_y ? Y.data_ptr() : nullptr;
  a.final_states = fin.data_ptr<float>();
  a.ws_dt = reinterpret_cast<float*>(base), a.ws_cum = reinterpret_cast<float*>(base + vec), a.ws_state = reinterpret_cast<float*>(base + 2 * vec);
  a.ws_state_in = base + 2 * vec + state_bytes;
  a.status = ssd_status(X.get_device()).data_ptr<int32_t>();
  run(ssm_ssd_fwd(&a, stream_of(X)));
  return {Y, fin};
}

// Differentiable call on the tensor cores; the backward runs in the dual form (see include/ssm_b200.h for its passes).
struct SsdCall final : Call {
  Tensor X_, dt_, A_, B_, C_;
  OptTensor D_, z_, bias_, init_;
  bool softplus;
  int64_t chunk;

  SsdCall(const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D, const OptTensor& z,
          const OptTensor& dt_bias, bool softplus_, const OptTensor& init, int64_t chunk_)
      : X_(X), dt_(dt), A_(A), B_(B), C_(C), D_(D), z_(z), bias_(dt_bias), init_(init), softplus(softplus_), chunk(chunk_) {
    for (const Tensor* t : {&X, &dt, &A, &B, &C}) input(*t);
    input(D), input(z), input(dt_bias), input(init);
  }
  variable_list forward(bool) override {
    auto [Y, fin] = ssd_run(X_, dt_, A_, B_, C_, D_, z_, bias_, softplus, init_, chunk, nullptr, true);
    return {Y, fin};
  }

  variable_list backward(const variable_list& grads) override {
    c10::cuda::CUDAGuard guard(X_.device());
    const int64_t nb = X_.size(0), nl = X_.size(1), nh = X_.size(2), np = X_.size(3), ng = B_.size(2), nn = B_.size(3), nchunks = (nl + chunk - 1) / chunk;
    const auto f32 = X_.options().dtype(at::kFloat).requires_grad(false);
    Tensor X = X_.detach().contiguous(), dt = like(dt_, X), B = like(B_, X), C = like(C_, X), A = f32c(A_);
    OptTensor D = f32c(D_), bias = f32c(bias_), init = f32c(init_), z;
    if (z_.has_value()) z = like(*z_, X);
    Tensor gy = grads[0].defined() ? like(grads[0], X) : at::zeros_like(X);
    OptTensor gfin;
    if (grads.size() > 1 && grads[1].defined()) gfin = f32c(grads[1]);
    const bool init_grad = init_.has_value() && init_->requires_grad();
    const int io = dtype_code(X, "ssd_scan");
    ssm_stream_t stream = stream_of(X);
    if (nl == 0) {  // the gradient of the final state is that of the initial one; everything else is empty or zero
      variable_list none;
      for (const Tensor* t : {&X_, &dt_, &A_, &B_, &C_}) none.push_back(at::zeros_like(*t));
      for (const OptTensor* t : {&D_, &z_, &bias_})
        if (t->has_value()) none.push_back(at::zeros_like(**t));
      if (init_.has_value()) none.push_back(!init_grad ? Tensor() : gfin.has_value() ? cast(gfin->clone(), init_->scalar_type()) : at::zeros_like(*init_));
      return none;
    }

    Tensor u, qd, dB, dC, dA, dD, dbias;
    ZeroPool work, coeffs, params;
    work.add(u, {nb, nl, nh}), work.add(qd, {nb, nl, nh});
    auto own = [&](const Tensor& t) -> ZeroPool& { return t.scalar_type() == at::kFloat ? coeffs : work; };  // in another type it is copied below
    own(B_).add(dB, {nb, nl, ng, nn}), own(C_).add(dC, {nb, nl, ng, nn});
    params.add(dA, {nh});
    if (D.has_value()) params.add(dD, D->sizes());
    if (bias.has_value()) params.add(dbias, {nh});
    work.make(f32), coeffs.make(f32), params.make(f32);
    Tensor dX = at::empty_like(X), ddt = at::empty_like(dt), dz, dinit, start0;

    ssm_ssd_bwd_args e{};
    e.batch = (int)nb, e.len = (int)nl, e.heads = (int)nh, e.headdim = (int)np, e.io_dtype = io, e.d_has_p = D.has_value() && D->dim() == 2;
    e.gY = gy.data_ptr(), e.z = ptr(z), e.X = X.data_ptr(), e.D = fptr(D), e.dX = dX.data_ptr(), e.dD = out_ptr(dD);
    Tensor dy = gy;
    if (z.has_value()) {
      dy = at::empty_like(X), dz = at::empty_like(X);
      e.dy = dy.data_ptr(), e.dz = dz.data_ptr();
      run(ssm_ssd_bwd_gate(&e, stream));
    }
    // forward again without skip and gate, then the adjoint pass on the same exponents
    const int64_t vec = nb * nh * nchunks * chunk * 4, fin_bytes = ssm_ssd_state_scratch_bytes((int)nb, (int)nl, (int)nh);
    const auto bytes = X.options().dtype(at::kByte);
    Tensor ws = at::empty({ssm_ssd_scratch_bytes((int)nb, (int)nl, (int)nh)}, bytes), ws_r = at::empty({ws.numel() - 2 * vec}, bytes);
    Tensor st32 = at::empty({nb, nchunks, nh, np * nn}, f32), ad32 = at::empty({nb, nchunks, nh, np * nn}, f32), y = at::empty_like(X), dx = at::empty_like(X), gstate;
    char *base = reinterpret_cast<char*>(ws.data_ptr()), *base_r = reinterpret_cast<char*>(ws_r.data_ptr());
    ssm_ssd_args a{};
    a.batch = (int)nb, a.len = (int)nl, a.heads = (int)nh, a.headdim = (int)np, a.nstate = (int)nn, a.groups = (int)ng, a.chunk_size = (int)chunk, a.io_dtype = io;
    a.dt_softplus = softplus, a.dt = dt.data_ptr(), a.A = A.data_ptr<float>(), a.dt_bias = fptr(bias);
    a.ws_dt = reinterpret_cast<float*>(base), a.ws_cum = reinterpret_cast<float*>(base + vec);
    a.status = ssd_status(X.get_device()).data_ptr<int32_t>();
    ssm_ssd_args f = a;
    f.X = X.data_ptr(), f.Bm = B.data_ptr(), f.Cm = C.data_ptr(), f.z = dy.data_ptr(), f.initial_states = fptr(init), f.Y = y.data_ptr();
    f.ws_state = reinterpret_cast<float*>(base + 2 * vec), f.ws_state_in = base + 2 * vec + fin_bytes;
    f.row_dots = u.data_ptr<float>(), f.ws_state_in_f32 = st32.data_ptr<float>();
    run(ssm_ssd_fwd(&f, stream));
    ssm_ssd_args r = a;
    r.reverse = 1, r.X = dy.data_ptr(), r.Bm = C.data_ptr(), r.Cm = B.data_ptr(), r.z = X.data_ptr(), r.initial_states = fptr(gfin), r.Y = dx.data_ptr();
    r.ws_state = reinterpret_cast<float*>(base_r), r.ws_state_in = base_r + fin_bytes;
    r.row_dots = qd.data_ptr<float>(), r.ws_state_in_f32 = ad32.data_ptr<float>();
    if (init.has_value()) gstate = at::empty({nb, nh, np, nn}, f32), r.final_states = gstate.data_ptr<float>();
    run(ssm_ssd_fwd(&r, stream));

    ssm_ssd_bc_args g{};
    g.batch = (int)nb, g.len = (int)nl, g.heads = (int)nh, g.groups = (int)ng, g.io_dtype = io;
    g.X = X.data_ptr(), g.dy = dy.data_ptr(), g.Bm = B.data_ptr(), g.Cm = C.data_ptr(), g.ws_dt = a.ws_dt, g.ws_cum = a.ws_cum;
    g.state_in = f.ws_state_in, g.adjoint_in = r.ws_state_in, g.dB = out_ptr(dB), g.dC = out_ptr(dC), g.status = a.status;
    run(ssm_ssd_bwd_bc(&g, stream));
    e.y_plain = y.data_ptr(), e.dx = dx.data_ptr();
    run(ssm_ssd_bwd_finish(&e, stream));
    if (init.has_value()) {  // the state before the first step: one decay further
      Tensor c0 = ws.narrow(0, vec, vec).view(at::kFloat).view({nb, nh, nchunks * chunk}).select(2, 0);
      dinit = gstate * at::exp2(c0).unsqueeze(-1).unsqueeze(-1);
      start0 = (dinit * *init).sum({-2, -1}).contiguous();
    }
    ssm_ssd_steps_args s{};
    s.batch = (int)nb, s.len = (int)nl, s.heads = (int)nh, s.io_dtype = io, s.dt_softplus = softplus;
    s.dt = dt.data_ptr(), s.dt_bias = fptr(bias), s.A = A.data_ptr<float>(), s.u = u.data_ptr<float>(), s.qd = qd.data_ptr<float>(), s.ws_cum = a.ws_cum;
    s.state_f32 = st32.data_ptr<float>(), s.adjoint_f32 = ad32.data_ptr<float>(), s.start0 = start0.defined() ? start0.data_ptr<float>() : nullptr;
    s.ddt = ddt.data_ptr(), s.dA = out_ptr(dA), s.ddt_bias = out_ptr(dbias);
    run(ssm_ssd_bwd_steps(&s, stream));

    auto to = [](const Tensor& grad, const Tensor& t) { return cast(grad, t.scalar_type()); };
    if (const auto type = B_.scalar_type(); type != at::kFloat && type == C_.scalar_type()) {  // neighbours at the end of the pool: one conversion
      const int64_t n = dB.numel();
      Tensor both = work.all.narrow(0, work.all.numel() - 2 * n, 2 * n).to(type);
      dB = both.narrow(0, 0, n).view(dB.sizes()), dC = both.narrow(0, n, n).view(dC.sizes());
    }
    variable_list res = {dX, to(ddt, dt_), to(dA, A_), to(dB, B_), to(dC, C_)};
    if (D_.has_value()) res.push_back(to(dD, *D_));
    if (z_.has_value()) res.push_back(to(dz, *z_));
    if (bias_.has_value()) res.push_back(to(dbias, *bias_));
    if (init_.has_value()) res.push_back(init_grad ? to(dinit, *init_) : Tensor());
    return res;
  }
};

std::tuple<Tensor, Tensor> ssd_scan(const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D,
                                    const OptTensor& z, const OptTensor& dt_bias, bool softplus, const OptTensor& init, int64_t chunk) {
  ValueErrors scope;
  ssd_check(X, dt, A, B, C, D, z, dt_bias, init);
  variable_list r = invoke_call(c10::make_intrusive<SsdCall>(X, dt, A, B, C, D, z, dt_bias, softplus, init, chunk));
  return {r[0], r[1]};
}

// ---------------------------------------------------------------------------------------------
// whole mixers
// ---------------------------------------------------------------------------------------------
// A mixer of a short sequence is bound by the host: as separate calls its projections and operators were two dozen autograd nodes, 0.95 ms
// of host time per training step for 0.12 ms of device time (d_model 256, 256 steps).  The calls below are the same products and
// operators behind one node; products that add into a gradient do so in their epilogue instead of a pass of their own.
//
// They stand for the composed form only where nothing can tell the difference: no tracing, autocast or saved-tensor hooks, plain types, no weight with a
// tangent, which a product behind the operators carries.
bool composed_only(const Tensor& x, std::initializer_list<const Tensor*> weights) {
  if (at::tracer::impl::is_dispatch_enabled() || at::autocast::is_autocast_enabled(at::kCUDA) || at::SavedTensorDefaultHooks::get_hooks().has_value()) return true;
  if (!x.is_cuda() || x.dim() != 3 || x.numel() == 0 || !io_dtype_ok(x)) return true;
  for (const Tensor* w : weights)
    if (w->scalar_type() != x.scalar_type() || w->dim() != 2 || w->device() != x.device() || w->_fw_grad(0).defined()) return true;
  return false;
}

struct Mamba1MixerCall final : Call {
  Tensor hidden, in_x, in_z, conv_w, x_proj, dt_proj, dt_bias, A_in, D, out_proj;
  OptTensor conv_b;
  bool a_log;
  int64_t nb, nl, dm, di, n, r;
  enum { kHidden, kInX, kInZ, kConvW, kConvB };
  int kXProj, kDtProj, kDtBias, kA, kD, kOut;  // the inputs behind the conv's bias, if it has one
  std::vector<bool> need;
  bool conv_live, scan_live;  // parts that a gradient flows back through
  // of the forward pass, what the backward reads
  Tensor h2, u2, xd, y2, A;
  c10::intrusive_ptr<ConvCall> conv;
  c10::intrusive_ptr<ScanCall> scan;

  Mamba1MixerCall(const Tensor& hidden_, const Tensor& in_x_, const Tensor& in_z_, const Tensor& conv_w_, const OptTensor& conv_b_, const Tensor& x_proj_,
                  const Tensor& dt_proj_, const Tensor& dt_bias_, const Tensor& A_, bool a_log_, const Tensor& D_, const Tensor& out_proj_)
      : hidden(hidden_), in_x(in_x_), in_z(in_z_), conv_w(conv_w_), x_proj(x_proj_), dt_proj(dt_proj_), dt_bias(dt_bias_), A_in(A_), D(D_), out_proj(out_proj_),
        conv_b(conv_b_), a_log(a_log_) {
    for (const Tensor* t : {&hidden, &in_x, &in_z, &conv_w}) input(*t);
    input(conv_b);
    for (const Tensor* t : {&x_proj, &dt_proj, &dt_bias, &A_in, &D, &out_proj}) input(*t);
    for (const Tensor& t : inputs) need.push_back(t.requires_grad());
    kXProj = kConvB + conv_b.has_value(), kDtProj = kXProj + 1, kDtBias = kXProj + 2, kA = kXProj + 3, kD = kXProj + 4, kOut = kXProj + 5;
    conv_live = need[kHidden] || need[kInX] || need[kConvW] || (conv_b.has_value() && need[kConvB]);
    scan_live = conv_live || need[kInZ];
    for (int i = kXProj; i < kOut; ++i) scan_live = scan_live || need[i];
    nb = hidden.size(0), nl = hidden.size(1), dm = hidden.size(2), di = in_x.size(0), r = dt_proj.size(1), n = (x_proj.size(0) - r) / 2;
  }
  Tensor rows(const Tensor& m) const { return m.view({m.size(0), nb, nl}).permute({1, 0, 2}); }                    // (C, B L) -> (B, C, L)
  Tensor flat(const Tensor& t) const { return t.permute({1, 0, 2}).reshape({t.size(1), nb * nl}); }                // and back

  bool survives_its_walk() const override { return false; }
  // The products are formed in the types of the forward pass, also where the backward runs inside autocast.
  using NoAutocast = c10::impl::ExcludeDispatchKeyGuard;
  // What the products and operators would keep one by one: a factor of a product where the other factor takes a gradient, all inputs of an
  // operator, A as it is formed (not its logarithm).
  bool reads(size_t input) const override {
    const int i = (int)input;
    if (i == kHidden) return need[kInX] || need[kInZ];
    if (i == kInX || i == kInZ) return need[kHidden];
    if (i <= kXProj) return conv_live;  // conv_w, conv_b, x_proj
    if (i == kDtProj) return conv_live || need[kXProj];
    return scan_live && !(i == kA && a_log);
  }

  // keep: for backward().  Else autograd records the parts wherever it records.
  Tensor evaluate(bool keep) {
    Tensor h = hidden.reshape({nb * nl, dm});
    Tensor x = at::mm(in_x, h.t()), z = at::mm(in_z, h.t());
    auto cv = c10::make_intrusive<ConvCall>(rows(x), conv_w, conv_b, "silu", OptTensor());
    Tensor u = (keep ? cv->forward(true) : invoke_call(cv))[0], uf = flat(u);
    Tensor xdbl = at::mm(x_proj, uf), delta = at::mm(dt_proj, xdbl.narrow(0, 0, r));
    auto coeff = [&](int64_t from) { return xdbl.narrow(0, from, n).view({n, nb, nl}).permute({1, 0, 2}).unsqueeze(1); };  // (B, 1, N, L)
    Tensor Av = a_log ? at::exp(A_in).neg() : A_in;
    auto sc = c10::make_intrusive<ScanCall>(u, rows(delta), Av, coeff(r), coeff(r + n), OptTensor(D), OptTensor(rows(z)), OptTensor(dt_bias), true, false, OptTensor(), false);
    Tensor yf = flat((keep ? sc->forward(scan_live) : invoke_call(sc))[0]);
    if (keep) {
      cv->inputs.clear(), sc->inputs.clear();
      sc->t_B = sc->t_C = at::kFloat;  // their gradients are converted where they are copied
      if (need[kInX] || need[kInZ]) h2 = h;
      if (need[kDtProj]) xd = xdbl;
      if (need[kXProj]) u2 = uf;
      if (need[kOut]) y2 = yf;
      if (need[kA]) A = Av;
      if (conv_live) conv = cv;
      if (scan_live) scan = sc;
    }
    return at::mm(yf.t(), out_proj.t()).view({nb, nl, dm});
  }

  variable_list forward(bool train) override {
    c10::cuda::CUDAGuard guard(out_proj.device());
    Tensor out = evaluate(train);
    if (train && !reads(kHidden)) {  // its values are not needed again; what hangs on its graph is an alias without any
      for (size_t i = 0; i < unread.size(); ++i)
        if (unread[i].first.is_same(hidden)) unread.erase(unread.begin() + i--);
      if (need[kHidden]) {
        at::AutoGradMode record(true);
        const Tensor none = hidden.narrow(0, 0, 0).clone();
        unread.emplace_back(none, none._version());
      }
      hidden = Tensor();
    }
    return {out};
  }

  // What can be differentiated twice (the products) has to be: the composed form again, for autograd to record.  Its inputs are aliases, so
  // that hooks on the real ones see one gradient each.
  variable_list backward_recorded(const variable_list& grads) override {
    bool edited = !hidden.defined();
    for (const auto& kept : unread) edited = edited || kept.first._version() != kept.second;
    if (edited || !grads[0].defined()) return Call::backward_recorded(grads);
    NoAutocast plain_types(c10::autocast_dispatch_keyset);
    c10::cuda::CUDAGuard guard(hidden.device());
    variable_list asked;
    size_t at_input = 0;
    auto alias = [&](const Tensor& t) {
      if (!need[at_input++]) return t.detach();
      asked.push_back(at::alias(t));
      if (!asked.back().requires_grad()) asked.back().requires_grad_();  // switched off since
      return asked.back();
    };
    const Tensor a_hidden = alias(hidden), a_in_x = alias(in_x), a_in_z = alias(in_z), a_conv_w = alias(conv_w);
    const OptTensor a_conv_b = conv_b.has_value() ? OptTensor(alias(*conv_b)) : conv_b;
    const Tensor a_x_proj = alias(x_proj), a_dt_proj = alias(dt_proj), a_dt_bias = alias(dt_bias), a_A = alias(A_in), a_D = alias(D), a_out_proj = alias(out_proj);
    Tensor out = c10::make_intrusive<Mamba1MixerCall>(a_hidden, a_in_x, a_in_z, a_conv_w, a_conv_b, a_x_proj, a_dt_proj, a_dt_bias, a_A, a_log, a_D, a_out_proj)->evaluate(false);
    const variable_list got = torch::autograd::grad({out}, asked, {cast(grads[0], out.scalar_type())}, true, true, true);
    variable_list res;
    size_t next = 0;
    for (bool wanted : need) res.push_back(wanted ? got[next++] : Tensor());
    return res;
  }

  // Each tensor goes with its last use, on the walk that ends the graph those of the forward pass too.
  variable_list backward(const variable_list& grads) override {
    c10::cuda::CUDAGuard guard(out_proj.device());
    NoAutocast plain_types(c10::autocast_dispatch_keyset);
    const bool ends = !torch::autograd::get_current_graph_task_keep_graph();
    auto drop = [&](auto& kept) {
      if (ends) kept = std::decay_t<decltype(kept)>();
    };
    variable_list res(kOut + 1);
    if (!grads[0].defined()) return res;
    Tensor g = cast(grads[0], out_proj.scalar_type()).reshape({nb * nl, dm});
    if (need[kOut]) res[kOut] = at::mm(g.t(), y2.t());
    drop(y2);
    if (!scan_live) return res;
    variable_list s = scan->backward({rows(at::mm(out_proj.detach().t(), g.t()))});  // u, delta, A, B, C, D, z, dt_bias
    drop(scan);
    Tensor du = flat(s[0]), dd = flat(s[1]), dz = flat(s[6]);
    s[0] = s[1] = s[6] = g = Tensor();
    if (need[kA]) res[kA] = cast(a_log ? s[2].mul_(A) : s[2], A_in.scalar_type());
    if (need[kD]) res[kD] = cast(s[5], D.scalar_type());
    if (need[kDtBias]) res[kDtBias] = cast(s[7], dt_bias.scalar_type());
    if (need[kInZ]) res[kInZ] = at::mm(dz, h2);
    if (!need[kHidden]) dz = Tensor();
    if (need[kDtProj]) res[kDtProj] = at::mm(dd, xd.narrow(0, 0, r).t());
    drop(xd);
    if (!(conv_live || need[kXProj])) return res;
    Tensor dxd = at::empty({r + 2 * n, nb * nl}, du.options()), low = dxd.narrow(0, 0, r);
    at::mm_out(low, dt_proj.detach().t(), dd);
    dd = Tensor();
    dxd.narrow(0, r, n).view({n, nb, nl}).copy_(s[3].squeeze(1).permute({1, 0, 2}));
    dxd.narrow(0, r + n, n).view({n, nb, nl}).copy_(s[4].squeeze(1).permute({1, 0, 2}));
    s.clear();
    if (need[kXProj]) res[kXProj] = at::mm(dxd, u2.t());
    drop(u2);
    if (!conv_live) return res;
    du.addmm_(x_proj.detach().t(), dxd);
    variable_list c = conv->backward({rows(du)});
    drop(conv);
    du = dxd = Tensor();
    if (need[kConvW]) res[kConvW] = c[1];
    if (conv_b.has_value() && need[kConvB]) res[kConvB] = c[2];
    Tensor dx = flat(c[0]);
    c.clear();
    if (need[kInX]) res[kInX] = at::mm(dx, h2);
    drop(h2);
    if (need[kHidden]) {
      Tensor dh = at::mm(dx.t(), in_x.detach());
      dh.addmm_(dz.t(), in_z.detach());
      res[kHidden] = dh.view({nb, nl, dm});
    }
    return res;
  }
};

// hidden (B, L, d_model) through a Mamba-1 mixer; None where the composed form has to serve.
py::object mamba1_mixer(const Tensor& hidden, const Tensor& in_x, const Tensor& in_z, const Tensor& conv_w, const OptTensor& conv_b, const Tensor& x_proj,
                        const Tensor& dt_proj, const Tensor& dt_bias, const Tensor& A, bool a_log, const Tensor& D, const Tensor& out_proj) {
  ValueErrors scope;
  if (composed_only(hidden, {&in_x, &in_z, &x_proj, &dt_proj, &out_proj})) return py::none();
  const int64_t dm = hidden.size(2), di = in_x.size(0), r = dt_proj.size(1), rest = x_proj.size(0) - r;
  if (in_x.size(1) != dm || in_z.sizes() != in_x.sizes() || x_proj.size(1) != di || dt_proj.size(0) != di || out_proj.size(0) != dm || out_proj.size(1) != di ||
      r < 1 || rest < 2 || rest % 2 != 0 || A.dim() != 2 || A.size(0) != di || A.size(1) != rest / 2 || conv_w.size(0) != di)
    return py::none();
  return py::cast(invoke_call(c10::make_intrusive<Mamba1MixerCall>(hidden, in_x, in_z, conv_w, conv_b, x_proj, dt_proj, dt_bias, A, a_log, D, out_proj))[0]);
}

// u (B, L, d_model), normed, through a Mamba-2 mixer on the tensor-core scan, without gradients; None where the composed form has to serve.
py::object mamba2_mixer(const Tensor& u, const Tensor& in_z, const Tensor& in_x, const Tensor& in_B, const Tensor& in_C, const Tensor& in_dt, const Tensor& wx,
                        const OptTensor& bx, const Tensor& wB, const OptTensor& bB, const Tensor& wC, const OptTensor& bC, const Tensor& dt_bias, const Tensor& A_log,
                        const Tensor& D, const Tensor& norm_w, const Tensor& out_proj, int64_t nh, int64_t hp, int64_t n, int64_t g, int64_t chunk, double eps) {
  ValueErrors scope;
  if (at::GradMode::is_enabled() || composed_only(u, {&in_z, &in_x, &in_B, &in_C, &in_dt, &out_proj})) return py::none();
  const int64_t nb = u.size(0), nl = u.size(1), dm = u.size(2), di = nh * hp;
  if (!ssm_ssd_supported((int)hp, (int)n, (int)chunk, dtype_code(u, "mamba2_mixer")) || in_x.size(0) != di || in_x.size(1) != dm) return py::none();
  c10::cuda::CUDAGuard guard(u.device());
  Tensor u2 = u.reshape({nb * nl, dm});
  auto proj = [&](const Tensor& w) { return at::mm(u2, w.t()).view({nb, nl, w.size(0)}); };
  auto conv = [&](const Tensor& t, const Tensor& w, const OptTensor& b) {
    const bool square = nl == t.size(2);  // as many steps as channels: (B, L, C) would be taken for (B, C, L)
    Tensor y = invoke_call(c10::make_intrusive<ConvCall>(square ? t.transpose(1, 2) : t, w, b, "silu", OptTensor()))[0];
    return square ? y.transpose(1, 2).contiguous() : y;
  };
  Tensor x = conv(proj(in_x), wx, bx).view({nb, nl, nh, hp}), B = conv(proj(in_B), wB, bB).view({nb, nl, g, n}), C = conv(proj(in_C), wC, bC).view({nb, nl, g, n});
  Tensor z = proj(in_z).view({nb, nl, nh, hp}), dt = proj(in_dt);
  Tensor y = std::get<0>(ssd_scan(x, dt, at::exp(A_log).neg_(), B, C, D, z, dt_bias, true, OptTensor(), chunk));
  y = invoke_call(c10::make_intrusive<NormCall>(y.view({nb, nl, di}), norm_w, OptTensor(), OptTensor(), true, eps, true, false, true))[0];
  return py::cast(at::mm(y.view({nb * nl, di}), out_proj.t()).view({nb, nl, dm}));
}

// Packed sequences.  reset: Y restarts at every boundary; without it Y is the scan through all of them.  -> (Y, last state, states)
std::tuple<Tensor, Tensor, Tensor> ssd_packed(const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D,
                                              const OptTensor& z, const OptTensor& dt_bias, bool softplus, const OptTensor& init, int64_t chunk,
                                              const Tensor& cu_seqlens, bool reset) {
  ValueErrors scope;
  // Boundaries on the device: the kernels are enqueued behind a table formed there, and the copy that the boundaries are checked on is awaited
  // only then, so that the device does not stand idle while the host reads them (35 us for 24 sequences in 16384 steps of 48 heads, 20 us at 4 to
  // 512 sequences in 512 to 16384).  The table has room for a chunk per sequence, 18 KB of scratch per head even where the sequence is
  // empty (boundaries padded to a fixed number: 1024 entries, 48 heads 0.9 GB): with more than four sequences to a chunk, and more than
  // 64, the host counts the chunks.
  const int64_t seqs = cu_seqlens.dim() == 1 ? cu_seqlens.numel() - 1 : 0, whole_chunks = X.size(1) / chunk, chunk_slots = whole_chunks + seqs;
  if (reset && seqs >= 1 && seqs <= std::max<int64_t>(64, 4 * whole_chunks) && cu_seqlens.is_cuda() && cu_seqlens.get_device() == X.get_device() && chunk_slots <= 65535 && X.size(1) > 0 && X.size(1) < (1 << 30)) {
    c10::cuda::CUDAGuard guard(X.device());
    const Tensor bounds = cu_seqlens.scalar_type() == at::kInt ? cu_seqlens.contiguous() : cu_seqlens.to(at::kLong).contiguous();
    Tensor host = at::empty(bounds.sizes(), bounds.options().device(at::kCPU).pinned_memory(true));
    host.copy_(bounds, true);
    at::cuda::CUDAEvent copied;
    copied.record(at::cuda::getCurrentCUDAStream(X.get_device()));
    auto [Y, states] = ssd_run(X, dt, A, B, C, D, z, dt_bias, softplus, c10::nullopt, chunk, nullptr, true, bounds);
    Tensor last = states.slice(0, states.size(0) - 1).clone();
    {
      py::gil_scoped_release unlocked;
      copied.synchronize();
    }
    seq_bounds(host, X.size(1));
    return {Y, last, states};
  }
  const std::vector<int64_t> cu = seq_bounds(cu_seqlens, X.size(1));
  // One set of launches takes up to 65535 sequences and chunks (a grid axis each); beyond that, groups of sequences one after the other.
  constexpr int64_t kMost = 65535;
  const int64_t nseq = (int64_t)cu.size() - 1;
  std::vector<Tensor> Ys, all;
  for (int64_t s0 = 0, s1; s0 < nseq; s0 = s1) {
    int64_t chunks = 0;
    for (s1 = s0; s1 < nseq && s1 - s0 < kMost; ++s1) {
      const int64_t more = (cu[s1 + 1] - cu[s1] + chunk - 1) / chunk;
      if (s1 > s0 && chunks + more > kMost) break;
      chunks += more;
    }
    const bool whole = s1 - s0 == nseq;
    const int64_t t0 = cu[s0], len = cu[s1] - t0;
    if (len == 0) {  // nothing but empty sequences
      all.push_back(at::zeros({s1 - s0, X.size(2), X.size(3), B.size(3)}, X.options().dtype(at::kFloat)));
      continue;
    }
    auto rows = [&](const Tensor& t) { return whole ? t : t.narrow(1, t0, len); };
    std::vector<int64_t> part(cu.begin() + s0, cu.begin() + s1 + 1);
    for (int64_t& v : part) v -= t0;
    auto [y, st] = ssd_run(rows(X), rows(dt), A, rows(B), rows(C), D, z.has_value() ? OptTensor(rows(*z)) : z, dt_bias, softplus, c10::nullopt, chunk, &part, reset);
    if (reset) Ys.push_back(y);
    all.push_back(st);
  }
  Tensor Y, last, states = all.size() == 1 ? all[0] : at::cat(all);
  if (reset) Y = Ys.size() == 1 ? Ys[0] : at::cat(Ys, 1);
  if (reset) last = states.slice(0, states.size(0) - 1).clone();
  else std::tie(Y, last) = ssd_run(X, dt, A, B, C, D, z, dt_bias, softplus, init, chunk, nullptr, true);
  return {Y, last, states};
}

}  // namespace

void bind_operators(py::module& m) {
  auto ops = m.def_submodule("operators", "the operator surface of ssm_b200.ops");
  ops.def("selective_scan", &selective_scan);
  ops.def("state_step", &state_step);
  ops.def("state_step_heads", &state_step_heads);
  ops.def("ssd_chunk_scan", &ssd_chunk_scan);
  ops.def("dw_causal_conv", &dw_causal_conv);
  ops.def("dw_causal_conv_update", &dw_causal_conv_update);
  ops.def("fused_layer_norm", &fused_layer_norm);
  ops.def("mamba1_step", &mamba1_step);
  ops.def("mamba2_step", &mamba2_step);
  ops.def("mamba1_mixer", &mamba1_mixer);
  ops.def("mamba2_mixer", &mamba2_mixer);
  ops.def("ssd_scan", &ssd_scan);
  ops.def("ssd_packed", &ssd_packed);
  ops.def("ssd_status", &ssd_status);
  ops.def("ssd_poll", &ssd_poll);
}

}  // namespace ssm_ext
