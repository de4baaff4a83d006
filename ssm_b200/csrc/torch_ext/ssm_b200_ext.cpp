// Thin PyTorch extension over the C ABI of include/ssm_b200.h.
//
// It exports the ten callables that upstream's facade (src/ssm/ops/__init__.py) invokes on
// its compiled CUDA backend, with the names, keyword arguments, defaults and return tuples
// that src/ssm/ops/cuda/bindings.cpp:96-152 fixes (selective_scan -> 3-tuple,
// selective_scan_backward -> 8-tuple, selective_state_step_backward -> the 9 values the
// facade zips with its nine requires_grad flags at src/ssm/ops/__init__.py:669-676, ...).
// Each function validates shapes the way the specification does (reference.py:22-84 and the
// operator bodies), allocates its outputs with ATen, fills the plain C struct of the matching
// entry point from data_ptr() / stride(), and launches on the current CUDA stream of the
// tensors' device.  Violations are reported with TORCH_CHECK, i.e. as RuntimeError, which the
// facade turns into ValueError (src/ssm/ops/__init__.py:1244-1252).  There is no fallback of
// any kind: CPU tensors are rejected.
#include "operands.h"

namespace ssm_ext {
void bind_operators(pybind11::module& m);  // operators.cpp
}

using namespace ssm_ext;

namespace {

// ---------------------------------------------------------------------------------------------
// selective scan
// ---------------------------------------------------------------------------------------------
std::tuple<Tensor, Tensor, Tensor> selective_scan(const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C,
                                                  const OptTensor& D, const OptTensor& z, const OptTensor& dt_bias, bool softplus,
                                                  bool return_last_state) {
  ScanCtx c(u, delta, A, B, C, D, z, dt_bias, softplus);
  c10::cuda::CUDAGuard guard(c.u.device());
  Tensor out = at::empty_like(c.u);
  Tensor last = return_last_state ? at::empty({c.nb, c.nd, c.nn}, c.u.options()) : at::empty({0}, c.u.options());
  Tensor cache = scan_checkpoints(c);
  ssm_scan_fwd_args a{};
  c.fill(a);
  a.out = out.data_ptr();
  a.last_state = return_last_state ? last.data_ptr() : nullptr;
  a.last_dtype = a.io_dtype;
  a.checkpoints = cache.data_ptr<float>();
  const int nseg = ssm_scan_split_segments((int)c.nb, (int)c.nd, (int)c.nl, (int)c.nn);  // > 1: cut the sequence into parallel segments
  Tensor split;
  if (nseg > 1) {
    split = at::empty({2 * c.nb * c.nd * nseg * c.nn}, c.u.options().dtype(at::kFloat));
    a.split_scratch = split.data_ptr<float>(), a.split_segments = nseg;
  }
  run(ssm_selective_scan_fwd(&a, stream_of(c.u)));
  return {out, last, cache};
}

// gradient buffer of a coefficient, folded back to the shape / dtype of the tensor the caller passed
Tensor fold_coeff_grad(const Tensor& grad, const Tensor& like_) {
  Tensor g = grad;
  if (g.sizes() != like_.sizes()) {  // the coefficient had been regrouped: sum the repeats back
    const int64_t rep = g.size(1) / like_.size(1);
    g = g.view({like_.size(0), like_.size(1), rep, like_.size(2), like_.size(3)}).sum(2);
  }
  return g.to(like_.scalar_type());
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, OptTensor, OptTensor, OptTensor> selective_scan_backward(
    const Tensor& grad_output, const OptTensor& grad_last_state, const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B,
    const Tensor& C, const OptTensor& D, const OptTensor& z, const OptTensor& dt_bias, bool softplus, const OptTensor& forward_output,
    const OptTensor& cache) {
  (void)forward_output;  // the kernel rebuilds what it needs from the checkpoints
  ScanCtx c(u, delta, A, B, C, D, z, dt_bias, softplus);
  c10::cuda::CUDAGuard guard(c.u.device());
  TORCH_CHECK(grad_output.sizes() == c.u.sizes(), "grad_output must have the shape of u.");
  Tensor ck;
  ssm_scan_bwd_args g{};
  c.fill(g.fwd);
  if (cache.has_value() && cache->numel() > 0) {
    ck = f32c(*cache);
  } else {  // no checkpoints handed over: one forward pass produces them
    ck = scan_checkpoints(c);
    Tensor scratch_out = at::empty_like(c.u);
    ssm_scan_fwd_args f = g.fwd;
    f.out = scratch_out.data_ptr(), f.checkpoints = ck.data_ptr<float>();
    run(ssm_selective_scan_fwd(&f, stream_of(c.u)));
  }
  g.fwd.checkpoints = ck.data_ptr<float>();
  const auto f32 = c.u.options().dtype(at::kFloat);
  Tensor go = like(grad_output, c.u);
  OptTensor gl = f32c(grad_last_state);
  if (gl.has_value()) TORCH_CHECK(gl->dim() == 3 && gl->size(0) == c.nb && gl->size(1) == c.nd && gl->size(2) == c.nn, "grad_last_state must have shape (B, D, N).");
  Tensor du = at::empty_like(c.u), dd = at::empty_like(c.u);
  OptTensor dz = c.z.has_value() ? OptTensor(at::empty_like(c.u)) : OptTensor();
  Tensor dA = at::zeros({c.nd, c.nn}, f32), dB = at::zeros(c.B.t.sizes(), f32), dC = at::zeros(c.C.t.sizes(), f32);
  OptTensor dD = c.D.has_value() ? OptTensor(at::zeros({c.nd}, f32)) : OptTensor();
  OptTensor db = c.bias.has_value() ? OptTensor(at::zeros({c.nd}, f32)) : OptTensor();
  g.dout = go.data_ptr(), g.dlast_state = fptr(gl);
  g.du = du.data_ptr(), g.ddelta = dd.data_ptr(), g.dz = dz.has_value() ? dz->data_ptr() : nullptr;
  g.dA = dA.data_ptr<float>(), g.dB = dB.data_ptr<float>(), g.dC = dC.data_ptr<float>();
  g.db_sb = c.B.sb, g.db_sg = c.B.sg, g.db_sn = c.B.sn, g.db_st = c.B.st;
  g.dc_sb = c.C.sb, g.dc_sg = c.C.sg, g.dc_sn = c.C.sn, g.dc_st = c.C.st;
  g.dD = fptr_mut(dD), g.ddt_bias = fptr_mut(db), g.dinitial_state = nullptr;
  if (c.nb * c.nd * c.nl > 0) run(ssm_selective_scan_bwd(&g, stream_of(c.u)));
  else du.zero_(), dd.zero_();
  auto cast = [](const OptTensor& grad, const OptTensor& src) { return grad.has_value() ? OptTensor(grad->to(src->scalar_type())) : OptTensor(); };
  return {du.to(u.scalar_type()), dd.to(delta.scalar_type()), dA.to(A.scalar_type()), fold_coeff_grad(dB, B.dim() == 4 ? B : dB).to(B.scalar_type()),
          fold_coeff_grad(dC, C.dim() == 4 ? C : dC).to(C.scalar_type()), cast(dD, D), cast(dz, z), cast(db, dt_bias)};
}

// ---------------------------------------------------------------------------------------------
// single-token state step
// ---------------------------------------------------------------------------------------------
Tensor selective_state_step(Tensor state, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D,
                            const OptTensor& z, const OptTensor& dt_bias, bool softplus) {
  StepCtx c(state, x, dt, A, B, C, D, z, dt_bias, softplus);
  c10::cuda::CUDAGuard guard(state.device());
  const bool direct = state.scalar_type() == at::kFloat && state.is_contiguous();
  Tensor work = direct ? state.detach() : f32c(state);
  Tensor out = at::empty_like(c.x);
  ssm_step_args a{};
  c.fill(a, work);
  a.out = out.data_ptr();
  if (c.nb * c.nd > 0) run(ssm_selective_state_step(&a, stream_of(state)));
  if (!direct) state.detach().copy_(work);
  return out;
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, OptTensor, OptTensor, OptTensor> selective_state_step_backward(
    const Tensor& grad_output, const OptTensor& grad_state, const Tensor& state, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B,
    const Tensor& C, const OptTensor& D, const OptTensor& z, const OptTensor& dt_bias, bool softplus) {
  StepCtx c(state, x, dt, A, B, C, D, z, dt_bias, softplus);
  c10::cuda::CUDAGuard guard(state.device());
  const auto f32 = c.x.options().dtype(at::kFloat);
  Tensor old = f32c(state);  // the state BEFORE the step
  Tensor go = like(grad_output, c.x);
  OptTensor gs = f32c(grad_state);
  Tensor dstate = at::empty({c.nb, c.nd, c.nn}, f32), dx = at::empty_like(c.x), ddt = at::empty_like(c.x);
  OptTensor dz = c.z.has_value() ? OptTensor(at::empty_like(c.x)) : OptTensor();
  Tensor dA = at::zeros({c.nd, c.nn}, f32), dB = at::zeros(c.B.sizes(), f32), dC = at::zeros(c.C.sizes(), f32);
  OptTensor dD = c.D.has_value() ? OptTensor(at::zeros({c.nd}, f32)) : OptTensor();
  OptTensor db = c.bias.has_value() ? OptTensor(at::zeros({c.nd}, f32)) : OptTensor();
  ssm_step_bwd_args g{};
  c.fill(g.fwd, old);
  g.dout = go.data_ptr(), g.dnew_state = fptr(gs), g.dstate = dstate.data_ptr<float>();
  g.dx = dx.data_ptr(), g.ddt = ddt.data_ptr(), g.dz = dz.has_value() ? dz->data_ptr() : nullptr;
  g.dA = dA.data_ptr<float>(), g.dB = dB.data_ptr<float>(), g.dC = dC.data_ptr<float>(), g.dD = fptr_mut(dD), g.ddt_bias = fptr_mut(db);
  if (c.nb * c.nd > 0) run(ssm_selective_state_step_bwd(&g, stream_of(state)));
  else dstate.zero_();
  auto fold = [&](Tensor grad, const Tensor& src) {
    if (grad.sizes() != src.sizes()) {  // grouped (B, G, N) had been expanded to (B, D, N)
      const int64_t rep = grad.size(1) / src.size(1);
      grad = grad.view({src.size(0), src.size(1), rep, src.size(2)}).sum(2);
    }
    return grad.to(src.scalar_type());
  };
  auto cast = [](const OptTensor& grad, const OptTensor& src) { return grad.has_value() ? OptTensor(grad->to(src->scalar_type())) : OptTensor(); };
  return {dstate.to(state.scalar_type()), dx, ddt.to(dt.scalar_type()), dA.to(A.scalar_type()), fold(dB, B), fold(dC, C), cast(dD, D), cast(dz, z),
          cast(db, dt_bias)};
}

// ---------------------------------------------------------------------------------------------
// element-wise chunked recurrence
// ---------------------------------------------------------------------------------------------
Tensor ssd_chunk_scan(const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk_size, const OptTensor& D,
                      const OptTensor& z, const OptTensor& seq_lens, const OptTensor& cu_seqlens, const OptTensor& initial_states) {
  ChunkCtx c(X, dt, A, B, C, chunk_size, D, z, seq_lens, cu_seqlens, initial_states);
  c10::cuda::CUDAGuard guard(c.X.device());
  Tensor Y = at::empty_like(c.X);
  const int64_t n = ssm_chunk_scan_scratch_floats((int)c.nb, (int)c.nl, (int)c.nh, (int)c.np, c.chunk);
  Tensor scratch = at::empty({std::max<int64_t>(n, 1)}, c.X.options().dtype(at::kFloat));
  ssm_chunk_args a{};
  c.fill(a);
  a.Y = Y.data_ptr(), a.final_state = nullptr, a.scratch = scratch.data_ptr<float>();
  run(ssm_chunk_scan_fwd(&a, stream_of(c.X)));
  return Y;
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, OptTensor, OptTensor, OptTensor> ssd_chunk_scan_backward(
    const Tensor& grad_output, const Tensor& X, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk_size,
    const OptTensor& D, const OptTensor& z, const OptTensor& seq_lens, const OptTensor& cu_seqlens, const OptTensor& initial_states) {
  ChunkCtx c(X, dt, A, B, C, chunk_size, D, z, seq_lens, cu_seqlens, initial_states);
  c10::cuda::CUDAGuard guard(c.X.device());
  TORCH_CHECK(grad_output.sizes() == c.X.sizes(), "grad_output must have the shape of X.");
  const auto f32 = c.X.options().dtype(at::kFloat);
  auto zeros_like = [&](const OptTensor& t) { return t.has_value() ? OptTensor(at::zeros(t->sizes(), f32)) : OptTensor(); };
  Tensor dX = at::empty_like(c.X), ddt = at::zeros({c.nb, c.nl, c.nh}, f32);
  // per-token B / C / z: the kernel writes their gradients in the tensor's own type (no zero-fill, no fp32 copy to convert)
  int typed = 0;
  auto own = [&](const OptTensor& t, Kind k, int bit) {
    if (!t.has_value() || k != Kind::BLHP) return zeros_like(t);
    typed |= bit;
    return OptTensor(at::empty_like(*t));
  };
  OptTensor dA = zeros_like(c.A), dB = own(c.B, c.kB, 1), dC = own(c.C, c.kC, 2), dD = zeros_like(c.D), dz = own(c.z, c.kz, 4), dI = zeros_like(c.init);
  Tensor hist = at::empty({c.nb, std::max<int64_t>(c.nl, 1), c.nh, c.np}, f32);
  Tensor gy = like(grad_output, c.X);
  ssm_chunk_bwd_args g{};
  c.fill(g.fwd);
  g.fwd.typed_grads = typed;
  Tensor scratch = at::empty({std::max<int64_t>(1, ssm_chunk_scan_bwd_scratch_floats((int)c.nb, (int)c.nl, (int)c.nh, (int)c.np, c.chunk))}, f32);
  g.dY = gy.data_ptr(), g.dX = dX.data_ptr(), g.ddt = ddt.data_ptr<float>(), g.history = hist.data_ptr<float>();
  g.scratch = scratch.data_ptr<float>();
  set_bc4(g.dA, dA, c.kA), set_bc4(g.dB, dB, c.kB), set_bc4(g.dC, dC, c.kC), set_bc4(g.dD, dD, c.kD), set_bc4(g.dz, dz, c.kz),
      set_bc4(g.dinitial, dI, Kind::BHP);
  run(ssm_chunk_scan_bwd(&g, stream_of(c.X)));
  auto cast = [](const OptTensor& grad, const OptTensor& src) { return grad.has_value() ? OptTensor(grad->to(src->scalar_type())) : OptTensor(); };
  return {dX, ddt.to(dt.scalar_type()), dA->to(A.scalar_type()), dB->to(B.scalar_type()), dC->to(C.scalar_type()), cast(dD, D), cast(dz, z),
          cast(dI, initial_states)};
}

// ---------------------------------------------------------------------------------------------
// depthwise causal conv
// ---------------------------------------------------------------------------------------------
Tensor dw_causal_conv(const Tensor& x, const Tensor& weight, const OptTensor& bias, const std::string& activation) {
  ConvCtx c(x, weight, bias, activation);
  c10::cuda::CUDAGuard guard(c.x.device());
  Tensor y = at::empty_like(c.x);
  ssm_conv_args a{};
  c.fill(a);
  a.y = y.data_ptr();
  run(ssm_dw_causal_conv_fwd(&a, stream_of(c.x)));
  return y;
}

std::tuple<Tensor, Tensor, OptTensor> dw_causal_conv_backward(const Tensor& grad_output, const Tensor& x, const Tensor& weight, const OptTensor& bias,
                                                             const std::string& activation) {
  ConvCtx c(x, weight, bias, activation);
  c10::cuda::CUDAGuard guard(c.x.device());
  TORCH_CHECK(grad_output.sizes() == c.x.sizes(), "grad_output must have the shape of x.");
  const auto f32 = c.x.options().dtype(at::kFloat);
  Tensor dx = at::empty_like(c.x), dw = at::zeros({c.nc, c.k}, f32);
  OptTensor db = c.b.has_value() ? OptTensor(at::zeros({c.nc}, f32)) : OptTensor();
  Tensor go = like(grad_output, c.x);
  ssm_conv_bwd_args g{};
  c.fill(g.fwd);
  g.dy = go.data_ptr(), g.dx = dx.data_ptr(), g.dweight = dw.data_ptr<float>(), g.dbias = fptr_mut(db);
  run(ssm_dw_causal_conv_bwd(&g, stream_of(c.x)));
  return {dx, dw.view(weight.sizes()).to(weight.scalar_type()), db.has_value() ? OptTensor(db->to(bias->scalar_type())) : OptTensor()};
}

// ---------------------------------------------------------------------------------------------
// fused residual add + LayerNorm / RMSNorm
// ---------------------------------------------------------------------------------------------
Tensor fused_layer_norm(const Tensor& x, const Tensor& weight, const OptTensor& bias, const OptTensor& residual, bool is_rms, double eps, bool prenorm,
                        bool residual_in_fp32) {
  (void)residual_in_fp32;  // all arithmetic is fp32 for fp32 / bf16 / fp16 inputs, whatever this flag says
  NormCtx c(x, weight, bias, residual, is_rms, eps, prenorm);
  c10::cuda::CUDAGuard guard(c.x.device());
  Tensor y = at::empty_like(c.x);
  ssm_norm_args a{};
  c.fill(a);
  a.y = y.data_ptr(), a.residual_out = nullptr;
  run(ssm_fused_add_norm_fwd(&a, stream_of(c.x)));
  return y;
}

std::tuple<Tensor, Tensor, Tensor, Tensor> fused_layer_norm_backward(const Tensor& grad_output, const Tensor& x, const Tensor& weight, const OptTensor& bias,
                                                                     const OptTensor& residual, bool is_rms, double eps, bool prenorm,
                                                                     bool residual_in_fp32) {
  (void)residual_in_fp32;
  NormCtx c(x, weight, bias, residual, is_rms, eps, prenorm);
  c10::cuda::CUDAGuard guard(c.x.device());
  TORCH_CHECK(grad_output.sizes() == c.x.sizes(), "grad_output must have the shape of x.");
  const auto f32 = c.x.options().dtype(at::kFloat);
  const int64_t rows = c.x.size(0) * c.x.size(1), hidden = c.x.size(2);
  Tensor dx = at::empty_like(c.x), dw = at::empty({hidden}, f32);
  Tensor db = c.b.has_value() ? at::empty({hidden}, f32) : at::empty({0}, c.x.options());
  Tensor dres = c.res.has_value() ? at::empty_like(*c.res) : at::empty({0}, c.x.options());
  Tensor partial = at::empty({ssm_norm_bwd_scratch_floats(rows, (int)hidden)}, f32);
  Tensor go = like(grad_output, c.x);
  ssm_norm_bwd_args g{};
  c.fill(g.fwd);
  g.dy = go.data_ptr(), g.dx = dx.data_ptr(), g.dresidual = c.res.has_value() ? dres.data_ptr() : nullptr;
  g.dweight = dw.data_ptr(), g.dbias = c.b.has_value() ? db.data_ptr() : nullptr, g.partial = partial.data_ptr<float>();
  g.dresidual_out = nullptr;
  run(ssm_fused_add_norm_bwd(&g, stream_of(c.x)));
  // absent inputs give empty tensors, as upstream's extension does
  return {dx, dw.to(weight.scalar_type()), c.b.has_value() ? db.to(bias->scalar_type()) : db, dres};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  m.doc() = "ssm.ops CUDA backend for B200 (sm_100a): the ten entry points of upstream's compiled extension, on libssm_b200";
  ssm_ext::bind_operators(m);
  m.def("abi_version", []() { return ssm_b200_abi_version(); });
  m.def("selective_scan", &selective_scan, py::arg("u"), py::arg("delta"), py::arg("A"), py::arg("B"), py::arg("C"), py::arg("D") = c10::nullopt,
        py::arg("z") = c10::nullopt, py::arg("dt_bias") = c10::nullopt, py::arg("softplus") = false, py::arg("return_last_state") = false);
  m.def("selective_scan_backward", &selective_scan_backward, py::arg("grad_output"), py::arg("grad_last_state") = c10::nullopt, py::arg("u"),
        py::arg("delta"), py::arg("A"), py::arg("B"), py::arg("C"), py::arg("D") = c10::nullopt, py::arg("z") = c10::nullopt,
        py::arg("dt_bias") = c10::nullopt, py::arg("softplus") = false, py::arg("forward_output") = c10::nullopt, py::arg("cache") = c10::nullopt);
  m.def("selective_state_step", &selective_state_step, py::arg("state"), py::arg("x"), py::arg("dt"), py::arg("A"), py::arg("B"), py::arg("C"),
        py::arg("D") = c10::nullopt, py::arg("z") = c10::nullopt, py::arg("dt_bias") = c10::nullopt, py::arg("softplus") = true);
  m.def("selective_state_step_backward", &selective_state_step_backward, py::arg("grad_output"), py::arg("grad_state") = c10::nullopt, py::arg("state"),
        py::arg("x"), py::arg("dt"), py::arg("A"), py::arg("B"), py::arg("C"), py::arg("D") = c10::nullopt, py::arg("z") = c10::nullopt,
        py::arg("dt_bias") = c10::nullopt, py::arg("softplus") = true);
  m.def("ssd_chunk_scan", &ssd_chunk_scan, py::arg("X"), py::arg("dt"), py::arg("A"), py::arg("B"), py::arg("C"), py::arg("chunk_size"),
        py::arg("D") = c10::nullopt, py::arg("z") = c10::nullopt, py::arg("seq_lens") = c10::nullopt, py::arg("cu_seqlens") = c10::nullopt,
        py::arg("initial_states") = c10::nullopt);
  m.def("ssd_chunk_scan_backward", &ssd_chunk_scan_backward, py::arg("grad_output"), py::arg("X"), py::arg("dt"), py::arg("A"), py::arg("B"),
        py::arg("C"), py::arg("chunk_size"), py::arg("D") = c10::nullopt, py::arg("z") = c10::nullopt, py::arg("seq_lens") = c10::nullopt,
        py::arg("cu_seqlens") = c10::nullopt, py::arg("initial_states") = c10::nullopt);
  m.def("dw_causal_conv", &dw_causal_conv, py::arg("x"), py::arg("weight"), py::arg("bias") = c10::nullopt, py::arg("activation") = "silu");
  m.def("dw_causal_conv_backward", &dw_causal_conv_backward, py::arg("grad_output"), py::arg("x"), py::arg("weight"), py::arg("bias") = c10::nullopt,
        py::arg("activation") = "silu");
  m.def("fused_layer_norm", &fused_layer_norm, py::arg("x"), py::arg("weight"), py::arg("bias") = c10::nullopt, py::arg("residual") = c10::nullopt,
        py::arg("is_rms") = false, py::arg("eps") = 1e-5, py::arg("prenorm") = true, py::arg("residual_in_fp32") = true);
  m.def("fused_layer_norm_backward", &fused_layer_norm_backward, py::arg("grad_output"), py::arg("x"), py::arg("weight"), py::arg("bias") = c10::nullopt,
        py::arg("residual") = c10::nullopt, py::arg("is_rms") = false, py::arg("eps") = 1e-5, py::arg("prenorm") = true,
        py::arg("residual_in_fp32") = true);
}
