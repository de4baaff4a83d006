// Operands of the five operators as the C ABI wants them: shape checks, dtype and layout normalisation, and the filling of
// the argument structs.  Shared by the ten upstream-named functions (ssm_b200_ext.cpp) and by the package's own operator
// surface (operators.cpp).
#pragma once

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <string>
#include <tuple>
#include <vector>

#include "../../../include/ssm_b200.h"

namespace ssm_ext {

using at::Tensor;
using OptTensor = c10::optional<at::Tensor>;

// A rejected argument is a RuntimeError in the upstream-named functions (their facade turns it into ValueError) and a
// ValueError in the package's own operators, which set this flag for the duration of a call.
inline thread_local bool value_errors = false;
struct ValueErrors {
  bool before;
  ValueErrors() : before(value_errors) { value_errors = true; }
  ~ValueErrors() { value_errors = before; }
};
[[noreturn]] inline void reject(const std::string& msg) {
  if (value_errors) throw pybind11::value_error(msg);
  TORCH_CHECK(false, msg);
}
#define SSM_ARG(cond, ...)                                      \
  do {                                                          \
    if (!(cond)) ::ssm_ext::reject(c10::str(__VA_ARGS__));      \
  } while (0)

inline int dtype_code(const Tensor& t, const char* what) {
  switch (t.scalar_type()) {
    case at::kFloat: return SSM_F32;
    case at::kBFloat16: return SSM_BF16;
    case at::kHalf: return SSM_F16;
    default: reject(c10::str(what, ": dtype ", t.scalar_type(), " is not built (float32, bfloat16 and float16 are)"));
  }
  return -1;
}
inline bool io_dtype_ok(const Tensor& t) { return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf; }

inline void need_cuda(const Tensor& ref, std::initializer_list<const OptTensor*> rest) {
  TORCH_CHECK(ref.is_cuda(), "ssm_b200 operators run on CUDA tensors only; there is no CPU fallback");
  for (const OptTensor* t : rest)
    if (t->has_value()) {
      TORCH_CHECK((*t)->is_cuda(), "ssm_b200 operators run on CUDA tensors only; there is no CPU fallback");
      SSM_ARG((*t)->device() == ref.device(), "all tensors must be on the same CUDA device");
    }
}
inline void same_device(const Tensor& ref, std::initializer_list<const Tensor*> rest) {
  TORCH_CHECK(ref.is_cuda(), "ssm_b200 operators run on CUDA tensors only; there is no CPU fallback");
  for (const Tensor* t : rest) {
    TORCH_CHECK(t->is_cuda(), "ssm_b200 operators run on CUDA tensors only; there is no CPU fallback");
    SSM_ARG(t->device() == ref.device(), "all tensors must be on the same CUDA device");
  }
}

inline Tensor f32c(const Tensor& t) { return t.detach().to(at::kFloat).contiguous(); }
inline OptTensor f32c(const OptTensor& t) { return t.has_value() ? OptTensor(f32c(*t)) : OptTensor(); }
inline Tensor like(const Tensor& t, const Tensor& ref) { return t.detach().to(ref.scalar_type()).contiguous(); }

// A (B, D, L) activation in one of the two row layouts the kernels address directly: dense (B, D, L), or a dense (D, B, L)
// buffer viewed as (B, D, L).  Anything else is copied to dense.
inline Tensor rows(const Tensor& t) {
  Tensor d = t.detach();
  if (d.is_contiguous()) return d.dim() == 3 ? d.as_strided(d.sizes(), {d.size(1) * d.size(2), d.size(2), 1}) : d;  // an extent of one may have any stride
  if (d.dim() == 3 && d.stride(2) == 1 && d.stride(0) == d.size(2) && d.stride(1) == d.size(0) * d.size(2)) return d;
  return d.contiguous();
}
// `t` with the dtype and exactly the strides of `ref` (copied only when it differs)
inline Tensor rows_like(const Tensor& t, const Tensor& ref) {
  Tensor d = t.detach();
  if (d.scalar_type() == ref.scalar_type() && d.strides() == ref.strides()) return d;
  Tensor out = at::empty_like(ref);
  out.copy_(d);
  return out;
}
inline const void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }
inline const float* fptr(const OptTensor& t) { return t.has_value() ? t->data_ptr<float>() : nullptr; }
inline float* fptr_mut(OptTensor& t) { return t.has_value() ? t->data_ptr<float>() : nullptr; }

inline void run(int rc) {
  if (rc == 0) return;
  const char* msg = ssm_b200_last_error();
  const std::string text = std::string((msg && *msg) ? msg : "libssm_b200 call failed") + " (code " + std::to_string(rc) + ")";
  if (rc < 0) reject(text);
  TORCH_CHECK(false, text);
}
inline ssm_stream_t stream_of(const Tensor& t) { return reinterpret_cast<ssm_stream_t>(at::cuda::getCurrentCUDAStream(t.get_device()).stream()); }

// ---------------------------------------------------------------------------------------------
// selective scan
// ---------------------------------------------------------------------------------------------
struct Coeff {
  Tensor t;
  int groups;
  int64_t sb, sg, sn, st;
};

// B / C in one of the layouts of reference.py:22-56 -> tensor + group count + element strides
inline Coeff scan_coeff(const char* name, const Tensor& p, int64_t nb, int64_t nd, int64_t nn, int64_t nl) {
  if (p.dim() == 2) {
    SSM_ARG(p.size(0) == nd && p.size(1) == nn, name, " must have shape (D, N).");
    return {f32c(p), (int)nd, 0, nn, 1, 0};
  }
  if (p.dim() == 3) {
    SSM_ARG(p.size(0) == nb && p.size(1) == nd && p.size(2) == nn, name, " must have shape (B, D, N) when 3-D.");
    return {f32c(p), (int)nd, nd * nn, nn, 1, 0};
  }
  SSM_ARG(p.dim() == 4, "Unsupported rank for ", name, ".");
  SSM_ARG(p.size(0) == nb && p.size(3) == nl, name, " must have shape (B, G, N, L) when 4-D.");
  const int64_t g = p.size(1);
  SSM_ARG(g > 0 && nd % g == 0, "Group dimension must divide D.");
  SSM_ARG(p.size(2) == nn, name, " has mismatched state dimension.");
  Tensor t = io_dtype_ok(p) ? p.detach().contiguous() : f32c(p);
  return {t, (int)g, g * nn * nl, nn * nl, nl, 1};
}

struct ScanCtx {
  int64_t nb, nd, nl, nn;
  Tensor u, delta, A;
  OptTensor z, D, bias, init;
  Coeff B, C;
  bool softplus;

  ScanCtx(const Tensor& u_, const Tensor& delta_, const Tensor& A_, const Tensor& B_, const Tensor& C_, const OptTensor& D_, const OptTensor& z_,
          const OptTensor& bias_, bool softplus_, const OptTensor& init_ = c10::nullopt, bool keep_rows = false)
      : softplus(softplus_) {
    SSM_ARG(u_.dim() == 3 && delta_.dim() == 3, "u and delta must have shape (B, D, L).");
    nb = u_.size(0), nd = u_.size(1), nl = u_.size(2);
    SSM_ARG(delta_.sizes() == u_.sizes(), "delta must match the shape of u.");
    SSM_ARG(A_.dim() == 2 && A_.size(0) == nd, "A must have shape (D, N).");
    SSM_ARG(!A_.is_complex(), "selective_scan: complex A is not built");
    nn = A_.size(1);
    SSM_ARG(nn >= 1 && nn <= 256, "selective_scan: the state dimension must be in [1, 256].");
    same_device(u_, {&delta_, &A_, &B_, &C_});
    need_cuda(u_, {&D_, &z_, &bias_, &init_});
    dtype_code(u_, "selective_scan");
    u = keep_rows ? rows(u_) : u_.detach().contiguous();
    delta = rows_like(delta_, u);
    A = f32c(A_);
    B = scan_coeff("B", B_, nb, nd, nn, nl);
    C = scan_coeff("C", C_, nb, nd, nn, nl);
    if (B.groups != C.groups) {  // expand the coarser grouping so that one group map serves both
      const int g = std::max(B.groups, C.groups);
      SSM_ARG(g % std::min(B.groups, C.groups) == 0, "B and C group dimensions must nest.");
      Coeff& low = B.groups < g ? B : C;
      SSM_ARG(low.st != 0, "B and C group dimensions must nest.");
      low.t = low.t.repeat_interleave(g / low.groups, 1).contiguous();
      low.groups = g, low.sb = g * nn * nl, low.sg = nn * nl, low.sn = nl, low.st = 1;
    }
    if (B.t.scalar_type() != C.t.scalar_type()) B.t = B.t.to(at::kFloat), C.t = C.t.to(at::kFloat);
    if (D_.has_value()) SSM_ARG(D_->dim() == 1 && D_->size(0) == nd, "D must have shape (D,).");
    if (z_.has_value()) SSM_ARG(z_->sizes() == u_.sizes(), "z must have shape (B, D, L).");
    if (bias_.has_value()) SSM_ARG(bias_->dim() == 1 && bias_->size(0) == nd, "dt_bias must have shape (D,).");
    if (init_.has_value()) SSM_ARG(init_->dim() == 3 && init_->size(0) == nb && init_->size(1) == nd && init_->size(2) == nn, "initial_state must have shape (B, D, N).");
    D = f32c(D_), bias = f32c(bias_), init = f32c(init_);
    if (z_.has_value()) z = rows_like(*z_, u);
  }

  void fill(ssm_scan_fwd_args& a) const {
    a.batch = (int)nb, a.dim = (int)nd, a.len = (int)nl, a.nstate = (int)nn;
    a.io_dtype = dtype_code(u, "selective_scan"), a.bc_dtype = dtype_code(B.t, "selective_scan B/C");
    a.delta_softplus = softplus;
    a.u = u.data_ptr(), a.delta = delta.data_ptr(), a.z = ptr(z), a.A = A.data_ptr<float>();
    a.Bm = B.t.data_ptr(), a.Cm = C.t.data_ptr(), a.bc_groups = B.groups;
    a.b_sb = B.sb, a.b_sg = B.sg, a.b_sn = B.sn, a.b_st = B.st;
    a.c_sb = C.sb, a.c_sg = C.sg, a.c_sn = C.sn, a.c_st = C.st;
    a.D = fptr(D), a.dt_bias = fptr(bias), a.initial_state = fptr(init);
    const bool any = u.numel() > 0;
    a.row_sb = any ? u.stride(0) : nd * nl, a.row_sd = any ? u.stride(1) : nl;
  }
};

inline Tensor scan_checkpoints(const ScanCtx& c) {
  const int iv = ssm_scan_checkpoint_interval();
  return at::empty({c.nb, c.nd, std::max<int64_t>(1, (c.nl + iv - 1) / iv), c.nn}, c.u.options().dtype(at::kFloat));
}

// ---------------------------------------------------------------------------------------------
// single-token state step
// ---------------------------------------------------------------------------------------------
struct StepCoeff {
  int groups;
  int64_t sb, sg, sn;
};
inline StepCoeff step_coeff(const char* name, const Tensor& p, int64_t nb, int64_t nd, int64_t nn) {
  if (p.dim() == 2) {
    SSM_ARG(p.size(0) == nd && p.size(1) == nn, name, " must have shape (D, N).");
    return {(int)nd, 0, nn, 1};
  }
  SSM_ARG(p.dim() == 3 && p.size(0) == nb, name, " must have shape (D, N), (B, D, N) or (B, G, N).");
  const int64_t g = p.size(1);
  SSM_ARG(p.size(2) == nn, name, " must have matching state dimension.");
  SSM_ARG(g > 0 && nd % g == 0, name, " group dimension must divide D.");
  return {(int)g, g * nn, nn, 1};
}

struct StepCtx {
  int64_t nb, nd, nn;
  Tensor x, dt, A, B, C;
  OptTensor z, D, bias;
  StepCoeff cb, cc;
  bool softplus;

  StepCtx(const Tensor& state, const Tensor& x_, const Tensor& dt_, const Tensor& A_, const Tensor& B_, const Tensor& C_, const OptTensor& D_,
          const OptTensor& z_, const OptTensor& bias_, bool softplus_,
          bool keep_views = false)
      : softplus(softplus_) {
    SSM_ARG(state.dim() == 3, "state must have shape (B, D, N).");
    SSM_ARG(x_.dim() == 2 && dt_.dim() == 2, "x and dt must have shape (B, D).");
    nb = state.size(0), nd = state.size(1), nn = state.size(2);
    SSM_ARG(x_.size(0) == nb && x_.size(1) == nd && dt_.sizes() == x_.sizes(), "x and dt must match the first two dimensions of state.");
    SSM_ARG(A_.dim() == 2 && A_.size(0) == nd && A_.size(1) == nn, "A must have shape (D, N).");
    same_device(state, {&x_, &dt_, &A_, &B_, &C_});
    need_cuda(state, {&D_, &z_, &bias_});
    dtype_code(x_, "selective_state_step");
    cb = step_coeff("B", B_, nb, nd, nn), cc = step_coeff("C", C_, nb, nd, nn);
    // keep_views: a (B, G, N) view with contiguous states (a slice of a wider projection) is addressed where it lies.  Not for
    // the backward pass, whose gradient buffers share the strides of B and C.
    auto states = [&](const Tensor& t, StepCoeff& sc) {
      Tensor d = t.detach();
      if (keep_views && d.dim() == 3 && d.stride(2) == 1) {
        sc.sb = d.stride(0), sc.sg = d.stride(1);
        return d;
      }
      return d.contiguous();
    };
    B = states(B_, cb), C = states(C_, cc);
    if (cb.groups != cc.groups || B.scalar_type() != C.scalar_type() || !io_dtype_ok(B)) {
      auto expand = [&](Tensor t, StepCoeff& sc) {  // bring to per-channel fp32 (B, D, N) / (D, N)
        t = t.to(at::kFloat);
        if (t.dim() == 3 && sc.groups != nd) t = t.repeat_interleave(nd / sc.groups, 1);
        sc = t.dim() == 2 ? StepCoeff{(int)nd, 0, nn, 1} : StepCoeff{(int)nd, nd * nn, nn, 1};
        return t.contiguous();
      };
      B = expand(B, cb), C = expand(C, cc);  // contiguous
    }
    if (D_.has_value()) SSM_ARG(D_->dim() == 1 && D_->size(0) == nd, "D must have shape (D,).");
    if (z_.has_value()) SSM_ARG(z_->sizes() == x_.sizes(), "z must have shape (B, D).");
    if (bias_.has_value()) SSM_ARG(bias_->dim() == 1 && bias_->size(0) == nd, "dt_bias must have shape (D,).");
    x = x_.detach().contiguous(), dt = like(dt_, x), A = f32c(A_), D = f32c(D_), bias = f32c(bias_);
    if (z_.has_value()) z = like(*z_, x);
  }

  void fill(ssm_step_args& a, Tensor& state32) const {
    a.batch = (int)nb, a.dim = (int)nd, a.nstate = (int)nn, a.io_dtype = dtype_code(x, "selective_state_step");
    a.bc_dtype = dtype_code(B, "selective_state_step B/C"), a.bc_groups = cb.groups, a.dt_softplus = softplus, a.param_heads = 0;
    a.state = state32.data_ptr<float>(), a.x = x.data_ptr(), a.dt = dt.data_ptr(), a.z = ptr(z), a.A = A.data_ptr<float>();
    a.Bm = B.data_ptr(), a.Cm = C.data_ptr();
    a.b_sb = cb.sb, a.b_sg = cb.sg, a.b_sn = cb.sn, a.c_sb = cc.sb, a.c_sg = cc.sg, a.c_sn = cc.sn;
    a.D = fptr(D), a.dt_bias = fptr(bias);
  }
};

// ---------------------------------------------------------------------------------------------
// element-wise chunked recurrence
// ---------------------------------------------------------------------------------------------
enum class Kind { H, HP, BHP, BLH, BLHP };
inline void set_bc4(ssm_bcast4& d, const OptTensor& t, Kind k) {
  d.ptr = nullptr, d.sb = d.st = d.sh = d.sq = 0;
  if (!t.has_value()) return;
  d.ptr = t->data_ptr();
  switch (k) {
    case Kind::H: d.sh = 1; break;
    case Kind::HP: d.sh = t->size(1), d.sq = 1; break;
    case Kind::BHP: d.sb = t->size(1) * t->size(2), d.sh = t->size(2), d.sq = 1; break;
    case Kind::BLH: d.sb = t->size(1) * t->size(2), d.st = t->size(2), d.sh = 1; break;
    case Kind::BLHP: d.sb = t->size(1) * t->size(2) * t->size(3), d.st = t->size(2) * t->size(3), d.sh = t->size(3), d.sq = 1; break;
  }
}

struct ChunkCtx {
  int64_t nb, nl, nh, np;
  int chunk;
  Tensor X, dt;
  OptTensor A, B, C, D, z, init, lens;
  Kind kA, kB, kC, kD = Kind::H, kz = Kind::BLH;
  int par;

  ChunkCtx(const Tensor& X_, const Tensor& dt_, const Tensor& A_, const Tensor& B_, const Tensor& C_, int64_t chunk_size, const OptTensor& D_,
           const OptTensor& z_, const OptTensor& seq_lens, const OptTensor& cu_seqlens, const OptTensor& init_) {
    SSM_ARG(X_.dim() == 4, "X must have shape (B, L, H, P).");
    SSM_ARG(dt_.dim() == 3, "dt must have shape (B, L, H).");
    nb = X_.size(0), nl = X_.size(1), nh = X_.size(2), np = X_.size(3);
    SSM_ARG(dt_.size(0) == nb && dt_.size(1) == nl && dt_.size(2) == nh, "dt must align with (B, L, H).");
    SSM_ARG(chunk_size > 0, "chunk_size must be positive.");
    chunk = (int)std::min<int64_t>(chunk_size, 1 << 30);
    same_device(X_, {&dt_, &A_, &B_, &C_});
    need_cuda(X_, {&D_, &z_, &init_});
    dtype_code(X_, "ssd_chunk_scan");
    X = X_.detach().contiguous(), dt = like(dt_, X);
    if (A_.dim() == 1) {
      SSM_ARG(A_.size(0) == nh, "A must have shape (H,) when 1-D.");
      kA = Kind::H;
    } else {
      SSM_ARG(A_.dim() == 2, "A must be 1-D or 2-D.");
      SSM_ARG(A_.size(0) == nh && A_.size(1) == np, "A must have shape (H, P) when 2-D.");
      kA = Kind::HP;
    }
    A = f32c(A_);
    auto coeff = [&](const char* name, const Tensor& p) {
      if (p.dim() == 2) {
        SSM_ARG(p.size(0) == nh && p.size(1) == np, name, " must have shape (H, P).");
        return Kind::HP;
      }
      if (p.dim() == 3) {
        SSM_ARG(p.size(0) == nb && p.size(1) == nh && p.size(2) == np, name, " must be (B, H, P) when 3-D.");
        return Kind::BHP;
      }
      SSM_ARG(p.dim() == 4, "Unsupported rank for ", name, ".");
      SSM_ARG(p.sizes() == X_.sizes(), name, " must have shape (B, L, H, P) when 4-D.");
      return Kind::BLHP;
    };
    kB = coeff("B", B_), kC = coeff("C", C_);
    if (D_.has_value()) {
      if (D_->dim() == 1 && D_->size(0) == nh) kD = Kind::H;
      else if (D_->dim() == 2 && D_->size(0) == nh && D_->size(1) == np) kD = Kind::HP;
      else SSM_ARG(false, "D must have shape (H,) or (H, P).");
    }
    if (z_.has_value()) {
      if (z_->dim() == 3 && z_->size(0) == nb && z_->size(1) == nl && z_->size(2) == nh) kz = Kind::BLH;
      else if (z_->dim() == 4 && z_->sizes() == X_.sizes()) kz = Kind::BLHP;
      else SSM_ARG(false, "z must have shape (B, L, H) or (B, L, H, P).");
    }
    if (init_.has_value()) SSM_ARG(init_->dim() == 3 && init_->size(0) == nb && init_->size(1) == nh && init_->size(2) == np, "initial_states must have shape (B, H, P).");
    // B, C and z share one run-time element type inside the kernel
    at::ScalarType pd = X_.scalar_type();  // the kernels take X's element type or fp32
    const bool same = B_.scalar_type() == pd && C_.scalar_type() == pd && (!z_.has_value() || z_->scalar_type() == pd);
    if (!same) pd = at::kFloat;
    par = pd == at::kFloat ? SSM_F32 : pd == at::kBFloat16 ? SSM_BF16 : SSM_F16;
    B = B_.detach().to(pd).contiguous(), C = C_.detach().to(pd).contiguous();
    if (z_.has_value()) z = z_->detach().to(pd).contiguous();
    D = f32c(D_), init = f32c(init_);
    // valid lengths per row, on the device (reference.py:413-428); never copied to the host
    if (cu_seqlens.has_value()) {
      SSM_ARG(cu_seqlens->numel() == nb + 1, "cu_seqlens must have length B + 1.");
      Tensor cu = cu_seqlens->to(X.device(), at::kLong);
      lens = (cu.slice(0, 1) - cu.slice(0, 0, nb)).contiguous();
    } else if (seq_lens.has_value()) {
      SSM_ARG(seq_lens->numel() == nb, "seq_lens must have length B.");
      lens = seq_lens->to(X.device(), at::kLong).contiguous();
    }
  }

  void fill(ssm_chunk_args& a) const {
    a.batch = (int)nb, a.len = (int)nl, a.heads = (int)nh, a.proj = (int)np;
    a.io_dtype = dtype_code(X, "ssd_chunk_scan"), a.par_dtype = par, a.chunk_size = chunk;
    a.X = X.data_ptr(), a.dt = dt.data_ptr();
    set_bc4(a.A, A, kA), set_bc4(a.Bm, B, kB), set_bc4(a.Cm, C, kC), set_bc4(a.D, D, kD), set_bc4(a.z, z, kz), set_bc4(a.initial, init, Kind::BHP);
    a.seq_lens = lens.has_value() ? lens->data_ptr<int64_t>() : nullptr;
  }
};

// ---------------------------------------------------------------------------------------------
// depthwise causal conv
// ---------------------------------------------------------------------------------------------
inline bool is_silu(const std::string& activation) {
  std::string act = activation;
  for (auto& ch : act) ch = (char)std::tolower((unsigned char)ch);
  SSM_ARG(act == "silu" || act == "swish" || act == "identity" || act == "none", "Unsupported activation '", activation, "'.");
  return act == "silu" || act == "swish";
}

struct ConvCtx {
  bool first, silu;
  int64_t nb, nc, nl, k;
  Tensor x, w;
  OptTensor b, halo;

  ConvCtx(const Tensor& x_, const Tensor& weight, const OptTensor& bias, const std::string& activation, const OptTensor& halo_ = c10::nullopt,
          bool keep_rows = false) {
    SSM_ARG(x_.dim() == 3, "x must have shape (B, C, L) or (B, L, C).");
    nc = weight.size(0);
    if (x_.size(1) == nc) first = true;
    else if (x_.size(2) == nc) first = false;
    else SSM_ARG(false, "weight channel dimension must match x.");
    Tensor w2;
    if (weight.dim() == 3) {
      SSM_ARG(weight.size(1) == 1, "Expected depthwise weights with shape (C, 1, K).");
      w2 = weight.select(1, 0);
    } else {
      SSM_ARG(weight.dim() == 2, "weight must have 2 or 3 dimensions.");
      w2 = weight;
    }
    if (bias.has_value()) SSM_ARG(bias->dim() == 1 && bias->size(0) == nc, "bias must have shape (C,).");
    silu = is_silu(activation);
    k = w2.size(1);
    SSM_ARG(k >= 1 && k <= 8, "dw_causal_conv: kernel width must be in [1, 8].");
    same_device(x_, {&weight});
    need_cuda(x_, {&bias, &halo_});
    dtype_code(x_, "dw_causal_conv");
    x = first && keep_rows ? rows(x_) : x_.detach().contiguous();
    if (io_dtype_ok(w2) && (!bias.has_value() || bias->scalar_type() == w2.scalar_type())) {  // as they are
      w = w2.detach().contiguous();
      if (bias.has_value()) b = bias->detach().contiguous();
    } else {
      w = f32c(w2), b = f32c(bias);
    }
    nb = x_.size(0), nl = first ? x_.size(2) : x_.size(1);
    if (halo_.has_value())
      SSM_ARG(halo_->dim() == 3 && halo_->size(0) == nb && halo_->size(1) == nc && halo_->size(2) == k - 1, "halo must have shape (B, C, K-1).");
    halo = f32c(halo_);
  }
  void fill(ssm_conv_args& a) const {
    a.batch = (int)nb, a.channels = (int)nc, a.len = (int)nl, a.width = (int)k;
    a.io_dtype = dtype_code(x, "dw_causal_conv"), a.channels_first = first, a.silu = silu;
    a.x = x.data_ptr(), a.weight = w.data_ptr(), a.bias = ptr(b), a.halo = fptr(halo);
    a.param_dtype = dtype_code(w, "dw_causal_conv");
    const bool own = first && x.numel() > 0;
    a.row_sb = own ? x.stride(0) : nc * nl, a.row_sc = own ? x.stride(1) : nl;
  }
};

// ---------------------------------------------------------------------------------------------
// fused residual add + LayerNorm / RMSNorm
// ---------------------------------------------------------------------------------------------
struct NormCtx {
  Tensor x, w;
  OptTensor b, res;
  bool is_rms, prenorm;
  double eps;

  NormCtx(const Tensor& x_, const Tensor& weight, const OptTensor& bias, const OptTensor& residual, bool is_rms_, double eps_, bool prenorm_)
      : is_rms(is_rms_), prenorm(prenorm_), eps(eps_) {
    SSM_ARG(x_.dim() == 3, "x must have shape (B, L, D).");
    SSM_ARG(weight.dim() == 1 && weight.size(0) == x_.size(2), "weight must match the last dimension of x.");
    if (bias.has_value()) SSM_ARG(bias->dim() == 1 && bias->size(0) == x_.size(2), "bias must match the last dimension of x.");
    if (residual.has_value()) SSM_ARG(residual->sizes() == x_.sizes(), "residual must match the shape of x.");
    same_device(x_, {&weight});
    need_cuda(x_, {&bias, &residual});
    dtype_code(x_, "fused_layer_norm");
    x = x_.detach().contiguous();
    // weight and bias go in as they are when they share a type that the kernels read
    if (io_dtype_ok(weight) && (!bias.has_value() || bias->scalar_type() == weight.scalar_type())) {
      w = weight.detach().contiguous();
      if (bias.has_value()) b = bias->detach().contiguous();
    } else {
      w = f32c(weight), b = f32c(bias);
    }
    if (residual.has_value()) {
      dtype_code(*residual, "fused_layer_norm residual");
      res = residual->detach().contiguous();
    }
  }
  void fill(ssm_norm_args& a) const {
    a.rows = x.size(0) * x.size(1), a.hidden = (int)x.size(2);
    a.io_dtype = dtype_code(x, "fused_layer_norm"), a.res_dtype = res.has_value() ? dtype_code(*res, "fused_layer_norm residual") : 0;
    a.is_rms = is_rms, a.prenorm = prenorm, a.eps = (float)eps;
    a.x = x.data_ptr(), a.residual = ptr(res), a.weight = w.data_ptr(), a.bias = ptr(b);
    a.param_dtype = dtype_code(w, "fused_layer_norm");
  }
};

}  // namespace ssm_ext
