"""The five state-space operators on the B200 CUDA library, with the upstream signatures.

``selective_scan``, ``selective_state_step``, ``ssd_chunk_scan``, ``dw_causal_conv`` and
``fused_layer_norm`` take the arguments of ``ssm.ops`` in b-vitamins/ssm
(src/ssm/ops/__init__.py:1255-1690; semantics src/ssm/ops/python/reference.py), accept CUDA
tensors only, and are differentiable: forward and backward both run hand-written sm_100a
kernels behind the C ABI of ``include/ssm_b200.h``.  What lies between a call and its launches
(checks, layout and dtype normalisation, allocation, the autograd node) is C++
(``csrc/torch_ext/operators.cpp``).  Contract violations raise ``ValueError`` as upstream does.
There is no CPU path and no PyTorch fallback: a missing library or a CPU tensor is an error.

Additive keyword arguments that upstream does not have are marked "extension" below; their
defaults reproduce upstream behaviour.
"""

from __future__ import annotations

import ctypes as C
import math
from typing import Any, Optional

import torch

from . import _lib as L

Tensor = torch.Tensor

_CODES = {torch.float32: L.F32, torch.bfloat16: L.BF16, torch.float16: L.F16}


_ops = None


def _native():
    """The compiled operator surface (loaded once; raises if it has not been built)."""
    global _ops
    if _ops is None:
        from .backend import load_extension

        _ops = load_extension().operators
    return _ops


class _Traced(torch.autograd.Function):
    """One call inside ``torch.jit.trace``: a Python node of the traced graph, which makes the call again whenever the graph runs.
    (The allocations of a compiled call would be recorded without its launches.)  Its backward is that of the call inside."""

    @staticmethod
    def forward(ctx, name, *args):
        with torch.enable_grad():
            ctx.leaves = [a.detach().requires_grad_(a.requires_grad) if isinstance(a, Tensor) else a for a in args]
            out = getattr(_native(), name)(*ctx.leaves)
        ctx.outs = out if isinstance(out, tuple) else (out,)
        res = tuple(t.detach() for t in ctx.outs)
        return res if isinstance(out, tuple) else res[0]

    @staticmethod
    def backward(ctx, *grads):
        live = [a for a in ctx.leaves if isinstance(a, Tensor) and a.requires_grad]
        pairs = [(o, g) for o, g in zip(ctx.outs, grads) if g is not None and o.requires_grad]
        got = iter(torch.autograd.grad([o for o, _ in pairs], live, [g for _, g in pairs], retain_graph=True, allow_unused=True))
        return (None, *(next(got) if isinstance(a, Tensor) and a.requires_grad else None for a in ctx.leaves))


def _run(name: str, *args):
    """A differentiable call of the compiled operator surface."""
    if torch._C._get_tracing_state() is None:
        return getattr(_native(), name)(*args)
    return _Traced.apply(name, *args)


def _code(t: Tensor, what: str) -> int:
    try:
        return _CODES[t.dtype]
    except KeyError:
        raise ValueError(f"{what}: dtype {t.dtype} is not built (float32, bfloat16 and float16 are)") from None


def _need_cuda(*ts: Optional[Tensor]) -> torch.device:
    dev = None
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("ssm_b200 operators run on CUDA tensors only; there is no CPU fallback")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise ValueError("all tensors must be on the same CUDA device")
    assert dev is not None
    return dev


def _p(t: Optional[Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _f32(t: Optional[Tensor]) -> Optional[Tensor]:
    if t is None:
        return None
    return t.detach().to(torch.float32).contiguous()


def _c(t: Optional[Tensor]) -> Optional[Tensor]:
    if t is None:
        return None
    t = t.detach()
    return t if t.is_contiguous() else t.contiguous()


def _guard(ctx, *tensors: Optional[Tensor]) -> None:
    """Remember the version counters of the tensors a backward pass will read again; `_check_guard`
    raises if one of them was modified in place in between (what autograd does for saved tensors)."""
    ctx._guarded = [(t, t._version) for t in tensors if t is not None]


def _check_guard(ctx) -> None:
    for t, v in getattr(ctx, "_guarded", ()):
        if t._version != v:
            raise RuntimeError("one of the tensors needed for the backward pass of an ssm_b200 operator has been modified in place "
                               f"(shape {tuple(t.shape)}, version {t._version}, expected {v})")


class _DeviceStatus:
    """The word that the tensor-core kernels set when one of their bounded waits runs out: one per device, in pinned host
    memory that the kernels write directly.  `poll` reads it, so a timed-out wait surfaces at the next call without the hot
    path ever copying or synchronising.  `poll(sync=True)` waits for the device first."""

    _per_device: dict[int, "_DeviceStatus"] = {}

    def __init__(self, index: int):
        self.index = index
        self.word = _native().ssd_status(index)

    @classmethod
    def of(cls, device: torch.device) -> "_DeviceStatus":
        idx = device.index if device.index is not None else torch.cuda.current_device()
        st = cls._per_device.get(idx)
        if st is None:
            st = cls._per_device[idx] = cls(idx)
        return st

    def poll(self, sync: bool = False) -> None:
        if sync and not torch.cuda.is_current_stream_capturing():
            torch.cuda.synchronize(self.index)
        _native().ssd_poll(self.index)


def ssd_check_status(device: Optional[torch.device] = None) -> None:
    """Wait for ``device`` and raise if a bounded wait of a tensor-core SSD launch ran out."""
    _DeviceStatus.of(torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)).poll(sync=True)


def ssd_wait_selftest(probes: int = 100, device: Optional[torch.device] = None) -> None:
    """Launch the library's wait self-test on ``device``: a warp waits on a barrier nothing arms and gives up after ``probes``
    probes, recording status 3 like a tensor-core kernel whose copy never landed.  The next ``ssd_scan`` call (or
    :func:`ssd_check_status`) then raises; the device and the context stay usable."""
    st = _DeviceStatus.of(torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device))
    with torch.cuda.device(st.index):
        L.check(L.load().ssm_ssd_wait_selftest(st.word.data_ptr(), int(probes), _stream()))


def _call(fn, args) -> None:
    try:
        L.check(fn(C.byref(args), _stream()))
    except L.BackendError as exc:
        if exc.code < 0:
            raise ValueError(str(exc)) from None
        raise


# =========================================================================================
# selective_scan
# =========================================================================================


def selective_scan(
    u: Tensor,
    delta: Tensor,
    A: Tensor,
    B: Tensor,
    C: Tensor,
    D: Optional[Tensor] = None,
    z: Optional[Tensor] = None,
    dt_bias: Optional[Tensor] = None,
    softplus: bool = False,
    return_last_state: bool = False,
    initial_state: Optional[Tensor] = None,
    keep_state_fp32: bool = False,
):
    """Mamba-1 selective scan (upstream ``ssm.ops.selective_scan``, reference.py:87-194).

    Extensions: ``initial_state`` ``(B, D, N)`` starts the recurrence from a given state (it
    receives a gradient like any other input); ``keep_state_fp32`` returns the last state in
    fp32 instead of ``u.dtype``.
    """
    if u.dtype == torch.float64:  # double-precision kernels, meant for gradient checks (ops_f64.py)
        from . import ops_f64
        return ops_f64.selective_scan(u, delta, A, B, C, D, z, dt_bias, softplus, return_last_state, initial_state)
    return _run("selective_scan", u, delta, A, B, C, D, z, dt_bias, softplus, return_last_state, initial_state, keep_state_fp32)


# =========================================================================================
# selective_state_step
# =========================================================================================


def _step_coeff(name: str, p: Tensor, nb: int, nd: int, nn: int):
    if p.dim() == 2:
        if tuple(p.shape) != (nd, nn):
            raise ValueError(f"{name} must have shape (D, N).")
        return nd, (0, nn, 1)
    if p.dim() == 3 and p.shape[0] == nb:
        g = p.shape[1]
        if p.shape[2] != nn:
            raise ValueError(f"{name} must have matching state dimension.")
        if g == 0 or nd % g != 0:
            raise ValueError(f"{name} group dimension must divide D.")
        return g, (g * nn, nn, 1)
    raise ValueError(f"{name} must have shape (D, N), (B, D, N) or (B, G, N).")


class _StepCtx:
    def __init__(self, state, x, dt, A, B, C_, D, z, dt_bias, softplus):
        if state.ndim != 3:
            raise ValueError("state must have shape (B, D, N).")
        if x.ndim != 2 or dt.ndim != 2:
            raise ValueError("x and dt must have shape (B, D).")
        nb, nd, nn = state.shape
        if tuple(x.shape) != (nb, nd) or tuple(dt.shape) != (nb, nd):
            raise ValueError("x and dt must match the first two dimensions of state.")
        if tuple(A.shape) != (nd, nn):
            raise ValueError("A must have shape (D, N).")
        _need_cuda(state, x, dt, A, B, C_, D, z, dt_bias)
        self.shape = (nb, nd, nn)
        self.io = _code(x, "selective_state_step")
        gb, self.sB = _step_coeff("B", B, nb, nd, nn)
        gc, self.sC = _step_coeff("C", C_, nb, nd, nn)
        Bt, Ct = _c(B), _c(C_)
        if gb != gc or Bt.dtype != Ct.dtype or Bt.dtype not in _CODES:
            # bring both to per-channel fp32 (B, D, N) / (D, N) form
            Bt, gb, self.sB = _expand_step(Bt, gb, nb, nd, nn)
            Ct, gc, self.sC = _expand_step(Ct, gc, nb, nd, nn)
        self.B, self.C, self.groups = Bt, Ct, gb
        if D is not None and tuple(D.shape) != (nd,):
            raise ValueError("D must have shape (D,).")
        if z is not None and tuple(z.shape) != (nb, nd):
            raise ValueError("z must have shape (B, D).")
        if dt_bias is not None and tuple(dt_bias.shape) != (nd,):
            raise ValueError("dt_bias must have shape (D,).")
        self.x, self.dt = _c(x), _c(dt.to(x.dtype))
        self.z = None if z is None else _c(z.to(x.dtype))
        self.A, self.D, self.dt_bias = _f32(A), _f32(D), _f32(dt_bias)
        self.softplus = bool(softplus)

    def fill(self, a: L.StepArgs, state32: Tensor) -> None:
        nb, nd, nn = self.shape
        a.batch, a.dim, a.nstate, a.io_dtype = nb, nd, nn, self.io
        a.bc_dtype, a.bc_groups, a.dt_softplus, a.param_heads = _CODES[self.B.dtype], self.groups, int(self.softplus), 0
        a.state, a.x, a.dt, a.z, a.A = _p(state32), _p(self.x), _p(self.dt), _p(self.z), _p(self.A)
        a.Bm, a.Cm = _p(self.B), _p(self.C)
        a.b_sb, a.b_sg, a.b_sn = self.sB
        a.c_sb, a.c_sg, a.c_sn = self.sC
        a.D, a.dt_bias = _p(self.D), _p(self.dt_bias)


def _expand_step(t: Tensor, g: int, nb: int, nd: int, nn: int):
    t = t.float()
    if t.dim() == 3 and g != nd:
        t = t.repeat_interleave(nd // g, dim=1)
    t = t.contiguous()
    return t, nd, ((0, nn, 1) if t.dim() == 2 else (nd * nn, nn, 1))


def _step_forward(sc: _StepCtx, state: Tensor) -> Tensor:
    """Runs the step; ``state`` is updated in place (through an fp32 copy if it is not fp32)."""
    lib = L.load()
    direct = state.dtype == torch.float32 and state.is_contiguous()
    work = state.detach() if direct else state.detach().float().contiguous()
    out = torch.empty_like(sc.x)
    a = L.StepArgs()
    sc.fill(a, work)
    a.out = _p(out)
    _call(lib.ssm_selective_state_step, a)
    if not direct:
        state.detach().copy_(work)
    return out


class _StateStepFn(torch.autograd.Function):
    """Out-of-place form used when gradients are needed: returns (y, new_state)."""

    @staticmethod
    def forward(ctx, state, x, dt, A, B, C_, D, z, dt_bias, softplus):
        sc = _StepCtx(state, x, dt, A, B, C_, D, z, dt_bias, softplus)
        old = state.detach().float().contiguous()
        new = old.clone()
        y = _step_forward(sc, new)
        ctx.sc, ctx.old = sc, old
        ctx.like = (state, dt, A, B, C_, D, z, dt_bias)
        _guard(ctx, x, dt, A, B, C_, D, z, dt_bias)
        return y, new.to(state.dtype)

    @staticmethod
    def backward(ctx, gy, gstate):
        _check_guard(ctx)
        sc: _StepCtx = ctx.sc
        state, dt, A, B, C_, D, z, dt_bias = ctx.like
        nb, nd, nn = sc.shape
        lib = L.load()
        dev = sc.x.device
        g = L.StepBwdArgs()
        sc.fill(g.fwd, ctx.old)
        gy = torch.zeros_like(sc.x) if gy is None else _c(gy.to(sc.x.dtype))
        gs = _f32(gstate)
        dstate = torch.empty(nb, nd, nn, dtype=torch.float32, device=dev)
        dx, ddt = torch.empty_like(sc.x), torch.empty_like(sc.x)
        dz = torch.empty_like(sc.x) if sc.z is not None else None
        dA = torch.zeros(nd, nn, dtype=torch.float32, device=dev)
        dB = torch.zeros(sc.B.shape, dtype=torch.float32, device=dev)
        dC = torch.zeros(sc.C.shape, dtype=torch.float32, device=dev)
        dD = torch.zeros(nd, dtype=torch.float32, device=dev) if sc.D is not None else None
        db = torch.zeros(nd, dtype=torch.float32, device=dev) if sc.dt_bias is not None else None
        g.dout, g.dnew_state, g.dstate = _p(gy), _p(gs), _p(dstate)
        g.dx, g.ddt, g.dz = _p(dx), _p(ddt), _p(dz)
        g.dA, g.dB, g.dC, g.dD, g.ddt_bias = _p(dA), _p(dB), _p(dC), _p(dD), _p(db)
        _call(lib.ssm_selective_state_step_bwd, g)

        def fold(grad: Tensor, like: Tensor) -> Tensor:
            if grad.shape != like.shape:  # grouped (B, G, N) had been expanded to (B, D, N)
                rep = grad.shape[1] // like.shape[1]
                grad = grad.view(like.shape[0], like.shape[1], rep, like.shape[2]).sum(2)
            return grad.to(like.dtype)

        return (
            dstate.to(state.dtype), dx, ddt.to(dt.dtype), dA.to(A.dtype), fold(dB, B), fold(dC, C_),
            None if D is None else dD.to(D.dtype),
            None if z is None else dz.to(z.dtype),
            None if dt_bias is None else db.to(dt_bias.dtype),
            None,
        )


def selective_state_step(
    state: Tensor,
    x: Tensor,
    dt: Tensor,
    A: Tensor,
    B: Tensor,
    C: Tensor,
    D: Optional[Tensor] = None,
    z: Optional[Tensor] = None,
    dt_bias: Optional[Tensor] = None,
    softplus: bool = True,
) -> Tensor:
    """One decode token; ``state`` ``(B, D, N)`` is overwritten in place (upstream
    ``ssm.ops.selective_state_step``, reference.py:197-309)."""
    if x.dtype == torch.float64:
        from . import ops_f64
        return ops_f64.selective_state_step(state, x, dt, A, B, C, D, z, dt_bias, softplus)
    if any(t is not None and t.requires_grad for t in (state, x, dt, A, B, C, D, z, dt_bias)) and torch.is_grad_enabled():
        y, new = _StateStepFn.apply(state, x, dt, A, B, C, D, z, dt_bias, softplus)
        with torch.no_grad():
            state.copy_(new)
        return y
    return _native().state_step(state, x, dt, A, B, C, D, z, dt_bias, softplus, False)


def selective_state_step_heads(
    state: Tensor, x: Tensor, dt: Tensor, A: Tensor, B: Tensor, C: Tensor,
    D: Optional[Tensor] = None, z: Optional[Tensor] = None, dt_bias: Optional[Tensor] = None, softplus: bool = True,
) -> Tensor:
    """Extension: Mamba-2 decode step.  ``state (B, H, P, N)`` fp32 in place, ``x, z (B, H, P)``,
    ``dt (B, H)``, ``A, D, dt_bias (H,)``, ``B, C (B, G, N)``; returns ``(B, H, P)``.  Equivalent to
    the upstream step on ``H*P`` flattened channels with per-head parameters broadcast."""
    return _native().state_step_heads(state, x, dt, A, B, C, D, z, dt_bias, softplus, False)


def mamba1_step(tok: Tensor, residual: Optional[Tensor], conv_state: Tensor, ssm_state: Tensor, w: dict, norm_w: Optional[Tensor] = None,
                eps: float = 1e-5):
    """Extension: one decode token through a Mamba-1 mixer, and with ``norm_w`` the residual add and RMSNorm behind it
    (then the result is ``(normed, residual)``).  ``tok (B, d_model)``; ``w`` as in `ssm_b200.mixer`, with ``A_log`` or ``A``;
    states fp32, in place; no gradients.  Up to 16 sequences run as one launch."""
    a_log = "A_log" in w
    return _native().mamba1_step(tok, residual, conv_state, ssm_state, w["in_x"], w["in_z"], w["conv_w"], w["conv_b"], w["x_proj"], w["dt_proj"],
                                 w["dt_bias"], w["A_log"] if a_log else w["A"], a_log, w["D"], w["out_proj"], norm_w, eps)


def mamba2_step(tok: Tensor, conv_states: tuple, ssm_state: Tensor, w: dict, eps: float = 1e-5) -> Tensor:
    """Extension: one decode token through a Mamba-2 mixer; the counterpart of :func:`mamba1_step`."""
    return _native().mamba2_step(tok, *conv_states, ssm_state, w["in_z"], w["in_x"], w["in_B"], w["in_C"], w["in_dt"], w["conv_x"], w["conv_x_b"],
                                 w["conv_B"], w["conv_B_b"], w["conv_C"], w["conv_C_b"], w["dt_bias"], w["A_log"], True, w["D"], w["norm_w"],
                                 w["out_proj"], eps)


_PLAIN_TENSORS = (Tensor, torch.nn.Parameter)  # a subclass may answer torch's own functions in its own way


def mamba1_mixer(hidden: Tensor, w: dict) -> Optional[Tensor]:
    """Extension: a whole Mamba-1 mixer behind one autograd node; ``hidden (B, L, d_model)``, ``w`` as for :func:`mamba1_step`.  ``None`` where
    the operators have to be composed instead (tracing, forward mode, autocast, saved-tensor hooks, mixed types, tensor subclasses)."""
    a_log = "A_log" in w
    for t in (hidden, w["in_x"], w["in_z"], w["x_proj"], w["dt_proj"], w["A_log"] if a_log else w["A"], w["out_proj"]):
        if type(t) not in _PLAIN_TENSORS:
            return None
    return _native().mamba1_mixer(hidden, w["in_x"], w["in_z"], w["conv_w"], w["conv_b"], w["x_proj"], w["dt_proj"], w["dt_bias"], w["A_log"] if a_log else w["A"],
                                  a_log, w["D"], w["out_proj"])


def mamba2_mixer(u: Tensor, w: dict, cfg: dict) -> Optional[Tensor]:
    """Extension: a whole Mamba-2 mixer on the tensor-core scan, without gradients; ``None`` as for :func:`mamba1_mixer`, with gradients enabled
    and for shapes that the scan is not built for."""
    for t in (u, w["in_z"], w["in_x"], w["in_B"], w["in_C"], w["in_dt"], w["A_log"], w["out_proj"]):
        if type(t) not in _PLAIN_TENSORS:
            return None
    return _native().mamba2_mixer(u, w["in_z"], w["in_x"], w["in_B"], w["in_C"], w["in_dt"], w["conv_x"], w["conv_x_b"], w["conv_B"], w["conv_B_b"], w["conv_C"],
                                  w["conv_C_b"], w["dt_bias"], w["A_log"], w["D"], w["norm_w"], w["out_proj"], cfg["heads"], cfg["headdim"], cfg["d_state"],
                                  cfg["groups"], cfg.get("chunk_size", 256), cfg.get("eps", 1e-5))


# =========================================================================================
# ssd_chunk_scan (element-wise chunked recurrence)
# =========================================================================================


def ssd_chunk_scan(
    X: Tensor,
    dt: Tensor,
    A: Tensor,
    B: Tensor,
    C: Tensor,
    chunk_size: int,
    D: Optional[Tensor] = None,
    z: Optional[Tensor] = None,
    seq_meta: Optional[dict[str, Any]] = None,
    initial_states: Optional[Tensor] = None,
) -> Tensor:
    """Element-wise chunked recurrence over ``(B, L, H, P)`` (upstream ``ssm.ops.ssd_chunk_scan``,
    reference.py:312-463)."""
    if X.dtype == torch.float64:
        from . import ops_f64
        return ops_f64.ssd_chunk_scan(X, dt, A, B, C, chunk_size, D, z, seq_meta, initial_states)
    lens = cu = None
    if seq_meta:  # valid lengths per row (reference.py:413-428)
        lens, cu = seq_meta.get("seq_lens"), seq_meta.get("cu_seqlens")
        if cu is None and lens is None:
            raise ValueError("seq_meta must provide cu_seqlens or seq_lens.")
        cu = None if cu is None else torch.as_tensor(cu)
        lens = None if lens is None or cu is not None else torch.as_tensor(lens)
    return _run("ssd_chunk_scan", X, dt, A, B, C, int(chunk_size), D, z, lens, cu, initial_states)


# =========================================================================================
# dw_causal_conv
# =========================================================================================


def dw_causal_conv(x: Tensor, weight: Tensor, bias: Optional[Tensor] = None, activation: str = "silu",
                   halo: Optional[Tensor] = None) -> Tensor:
    """Depthwise causal conv1d with optional SiLU (upstream ``ssm.ops.dw_causal_conv``,
    reference.py:466-537).  Extension: ``halo`` ``(B, C, K-1)`` supplies the inputs that precede
    ``t = 0`` (sequence-sharded prefill) instead of zeros; no gradient flows into it."""
    if x.dtype == torch.float64:
        if halo is not None:
            raise ValueError("dw_causal_conv in float64 takes no halo.")
        from . import ops_f64
        return ops_f64.dw_causal_conv(x, weight, bias, activation)
    return _run("dw_causal_conv", x, weight, bias, str(activation), halo)


def dw_causal_conv_update(conv_state: Tensor, x: Tensor, weight: Tensor, bias: Optional[Tensor] = None,
                          activation: str = "silu") -> Tensor:
    """Extension: decode-time conv.  Rolls ``conv_state (B, C, K)`` (fp32, in place) left by one,
    appends ``x (B, C)`` and returns ``act(bias + <conv_state, weight>)`` (what upstream's
    ``Mamba1.step`` does with ``torch.roll``, modules/mamba1.py:345-353)."""
    return _native().dw_causal_conv_update(conv_state, x, weight, bias, str(activation))


# =========================================================================================
# fused_layer_norm
# =========================================================================================


class _NormCtx:
    """Operands of a norm call for direct use of the C ABI: the allocation-free backward has no operator of its own."""

    def __init__(self, x, weight, bias, residual, is_rms, eps, prenorm):
        if x.ndim != 3:
            raise ValueError("x must have shape (B, L, D).")
        if tuple(weight.shape) != (x.shape[-1],):
            raise ValueError("weight must match the last dimension of x.")
        if bias is not None and tuple(bias.shape) != (x.shape[-1],):
            raise ValueError("bias must match the last dimension of x.")
        if residual is not None and residual.shape != x.shape:
            raise ValueError("residual must match the shape of x.")
        _need_cuda(x, weight, bias, residual)
        self.io = _code(x, "fused_layer_norm")
        self.x, self.w, self.b = _c(x), _f32(weight), _f32(bias)
        self.res = _c(residual)
        if self.res is not None:
            _code(self.res, "fused_layer_norm residual")
        self.is_rms, self.eps, self.prenorm = bool(is_rms), float(eps), bool(prenorm)

    def fill(self, a: L.NormArgs) -> None:
        a.rows, a.hidden = self.x.shape[0] * self.x.shape[1], self.x.shape[2]
        a.io_dtype = self.io
        a.res_dtype = _CODES[self.res.dtype] if self.res is not None else 0
        a.is_rms, a.prenorm, a.eps = int(self.is_rms), int(self.prenorm), self.eps
        a.x, a.residual, a.weight, a.bias = _p(self.x), _p(self.res), _p(self.w), _p(self.b)


def fused_layer_norm(
    x: Tensor,
    weight: Tensor,
    bias: Optional[Tensor],
    residual: Optional[Tensor] = None,
    is_rms: bool = False,
    eps: float = 1e-5,
    prenorm: bool = True,
    residual_in_fp32: bool = True,
    return_residual: bool = False,
):
    """Residual add fused with LayerNorm / RMSNorm (upstream ``ssm.ops.fused_layer_norm``,
    reference.py:540-609).  All arithmetic is fp32, which is what upstream does for fp32, bf16
    and fp16 inputs whatever ``residual_in_fp32`` says.  Extension: ``return_residual`` also
    returns ``x + residual`` (fp32 when ``residual_in_fp32``, else ``x.dtype``), the residual
    stream a stack of blocks passes on; gradients flow back through both outputs."""
    if x.dtype == torch.float64:
        from . import ops_f64
        return ops_f64.fused_layer_norm(x, weight, bias, residual, is_rms, eps, prenorm, residual_in_fp32, return_residual)
    return _run("fused_layer_norm", x, weight, bias, residual, is_rms, float(eps), prenorm, residual_in_fp32, return_residual)


# =========================================================================================
# ssd_scan: state-space-dual scan with a d_state axis (Mamba-2 layout)
# =========================================================================================


def _ssd_check(X, dt, A, B, C_, D, z, dt_bias, initial_states):
    if X.ndim != 4 or dt.ndim != 3:
        raise ValueError("X must be (B, L, H, P) and dt (B, L, H).")
    nb, nl, nh, npj = X.shape
    if tuple(dt.shape) != (nb, nl, nh):
        raise ValueError("dt must align with (B, L, H).")
    if tuple(A.shape) != (nh,):
        raise ValueError("A must have shape (H,).")
    if B.ndim != 4 or B.shape[0] != nb or B.shape[1] != nl or B.shape != C_.shape:
        raise ValueError("B and C must have shape (B, L, G, N).")
    ng, nn = B.shape[2], B.shape[3]
    if ng == 0 or nh % ng != 0:
        raise ValueError("Group dimension must divide H.")
    if D is not None and tuple(D.shape) not in ((nh,), (nh, npj)):
        raise ValueError("D must have shape (H,) or (H, P).")
    if z is not None and z.shape != X.shape:
        raise ValueError("z must have shape (B, L, H, P).")
    if dt_bias is not None and tuple(dt_bias.shape) != (nh,):
        raise ValueError("dt_bias must have shape (H,).")
    if initial_states is not None and tuple(initial_states.shape) != (nb, nh, npj, nn):
        raise ValueError("initial_states must have shape (B, H, P, N).")
    _need_cuda(X, dt, A, B, C_, D, z, dt_bias, initial_states)
    return nb, nl, nh, npj, ng, nn


def _ssd_via_scan(X, dt, A, B, C_, D, z, dt_bias, dt_softplus, initial_states):
    """The same recurrence through the selective-scan kernels on the ``H*P`` flattened channels
    (any shape and dtype the scan supports; differentiable).  Returns ``(Y, final_states fp32)``."""
    nb, nl, nh, npj = X.shape
    nn = B.shape[3]
    u = X.permute(0, 2, 3, 1).reshape(nb, nh * npj, nl)
    delta = dt.permute(0, 2, 1).repeat_interleave(npj, dim=1)
    A_full = A.float()[:, None, None].expand(nh, npj, nn).reshape(nh * npj, nn)
    Bs, Cs = B.permute(0, 2, 3, 1), C_.permute(0, 2, 3, 1)
    D_flat = None if D is None else (D.reshape(-1) if D.ndim == 2 else D[:, None].expand(nh, npj).reshape(-1))
    z_flat = None if z is None else z.permute(0, 2, 3, 1).reshape(nb, nh * npj, nl)
    b_flat = None if dt_bias is None else dt_bias[:, None].expand(nh, npj).reshape(-1)
    init = None if initial_states is None else initial_states.reshape(nb, nh * npj, nn)
    y, last = selective_scan(u, delta, A_full, Bs, Cs, D=D_flat, z=z_flat, dt_bias=b_flat, softplus=dt_softplus,
                             return_last_state=True, initial_state=init, keep_state_fp32=True)
    return y.reshape(nb, nh, npj, nl).permute(0, 3, 1, 2).contiguous(), last.reshape(nb, nh, npj, nn)


class _SsdWorkspace:
    """Scratch and bookkeeping of one tensor-core SSD call, kept so that a sequence shard can run
    the state phase, exchange states, and then finish from the same scratch."""

    def __init__(self, X, dt, A, B, C_, D, z, dt_bias, dt_softplus, chunk_size):
        nb, nl, nh, npj = X.shape
        self.shape = (nb, nl, nh, npj, B.shape[2], B.shape[3])
        io = X.dtype
        self.io, self.chunk = io, int(chunk_size)
        self.X, self.B, self.C = _c(X), _c(B.to(io)), _c(C_.to(io))
        self.dt = _c(dt.to(io))
        self.z = None if z is None else _c(z.to(io))
        self.A, self.D, self.bias = _f32(A), _f32(D), _f32(dt_bias)
        self.d_has_p = int(D is not None and D.ndim == 2)
        self.softplus = int(bool(dt_softplus))
        self.nchunks = (nl + self.chunk - 1) // self.chunk
        self.ws = torch.empty(int(L.load().ssm_ssd_scratch_bytes(nb, nl, nh)), dtype=torch.uint8, device=X.device)
        self._status = _DeviceStatus.of(X.device)
        self._status.poll()  # a wait that ran out in an earlier launch surfaces here, without a synchronisation
        self.status = self._status.word

    def run(self, phase: int, initial_states: Optional[Tensor], want_y: bool):
        nb, nl, nh, npj, ng, nn = self.shape
        dev = self.X.device
        init32 = _f32(initial_states)
        Y = torch.empty(nb, nl, nh, npj, dtype=self.io, device=dev) if want_y else None
        final = torch.empty(nb, nh, npj, nn, dtype=torch.float32, device=dev)
        vec = nb * nh * self.nchunks * self.chunk * 4
        fin = int(L.load().ssm_ssd_state_scratch_bytes(nb, nl, nh))
        a = L.SsdArgs()
        a.batch, a.len, a.heads, a.headdim = nb, nl, nh, npj
        a.nstate, a.groups, a.chunk_size, a.io_dtype = nn, ng, self.chunk, _CODES[self.io]
        a.dt_softplus, a.d_has_p, a.phase = self.softplus, self.d_has_p, phase
        a.X, a.dt, a.A, a.Bm, a.Cm = _p(self.X), _p(self.dt), _p(self.A), _p(self.B), _p(self.C)
        a.D, a.z, a.dt_bias, a.initial_states = _p(self.D), _p(self.z), _p(self.bias), _p(init32)
        a.Y, a.final_states = _p(Y), _p(final)
        base = self.ws.data_ptr()
        a.ws_dt, a.ws_cum, a.ws_state, a.ws_state_in = base, base + vec, base + 2 * vec, base + 2 * vec + fin
        a.status = _p(self.status)
        _call(L.load().ssm_ssd_fwd, a)
        return Y, final

    def shard_summary(self) -> Tensor:
        """Flat fp32 view of what phase 1 left for the other ranks: the final state from a zero start, then (B, H) total log-decay."""
        nb, nl, nh, _, _, _ = self.shape
        vec = nb * nh * self.nchunks * self.chunk * 4
        n = int(L.load().ssm_ssd_shard_summary_floats(nb, nh))
        return self.ws[2 * vec: 2 * vec + n * 4].view(torch.float32)

    def total_log_decay(self) -> Tensor:
        """(B, H) sum over the shard of delta * A, read from the cumulative sums left in scratch."""
        nb, nl, nh, _, _, _ = self.shape
        vec = nb * nh * self.nchunks * self.chunk
        cum = self.ws[vec * 4: 2 * vec * 4].view(torch.float32).view(nb, nh, self.nchunks, self.chunk)
        return cum[..., -1].sum(-1) * math.log(2.0)  # the scratch holds base-2 exponents


def ssd_tensor_core_supported(X: Tensor, B: Tensor, chunk_size: int) -> bool:
    """True when :func:`ssd_scan` runs on the tcgen05 kernels for these operands."""
    return bool(X.is_cuda and X.dtype in (torch.bfloat16, torch.float16)
                and L.load().ssm_ssd_supported(X.shape[3], B.shape[3], int(chunk_size), _CODES[X.dtype]))



class _SsdFn(torch.autograd.Function):
    """The scan whose backward goes through the selective-scan kernels: shapes the tensor-core kernels are not built for, and
    ``backward="scan"``."""

    @staticmethod
    def forward(ctx, X, dt, A, B, C_, D, z, dt_bias, dt_softplus, initial_states, chunk_size):
        _ssd_check(X, dt, A, B, C_, D, z, dt_bias, initial_states)
        ctx.args = (X, dt, A, B, C_, D, z, dt_bias, dt_softplus, initial_states)
        _guard(ctx, X, dt, A, B, C_, D, z, dt_bias, initial_states)
        with torch.no_grad():
            if ssd_tensor_core_supported(X, B, chunk_size):
                return _native().ssd_scan(X, dt, A, B, C_, D, z, dt_bias, dt_softplus, initial_states, int(chunk_size))
            return _ssd_via_scan(X, dt, A, B, C_, D, z, dt_bias, dt_softplus, initial_states)

    @staticmethod
    def backward(ctx, gY, gfinal):
        _check_guard(ctx)
        X, dt, A, B, C_, D, z, dt_bias, dt_softplus, init = ctx.args
        leaves = [None if t is None else t.detach().requires_grad_(t.requires_grad) for t in (X, dt, A, B, C_, D, z, dt_bias, init)]
        with torch.enable_grad():
            Y, final = _ssd_via_scan(*leaves[:8], dt_softplus, leaves[8])
        live = [t for t in leaves if t is not None and t.requires_grad]
        outs, gouts = [Y], [gY if gY is not None else torch.zeros_like(Y)]
        if gfinal is not None:
            outs.append(final)
            gouts.append(gfinal)
        grads = iter(torch.autograd.grad(outs, live, gouts, allow_unused=True))
        res = [next(grads) if (t is not None and t.requires_grad) else None for t in leaves]
        return (*res[:8], None, res[8], None)


def _ssd_call(X, dt, A, B, C_, D, z, dt_bias, dt_softplus, init, chunk_size, check_status, dual):
    """``(Y, final_states)`` of one dense scan."""
    _need_cuda(X)
    if dual and X.ndim == 4 and B.ndim == 4 and ssd_tensor_core_supported(X, B, chunk_size):
        out = _run("ssd_scan", X, dt, A, B, C_, D, z, dt_bias, dt_softplus, init, int(chunk_size))
    else:
        out = _SsdFn.apply(X, dt, A, B, C_, D, z, dt_bias, dt_softplus, init, int(chunk_size))
    if check_status:
        ssd_check_status(X.device)
    return out


def ssd_scan(
    X: Tensor,
    dt: Tensor,
    A: Tensor,
    B: Tensor,
    C: Tensor,
    chunk_size: int = 256,
    D: Optional[Tensor] = None,
    z: Optional[Tensor] = None,
    dt_bias: Optional[Tensor] = None,
    dt_softplus: bool = False,
    initial_states: Optional[Tensor] = None,
    return_final_states: bool = False,
    check_status: bool = False,
    backward: str = "dual",
    cu_seqlens: Optional[Tensor] = None,
    seq_reset: bool = True,
    return_varlen_states: bool = False,
):
    """Extension: state-space-dual scan with a ``d_state`` axis (Mamba-2 layout).

    ``X (B,L,H,P)``, ``dt (B,L,H)``, ``A (H,)``, ``B/C (B,L,G,N)``, ``D (H,)|(H,P)``, ``z (B,L,H,P)``,
    state ``(B,H,P,N)`` fp32.  It is upstream's ``selective_scan`` recurrence (reference.py:173-188)
    on channel ``h*P+p`` with per-head ``dt`` and ``A``.  For headdim 64, d_state 128, chunk 256 and
    bf16 / fp16 operands the forward runs as chunked GEMMs on the tcgen05 tensor cores, and so does the
    backward (``backward="dual"``: the same kernels again and mirrored in time, and a kernel for the gradients of B and C; its
    gradients carry the rounding of 16-bit operands, about 0.3 % of each contraction).  ``cu_seqlens (S + 1,)``
    marks ``S`` sequences packed along ``L`` of a batch of one: ``return_varlen_states`` adds the state after the last
    token of every sequence ``(S, H, P, N)``, each scanned from zero, and with ``seq_reset`` (default) ``Y`` restarts at
    every boundary too (without it ``Y`` runs through, as upstream mamba-ssm does when given no ``seq_idx``).  Any other shape or
    dtype, and ``backward="scan"``, goes through the selective-scan kernels on the flattened channels
    (fp32 arithmetic, an order of magnitude slower at these shapes).  A bounded device-side wait that runs out (it never should) is reported by the next
    ``ssd_scan`` call on the device, or at once by ``check_status=True`` / :func:`ssd_check_status`, which synchronise.
    """
    if backward not in ("dual", "scan"):
        raise ValueError('backward must be "dual" or "scan".')
    dual = backward == "dual"
    if cu_seqlens is None:
        if return_varlen_states:
            raise ValueError("return_varlen_states needs cu_seqlens.")
        Y, final = _ssd_call(X, dt, A, B, C, D, z, dt_bias, dt_softplus, initial_states, chunk_size, check_status, dual)
        return (Y, final) if return_final_states else Y
    # packed sequences: every sequence is its own scan from a zero state (chunks counted from its first token).  Without gradients the
    # tensor-core kernels take them all at once (boundaries on the device are used where they lie and checked behind the launches); otherwise
    # they are read by the host and the scans are separate dense problems
    if X.ndim != 4 or X.shape[0] != 1:
        raise ValueError("cu_seqlens needs a batch of one (sequences packed along L).")
    if initial_states is not None and seq_reset:
        raise ValueError("initial_states cannot be combined with sequences that restart at cu_seqlens.")
    grads = torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (X, dt, A, B, C, D, z, dt_bias, initial_states))
    if not grads and X.shape[1] > 0 and ssd_tensor_core_supported(X, B, chunk_size):  # all sequences in one set of launches
        Y, final, varlen = _run("ssd_packed", X, dt, A, B, C, D, z, dt_bias, dt_softplus, initial_states, int(chunk_size), torch.as_tensor(cu_seqlens),
                                seq_reset)
        if check_status:
            ssd_check_status(X.device)
        out = (Y,) + ((final,) if return_final_states else ()) + ((varlen,) if return_varlen_states else ())
        return out[0] if len(out) == 1 else out
    cu = [int(v) for v in torch.as_tensor(cu_seqlens).tolist()]
    if len(cu) < 2 or cu[0] != 0 or cu[-1] != X.shape[1] or any(b < a for a, b in zip(cu, cu[1:])):
        raise ValueError("cu_seqlens must rise from 0 to L.")
    cut = lambda t, a, b: None if t is None else t[:, a:b]  # noqa: E731
    parts, states = [], []
    for a, b in zip(cu, cu[1:]):
        if b == a:
            states.append(torch.zeros(X.shape[2], X.shape[3], B.shape[3], dtype=torch.float32, device=X.device))
            continue
        y_k, s_k = _ssd_call(cut(X, a, b), cut(dt, a, b), A, cut(B, a, b), cut(C, a, b), D, cut(z, a, b), dt_bias, dt_softplus, None, chunk_size,
                             check_status, dual)
        parts.append(y_k)
        states.append(s_k[0])
    varlen = torch.stack(states)
    if seq_reset:
        Y, final = (torch.cat(parts, 1) if parts else torch.empty_like(X)), varlen[-1:].clone()
    else:  # upstream mamba-ssm given cu_seqlens without seq_idx: Y runs through the boundaries, only the states are per sequence
        Y, final = _ssd_call(X, dt, A, B, C, D, z, dt_bias, dt_softplus, initial_states, chunk_size, check_status, dual)
    out = [Y]
    if return_final_states:
        out.append(final)
    if return_varlen_states:
        out.append(varlen)
    return out[0] if len(out) == 1 else tuple(out)


__all__ = [
    "selective_scan",
    "selective_state_step",
    "selective_state_step_heads",
    "mamba1_step",
    "mamba2_step",
    "ssd_chunk_scan",
    "dw_causal_conv",
    "dw_causal_conv_update",
    "fused_layer_norm",
    "ssd_scan",
    "ssd_check_status",
    "ssd_wait_selftest",
    "ssd_tensor_core_supported",
]
