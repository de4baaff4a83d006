"""Fused add + norm at the row widths where the number of threads or chunks per row changes, parameters in their own type."""

from __future__ import annotations

import pytest
import torch

from oracle import ssm_oracle as orc
from tests.gpu_util import FP32_TOL, HALF_TOL, close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,dtype", [(264, torch.bfloat16), (776, torch.float16), (1600, torch.bfloat16), (3080, torch.float16), (5000, torch.float32),
                                          (8192, torch.float32), (8200, torch.bfloat16), (502, torch.float32)])
@pytest.mark.parametrize("is_rms", [True, False])
def test_widths_match_oracle(hidden, dtype, is_rms):
    from ssm_b200 import ops

    gen = torch.Generator().manual_seed(hidden)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    ins = {"x": rnd(2, 5, hidden).to(dtype), "weight": (1 + 0.1 * rnd(hidden)).to(dtype), "bias": (0.1 * rnd(hidden)).to(dtype), "residual": rnd(2, 5, hidden)}
    wy, wr = rnd(2, 5, hidden).to(dtype).float(), rnd(2, 5, hidden)
    lg = {k: v.cuda().requires_grad_() for k, v in ins.items()}
    lo = {k: v.float().requires_grad_() for k, v in ins.items()}
    yg, rg = ops.fused_layer_norm(lg["x"], lg["weight"], lg["bias"], residual=lg["residual"], is_rms=is_rms, return_residual=True)
    yo = orc.fused_layer_norm(lo["x"], lo["weight"], lo["bias"], residual=lo["residual"], is_rms=is_rms)
    ro = lo["x"] + lo["residual"]
    tol = FP32_TOL if dtype == torch.float32 else HALF_TOL
    close(yg, yo, **tol, what="y"), close(rg, ro, **FP32_TOL, what="residual")
    gg = torch.autograd.grad((yg.float() * wy.cuda()).sum() + (rg * wr.cuda()).sum(), list(lg.values()))
    go = torch.autograd.grad((yo * wy).sum() + (ro * wr).sum(), list(lo.values()))
    for k, a, b in zip(ins, gg, go):
        assert a.dtype == ins[k].dtype
        close(a, b, **tol, what=f"d{k}", reduced=k in ("weight", "bias"))


@pytest.mark.parametrize("hidden,dtype", [(136, torch.bfloat16), (520, torch.float32), (1032, torch.bfloat16), (1600, torch.float32), (2560, torch.bfloat16),
                                          (4104, torch.float16), (8200, torch.float32), (16384, torch.bfloat16)])
@pytest.mark.parametrize("residual,out_f32", [(None, False), ("own", False), ("fp32", True), (None, True)])
def test_many_rows_per_block(hidden, dtype, residual, out_f32):
    """Every block takes several rows (the last round only for some), with and without the residual stream, in either type."""
    from ssm_b200 import ops

    rows = 148 * (16 if hidden < 1100 else 4 if hidden <= 4104 else 1) * 3 + 5
    gen = torch.Generator(device="cuda").manual_seed(hidden)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    ins = {"x": rnd(1, rows, hidden).to(dtype), "weight": (1 + 0.1 * rnd(hidden)), "bias": 0.1 * rnd(hidden)}
    if residual:
        ins["residual"] = rnd(1, rows, hidden).to(torch.float32 if residual == "fp32" else dtype)
    wy, wr = rnd(1, rows, hidden).to(dtype), rnd(1, rows, hidden)
    lg = {k: v.clone().requires_grad_() for k, v in ins.items()}
    lo = {k: v.double().requires_grad_() for k, v in ins.items()}
    yg, rg = ops.fused_layer_norm(lg["x"], lg["weight"], lg["bias"], residual=lg.get("residual"), return_residual=True, residual_in_fp32=out_f32)
    so = lo["x"] + lo["residual"] if residual else lo["x"]
    yo = torch.nn.functional.layer_norm(so, (hidden,), lo["weight"], lo["bias"], 1e-5)
    gg = torch.autograd.grad([yg, rg], list(lg.values()), [wy, wr.to(rg.dtype)])
    go = torch.autograd.grad([yo, so], list(lo.values()), [wy.double(), wr.to(rg.dtype).double()])
    tol = FP32_TOL if dtype == torch.float32 else HALF_TOL
    for k, a, b in zip(ins, gg, go):
        assert a.dtype == ins[k].dtype
        close(a, b, **tol, what=f"d{k}", reduced=k in ("weight", "bias"))
