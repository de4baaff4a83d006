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
