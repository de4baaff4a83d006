"""Depthwise conv where rows, pieces and tiles end: channels-first rows that start off a 16-byte boundary, warps of pieces whose
first and last serve their neighbours, channels-last tiles of every remainder; forward and all gradients."""

from __future__ import annotations

import pytest
import torch

from oracle import ssm_oracle as orc
from tests.gpu_util import FP32_TOL, HALF_TOL, close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("nl,nc,k,dtype", [(1, 8, 4, torch.bfloat16), (7, 4, 4, torch.float32), (9, 16, 4, torch.float16), (241, 24, 4, torch.bfloat16),
                                           (250, 12, 4, torch.float32), (965, 8, 3, torch.bfloat16), (130, 5, 4, torch.float16), (123, 8, 8, torch.float32),
                                           (259, 40, 2, torch.float16), (1030, 516, 4, torch.bfloat16)])
def test_conv_edges_match_oracle(first, nl, nc, k, dtype):
    from ssm_b200 import ops

    gen = torch.Generator().manual_seed(nl)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    shape = (3, nc, nl) if first else (3, nl, nc)
    if nl == nc:
        pytest.skip("ambiguous layout")
    ins = {"x": rnd(*shape).to(dtype), "weight": (rnd(nc, k) * 0.4).to(dtype), "bias": (rnd(nc) * 0.1).to(dtype)}
    wy = rnd(*shape).to(dtype).float()
    lg = {n: v.cuda().requires_grad_() for n, v in ins.items()}
    lo = {n: v.float().requires_grad_() for n, v in ins.items()}
    yg, yo = ops.dw_causal_conv(*lg.values(), "silu"), orc.dw_causal_conv(*lo.values(), "silu")
    tol = FP32_TOL if dtype == torch.float32 else HALF_TOL
    close(yg, yo, **tol, what="y")
    gg = torch.autograd.grad((yg.float() * wy.cuda()).sum(), list(lg.values()))
    go = torch.autograd.grad((yo * wy).sum(), list(lo.values()))
    for n, a, b in zip(ins, gg, go):
        assert a.dtype == ins[n].dtype
        close(a, b, **tol, what=f"d{n}", reduced=n != "x")
