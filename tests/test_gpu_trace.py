"""Operators inside ``torch.jit.trace``: the traced function runs them on what it is given."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _cases():
    from ssm_b200 import ops

    r = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    A, w, nw = -torch.rand(8, 16, device="cuda"), r(8, 4), r(64)
    A2, Am = -torch.ones(2, device="cuda"), -torch.rand(2, 8, device="cuda")
    half = lambda *s: r(*s).bfloat16()  # noqa: E731
    return {
        "scan": (lambda u, d, B, C: ops.selective_scan(u, d, A, B, C, softplus=True, return_last_state=True)[0], lambda: (r(1, 8, 40), r(1, 8, 40), r(1, 1, 16, 40), r(1, 1, 16, 40))),
        "chunk": (lambda X, d, B, C: ops.ssd_chunk_scan(X, d.abs(), Am, B, C, 32), lambda: (r(1, 40, 2, 8), r(1, 40, 2), r(1, 40, 2, 8), r(1, 40, 2, 8))),
        "conv": (lambda x: ops.dw_causal_conv(x, w, None, "silu") * 2, lambda: (r(1, 8, 40),)),
        "norm": (lambda x, res: sum(ops.fused_layer_norm(x, nw, None, residual=res, return_residual=True)), lambda: (r(1, 3, 64), r(1, 3, 64))),
        "ssd": (lambda X, d, B, C: ops.ssd_scan(X, d, A2, B, C, 256, dt_softplus=True), lambda: (half(1, 300, 2, 64), half(1, 300, 2), half(1, 300, 1, 128), half(1, 300, 1, 128))),
    }


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("op", ["scan", "chunk", "conv", "norm", "ssd"])
def test_traced_operators_run_on_their_arguments(op, grad):
    fn, make = _cases()[op]
    torch.manual_seed(1)
    traced = torch.jit.trace(fn, make(), check_trace=False)
    ins = [t.requires_grad_(grad) for t in make()]
    want = fn(*ins)
    junk = [torch.full_like(want, 7.0) for _ in range(4)]  # memory that an output left unwritten would show
    del junk
    got = traced(*ins)
    assert torch.equal(got, want)
    if grad:
        weight = torch.randn_like(want)
        for a, b in zip(torch.autograd.grad((got * weight).sum(), ins), torch.autograd.grad((want * weight).sum(), ins)):
            torch.testing.assert_close(a, b, rtol=2e-2 if op == "ssd" else 1e-4, atol=1e-2 if op == "ssd" else 1e-4)
