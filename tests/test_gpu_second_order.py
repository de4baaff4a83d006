"""Gradients formed with ``create_graph=True``: the values are those of an ordinary backward pass, and what the kernels cannot differentiate
a second time raises instead of counting as a constant."""

from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F

from ssm_b200 import ops
from ssm_b200.mixer import Mamba1Block

pytestmark = pytest.mark.gpu


def _case(op):
    torch.manual_seed(3)
    r = lambda *s, t=torch.float32: torch.randn(*s, device="cuda").to(t).requires_grad_()  # noqa: E731
    half = lambda *s: r(*s, t=torch.bfloat16)  # noqa: E731
    A, Am, A2 = -torch.rand(8, 16, device="cuda"), -torch.rand(2, 8, device="cuda"), -torch.ones(2, device="cuda")
    return {
        "scan": (lambda u, d, B, C: ops.selective_scan(u, d, A, B, C, softplus=True), (r(1, 8, 40), r(1, 8, 40), r(1, 1, 16, 40), r(1, 1, 16, 40))),
        "chunk": (lambda X, d, B: ops.ssd_chunk_scan(X, F.softplus(d), Am, B, B, 32), (r(1, 40, 2, 8), r(1, 40, 2), r(1, 40, 2, 8))),
        "conv": (lambda x, w, b: ops.dw_causal_conv(x, w, b, "silu"), (r(1, 8, 40), r(8, 4), r(8))),
        "norm": (lambda x, w, res: ops.fused_layer_norm(x, w, None, residual=res), (r(1, 3, 64), r(64), r(1, 3, 64))),
        "ssd": (lambda X, d, B: ops.ssd_scan(X, d, A2, B, B, 256, dt_softplus=True), (half(1, 300, 2, 64), half(1, 300, 2), half(1, 300, 1, 128))),
    }[op]


@pytest.mark.parametrize("op", ["scan", "chunk", "conv", "norm", "ssd"])
def test_an_operators_gradient_is_no_constant(op):
    fn, ins = _case(op)
    out = fn(*ins)
    go = torch.randn_like(out).requires_grad_()
    plain = torch.autograd.grad(out, ins, go, retain_graph=True)
    recorded = torch.autograd.grad(out, ins, go, create_graph=True)
    for a, b in zip(plain, recorded):  # sums over blocks by atomics: not always in one order
        torch.testing.assert_close(a, b.detach(), rtol=1e-2 if op == "ssd" else 1e-4, atol=1e-2 if op == "ssd" else 1e-4)
        assert b.requires_grad
    for g in recorded:
        for wrt in (ins[0], go):
            with pytest.raises(RuntimeError, match="differentiable once"):
                torch.autograd.grad(g.float().square().sum(), wrt, retain_graph=True)


def test_a_gradient_that_is_not_asked_for_stays_absent():
    x, w = torch.randn(1, 8, 40, device="cuda").requires_grad_(), torch.randn(8, 4, device="cuda")
    y = ops.dw_causal_conv(x, w, None, "silu").square().sum()
    y.backward(create_graph=True)
    assert x.grad.requires_grad and w.grad is None


def _mixer_second_order(block, hidden, go, penalised):
    out = block.mixer_forward(hidden)
    (g,) = torch.autograd.grad(out, penalised, go, create_graph=True)
    wrt = [hidden, go, *block.parameters()]
    return g, torch.autograd.grad(g.square().sum(), wrt, allow_unused=True)


def test_a_penalty_on_the_out_projections_gradient_reaches_everything_in_front_of_it():
    """The product is differentiated twice, the operators before it once: as exact as in the composed form."""
    torch.manual_seed(0)
    block = Mamba1Block(64, device="cuda", dtype=torch.float32)
    hidden, go = torch.randn(2, 33, 64, device="cuda").requires_grad_(), torch.randn(2, 33, 64, device="cuda").requires_grad_()
    calls = []
    hook = block.out_proj.register_hook(lambda g: calls.append(1))
    g, got = _mixer_second_order(block, hidden, go, block.out_proj)
    assert len(calls) == 1
    hook.remove()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t):  # the composed form
        gc, want = _mixer_second_order(block, hidden, go, block.out_proj)
    torch.testing.assert_close(g, gc, rtol=1e-4, atol=1e-4)
    for name, a, b in zip(["hidden", "go", *(n for n, _ in block.named_parameters())], got, want):
        assert (a is None) == (b is None), name
        if b is not None:
            assert (a - b).norm() <= 1e-4 * b.norm(), name
    assert got[0] is not None and got[1] is not None


def test_a_penalty_on_a_gradient_behind_the_scan_raises():
    block = Mamba1Block(64, device="cuda", dtype=torch.float32)
    hidden, go = torch.randn(2, 33, 64, device="cuda").requires_grad_(), torch.randn(2, 33, 64, device="cuda").requires_grad_()
    with pytest.raises(RuntimeError, match="differentiable once"):
        _mixer_second_order(block, hidden, go, block.in_x)


def test_a_mixers_gradient_after_an_edit_of_what_it_does_not_read_raises_when_differentiated():
    """Its composed form cannot be formed again then."""
    block = Mamba1Block(64, device="cuda", dtype=torch.float32)
    hidden, go = torch.randn(2, 33, 64, device="cuda").requires_grad_(), torch.randn(2, 33, 64, device="cuda")
    out = block.mixer_forward(hidden)
    (want,) = torch.autograd.grad(out, block.out_proj, go, retain_graph=True)
    with torch.no_grad():
        block.A_log.mul_(0.5)
    (g,) = torch.autograd.grad(out, block.out_proj, go, create_graph=True)
    torch.testing.assert_close(g.detach(), want, rtol=1e-4, atol=1e-4)
    for wrt in (hidden, block.in_x):
        with pytest.raises(RuntimeError, match="differentiable once"):
            torch.autograd.grad(g.square().sum(), wrt, retain_graph=True)
