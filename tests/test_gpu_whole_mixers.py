"""Mixers behind one call against the same operators composed one by one: outputs, every gradient, any subset of inputs that takes one, and
the modes in which the composed form has to serve."""

from __future__ import annotations

import contextlib
import types

import pytest
import torch

from ssm_b200 import ops
from ssm_b200.mixer import Mamba1Block, Mamba2Block

pytestmark = pytest.mark.gpu

# the composed form, which torch has to record node by node
composed = lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t)  # noqa: E731


def _near(a, b, dtype, what):
    # 16-bit chains that differ where a gradient is added in a product's epilogue instead of after a rounding of its own
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    assert a.dtype == b.dtype and a.shape == b.shape, what
    assert (a.double() - b.double()).norm() <= tol * b.double().norm() + 1e-6, what


@pytest.mark.parametrize("nb,nl,dm,dtype", [(2, 40, 96, torch.bfloat16), (1, 1, 64, torch.float16), (3, 77, 64, torch.float32), (2, 300, 256, torch.bfloat16)])
def test_mamba1_matches_composed_operators(nb, nl, dm, dtype):
    torch.manual_seed(nl)
    block = Mamba1Block(dm, device="cuda", dtype=dtype)
    hidden = torch.randn(nb, nl, dm, device="cuda").to(dtype).requires_grad_()
    res = torch.randn(nb, nl, dm, device="cuda").requires_grad_()
    go, gr = torch.randn(nb, nl, dm, device="cuda").to(dtype), torch.randn(nb, nl, dm, device="cuda")
    names = ["hidden", "residual", *(n for n, _ in block.named_parameters())]

    def run():
        out, new = block(hidden, res)
        return out, new, torch.autograd.grad((out, new), [hidden, res, *block.parameters()], (go, gr))

    assert ops.mamba1_mixer(hidden, block._step_weights()) is not None
    got = run()
    with composed():
        assert ops.mamba1_mixer(hidden, block._step_weights()) is None
        want = run()
    with torch.no_grad():
        plain = block(hidden, res)
    _near(got[0], want[0], dtype, "out"), _near(got[1], want[1], dtype, "residual"), _near(plain[0], want[0], dtype, "out without gradients")
    for n, a, b in zip(names, got[2], want[2]):
        _near(a, b, dtype, n)


@pytest.mark.parametrize("live", [["hidden"], ["out_proj"], ["in_z", "conv_b"], ["A_log", "dt_proj"], ["x_proj"], ["hidden", "in_x", "conv_w", "D", "dt_bias"]])
def test_mamba1_gradients_of_a_subset(live):
    torch.manual_seed(0)
    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    hidden = torch.randn(2, 33, 64, device="cuda").bfloat16().requires_grad_("hidden" in live)
    for n, p in block.named_parameters():
        p.requires_grad_(n in live)
    go = torch.randn(2, 33, 64, device="cuda").bfloat16()
    leaves = [hidden if n == "hidden" else getattr(block, n) for n in live]
    got = torch.autograd.grad(block.mixer_forward(hidden), leaves, go)
    with composed():
        want = torch.autograd.grad(block.mixer_forward(hidden), leaves, go)
    for n, a, b in zip(live, got, want):
        _near(a, b, torch.bfloat16, n)


def test_mamba1_edits_in_place_are_seen_and_a_graph_can_be_walked_twice():
    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    hidden = torch.randn(1, 20, 64, device="cuda").bfloat16().requires_grad_()
    out = block.mixer_forward(hidden)
    a = torch.autograd.grad(out.sum(), [hidden, block.in_x], retain_graph=True)
    b = torch.autograd.grad(out.sum(), [hidden, block.in_x], retain_graph=True)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    with torch.no_grad():
        block.out_proj.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified in place"):
        torch.autograd.grad(out.sum(), hidden)


@pytest.mark.parametrize("whole", [True, False])
def test_mamba1_graph_is_walked_once_unless_it_is_retained(whole):
    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    hidden = torch.randn(1, 20, 64, device="cuda").bfloat16().requires_grad_()
    with contextlib.nullcontext() if whole else composed():
        out = block.mixer_forward(hidden).float().sum()
        out.backward(retain_graph=True)
        out.backward()
        grad = hidden.grad.clone()
        with pytest.raises(RuntimeError, match="backward through the graph a second time"):
            out.backward()
    assert torch.equal(hidden.grad, grad)


# parameters without a gradient; what is edited between forward and backward; whether the backward reads it
@pytest.mark.parametrize("frozen,edited,read", [
    (["in_x", "in_z"], "hidden", False), (["in_x"], "hidden", True), ([], "A_log", False), ([], "in_x", True), (["hidden"], "in_x", False), (["hidden"], "x_proj", True),
    (["hidden", "in_x", "conv_w", "conv_b"], "x_proj", False), (["hidden", "in_x", "conv_w", "conv_b", "x_proj"], "dt_proj", False), ([], "out_proj", True), ([], "dt_bias", True)])
def test_mamba1_inputs_that_the_backward_does_not_read_may_be_edited(frozen, edited, read):
    torch.manual_seed(1)
    block = Mamba1Block(64, device="cuda", dtype=torch.float32)
    leaf = torch.randn(1, 20, 64, device="cuda").requires_grad_("hidden" not in frozen)
    for n, p in block.named_parameters():
        p.requires_grad_(n not in frozen)
    live = [p for p in [leaf, *block.parameters()] if p.requires_grad and p is not block.norm_w]

    def run():
        hidden = leaf * 1.0
        out = block.mixer_forward(hidden)
        with torch.no_grad():
            (hidden if edited == "hidden" else getattr(block, edited)).mul_(1.0)
        return torch.autograd.grad(out.square().sum(), live)

    results = []
    for namespace in (ops, types.SimpleNamespace(**{n: getattr(ops, n) for n in ops.__all__})):  # the second without whole mixers
        block._ops = namespace
        if read:
            with pytest.raises(RuntimeError, match="modified in place|modified by an inplace"):
                run()
        else:
            results.append(run())
    for a, b in zip(*results):
        _near(a, b, torch.float32, edited)


def test_mamba1_in_place_residual_trains():
    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    block.in_x.requires_grad_(False), block.in_z.requires_grad_(False)
    leaf = torch.randn(1, 20, 64, device="cuda").bfloat16().requires_grad_()
    h = leaf * 1.0
    h += block.mixer_forward(h)
    h.float().sum().backward()
    assert leaf.grad.isfinite().all() and block.out_proj.grad is not None


@pytest.mark.parametrize("frozen", [[], ["out_proj"], ["in_x", "in_z"], ["x_proj", "dt_proj"], ["but out_proj"]])
def test_mamba1_keeps_no_more_than_composed_operators(frozen):
    """Bytes held after the forward pass, at the worst in the backward, and after it while the loss is alive."""
    block = Mamba1Block(256, device="cuda", dtype=torch.bfloat16)
    for n, p in block.named_parameters():
        p.requires_grad_(n == "out_proj" if frozen == ["but out_proj"] else n not in frozen)

    def run(namespace):
        block._ops = namespace
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        leaf = torch.randn(8, 1024, 256, device="cuda").bfloat16().requires_grad_(frozen != ["but out_proj"])
        loss = block.mixer_forward(leaf * 1.0).float().sum()
        kept = torch.cuda.memory_allocated() - before
        torch.cuda.reset_peak_memory_stats()
        loss.backward()
        peak, left = torch.cuda.max_memory_allocated() - before, torch.cuda.memory_allocated() - before
        for p in block.parameters():
            p.grad = None
        assert loss.isfinite()
        return kept, peak, left

    whole, apart = ops, types.SimpleNamespace(**{n: getattr(ops, n) for n in ops.__all__})
    run(whole), run(apart)  # library workspaces
    got, want = run(whole), run(apart)
    gradient = 8 * 1024 * 256 * 2  # the incoming one, which autograd holds while the node runs
    for what, a, b in zip(("kept", "peak", "left"), got, want):
        assert a <= b + 65536 + (gradient if what == "peak" else 0), (what, got, want)  # (small tensors round up to blocks of their own)


@pytest.mark.parametrize("create_graph", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_mamba1_backward_inside_autocast(dtype, create_graph):
    """The forward pass ran outside: the gradients are those of its types."""
    torch.manual_seed(2)
    block = Mamba1Block(64, device="cuda", dtype=dtype)
    hidden = torch.randn(2, 33, 64, device="cuda").to(dtype).requires_grad_()
    go = torch.randn(2, 33, 64, device="cuda").to(dtype)
    leaves = [hidden, *(p for n, p in block.named_parameters() if n != "norm_w")]
    want = torch.autograd.grad(block.mixer_forward(hidden), leaves, go)
    out = block.mixer_forward(hidden)
    with torch.autocast("cuda", torch.float16):
        got = torch.autograd.grad(out, leaves, go, create_graph=create_graph)
    for a, b in zip(got, want):
        _near(a.detach(), b, dtype, "gradient")


def test_mamba1_modes_that_compose():
    block = Mamba1Block(64, device="cuda", dtype=torch.float32)
    hidden = torch.randn(1, 20, 64, device="cuda")
    with torch.autocast("cuda", torch.bfloat16):
        assert ops.mamba1_mixer(hidden, block._step_weights()) is None
        assert block.mixer_forward(hidden).dtype == torch.bfloat16
    assert ops.mamba1_mixer(hidden.bfloat16(), block._step_weights()) is None  # other types than the weights'
    assert ops.mamba1_mixer(hidden[:, :0], block._step_weights()) is None
    half = Mamba1Block(64, device="cuda", dtype=torch.bfloat16).requires_grad_(False)
    with torch.no_grad():
        traced = torch.jit.trace(lambda t: half.mixer_forward(t), hidden.bfloat16(), check_trace=False)
        _near(traced(hidden.bfloat16() * 2), half.mixer_forward(hidden.bfloat16() * 2), torch.bfloat16, "traced")


@pytest.mark.parametrize("nb,nl,dm,groups,dtype", [(2, 300, 128, 1, torch.bfloat16), (1, 1, 64, 1, torch.float16), (1, 513, 256, 2, torch.bfloat16)])
def test_mamba2_matches_composed_operators(nb, nl, dm, groups, dtype):
    torch.manual_seed(nl)
    block = Mamba2Block(dm, ngroups=groups, device="cuda", dtype=dtype)
    hidden, res = torch.randn(nb, nl, dm, device="cuda").to(dtype), torch.randn(nb, nl, dm, device="cuda")
    with torch.no_grad():
        assert ops.mamba2_mixer(hidden, block._weights(), block._cfg()) is not None
        got = block(hidden, res)
        with composed():
            assert ops.mamba2_mixer(hidden, block._weights(), block._cfg()) is None
            want = block(hidden, res)
    assert ops.mamba2_mixer(hidden, block._weights(), block._cfg()) is None  # gradients enabled
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("nl", [128, 256])  # as many steps as channels of B and C, of x
def test_mamba2_of_as_many_steps_as_channels(nl, grad):
    torch.manual_seed(4)
    block = Mamba2Block(128, device="cuda", dtype=torch.bfloat16)
    u = torch.randn(2, nl + 1, 128, device="cuda").bfloat16()
    with torch.set_grad_enabled(grad):
        got, want = block.mixer_forward(u[:, :nl]), block.mixer_forward(u)[:, :nl]
    _near(got.detach(), want.detach(), torch.bfloat16, "out")


def _other_out_proj(block):
    """Weights without gradients and another output projection, in which a mixer is linear."""
    w = {n: p.detach() for n, p in block.named_parameters()}
    return w, torch.randn_like(w["out_proj"])


@pytest.mark.parametrize("train", [False, True])
def test_mamba1_tangent_of_the_output_projection(train):
    import torch.autograd.forward_ad as fwd
    from ssm_b200.mixer import mamba1_mixer_forward

    torch.manual_seed(5)
    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    w, other = _other_out_proj(block)
    hidden = torch.randn(2, 33, 64, device="cuda").bfloat16().requires_grad_(train)
    cfg = dict(d_state=block.d_state, dt_rank=block.dt_rank)
    want = mamba1_mixer_forward(ops, {**w, "out_proj": other}, cfg, hidden)
    with fwd.dual_level():
        got = mamba1_mixer_forward(ops, {**w, "out_proj": fwd.make_dual(w["out_proj"], other)}, cfg, hidden)
        _near(fwd.unpack_dual(got).tangent.detach(), want.detach(), torch.bfloat16, "tangent")


@pytest.mark.parametrize("train", [False, True])
def test_mamba1_batched_output_projection(train):
    """torch.vmap over the last product's weight; the operators in front of it see plain tensors."""
    from ssm_b200.mixer import mamba1_mixer_forward

    torch.manual_seed(6)
    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    w, other = _other_out_proj(block)
    hidden, cfg = torch.randn(2, 33, 64, device="cuda").bfloat16(), dict(d_state=block.d_state, dt_rank=block.dt_rank)
    both = torch.stack([w["out_proj"], other]).requires_grad_(train)
    got = torch.vmap(lambda o: mamba1_mixer_forward(ops, {**w, "out_proj": o}, cfg, hidden))(both)
    assert got.requires_grad == train
    for a, o in zip(got, both):
        _near(a.detach(), mamba1_mixer_forward(ops, {**w, "out_proj": o.detach()}, cfg, hidden), torch.bfloat16, "out")



class _Doubled(torch.Tensor):
    """A weight that stands for twice its values."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        plain = lambda t: t.as_subclass(torch.Tensor) if isinstance(t, cls) else t  # noqa: E731
        if func is torch.Tensor.t:
            return plain(args[0]).t().as_subclass(cls)
        if func is torch.matmul:
            return torch.matmul(*(2 * plain(t) if isinstance(t, cls) else t for t in args))
        return func(*map(plain, args), **(kwargs or {}))


@pytest.mark.parametrize("cls", [Mamba1Block, Mamba2Block])
def test_weights_of_a_tensor_subclass(cls):
    from ssm_b200 import mixer

    torch.manual_seed(7)
    block = cls(128, device="cuda", dtype=torch.bfloat16).requires_grad_(False)
    w = dict(block.named_parameters())
    hidden = torch.randn(2, 33, 128, device="cuda").bfloat16()
    if cls is Mamba1Block:
        run = lambda w: mixer.mamba1_mixer_forward(ops, w, dict(d_state=block.d_state, dt_rank=block.dt_rank), hidden)  # noqa: E731
    else:
        run = lambda w: mixer.mamba2_mixer_forward(ops, w, block._cfg(), hidden)  # noqa: E731
    with torch.no_grad():
        got = run({**w, "out_proj": w["out_proj"].detach().as_subclass(_Doubled)})
        _near(got, 2 * run(w), torch.bfloat16, "out")
