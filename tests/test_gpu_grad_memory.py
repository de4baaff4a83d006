"""What a gradient keeps alive: the gradient of a small parameter holds no work buffer and no gradient of an activation."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, leaves, small):
    grads = dict(zip(leaves, torch.autograd.grad(out.float().sum(), list(leaves.values()))))
    room = sum(-(-grads[k].numel() // 64) * 256 for k in small)  # every small one on 256-byte lines of its own
    for k in small:
        assert grads[k].untyped_storage().nbytes() <= room, (k, grads[k].untyped_storage().nbytes())
    for k, g in grads.items():  # any gradient: at most a few others of its own size
        assert g.untyped_storage().nbytes() <= 4 * max(g.numel() * g.element_size(), 256) + room, k
    return grads


@pytest.mark.parametrize("bc", [torch.bfloat16, torch.float32])
def test_ssd_scan_parameter_gradients_hold_no_work_buffers(bc):
    from ssm_b200 import ops

    nl, nh = 1500, 8
    mk = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    t = {"X": mk(2, nl, nh, 64).bfloat16(), "dt": mk(2, nl, nh).bfloat16(), "A": -torch.rand(nh, device="cuda") - 0.5, "B": mk(2, nl, 1, 128).to(bc) / 11,
         "C": mk(2, nl, 1, 128).to(bc) / 11, "D": mk(nh), "dt_bias": mk(nh)}
    t = {k: v.requires_grad_() for k, v in t.items()}
    Y = ops.ssd_scan(t["X"], t["dt"], t["A"], t["B"], t["C"], 256, D=t["D"], dt_bias=t["dt_bias"], dt_softplus=True)
    _check(Y, t, ["A", "D", "dt_bias"])


@pytest.mark.parametrize("bkind", ["hp", "bhp", "blhp"])
@pytest.mark.parametrize("zkind", [None, "blh", "blhp"])
def test_chunk_scan_parameter_gradients_hold_no_step_gradients(bkind, zkind):
    from ssm_b200 import ops

    nb, nl, nh, p = 2, 4000, 4, 8
    mk = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    shapes = {"hp": (nh, p), "bhp": (nb, nh, p), "blhp": (nb, nl, nh, p), "blh": (nb, nl, nh)}
    t = {"X": mk(nb, nl, nh, p), "dt": torch.rand(nb, nl, nh, device="cuda") * 0.1, "A": -torch.rand(nh, p, device="cuda"), "B": mk(*shapes[bkind]),
         "C": mk(*shapes[bkind]), "D": mk(nh, p), "initial": mk(nb, nh, p)}
    if zkind:
        t["z"] = mk(*shapes[zkind])
    t = {k: v.requires_grad_() for k, v in t.items()}
    Y = ops.ssd_chunk_scan(t["X"], t["dt"], t["A"], t["B"], t["C"], 64, D=t["D"], z=t.get("z"), initial_states=t["initial"])
    _check(Y, t, ["A", "D"] + (["B", "C"] if bkind == "hp" else []))
