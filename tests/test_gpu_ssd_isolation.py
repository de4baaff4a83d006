"""Sequences packed end to end do not see each other: values that overflow in one leave every other sequence's outputs and states as
they are, wherever the boundary falls in the 32-step column, the 64-step stage, the 128-row block and the 256-step chunk."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
# the steep A puts chunks on the exact per-element form of the decay mask, whose cut columns are not formed as products
@pytest.mark.parametrize("first,steep", [(1, False), (31, True), (63, False), (65, True), (127, False), (128, False), (129, True), (192, False), (255, True),
                                         (256, False), (300, True)])
def test_nonfinite_neighbours_do_not_leak(first, steep, bad, dtype):
    from ssm_b200 import ops

    lens, nh, ng = [first, 200, 70], 4, 2
    nl = sum(lens)
    g = torch.Generator().manual_seed(first)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    X, z, dt = r(1, nl, nh, 64).to(dtype), r(1, nl, nh, 64).to(dtype), r(1, nl, nh).to(dtype)
    B, C = (r(1, nl, ng, 128) / 128 ** 0.5).to(dtype), (r(1, nl, ng, 128) / 128 ** 0.5).to(dtype)
    A, D = -torch.exp(r(nh)) * (40.0 if steep else 1.0), r(nh, 64) if first % 4 == 1 else r(nh)  # a skip weight per channel is another instance
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    clean = [t.cuda() for t in (X, dt, A, B, C)]
    kw = dict(D=D.cuda(), z=z.cuda(), dt_softplus=True, cu_seqlens=cu, return_final_states=True, return_varlen_states=True, check_status=True)
    Y, _, states = ops.ssd_scan(*clean, 256, **kw)
    assert torch.isfinite(Y).all() and torch.isfinite(states).all()
    a, b = lens[0], lens[0] + lens[1]
    for which in range(5):  # X, dt, B, C and z of the middle sequence, one at a time
        dirty = [t.clone() for t in clean]
        kw2 = dict(kw, z=kw["z"].clone())
        target = [dirty[0], dirty[1], dirty[3], dirty[4], kw2["z"]][which]
        target[:, a:b] = bad
        Yd, last, sd = ops.ssd_scan(*dirty, 256, **kw2)
        for s in (slice(0, a), slice(b, nl)):
            assert torch.equal(Yd[:, s], Y[:, s]), which
        assert torch.equal(sd[0], states[0]) and torch.equal(sd[2], states[2]) and torch.equal(last[0], states[2]), which


def test_a_step_of_zero_size_keeps_its_nonfinite_input():
    """0 x Inf inside a sequence is NaN in the packed form as in the separate scan."""
    from ssm_b200 import ops

    X = torch.ones(1, 96, 2, 64, dtype=torch.bfloat16, device="cuda")
    dt = torch.full((1, 96, 2), 0.1, dtype=torch.bfloat16, device="cuda")
    B = torch.ones(1, 96, 1, 128, dtype=torch.bfloat16, device="cuda")
    A = -torch.ones(2, device="cuda")
    X[:, 10], dt[:, 10] = float("inf"), 0.0
    cu = torch.tensor([0, 40, 96], device="cuda")
    _, packed = ops.ssd_scan(X, dt, A, B, B, 256, cu_seqlens=cu, return_varlen_states=True)
    _, alone = ops.ssd_scan(X[:, :40], dt[:, :40], A, B[:, :40], B[:, :40], 256, return_final_states=True)
    assert torch.equal(torch.isnan(packed[0]), torch.isnan(alone[0])) and torch.isnan(alone).any() and torch.isfinite(packed[1]).all()
