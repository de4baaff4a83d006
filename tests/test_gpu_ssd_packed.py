"""Packed sequences of the state-space-dual scan in one set of launches: lengths around the 128-row block and the 256-step
chunk, empty sequences, several groups and a skip weight per channel, against the CPU oracle sequence by sequence."""

from __future__ import annotations

import pytest
import torch

from oracle import ssm_oracle as orc
from tests.gpu_util import close

pytestmark = pytest.mark.gpu

SSD_TOL = dict(rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("lens,nh,ng,dtype,per_channel", [([1, 127, 128, 129, 0, 255, 256, 257, 3], 2, 1, torch.bfloat16, False), ([513, 0], 4, 2, torch.float16, True),
                                                          ([40] * 9, 6, 1, torch.bfloat16, False)])
@pytest.mark.parametrize("reset", [True, False])
def test_packed_sequences_match_oracle(lens, nh, ng, dtype, per_channel, reset):
    from ssm_b200 import ops

    nl = sum(lens)
    gen = torch.Generator().manual_seed(nl)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    X, z, dt = rnd(1, nl, nh, 64).to(dtype), rnd(1, nl, nh, 64).to(dtype), (rnd(1, nl, nh) - 2).to(dtype)
    B, C = (rnd(1, nl, ng, 128) / 128 ** 0.5).to(dtype), (rnd(1, nl, ng, 128) / 128 ** 0.5).to(dtype)
    A, D, bias = -torch.exp(torch.rand(nh, generator=gen) * 2.7), rnd(nh, 64) if per_channel else rnd(nh), rnd(nh) * 0.3
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    g = lambda t: t.cuda()  # noqa: E731
    Y, last, states = ops.ssd_scan(g(X), g(dt), g(A), g(B), g(C), 256, D=g(D), z=g(z), dt_bias=g(bias), dt_softplus=True, cu_seqlens=g(cu), seq_reset=reset,
                                   return_final_states=True, return_varlen_states=True, check_status=True)
    assert states.shape == (len(lens), nh, 64, 128)
    for k, (a, b) in enumerate(zip(cu[:-1].tolist(), cu[1:].tolist())):
        if a == b:
            assert not states[k].any()
            continue
        s = slice(a, b)
        yo, so = orc.ssd_scan(X[:, s], dt[:, s], A, B[:, s], C[:, s], 256, D=D, z=z[:, s], dt_bias=bias, dt_softplus=True, return_final_states=True)
        close(states[k], so[0], **SSD_TOL, what=f"state {k}", reduced=True)
        if reset:
            close(Y[:, s], yo, **SSD_TOL, what=f"Y of sequence {k}", reduced=True)
    if reset:
        assert torch.equal(last[0], states[-1])
    else:
        yo, so = orc.ssd_scan(X, dt, A, B, C, 256, D=D, z=z, dt_bias=bias, dt_softplus=True, return_final_states=True)
        close(Y, yo, **SSD_TOL, what="Y", reduced=True), close(last, so, **SSD_TOL, what="last state", reduced=True)
