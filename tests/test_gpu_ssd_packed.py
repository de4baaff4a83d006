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


@pytest.mark.parametrize("empty", [0, 66000])  # sequences of no step in front: a group of nothing else
def test_more_sequences_than_one_grid_takes(empty):
    """65536 chunks and more go in groups; each sequence as when it is scanned alone."""
    from ssm_b200 import ops

    ones, tail = 65700, 300
    nl = ones + tail
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    X, z, dt = r(1, nl, 1, 64).bfloat16(), r(1, nl, 1, 64).bfloat16(), (torch.rand(1, nl, 1, generator=g, device="cuda") + 0.1).bfloat16()
    B, C, A, D = r(1, nl, 1, 128).bfloat16() / 11, r(1, nl, 1, 128).bfloat16() / 11, -torch.ones(1, device="cuda"), r(1)
    cu = torch.cat([torch.zeros(empty, dtype=torch.long), torch.arange(ones + 1), torch.tensor([nl])]).cuda()
    with torch.no_grad():
        Y, states = ops.ssd_scan(X, dt, A, B, C, 256, D=D, z=z, cu_seqlens=cu, return_varlen_states=True, check_status=True)
        yt, st = ops.ssd_scan(X[:, ones:], dt[:, ones:], A, B[:, ones:], C[:, ones:], 256, D=D, z=z[:, ones:], return_final_states=True)
    assert states.shape[0] == empty + ones + 1 and not states[:empty].any()
    close(Y[:, ones:], yt, **SSD_TOL, what="Y of the last", reduced=True), close(states[-1], st[0], **SSD_TOL, what="state of the last", reduced=True)
    # one step from zero: S = dt x B^T, y = (dt B . C + D) x silu(z)
    x, b, c, d = X[0, :ones, 0].float(), B[0, :ones, 0].float(), C[0, :ones, 0].float(), dt[0, :ones].float()
    zz = z[0, :ones, 0].float()
    want = ((b * c).sum(-1, keepdim=True) * d + D) * x * torch.nn.functional.silu(zz)
    close(Y[0, :ones, 0], want, **SSD_TOL, what="Y", reduced=True)
    for a in range(0, ones, 10000):
        e = min(a + 10000, ones)
        close(states[empty + a:empty + e, 0], (d[a:e] * x[a:e])[:, :, None] * b[a:e, None, :], **SSD_TOL, what="states", reduced=True)
