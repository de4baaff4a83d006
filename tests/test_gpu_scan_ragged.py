"""Selective scan on rows that do not start on 16-byte boundaries, against the fp32 oracle: lengths around the tile of 32 steps and the
vector widths, a call that is cut in time, padded state counts, several B / C groups, and B / C with a stride over time."""

from __future__ import annotations

import pytest
import torch

from oracle import ssm_oracle as oracle
from ssm_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nb,dim,length,n,groups", [(2, 64, 1, 16, 1), (1, 32, 31, 16, 1), (2, 96, 33, 5, 1), (1, 64, 301, 16, 2), (3, 64, 95, 32, 1), (1, 32, 67, 3, 1)])
def test_ragged_rows(nb, dim, length, n, groups, dtype):
    g = torch.Generator().manual_seed(length)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    u, delta, z = (r(nb, dim, length).to(dtype) for _ in range(3))
    A, D, bias = -torch.exp(r(dim, n) * 0.5), r(dim), r(dim) * 0.3 - 1.0
    B, C = (r(nb, groups, n, length).to(dtype) for _ in range(2))
    go = r(nb, dim, length).to(dtype)

    def both(fn, dev, cast):
        t = [x.to(dev).to(cast(x)).requires_grad_() for x in (u, delta, A, B, C, D, z, bias)]
        out, last = fn(t[0], t[1], t[2], t[3], t[4], D=t[5], z=t[6], dt_bias=t[7], softplus=True, return_last_state=True)
        return [out, last, *torch.autograd.grad(out, t, go.to(dev).to(out.dtype))]

    got = both(ops.selective_scan, "cuda", lambda x: x.dtype)
    want = both(oracle.selective_scan, "cpu", lambda x: torch.float32)
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    for i, (a, b) in enumerate(zip(got, want)):
        b = b.reshape(a.shape).double()
        assert (a.cpu().double() - b).norm() <= tol * b.norm() + 1e-6, i
