"""Backward of the selective scan with two rows per lane, where its half tiles of 16 steps, its tiles of 32 and its buffers end: every way
in which the last tile can be cut, one to five tiles (each buffer reused), 5 to 16 states, with and without a gate, several B / C
groups, calls cut in time, coefficients of another type than the rows."""

from __future__ import annotations

import pytest
import torch

from oracle import ssm_oracle as oracle
from ssm_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,dim,length,n,groups,gate,bc_dtype,dtype", [
    (1, 32, 1, 16, 1, True, None, torch.bfloat16), (2, 32, 15, 16, 1, False, None, torch.float32), (1, 64, 16, 13, 2, True, None, torch.float16),
    (1, 32, 17, 16, 1, True, torch.float32, torch.bfloat16), (1, 32, 32, 5, 1, False, None, torch.bfloat16), (2, 64, 48, 16, 1, True, None, torch.float32),
    (150, 64, 65, 16, 2, True, None, torch.bfloat16), (80, 64, 160, 16, 1, True, None, torch.float16), (90, 128, 128, 8, 2, True, None, torch.bfloat16),
    (75, 128, 113, 7, 1, False, None, torch.float16), (140, 32, 96, 12, 1, True, torch.bfloat16, torch.float32), (1, 64, 520, 16, 1, True, None, torch.bfloat16)])
def test_gradients_match_oracle(nb, dim, length, n, groups, gate, bc_dtype, dtype):
    g = torch.Generator().manual_seed(length * n)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    u, delta = (r(nb, dim, length).to(dtype) for _ in range(2))
    z = r(nb, dim, length).to(dtype) if gate else None
    A, D, bias = -torch.exp(r(dim, n) * 0.5), r(dim), r(dim) * 0.3 - 1.0
    B, C = (r(nb, groups, n, length).to(bc_dtype or dtype) for _ in range(2))
    init, go, gl = r(nb, dim, n), r(nb, dim, length).to(dtype), r(nb, dim, n)

    def both(fn, dev, cast):
        t = [None if x is None else x.to(dev).to(cast(x)).requires_grad_() for x in (u, delta, A, B, C, D, z, bias, init)]
        out, last = fn(t[0], t[1], t[2], t[3], t[4], D=t[5], z=t[6], dt_bias=t[7], softplus=True, return_last_state=True, initial_state=t[8])
        return [out, last, *torch.autograd.grad((out, last), [x for x in t if x is not None], (go.to(dev).to(out.dtype), gl.to(dev).to(last.dtype)))]

    got = both(ops.selective_scan, "cuda", lambda x: x.dtype)
    want = both(oracle.selective_scan, "cpu", lambda x: torch.float32)
    tol = 1e-4 if dtype == torch.float32 and bc_dtype is None else 2e-2  # the bars of the other scan tests: fp32 sums, 16-bit values
    for i, (a, b) in enumerate(zip(got, want)):
        b = b.reshape(a.shape).double()
        assert (a.cpu().double() - b).norm() <= tol * b.norm() + 1e-6, i
