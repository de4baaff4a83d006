"""Selective scan on ragged rows and on calls that are cut in time, against the fp32 oracle: lengths around the tile of 32 steps and the
vector widths, whole vectors, padded state counts, several B / C groups, gradients of the first and last states across the cuts."""

from __future__ import annotations

import pytest
import torch

from oracle import ssm_oracle as oracle
from ssm_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nb,dim,length,n,groups", [(2, 64, 1, 16, 1), (1, 32, 31, 16, 1), (2, 96, 33, 5, 1), (1, 64, 301, 16, 2), (3, 64, 95, 32, 1), (1, 32, 67, 3, 1),
                                                    (1, 32, 64, 16, 1), (2, 32, 416, 16, 1), (1, 64, 1000, 8, 1), (1, 32, 129, 32, 1)])
def test_scan_edges(nb, dim, length, n, groups, dtype):
    g = torch.Generator().manual_seed(length)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    u, delta, z = (r(nb, dim, length).to(dtype) for _ in range(3))
    A, D, bias = -torch.exp(r(dim, n) * 0.5), r(dim), r(dim) * 0.3 - 1.0
    B, C = (r(nb, groups, n, length).to(dtype) for _ in range(2))
    init, go, gl = r(nb, dim, n), r(nb, dim, length).to(dtype), r(nb, dim, n)

    def both(fn, dev, cast):
        t = [x.to(dev).to(cast(x)).requires_grad_() for x in (u, delta, A, B, C, D, z, bias, init)]
        out, last = fn(t[0], t[1], t[2], t[3], t[4], D=t[5], z=t[6], dt_bias=t[7], softplus=True, return_last_state=True, initial_state=t[8])
        return [out, last, *torch.autograd.grad((out, last), t, (go.to(dev).to(out.dtype), gl.to(dev).to(last.dtype)))]

    got = both(ops.selective_scan, "cuda", lambda x: x.dtype)
    want = both(oracle.selective_scan, "cpu", lambda x: torch.float32)
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    for i, (a, b) in enumerate(zip(got, want)):
        b = b.reshape(a.shape).double()
        assert (a.cpu().double() - b).norm() <= tol * b.norm() + 1e-6, i


@pytest.mark.parametrize("op", ["scan", "conv"])
def test_one_row_of_any_stride(op):
    """An extent of one may have any stride, also one shorter than a row."""
    u = torch.randn(2, 40, 1, device="cuda").transpose(1, 2)  # (2, 1, 40) with strides (40, 1, 1)
    if op == "conv":
        w = torch.randn(1, 4, device="cuda")
        run = lambda t: ops.dw_causal_conv(t, w)  # noqa: E731
    else:
        A, BC = -torch.rand(1, 4, device="cuda"), torch.randn(2, 1, 4, 40, device="cuda")
        run = lambda t: ops.selective_scan(t, t.abs(), A, BC, BC)  # noqa: E731
    a, b = u.clone(memory_format=torch.preserve_format).requires_grad_(), torch.empty(2, 1, 40, device="cuda").copy_(u).requires_grad_()
    assert a.stride() == (40, 1, 1)
    ya, yb = run(a), run(b)
    assert torch.equal(ya, yb)
    for x, y in zip(torch.autograd.grad(ya.sum(), a), torch.autograd.grad(yb.sum(), b)):
        torch.testing.assert_close(x, y)
