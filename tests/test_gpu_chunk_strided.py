"""Backward of the element-wise chunked recurrence on rows that lie apart in memory (the C interface takes any strides) against the same
call on contiguous rows: two instances of its last pass that differ in nothing but their addresses."""

from __future__ import annotations

import ctypes

import pytest
import torch
import torch.nn.functional as F

from ssm_b200 import _lib
from tests.gpu_util import FP32_TOL, close

pytestmark = pytest.mark.gpu

CODES = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}


def _bcast(t, *strides):
    return _lib.Bcast4(t.data_ptr(), *strides)


@pytest.mark.parametrize("nl,nh,p,gate,dtype", [(33, 3, 64, True, torch.bfloat16), (97, 2, 4, False, torch.float32), (64, 5, 128, True, torch.float16), (65, 1, 8, True, torch.float32)])
def test_strided_rows_match_contiguous_rows(nl, nh, p, gate, dtype):
    lib = _lib.load()
    nb, pad = 2, 8
    gen = torch.Generator(device="cuda").manual_seed(nl)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    X, dY = rnd(nb, nl, nh, p).to(dtype), rnd(nb, nl, nh, p).to(dtype)
    dt, A, D = F.softplus(rnd(nb, nl, nh) - 2).to(dtype), -torch.exp(rnd(nh, p) * 0.5), rnd(nh, p)
    B, C, z = (rnd(nb, nl, nh, p).to(dtype) for _ in range(3))
    lens = torch.tensor([nl, nl - 3], device="cuda")

    def run(extra):
        q = p + extra  # elements from head to head
        wide = lambda t: F.pad(t, (0, extra)).contiguous()  # noqa: E731
        ins = {"Bm": wide(B), "Cm": wide(C), "z": wide(z)}
        grads = {k: torch.full((nb, nl, nh, q), 7.0, device="cuda", dtype=dtype) for k in ("dB", "dC", "dz")}
        dX, ddt = torch.empty_like(X), torch.empty_like(dt)
        dA, dD = torch.zeros_like(A), torch.zeros_like(D)
        g = _lib.ChunkBwdArgs()
        a = g.fwd
        a.batch, a.len, a.heads, a.proj, a.chunk_size = nb, nl, nh, p, 64
        a.io_dtype = a.par_dtype = CODES[dtype]
        a.X, a.dt, a.seq_lens = X.data_ptr(), dt.data_ptr(), lens.data_ptr()
        a.A, a.D = _bcast(A, 0, 0, p, 1), _bcast(D, 0, 0, p, 1)
        strides = (nl * nh * q, nh * q, q, 1)
        a.Bm, a.Cm = _bcast(ins["Bm"], *strides), _bcast(ins["Cm"], *strides)
        g.dB, g.dC = _bcast(grads["dB"], *strides), _bcast(grads["dC"], *strides)
        if gate:
            a.z, g.dz = _bcast(ins["z"], *strides), _bcast(grads["dz"], *strides)
        a.typed_grads = 15 if gate else 11
        g.dA, g.dD = _bcast(dA, 0, 0, p, 1), _bcast(dD, 0, 0, p, 1)
        g.dY, g.dX, g.ddt = dY.data_ptr(), dX.data_ptr(), ddt.data_ptr()
        scratch = torch.empty(lib.ssm_chunk_scan_bwd_scratch_floats(nb, nl, nh, p, 64), device="cuda")
        g.scratch = scratch.data_ptr()
        assert lib.ssm_chunk_scan_bwd_fused(ctypes.byref(g)) == 1
        assert lib.ssm_chunk_scan_bwd(ctypes.byref(g), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        for k, t in grads.items():
            if k != "dz" or gate:
                assert (t[..., p:] == 7.0).all(), f"{k}: written beyond its rows"
        return {"dX": dX, "ddt": ddt, "dA": dA, "dD": dD, **{k: t[..., :p] for k, t in grads.items()}}

    want, got = run(0), run(pad)
    for k in want:
        if k in ("dA", "dD"):  # sums over the CTAs in any order
            close(got[k], want[k], **FP32_TOL, what=k, reduced=True)
        else:
            assert torch.equal(got[k], want[k]), k
