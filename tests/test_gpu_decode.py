"""Whole-mixer decode steps: the one-launch kernels for small batches and the library-GEMM form above them, against the
CPU oracle's operator-by-operator step at the sizes where a tile, a batch row or a split can go wrong."""

from __future__ import annotations

import pytest
import torch

from oracle import ssm_oracle as orc
from tests.gpu_util import close

pytestmark = pytest.mark.gpu

TOL = dict(rtol=2e-2, atol=2e-2)  # chains of 16-bit projections


def _cpu_copy(block, cls, **kw):
    ref = cls(block.d_model, ops=orc, **kw)
    ref.load_state_dict({k: v.float().cpu() for k, v in block.state_dict().items()})
    return ref.float()


# one and two groups of eight token rows, the largest batch of one launch and the first beyond it; d_model 32: fewer tiles than SMs;
# 320: a dt_rank that is no multiple of eight; 96: dt_rank 6, which the one-launch kernel leaves to the other path
@pytest.mark.parametrize("nb,dm,dtype", [(1, 768, torch.bfloat16), (8, 320, torch.float16), (9, 64, torch.bfloat16), (16, 1024, torch.float16),
                                         (17, 128, torch.bfloat16), (2, 96, torch.float16)])
def test_mamba1_step_matches_oracle(nb, dm, dtype):
    from ssm_b200.mixer import Mamba1Block

    torch.manual_seed(nb * dm)
    block = Mamba1Block(dm, device="cuda", dtype=dtype)
    ref = _cpu_copy(block, Mamba1Block)
    cg, cc = block.allocate_inference_cache(nb), ref.allocate_inference_cache(nb)
    with torch.no_grad():
        for g, c in zip(cg, cc):
            c.normal_(std=0.1), g.copy_(c)
        for _ in range(2):
            hidden, res = torch.randn(nb, 1, dm).to(dtype), torch.randn(nb, 1, dm)
            out_g, res_g = block.step(hidden.cuda(), res.cuda(), *cg)
            out_c, res_c = ref.step(hidden.float(), res, *cc)
            close(out_g, out_c, **TOL, what="normed"), close(res_g, res_c, **TOL, what="residual")
        mix_g, mix_c = block.mixer_step(hidden[:, 0].cuda(), cg), ref.mixer_step(hidden[:, 0].float(), cc)
    close(mix_g, mix_c, **TOL, what="mixer output")
    close(cg[0], cc[0], **TOL, what="conv window"), close(cg[1], cc[1], **TOL, what="state")


@pytest.mark.parametrize("nb,dm,groups,dtype", [(1, 256, 1, torch.bfloat16), (8, 320, 2, torch.float16), (16, 96, 3, torch.bfloat16), (17, 128, 1, torch.float16)])
def test_mamba2_step_matches_oracle(nb, dm, groups, dtype):
    from ssm_b200.mixer import Mamba2Block

    torch.manual_seed(nb * dm)
    block = Mamba2Block(dm, ngroups=groups, device="cuda", dtype=dtype)
    ref = _cpu_copy(block, Mamba2Block, ngroups=groups)
    (wg, sg), (wc, sc) = block.allocate_inference_cache(nb), ref.allocate_inference_cache(nb)
    with torch.no_grad():
        for g, c in zip((*wg, sg), (*wc, sc)):
            c.normal_(std=0.1), g.copy_(c)
        for _ in range(2):
            tok = torch.randn(nb, dm).to(dtype)
            out_g, out_c = block.mixer_step(tok.cuda(), (wg, sg)), ref.mixer_step(tok.float(), (wc, sc))
            close(out_g, out_c, **TOL, what="mixer output")
    for g, c in zip((*wg, sg), (*wc, sc)):
        close(g, c, **TOL, what="cache")


# states of more than two pieces per resident warp (the streaming kernel), rows that do not fill the last piece, every state width
@pytest.mark.parametrize("n,dtype", [(16, torch.bfloat16), (32, torch.float32), (64, torch.float16), (128, torch.bfloat16), (256, torch.float32)])
def test_large_state_step_matches_oracle(n, dtype):
    from ssm_b200 import ops

    nb, nd = 3, 3_700_000 // n // 3 | 1
    gen = torch.Generator().manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    state, x, dt, z = rnd(nb, nd, n), rnd(nb, nd).to(dtype), rnd(nb, nd).to(dtype), rnd(nb, nd).to(dtype)
    A, B, C, D, bias = -torch.exp(rnd(nd, n) * 0.5), rnd(nb, 1, n).to(dtype), rnd(nb, 1, n).to(dtype), rnd(nd), rnd(nd)
    sg = state.cuda()
    c = lambda t: t.cuda()  # noqa: E731
    y = ops.selective_state_step(sg, c(x), c(dt), c(A), c(B), c(C), D=c(D), z=c(z), dt_bias=c(bias), softplus=True)
    yo = orc.selective_state_step(state, x, dt, A, B, C, D=D, z=z, dt_bias=bias, softplus=True)
    tol = dict(rtol=1e-4, atol=1e-4) if dtype == torch.float32 else dict(rtol=2e-2, atol=1e-2)
    close(y, yo, **tol, what="y"), close(sg, state, rtol=1e-4, atol=1e-4, what="state")


def test_large_state_step_with_parameters_per_head_matches_oracle():
    from ssm_b200 import ops

    nb, nh, p, n = 5, 100, 60, 128
    gen = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    state, x, dt, z = rnd(nb, nh, p, n), rnd(nb, nh, p).bfloat16(), rnd(nb, nh).bfloat16(), rnd(nb, nh, p).bfloat16()
    A, B, C, D, bias = -torch.exp(rnd(nh) * 0.5), rnd(nb, 2, n).bfloat16(), rnd(nb, 2, n).bfloat16(), rnd(nh), rnd(nh)
    sg = state.cuda()
    y = ops.selective_state_step_heads(sg, x.cuda(), dt.cuda(), A.cuda(), B.cuda(), C.cuda(), D=D.cuda(), z=z.cuda(), dt_bias=bias.cuda(), softplus=True)
    rep = lambda t: t[:, None].expand(nh, p).reshape(-1)  # noqa: E731
    flat = state.view(nb, nh * p, n)
    yo = orc.selective_state_step(flat, x.reshape(nb, -1), dt.repeat_interleave(p, 1), A[:, None, None].expand(nh, p, n).reshape(nh * p, n), B, C, D=rep(D),
                                  z=z.reshape(nb, -1), dt_bias=rep(bias), softplus=True)
    close(y.reshape(nb, -1), yo, rtol=2e-2, atol=1e-2, what="y"), close(sg.view_as(flat), flat, rtol=1e-4, atol=1e-4, what="state")
