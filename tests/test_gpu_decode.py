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
