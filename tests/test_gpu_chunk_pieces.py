"""Element-wise chunked recurrence where pieces, groups of steps and CTAs end: ragged lengths, valid lengths inside a piece, heads of
4 to 128 projections, lanes that do not fill a CTA, a skip weight per head or per channel, with and without gate."""

from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F

from oracle import ssm_oracle as orc
from tests.gpu_util import FP32_TOL, HALF_TOL, close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl,nh,p,gate,per_head,lens,dtype", [
    (33, 3, 64, True, False, None, torch.bfloat16), (100, 2, 4, False, True, None, torch.float32), (257, 5, 128, True, False, [257, 0, 31], torch.float16),
    (64, 1, 8, True, True, [1, 63, 40], torch.bfloat16), (1000, 9, 64, False, False, None, torch.float32), (70, 4, 12, True, True, None, torch.float16)])
def test_gradients_match_oracle(nl, nh, p, gate, per_head, lens, dtype):
    from ssm_b200 import ops

    nb = 3
    gen = torch.Generator().manual_seed(nl)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    ins = {"X": rnd(nb, nl, nh, p).to(dtype), "dt": F.softplus(rnd(nb, nl, nh) - 2).to(dtype), "A": -torch.exp(rnd(nh, p) * 0.5), "B": rnd(nb, nl, nh, p).to(dtype),
           "C": rnd(nb, nl, nh, p).to(dtype), "D": rnd(nh) if per_head else rnd(nh, p)}
    if gate:
        ins["z"] = rnd(nb, nl, nh, p).to(dtype)
    wy = rnd(nb, nl, nh, p).to(dtype).float()
    meta = None if lens is None else {"seq_lens": torch.tensor(lens)}
    lg = {k: v.cuda().requires_grad_() for k, v in ins.items()}
    lo = {k: v.float().requires_grad_() for k, v in ins.items()}

    def run(ops_, t):
        return ops_.ssd_chunk_scan(t["X"], t["dt"], t["A"], t["B"], t["C"], 64, D=t["D"], z=t.get("z"), seq_meta=meta)

    yg, yo = run(ops, lg), run(orc, lo)
    tol = FP32_TOL if dtype == torch.float32 else HALF_TOL
    close(yg, yo, **tol, what="y")
    gg = torch.autograd.grad((yg.float() * wy.cuda()).sum(), list(lg.values()))
    go = torch.autograd.grad((yo * wy).sum(), list(lo.values()))
    for k, a, b in zip(ins, gg, go):
        assert a.dtype == ins[k].dtype
        # ddt is a sum over the head's projections of terms of both signs
        close(a, b, **tol, what=f"d{k}", reduced=k in ("A", "D", "dt"))


# storage offsets in elements: 0 and 8 leave 16-bit rows on 16-byte boundaries (eight projections per lane), 4 on 8-byte ones (four), 1
# on none (one); projections that are no multiple of eight go the same ways
@pytest.mark.parametrize("offset", [0, 8, 4, 1])
@pytest.mark.parametrize("nl,nh,p,gate,lens,dtype", [(33, 3, 64, True, None, torch.bfloat16), (257, 5, 8, False, [257, 0, 31], torch.float16),
                                                     (100, 2, 24, True, [99, 100, 1], torch.bfloat16), (64, 4, 12, True, None, torch.float16), (96, 2, 20, True, [7, 96, 33], torch.float32)])
def test_forward_on_every_lane_width(nl, nh, p, gate, lens, dtype, offset):
    from ssm_b200 import ops

    nb = 3
    gen = torch.Generator().manual_seed(nl + p)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731

    def at(t):  # contiguous, `offset` elements into its allocation
        buf = torch.empty(t.numel() + offset, dtype=t.dtype, device="cuda")
        return buf[offset:].view(t.shape).copy_(t)

    X, B, C = (rnd(nb, nl, nh, p).to(dtype) for _ in range(3))
    z = rnd(nb, nl, nh, p).to(dtype) if gate else None
    dt, A, D, init = F.softplus(rnd(nb, nl, nh) - 2).to(dtype), -torch.exp(rnd(nh, p) * 0.5), rnd(nh, p), rnd(nb, nh, p)
    meta = None if lens is None else {"seq_lens": torch.tensor(lens)}
    with torch.no_grad():
        y = ops.ssd_chunk_scan(at(X), at(dt), A.cuda(), at(B), at(C), 64, D=D.cuda(), z=None if z is None else at(z), seq_meta=meta, initial_states=init.cuda())
        yo = orc.ssd_chunk_scan(X.float(), dt.float(), A, B.float(), C.float(), 64, D=D, z=None if z is None else z.float(), seq_meta=meta, initial_states=init)
    close(y, yo, **(FP32_TOL if dtype == torch.float32 else HALF_TOL), what="y")
