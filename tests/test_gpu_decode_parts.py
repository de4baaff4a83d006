"""Decode steps between the one-launch kernels and the library's: the product kernel at the edges of its tiles, columns and splits, the
window updates of four sequences per thread, the state step of a warp that keeps its channels, and whole steps."""

from __future__ import annotations

import ctypes

import pytest
import torch

from oracle import ssm_oracle as orc
from ssm_b200 import _lib
from tests.gpu_util import close
from tests.test_gpu_decode import TOL, _cpu_copy

pytestmark = pytest.mark.gpu


class _GemmArgs(ctypes.Structure):
    _fields_ = [("batch", ctypes.c_int32), ("k", ctypes.c_int32), ("mats", ctypes.c_int32), ("io_dtype", ctypes.c_int32), ("ldx", ctypes.c_int64),
                ("x", ctypes.c_void_p), ("w", ctypes.c_void_p * 5), ("rows", ctypes.c_int32 * 5), ("out", ctypes.c_void_p * 5), ("ldo", ctypes.c_int64 * 5),
                ("status", ctypes.c_void_p), ("weights_ahead", ctypes.c_int32), ("plan_rows", ctypes.c_int32), ("plan_splits", ctypes.c_int32),
                ("reserved0", ctypes.c_int32)]


# one element of everything; whole tiles; token rows, weight rows and columns that end inside one; an output whose rows start on no 8-byte
# boundary (odd row counts); rows of x that lie apart; more CTAs than SMs
@pytest.mark.parametrize("nb,k,rows,pad,dtype", [(1, 8, [1], 0, torch.bfloat16), (16, 64, [128], 0, torch.float16), (17, 72, [129, 5], 8, torch.bfloat16),
                                                 (33, 200, [300, 20, 7], 0, torch.float16), (255, 128, [128, 130], 24, torch.bfloat16), (256, 2112, [200], 0, torch.bfloat16),
                                                 (64, 5120, [192], 0, torch.float16), (100, 768, [1536, 1536, 128, 128, 24], 0, torch.bfloat16), (256, 160, [5120], 32, torch.bfloat16), (200, 128, [19300], 0, torch.float16)])
def test_rows_product_matches_double_precision(nb, k, rows, pad, dtype):
    _check_product(nb, k, rows, pad, dtype)


# every split over 2, 4 and 8 CTAs at 16 to 256 token rows of a CTA: one pass through the stages and several; columns that are no multiple of the
# split; token rows that end inside a CTA's; two CTAs on an SM (more CTAs than SMs, up to 208 token rows) and one with the whole ring (more)
@pytest.mark.parametrize("nb,k,rows,n,splits", [(17, 320, [130], 16, 2), (64, 5120, [2560], 64, 4), (128, 5120, [2560], 128, 2), (128, 2112, [200, 7], 64, 8), (255, 1032, [300], 256, 4),
                                                (256, 5120, [256], 256, 8), (100, 520, [129], 112, 8), (200, 640, [19200], 208, 1), (250, 640, [19200], 256, 1), (256, 640, [9600], 128, 4)])
def test_rows_product_of_every_split_matches_double_precision(nb, k, rows, n, splits):
    _check_product(nb, k, rows, 0, torch.bfloat16, n, splits)


@pytest.mark.parametrize("n,splits", [(8, 1), (24, 1), (272, 1), (16, 3), (16, 16), (32, 4)])
def test_plans_that_are_none_are_refused(n, splits):
    with pytest.raises(AssertionError):
        _check_product(32, 128, [128], 0, torch.bfloat16, n, splits)


def _check_product(nb, k, rows, pad, dtype, n=0, splits=0):
    lib = _lib.load()
    lib.ssmb_rows_gemm.restype = ctypes.c_int
    gen = torch.Generator(device="cuda").manual_seed(nb + k)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    x = rnd(nb, k + pad).to(dtype)
    ws = [(rnd(r, k) / k ** 0.5).to(dtype) for r in rows]
    outs = [torch.full((nb, r + 3), 9.0, device="cuda", dtype=dtype) for r in rows]  # rows that lie apart: nothing beyond them is written
    status = torch.zeros(1, dtype=torch.int32).pin_memory()
    a = _GemmArgs(batch=nb, k=k, mats=len(ws), io_dtype=1 if dtype == torch.bfloat16 else 2, ldx=k + pad, x=x.data_ptr(), status=status.data_ptr(),
                  plan_rows=n, plan_splits=splits)
    for i, (w, o) in enumerate(zip(ws, outs)):
        a.w[i], a.rows[i], a.out[i], a.ldo[i] = w.data_ptr(), w.shape[0], o.data_ptr(), o.stride(0)
    for ahead in (0, 1):
        a.weights_ahead = ahead
        assert lib.ssmb_rows_gemm(ctypes.byref(a), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        assert status.item() == 0
        for w, o in zip(ws, outs):
            xd, wd = x[:, :k].double(), w.double()
            want, terms = xd @ wd.t(), xd.abs() @ wd.abs().t()
            # one rounding to the type (half a unit of its last place: 2^-9, 2^-12) and fp32 sums of k products
            tol = want.abs() * 2.0 ** (-8 if dtype == torch.bfloat16 else -11) + terms * k * 2.0 ** -24 + 1e-7
            r = w.shape[0]
            assert ((o[:, :r].double() - want).abs() <= tol).all()
            assert (o[:, r:] == 9.0).all()
            o[:, :r] = 0


# d_model 320 and 96: dt_rank 20 and 6 (rows of dt_proj that start on no 16-byte boundary); 257 sequences: the library's products
@pytest.mark.parametrize("nb,dm,dtype", [(17, 320, torch.float16), (33, 96, torch.bfloat16), (129, 256, torch.bfloat16), (256, 128, torch.float16), (257, 64, torch.bfloat16)])
def test_mamba1_step_of_many_sequences_matches_oracle(nb, dm, dtype):
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


@pytest.mark.parametrize("nb,dm,groups,dtype", [(18, 96, 3, torch.bfloat16), (130, 256, 1, torch.float16), (256, 128, 2, torch.bfloat16), (300, 64, 1, torch.bfloat16)])
def test_mamba2_step_of_many_sequences_matches_oracle(nb, dm, groups, dtype):
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
            close(block.mixer_step(tok.cuda(), (wg, sg)), ref.mixer_step(tok.float(), (wc, sc)), **TOL, what="mixer output")
    for g, c in zip((*wg, sg), (*wc, sc)):
        close(g, c, **TOL, what="cache")


@pytest.mark.parametrize("nb,nc,k,dtype", [(259, 2600, 4, torch.bfloat16), (1025, 600, 4, torch.float32), (203, 3001, 3, torch.float16)])
def test_window_update_of_many_sequences_matches_oracle(nb, nc, k, dtype):
    from ssm_b200 import ops

    gen = torch.Generator().manual_seed(nb)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    state, x, w, b = rnd(nb, nc, k), rnd(nb, nc).to(dtype), rnd(nc, k).to(dtype), rnd(nc).to(dtype)
    sg = state.cuda()
    y = ops.dw_causal_conv_update(sg, x.cuda(), w.cuda(), b.cuda(), "silu")
    want = torch.cat([state[:, :, 1:], x.float()[:, :, None]], dim=2)
    pre = (want * w.float()).sum(-1) + b.float()
    tol = dict(rtol=1e-4, atol=1e-5) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-3)
    assert torch.equal(sg.cpu(), want)
    close(y, torch.nn.functional.silu(pre), **tol, what="y")


# enough sequences that a warp keeps its channels; the last slice of sequences is shorter than the others
@pytest.mark.parametrize("n,nd,groups,gate,a_dtype", [(16, 1024, 1, True, torch.bfloat16), (32, 512, 2, False, torch.float32), (64, 256, 1, True, torch.float16), (128, 128, 1, True, torch.bfloat16)])
def test_state_step_by_channels_matches_oracle(n, nd, groups, gate, a_dtype):
    from ssm_b200 import ops

    nb = 231
    gen = torch.Generator().manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    state, x, dt = rnd(nb, nd, n), rnd(nb, nd).to(a_dtype), rnd(nb, nd).to(a_dtype)
    z = rnd(nb, nd).to(a_dtype) if gate else None
    A, B, C, D, bias = -torch.exp(rnd(nd, n) * 0.5), rnd(nb, groups, n).to(a_dtype), rnd(nb, groups, n).to(a_dtype), rnd(nd), rnd(nd)
    sg = state.cuda()
    c = lambda t: None if t is None else t.cuda()  # noqa: E731
    y = ops.selective_state_step(sg, c(x), c(dt), c(A), c(B), c(C), D=c(D), z=c(z), dt_bias=c(bias), softplus=True)
    yo = orc.selective_state_step(state, x, dt, A, B, C, D=D, z=z, dt_bias=bias, softplus=True)
    tol = dict(rtol=1e-4, atol=1e-4) if a_dtype == torch.float32 else dict(rtol=2e-2, atol=1e-2)
    close(y, yo, **tol, what="y"), close(sg, state, rtol=1e-4, atol=1e-4, what="state")


@pytest.mark.parametrize("nb", [3, 20, 300])
def test_groups_that_cut_through_a_head_are_refused_before_anything_is_written(nb):
    from ssm_b200 import ops
    from ssm_b200.mixer import Mamba2Block

    w = dict(Mamba2Block(96, device="cuda", dtype=torch.bfloat16)._weights())  # three heads, here with two groups of states
    for k, shape in {"in_B": (256, 96), "in_C": (256, 96), "conv_B": (256, 4), "conv_C": (256, 4), "conv_B_b": (256,), "conv_C_b": (256,)}.items():
        w[k] = torch.randn(*shape, device="cuda").bfloat16()
    windows = [torch.zeros(nb, c, 4, device="cuda") for c in (192, 256, 256)]
    state = torch.zeros(nb, 3, 64, 128, device="cuda")
    with torch.no_grad(), pytest.raises(ValueError, match="G dividing H"):
        ops.mamba2_step(torch.randn(nb, 96, device="cuda").bfloat16(), tuple(windows), state, w)
    assert not any(t.any() for t in (*windows, state))


def test_windows_of_another_shape_are_refused():
    from ssm_b200 import ops
    from ssm_b200.mixer import Mamba2Block

    block = Mamba2Block(64, device="cuda", dtype=torch.bfloat16)
    (wx, wB, wC), state = block.allocate_inference_cache(20)
    with torch.no_grad(), pytest.raises(ValueError, match="conv_state must be"):
        ops.mamba2_step(torch.randn(20, 64, device="cuda").bfloat16(), (wx.view(20, 4, -1), wB, wC), state, block._weights())


def test_a_step_inside_autocast_to_another_type_answers_in_that_type():
    from ssm_b200.mixer import Mamba1Block

    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    tok, cache = torch.randn(20, 64, device="cuda").bfloat16(), block.allocate_inference_cache(20)
    with torch.no_grad(), torch.autocast("cuda", torch.float16):
        assert block.mixer_step(tok, cache).dtype == torch.float16
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        assert block.mixer_step(tok, cache).dtype == torch.bfloat16


def test_a_tangent_of_the_residual_is_refused():
    import torch.autograd.forward_ad as fwd
    from ssm_b200.mixer import Mamba1Block

    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    hidden, res, cache = torch.randn(20, 1, 64, device="cuda").bfloat16(), torch.randn(20, 1, 64, device="cuda"), block.allocate_inference_cache(20)
    with torch.no_grad(), fwd.dual_level(), pytest.raises(NotImplementedError, match="forward-mode"):
        block.step(hidden, fwd.make_dual(res, torch.ones_like(res)), *cache)


# the launches of a step that is captured: overlapped kernels, clusters and, at 256 sequences of a wide model, one of the library's products
@pytest.mark.parametrize("cls,nb,dm", [("Mamba1Block", 20, 320), ("Mamba1Block", 256, 2048), ("Mamba2Block", 130, 256)])
def test_captured_steps_match_plain_ones(cls, nb, dm):
    from ssm_b200 import mixer

    torch.manual_seed(0)
    block = getattr(mixer, cls)(dm, device="cuda", dtype=torch.bfloat16)
    flat = lambda cache: [cache[0], cache[1]] if cls == "Mamba1Block" else [*cache[0], cache[1]]  # noqa: E731
    toks = [torch.randn(nb, dm, device="cuda").bfloat16() for _ in range(3)]
    plain, captured = block.allocate_inference_cache(nb), block.allocate_inference_cache(nb)
    with torch.no_grad():
        want = [block.mixer_step(t, plain) for t in toks]
        tok = toks[0].clone()
        block.mixer_step(tok, block.allocate_inference_cache(nb))  # library handles and workspaces
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = block.mixer_step(tok, captured)
        for t, w in zip(toks, want):
            tok.copy_(t)
            graph.replay()
            assert torch.equal(out, w)
    for a, b in zip(flat(plain), flat(captured)):
        assert torch.equal(a, b)
    del graph


@pytest.mark.parametrize("cls", ["Mamba1Block", "Mamba2Block"])
def test_a_tangent_of_the_output_projection_goes_through_a_step(cls):
    import torch.autograd.forward_ad as fwd
    from ssm_b200 import mixer, ops

    torch.manual_seed(3)
    block = getattr(mixer, cls)(64, device="cuda", dtype=torch.bfloat16)
    w = {n: p.detach() for n, p in block.named_parameters()}
    other, tok = torch.randn_like(w["out_proj"]), torch.randn(20, 64, device="cuda").bfloat16()

    def step(out_proj):
        cache = block.allocate_inference_cache(20)
        if cls == "Mamba1Block":
            return ops.mamba1_step(tok, None, *cache, {**w, "out_proj": out_proj})
        return ops.mamba2_step(tok, *cache, {**w, "out_proj": out_proj})

    want = step(other)
    with fwd.dual_level():
        got = fwd.unpack_dual(step(fwd.make_dual(w["out_proj"], other))).tangent
    assert got is not None and (got.double() - want.double()).norm() <= 1e-2 * want.double().norm()


def test_a_tangent_of_the_gated_norm_is_refused():
    import torch.autograd.forward_ad as fwd
    from ssm_b200 import ops
    from ssm_b200.mixer import Mamba2Block

    block = Mamba2Block(64, device="cuda", dtype=torch.bfloat16)
    w = {n: p.detach() for n, p in block.named_parameters()}
    with fwd.dual_level(), pytest.raises(NotImplementedError, match="forward-mode"):
        dual = {**w, "norm_w": fwd.make_dual(w["norm_w"], torch.ones_like(w["norm_w"]))}
        ops.mamba2_step(torch.randn(20, 64, device="cuda").bfloat16(), *block.allocate_inference_cache(20), dual)
