"""The host side of the operators: what they refuse, what they hold up, and what they do when a launch is refused."""

from __future__ import annotations

import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 17])  # one launch, and the projections as separate calls
@pytest.mark.parametrize("which", ["in_x", "conv_w", "conv_b", "x_proj", "dt_proj", "dt_bias", "A_log", "D", "out_proj", "conv_state", "ssm_state", "residual", "norm_w"])
def test_mamba1_step_refuses_host_tensors(which, nb):
    from ssm_b200 import ops
    from ssm_b200.mixer import Mamba1Block

    block = Mamba1Block(64, device="cuda", dtype=torch.bfloat16)
    conv, state = block.allocate_inference_cache(nb)
    t = {**block._parameters, "conv_state": conv, "ssm_state": state, "residual": torch.zeros(nb, 64, device="cuda"), "norm_w": block.norm_w}
    t[which] = t[which].detach().cpu()
    with torch.no_grad(), pytest.raises((RuntimeError, ValueError)):
        ops.mamba1_step(torch.zeros(nb, 64, device="cuda", dtype=torch.bfloat16), t["residual"], t["conv_state"], t["ssm_state"], t, t["norm_w"])


@pytest.mark.parametrize("nb", [1, 17])
def test_decode_steps_refuse_short_vectors(nb):
    from ssm_b200 import ops
    from ssm_b200.mixer import Mamba1Block, Mamba2Block

    tok = torch.zeros(nb, 64, device="cuda", dtype=torch.bfloat16)
    b1, b2 = Mamba1Block(64, device="cuda", dtype=torch.bfloat16), Mamba2Block(64, device="cuda", dtype=torch.bfloat16)
    c1, (win, s2) = b1.allocate_inference_cache(nb), b2.allocate_inference_cache(nb)
    w1, w2 = dict(b1._parameters), dict(b2._parameters)
    norm = b1.norm_w.detach()
    with torch.no_grad():
        for key in ("conv_b", "dt_bias", "D"):
            with pytest.raises((RuntimeError, ValueError)):
                ops.mamba1_step(tok, None, *c1, dict(w1, **{key: w1[key].detach()[:16].clone()}), norm)
        with pytest.raises((RuntimeError, ValueError)):
            ops.mamba1_step(tok, None, *c1, w1, norm[:16].clone())
        for key in ("conv_x_b", "conv_B_b", "conv_C_b", "dt_bias", "D", "norm_w"):
            with pytest.raises((RuntimeError, ValueError)):
                ops.mamba2_step(tok, win, s2, dict(w2, **{key: w2[key].detach()[:1].clone()}))
        with pytest.raises((RuntimeError, ValueError)):
            ops.mamba2_step(tok, [t.cpu() for t in win], s2, w2)


def test_packed_scan_waits_without_the_interpreter_lock():
    from ssm_b200 import ops

    X = torch.randn(1, 600, 2, 64, device="cuda").bfloat16()
    dt, B, A = torch.rand(1, 600, 2, device="cuda").bfloat16(), torch.randn(1, 600, 1, 128, device="cuda").bfloat16(), -torch.ones(2, device="cuda")
    cu = torch.tensor([0, 300, 600], device="cuda")
    ops.ssd_scan(X, dt, A, B, B, 256, cu_seqlens=cu)
    torch.cuda.synchronize()
    beats, stop = [], threading.Event()

    def beat():
        while not stop.is_set():
            beats.append(time.perf_counter())
            time.sleep(0.002)

    th = threading.Thread(target=beat)
    th.start()
    try:
        torch.cuda._sleep(600_000_000)  # about 0.3 s of device time ahead of the read of cu_seqlens
        t0 = time.perf_counter()
        ops.ssd_scan(X, dt, A, B, B, 256, cu_seqlens=cu)
        t1 = time.perf_counter()
    finally:
        stop.set()
        th.join()
    assert t1 - t0 > 0.1, "the call was meant to wait"
    during = [b for b in beats if t0 < b < t1]
    assert len(during) > 0.1 * (t1 - t0) / 0.002, f"{len(during)} beats of another thread in {t1 - t0:.3f} s"


@pytest.mark.parametrize("op", ["scan", "chunk", "conv", "norm", "ssd"])
def test_forward_mode_is_refused(op):
    """No operator has a forward-mode rule: a tangent is an error and never dropped."""
    import torch.autograd.forward_ad as fwd

    from ssm_b200 import ops

    mk = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    with fwd.dual_level():
        dual = lambda *s: fwd.make_dual(mk(*s), mk(*s))  # noqa: E731
        with pytest.raises((RuntimeError, NotImplementedError)):
            if op == "scan":
                ops.selective_scan(dual(1, 8, 40), mk(1, 8, 40), -torch.rand(8, 16, device="cuda"), mk(1, 1, 16, 40), mk(1, 1, 16, 40))
            elif op == "chunk":
                ops.ssd_chunk_scan(dual(1, 40, 2, 8), torch.rand(1, 40, 2, device="cuda"), -torch.rand(2, 8, device="cuda"), mk(1, 40, 2, 8), mk(1, 40, 2, 8), 32)
            elif op == "conv":
                ops.dw_causal_conv(mk(1, 8, 40), dual(8, 4))
            elif op == "norm":
                ops.fused_layer_norm(mk(1, 3, 64), dual(64), None)
            else:
                X = fwd.make_dual(mk(1, 256, 2, 64).bfloat16(), mk(1, 256, 2, 64).bfloat16())
                B = mk(1, 256, 1, 128).bfloat16()
                ops.ssd_scan(X, torch.rand(1, 256, 2, device="cuda").bfloat16(), -torch.ones(2, device="cuda"), B, B, 256)


_REFUSED_STEP = """
import sys, torch
from ssm_b200.mixer import Mamba1Block, Mamba2Block
torch.manual_seed(0)
b1, b2 = Mamba1Block(64, device="cuda", dtype=torch.bfloat16), Mamba2Block(64, device="cuda", dtype=torch.bfloat16)
c1, c2 = b1.allocate_inference_cache(3), b2.allocate_inference_cache(3)
outs = []
with torch.no_grad():
    for _ in range(2):
        tok, res = torch.randn(3, 64, device="cuda").bfloat16(), torch.randn(3, 1, 64, device="cuda")
        outs += [*b1.step(tok[:, None], res, *c1), b1.mixer_step(tok, c1), b2.mixer_step(tok, c2)]
torch.save([t.float().cpu() for t in (*outs, *c1, *c2[0], c2[1])], sys.argv[1])
"""


def test_steps_run_when_the_one_launch_kernel_cannot(tmp_path):
    """The library's decode entry points are replaced by ones that answer "unsupported"; the step goes through the separate calls."""
    import os
    import subprocess
    import sys
    from pathlib import Path

    from tests.gpu_util import close

    (tmp_path / "refuse.c").write_text('#include <stdio.h>\nint ssm_mamba1_decode(void* a, void* s) { fputs("refused1\\n", stderr); return -5; }\n'
                                       'int ssm_mamba2_decode(void* a, void* s) { fputs("refused2\\n", stderr); return -5; }\n')
    (tmp_path / "step.py").write_text(_REFUSED_STEP)
    subprocess.run(["gcc", "-shared", "-fPIC", str(tmp_path / "refuse.c"), "-o", str(tmp_path / "refuse.so")], check=True)
    root = str(Path(__file__).resolve().parent.parent)
    got = {}
    for name, preload in (("one", ""), ("separate", str(tmp_path / "refuse.so"))):
        env = dict(os.environ, PYTHONPATH=root, **({"LD_PRELOAD": preload} if preload else {}))
        r = subprocess.run([sys.executable, str(tmp_path / "step.py"), str(tmp_path / name)], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got[name] = torch.load(tmp_path / name)
        assert r.stderr.count("refused1") == (4 if preload else 0) and r.stderr.count("refused2") == (2 if preload else 0)
    for i, (a, b) in enumerate(zip(got["one"], got["separate"])):
        close(a, b, rtol=2e-2, atol=2e-2, what=str(i))


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, t):
        return t.clone()

    @staticmethod
    def backward(ctx, g):
        return None


@pytest.mark.parametrize("op", ["scan", "chunk", "conv", "norm", "ssd"])
def test_a_node_that_returns_no_gradient_is_zero_upstream(op):
    from ssm_b200 import ops

    mk = lambda *s: torch.randn(*s, device="cuda", requires_grad=True)  # noqa: E731
    A = -torch.rand(8, 16, device="cuda")
    if op == "scan":
        x = mk(1, 8, 40)
        y = ops.selective_scan(x, mk(1, 8, 40), A, mk(1, 1, 16, 40), mk(1, 1, 16, 40))
    elif op == "chunk":
        x = mk(1, 40, 2, 8)
        y = ops.ssd_chunk_scan(x, torch.rand(1, 40, 2, device="cuda"), -torch.rand(2, 8, device="cuda"), mk(1, 40, 2, 8), mk(1, 40, 2, 8), 32)
    elif op == "conv":
        x = mk(1, 8, 40)
        y = ops.dw_causal_conv(x, mk(8, 4))
    elif op == "norm":
        x = mk(1, 3, 64)
        y = ops.fused_layer_norm(x, mk(64), None)
    else:
        x = torch.randn(1, 256, 2, 64, device="cuda").bfloat16().requires_grad_()
        B = torch.randn(1, 256, 1, 128, device="cuda").bfloat16()
        y = ops.ssd_scan(x, torch.rand(1, 256, 2, device="cuda").bfloat16(), -torch.ones(2, device="cuda"), B, B, 256)
    _NoGradient.apply(y).sum().backward()
    assert x.grad is None or not x.grad.any()
