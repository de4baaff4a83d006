"""Performance cases: the work that users of this package have it do, through its public entry points.

``listed()`` names a dozen passes over the range of sizes, directions and data types the package is used for: decoding
one token for one or for many sequences, prefill of a single prompt and of packed prompts, forward and backward of the
operators and of a whole block.  ``draw()`` gives further cases of the same ranges.  ``prepare()`` builds what a program
has in hand before the call (inputs from the seed, module weights, decode caches), ``run()`` makes one pass and returns
everything that it computes, ``work()`` states the bytes and operations that the pass cannot do without, and
``tolerance()`` how far another correct implementation of the same precision may be off.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from ssm_b200 import ops
from ssm_b200.mixer import Mamba1Block, Mamba2Block

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
HEADDIM, D_STATE2 = 64, 128  # Mamba-2: head width and state width
D_STATE1, D_CONV = 16, 4     # Mamba-1 state width; conv width of both


def listed():
    return [
        # decoding: one user at a small model (launches and host work), then a served batch at the width of a large one
        {"name": "mamba1_step_batch1", "kind": "mamba1_step", "batch": 1, "d_model": 768, "dtype": "bf16"},
        {"name": "mamba1_step_batch256", "kind": "mamba1_step", "batch": 256, "d_model": 2560, "dtype": "bf16"},
        {"name": "mamba2_step_batch256", "kind": "mamba2_step", "batch": 256, "d_model": 2560, "dtype": "bf16"},
        # the selective scan of one short fp32 prompt: few rows, a long chain
        {"name": "scan_prefill_f32", "kind": "scan_prefill", "batch": 1, "dim": 512, "len": 2048, "dtype": "f32"},
        # a Mamba-1 block in training
        {"name": "mamba1_block_train", "kind": "mamba1_block_train", "batch": 8, "len": 4096, "d_model": 768, "dtype": "bf16"},
        # the state-space-dual scan: prefill of full batches, training on a ragged length, and prompts packed end to end
        {"name": "ssd_prefill", "kind": "ssd_prefill", "batch": 8, "len": 8192, "heads": 48, "groups": 1, "dtype": "bf16"},
        {"name": "ssd_train_ragged", "kind": "ssd_train", "batch": 2, "len": 4001, "heads": 48, "groups": 1, "dtype": "bf16"},
        {"name": "ssd_packed_prompts", "kind": "ssd_packed", "sequences": 24, "len": 16384, "heads": 48, "groups": 1, "dtype": "bf16"},
        # one Mamba-2 block of a long prefill
        {"name": "mamba2_block_prefill", "kind": "mamba2_block_prefill", "batch": 2, "len": 16384, "d_model": 2560, "dtype": "bf16"},
        # the element-wise chunked recurrence, the convolution and the norm on their own, in training
        {"name": "chunk_scan_train", "kind": "chunk_scan_train", "batch": 8, "len": 2048, "heads": 16, "chunk": 128, "gate": True, "dtype": "bf16"},
        {"name": "conv_train_channels_last", "kind": "conv_train", "batch": 4, "len": 4093, "channels": 2560, "first": False, "dtype": "bf16"},
        {"name": "add_layer_norm_train", "kind": "norm_train", "batch": 8, "len": 2047, "hidden": 1600, "rms": False, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer of [lo, hi], a multiple of `step`, spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["mamba1_step", "mamba2_step", "scan_prefill", "mamba1_block_train", "ssd_prefill", "ssd_train", "ssd_packed",
                       "mamba2_block_prefill", "chunk_scan_train", "conv_train", "norm_train"])
    half = rng.choice(["bf16", "bf16", "f16"])
    anyt = rng.choice(["bf16", "f16", "f32"])
    if kind == "mamba1_step":
        return {"kind": kind, "batch": _log_int(rng, 1, 256), "d_model": _log_int(rng, 256, 2560, 64), "dtype": half}
    if kind == "mamba2_step":
        return {"kind": kind, "batch": _log_int(rng, 1, 256), "d_model": _log_int(rng, 256, 2560, 64), "dtype": half}
    if kind == "scan_prefill":
        dim = _log_int(rng, 256, 5120, 64)
        length = _log_int(rng, 64, 8192)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, min(8, (1 << 24) // (dim * length)))), "dim": dim, "len": length, "dtype": anyt}
    if kind == "mamba1_block_train":
        length = _log_int(rng, 256, 4096)
        return {"kind": kind, "batch": _log_int(rng, 1, 8), "len": length, "d_model": _log_int(rng, 256, 768, 64), "dtype": "bf16"}
    if kind in ("ssd_prefill", "ssd_train"):
        top = 8192 * 48 * 8 if kind == "ssd_prefill" else 4001 * 48 * 2  # heads x tokens
        heads = _log_int(rng, 8, 80, 4)
        length = _log_int(rng, 128, 16384 if kind == "ssd_prefill" else 4096)
        batch = _log_int(rng, 1, max(1, min(8, top // (heads * length))))
        return {"kind": kind, "batch": batch, "len": length, "heads": heads, "groups": rng.choice([1, 1, 2, 4]), "dtype": half}
    if kind == "ssd_packed":
        return {"kind": kind, "sequences": _log_int(rng, 2, 64), "len": _log_int(rng, 512, 16384), "heads": _log_int(rng, 8, 48, 4), "groups": 1, "dtype": half}
    if kind == "mamba2_block_prefill":
        return {"kind": kind, "batch": _log_int(rng, 1, 2), "len": _log_int(rng, 128, 16384), "d_model": _log_int(rng, 256, 2560, 64), "dtype": half}
    if kind == "chunk_scan_train":
        heads = _log_int(rng, 4, 32, 2)
        length = _log_int(rng, 128, 4096)
        batch = _log_int(rng, 1, max(1, min(8, (1 << 18) // (heads * length))))
        return {"kind": kind, "batch": batch, "len": length, "heads": heads, "chunk": rng.choice([64, 128, 256]), "gate": rng.random() < 0.7, "dtype": anyt}
    if kind == "conv_train":
        channels = _log_int(rng, 128, 5120, 16)
        length = _log_int(rng, 128, 8192)
        batch = _log_int(rng, 1, max(1, min(8, 41_900_000 // (channels * length))))
        return {"kind": kind, "batch": batch, "len": length, "channels": channels, "first": rng.random() < 0.5, "dtype": anyt}
    hidden = _log_int(rng, 256, 8192, 8)
    length = _log_int(rng, 32, 4096)
    batch = _log_int(rng, 1, max(1, min(8, 26_200_000 // (hidden * length))))
    return {"kind": "norm_train", "batch": batch, "len": length, "hidden": hidden, "rms": rng.random() < 0.5, "dtype": anyt}


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------


class _Draws:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, dtype=torch.float32, std=1.0, mean=0.0):
        t = torch.randn(*shape, generator=self.g, device="cuda")
        return t.mul_(std).add_(mean).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=self.g, device="cuda").mul_(hi - lo).add_(lo)


def _ssd_inputs(r, nb, nl, nh, ng, dt):
    """x and z of unit variance, steps softplus(N(-3, 1)), decays in [1, 16], B and C of unit length: what the projections and
    convolutions of a Mamba-2 layer hand to the scan."""
    return {
        "X": r.normal(nb, nl, nh, HEADDIM, dtype=dt), "dt": r.normal(nb, nl, nh, dtype=dt), "A": -torch.exp(r.uniform(nh, hi=math.log(16.0))),
        "B": r.normal(nb, nl, ng, D_STATE2, dtype=dt, std=D_STATE2 ** -0.5), "C": r.normal(nb, nl, ng, D_STATE2, dtype=dt, std=D_STATE2 ** -0.5),
        "D": r.normal(nh), "z": r.normal(nb, nl, nh, HEADDIM, dtype=dt), "dt_bias": r.normal(nh, std=0.3, mean=-3.0),
    }


def prepare(case, seed):
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    r = _Draws(seed)
    if kind in ("mamba1_step", "mamba2_step"):
        torch.manual_seed(seed)  # the modules draw their weights from torch's own generator
        nb, dm = case["batch"], case["d_model"]
        if kind == "mamba1_step":
            block = Mamba1Block(dm, d_state=D_STATE1, d_conv=D_CONV, device="cuda", dtype=dt)
            conv, ssm = block.allocate_inference_cache(nb)
            conv.copy_(r.normal(*conv.shape, std=0.1)), ssm.copy_(r.normal(*ssm.shape, std=0.1))
            return {"kind": kind, "block": block, "hidden": r.normal(nb, 1, dm, dtype=dt), "residual": r.normal(nb, 1, dm), "conv": conv, "ssm": ssm}
        block = Mamba2Block(dm, d_state=D_STATE2, headdim=HEADDIM, d_conv=D_CONV, device="cuda", dtype=dt)
        convs, ssm = block.allocate_inference_cache(nb)
        for t in (*convs, ssm):
            t.copy_(r.normal(*t.shape, std=0.1))
        return {"kind": kind, "block": block, "tok": r.normal(nb, dm, dtype=dt), "cache": (convs, ssm)}
    if kind == "scan_prefill":
        nb, nd, nl, n = case["batch"], case["dim"], case["len"], D_STATE1
        return {"kind": kind, "u": r.normal(nb, nd, nl, dtype=dt), "delta": F.softplus(r.normal(nb, nd, nl, mean=-2.0)).to(dt),
                "A": -torch.exp(r.normal(nd, n, std=0.5)), "B": r.normal(nb, 1, n, nl, dtype=dt), "C": r.normal(nb, 1, n, nl, dtype=dt),
                "D": r.normal(nd), "z": r.normal(nb, nd, nl, dtype=dt)}
    if kind == "mamba1_block_train":
        torch.manual_seed(seed)
        nb, nl, dm = case["batch"], case["len"], case["d_model"]
        block = Mamba1Block(dm, d_state=D_STATE1, d_conv=D_CONV, device="cuda", dtype=dt)
        return {"kind": kind, "block": block, "hidden": r.normal(nb, nl, dm, dtype=dt).requires_grad_(), "residual": r.normal(nb, nl, dm).requires_grad_(),
                "g_out": r.normal(nb, nl, dm, dtype=dt), "g_res": r.normal(nb, nl, dm)}
    if kind == "mamba2_block_prefill":
        torch.manual_seed(seed)
        nb, nl, dm = case["batch"], case["len"], case["d_model"]
        block = Mamba2Block(dm, d_state=D_STATE2, headdim=HEADDIM, d_conv=D_CONV, device="cuda", dtype=dt)
        return {"kind": kind, "block": block, "hidden": r.normal(nb, nl, dm, dtype=dt), "residual": r.normal(nb, nl, dm)}
    if kind == "ssd_prefill":
        return {"kind": kind, **_ssd_inputs(r, case["batch"], case["len"], case["heads"], case["groups"], dt)}
    if kind == "ssd_train":
        t = {k: v.requires_grad_() for k, v in _ssd_inputs(r, case["batch"], case["len"], case["heads"], case["groups"], dt).items()}
        return {"kind": kind, "inputs": t, "g_out": r.normal(case["batch"], case["len"], case["heads"], HEADDIM, dtype=dt)}
    if kind == "ssd_packed":
        cuts = torch.randperm(case["len"] - 1, generator=torch.Generator().manual_seed(seed))[: case["sequences"] - 1] + 1
        cu = torch.cat([torch.zeros(1, dtype=torch.long), cuts.sort().values, torch.tensor([case["len"]])]).to(torch.int32)
        return {"kind": kind, "cu_seqlens": cu.cuda(), **_ssd_inputs(r, 1, case["len"], case["heads"], case["groups"], dt)}
    if kind == "chunk_scan_train":
        nb, nl, nh, p = case["batch"], case["len"], case["heads"], HEADDIM
        t = {"X": r.normal(nb, nl, nh, p, dtype=dt), "dt": F.softplus(r.normal(nb, nl, nh, mean=-2.0)).to(dt), "A": -torch.exp(r.normal(nh, p, std=0.5)),
             "B": r.normal(nb, nl, nh, p, dtype=dt), "C": r.normal(nb, nl, nh, p, dtype=dt), "D": r.normal(nh, p)}
        if case["gate"]:
            t["z"] = r.normal(nb, nl, nh, p, dtype=dt)
        return {"kind": kind, "inputs": {k: v.requires_grad_() for k, v in t.items()}, "chunk": case["chunk"], "g_out": r.normal(nb, nl, nh, p, dtype=dt)}
    if kind == "conv_train":
        nb, nl, nc = case["batch"], case["len"], case["channels"]
        shape = (nb, nc, nl) if case["first"] else (nb, nl, nc)
        t = {"x": r.normal(*shape, dtype=dt), "weight": r.uniform(nc, D_CONV, lo=-0.5, hi=0.5).to(dt), "bias": r.normal(nc, dtype=dt, std=0.1)}
        return {"kind": kind, "inputs": {k: v.requires_grad_() for k, v in t.items()}, "g_out": r.normal(*shape, dtype=dt)}
    assert kind == "norm_train"
    nb, nl, nd = case["batch"], case["len"], case["hidden"]
    t = {"x": r.normal(nb, nl, nd, dtype=dt), "weight": r.normal(nd, dtype=dt, std=0.1, mean=1.0)}
    if not case["rms"]:
        t["bias"] = r.normal(nd, dtype=dt, std=0.1)
    t["residual"] = r.normal(nb, nl, nd)
    return {"kind": kind, "inputs": {k: v.requires_grad_() for k, v in t.items()}, "rms": case["rms"], "g_out": r.normal(nb, nl, nd, dtype=dt),
            "g_res": r.normal(nb, nl, nd)}


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind == "mamba1_step":  # one token of a pre-allocated decode cache; the states are updated in place
        with torch.no_grad():
            out, res = s["block"].step(s["hidden"], s["residual"], s["conv"], s["ssm"])
        return out, res, s["conv"], s["ssm"]
    if kind == "mamba2_step":
        with torch.no_grad():
            out = s["block"].mixer_step(s["tok"], s["cache"])
        return out, s["cache"]
    if kind == "scan_prefill":
        with torch.no_grad():
            return ops.selective_scan(s["u"], s["delta"], s["A"], s["B"], s["C"], D=s["D"], z=s["z"], return_last_state=True)
    if kind == "mamba1_block_train":
        out, res = s["block"](s["hidden"], s["residual"])
        return out, res, torch.autograd.grad((out, res), [s["hidden"], s["residual"], *s["block"].parameters()], (s["g_out"], s["g_res"]))
    if kind == "mamba2_block_prefill":
        with torch.no_grad():
            return s["block"](s["hidden"], s["residual"])
    if kind == "ssd_prefill":
        with torch.no_grad():
            return ops.ssd_scan(s["X"], s["dt"], s["A"], s["B"], s["C"], D=s["D"], z=s["z"], dt_bias=s["dt_bias"], dt_softplus=True, return_final_states=True)
    if kind == "ssd_packed":
        with torch.no_grad():
            return ops.ssd_scan(s["X"], s["dt"], s["A"], s["B"], s["C"], D=s["D"], z=s["z"], dt_bias=s["dt_bias"], dt_softplus=True,
                                cu_seqlens=s["cu_seqlens"], return_varlen_states=True)
    t = s["inputs"]
    if kind == "ssd_train":
        out = ops.ssd_scan(t["X"], t["dt"], t["A"], t["B"], t["C"], D=t["D"], z=t["z"], dt_bias=t["dt_bias"], dt_softplus=True)
        return out, torch.autograd.grad(out, list(t.values()), s["g_out"])
    if kind == "chunk_scan_train":
        out = ops.ssd_chunk_scan(t["X"], t["dt"], t["A"], t["B"], t["C"], s["chunk"], D=t["D"], z=t.get("z"))
        return out, torch.autograd.grad(out, list(t.values()), s["g_out"])
    if kind == "conv_train":
        out = ops.dw_causal_conv(t["x"], t["weight"], t["bias"], "silu")
        return out, torch.autograd.grad(out, list(t.values()), s["g_out"])
    out, res = ops.fused_layer_norm(t["x"], t["weight"], t.get("bias"), residual=t["residual"], is_rms=s["rms"], return_residual=True)
    return out, res, torch.autograd.grad((out, res), list(t.values()), (s["g_out"], s["g_res"]))


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------


def _ssd_work(tokens, heads, groups, states, io):
    """Forward: x, z, y, dt, B, C and the final states; the recurrence itself is 3 N P multiply-adds' worth per token and head."""
    rows = tokens * heads * HEADDIM
    by = 3 * rows * io + tokens * heads * io + 2 * tokens * groups * D_STATE2 * io + states * heads * HEADDIM * D_STATE2 * 4
    return by, 5 * rows * D_STATE2


def work(case):
    kind, io = case["kind"], 4 if case["dtype"] == "f32" else 2
    if kind in ("mamba1_step", "mamba2_step", "mamba1_block_train", "mamba2_block_prefill"):
        dm = case["d_model"]
        di, rank = 2 * dm, math.ceil(dm / 16)
        if kind.startswith("mamba1"):
            gemm = 2 * di * dm + (rank + 2 * D_STATE1) * di + di * rank + dm * di
        else:
            heads = di // HEADDIM
            gemm = (2 * di + 2 * D_STATE2 + heads) * dm + dm * di
    if kind == "mamba1_step":
        nb = case["batch"]
        by = gemm * io + nb * (2 * di * (D_STATE1 + D_CONV) * 4 + dm * (2 * io + 8)) + di * (D_STATE1 + 2) * 4 + di * (D_CONV + 1) * io
        return {"bytes": by, "flops": nb * (2 * gemm + di * (6 * D_STATE1 + 2 * D_CONV))}
    if kind == "mamba2_step":
        nb = case["batch"]
        by = gemm * io + nb * (2 * di * D_STATE2 * 4 + 2 * (di + 2 * D_STATE2) * D_CONV * 4 + 2 * dm * io)
        return {"bytes": by, "flops": nb * (2 * gemm + 6 * di * D_STATE2)}
    if kind == "scan_prefill":
        nb, nd, nl = case["batch"], case["dim"], case["len"]
        return {"bytes": 4 * nb * nd * nl * io + 2 * nb * D_STATE1 * nl * io + nb * nd * D_STATE1 * io + nd * (D_STATE1 + 1) * 4,
                "flops": nb * nd * nl * (6 * D_STATE1 + 8)}
    if kind == "mamba1_block_train":  # hidden and the fp32 residual in, both outputs, both gradients in and out, weights and their gradients
        tok = case["batch"] * case["len"]
        return {"bytes": tok * dm * (4 * io + 16) + 2 * gemm * io, "flops": tok * (6 * gemm + di * 18 * D_STATE1)}
    if kind == "mamba2_block_prefill":
        tok = case["batch"] * case["len"]
        return {"bytes": tok * dm * (2 * io + 8) + gemm * io, "flops": tok * (2 * gemm + 5 * di * D_STATE2)}
    if kind in ("ssd_prefill", "ssd_packed", "ssd_train"):
        tok = case["len"] * case.get("batch", 1)
        by, fl = _ssd_work(tok, case["heads"], case["groups"], case.get("sequences", case.get("batch", 1)), io)
        if kind == "ssd_train":  # also the gradient of y, and the gradients of x, z, dt, B and C
            by += 3 * tok * case["heads"] * HEADDIM * io + tok * case["heads"] * io + 2 * tok * case["groups"] * D_STATE2 * io
            by -= case["batch"] * case["heads"] * HEADDIM * D_STATE2 * 4
            fl *= 3
        return {"bytes": by, "flops": fl}
    if kind == "chunk_scan_train":  # X, B, C (z), dY in, Y, dX, dB, dC (dz) out; dt and ddt
        tok = case["batch"] * case["len"] * case["heads"]
        return {"bytes": tok * HEADDIM * io * (10 if case["gate"] else 8) + 2 * tok * io, "flops": tok * HEADDIM * 30}
    if kind == "conv_train":  # x, dy in, y, dx out
        n = case["batch"] * case["len"] * case["channels"]
        return {"bytes": 4 * n * io, "flops": n * (6 * D_CONV + 10)}
    n = case["batch"] * case["len"] * case["hidden"]  # x, dy in, y, dx out; the fp32 residual, its sum and their two gradients
    return {"bytes": n * (4 * io + 16), "flops": n * 20}


def tolerance(case):
    kind, dt = case["kind"], case["dtype"]
    if kind in ("scan_prefill", "chunk_scan_train", "conv_train", "norm_train"):  # fp32 arithmetic; 16-bit results are rounded once
        return {"rel": 2e-5, "max": 1e-3} if dt == "f32" else {"rel": 5e-3, "max": 2e-2}
    if kind in ("ssd_prefill", "ssd_packed"):  # products of 16-bit operands, fp32 sums
        return {"rel": 1e-2, "max": 0.2}
    if kind == "mamba1_step":  # the step itself is fp32, its inputs pass through 16-bit projections
        return {"rel": 1e-2, "max": 0.1}
    if kind == "ssd_train":  # the gradients of A and of dt_bias sum signed terms that largely cancel: 16-bit operands leave 1e-2 to 2e-2 of them
        return {"rel": 3e-2, "max": 0.9}
    return {"rel": 2e-2, "max": 0.5}  # chains of 16-bit operands, and gradients that are sums of cancelling terms
