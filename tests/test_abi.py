"""CPU-side checks of the C-ABI boundary: the library loads, exports every function the
header declares, and the ctypes mirrors have the C structs' sizes.  No kernel is launched."""

from __future__ import annotations

import ctypes
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HEADER = ROOT / "include" / "ssm_b200.h"


def _declared_functions() -> list[str]:
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(ssm_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from ssm_b200 import _lib

    lib = _lib.load()
    names = _declared_functions()
    assert len(names) >= 15
    for name in names:
        assert hasattr(lib, name), f"{name} is declared in the header but not exported"
        assert name in _lib.ENTRY_POINTS, f"{name} has no ctypes prototype"
    assert lib.ssm_b200_abi_version() == 4
    assert lib.ssm_scan_checkpoint_interval() == 32


def test_ctypes_structs_match_c_layout(tmp_path):
    from ssm_b200 import _lib

    pairs = {
        "ssm_scan_fwd_args": _lib.ScanFwdArgs, "ssm_scan_bwd_args": _lib.ScanBwdArgs,
        "ssm_step_args": _lib.StepArgs, "ssm_step_bwd_args": _lib.StepBwdArgs,
        "ssm_bcast4": _lib.Bcast4, "ssm_chunk_args": _lib.ChunkArgs, "ssm_chunk_bwd_args": _lib.ChunkBwdArgs,
        "ssm_conv_args": _lib.ConvArgs, "ssm_conv_bwd_args": _lib.ConvBwdArgs, "ssm_conv_update_args": _lib.ConvUpdateArgs,
        "ssm_norm_args": _lib.NormArgs, "ssm_norm_bwd_args": _lib.NormBwdArgs, "ssm_ssd_args": _lib.SsdArgs,
    }
    src = tmp_path / "sizes.c"
    body = "".join(f'  printf("{n} %zu\\n", sizeof({n}));\n' for n in pairs)
    src.write_text(f'#include <stdio.h>\n#include "{HEADER}"\nint main(void) {{\n{body}  return 0;\n}}\n')
    exe = tmp_path / "sizes"
    subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    for line in out.splitlines():
        name, size = line.split()
        assert ctypes.sizeof(pairs[name]) == int(size), name


def test_null_and_bad_arguments_are_rejected_without_a_gpu():
    from ssm_b200 import _lib

    lib = _lib.load()
    assert lib.ssm_selective_scan_fwd(None, None) == -1
    assert b"NULL" in lib.ssm_b200_last_error()
    a = _lib.ConvArgs()
    a.batch, a.channels, a.len, a.width = 1, 1, 1, 9
    assert lib.ssm_dw_causal_conv_fwd(ctypes.byref(a), None) == -5
    n = _lib.NormArgs()
    n.rows, n.hidden, n.io_dtype = 1, 8, 7
    assert lib.ssm_fused_add_norm_fwd(ctypes.byref(n), None) == -3
    assert lib.ssm_norm_bwd_scratch_floats(10, 768) == 2 * 768 * 592
    assert lib.ssm_chunk_scan_scratch_floats(2, 100, 3, 4, 32) == 2 * 2 * 4 * 12


def test_operators_refuse_cpu_tensors():
    import torch

    from ssm_b200 import ops

    x = torch.zeros(1, 2, 8)
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        ops.dw_causal_conv(x, torch.zeros(2, 4))
    with pytest.raises(ValueError):
        ops.dw_causal_conv(torch.zeros(2, 8), torch.zeros(2, 4))


def test_missing_library_is_a_loud_error(monkeypatch, tmp_path):
    from ssm_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "nope.so")
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        _lib.load()


def test_abi_version_stands_for_this_header():
    """The version is what a binding checks, so it has to move with the interface.  When this fails: raise SSM_B200_ABI_VERSION (and
    ABI_VERSION in _lib.py) unless it already is above the last released one, then record the digest printed here."""
    import hashlib

    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    version = int(re.search(r"#define SSM_B200_ABI_VERSION (\d+)", text).group(1))
    # structs, enums and prototypes without comments and spacing
    digest = hashlib.sha256("".join("".join(ln.split()) for ln in text.splitlines() if not ln.lstrip().startswith("#")).encode()).hexdigest()[:16]
    assert (version, digest) == (4, "e96543baf59aa5b9")


def test_fused_chunk_backward_looks_at_every_pointer_it_reads_in_pieces():
    """Host logic only: no pointer is followed."""
    from ssm_b200 import _lib

    lib = _lib.load()

    def fused(**moved):
        g = _lib.ChunkBwdArgs()
        f = g.fwd
        f.batch, f.len, f.heads, f.proj, f.chunk_size, f.io_dtype, f.par_dtype, f.typed_grads = 2, 100, 4, 64, 64, _lib.BF16, _lib.BF16, 7
        at = {k: 1 << 20 for k in ("X", "dt", "A", "Bm", "Cm", "z", "dY", "dX", "dB", "dC", "dz", "scratch", "fwd_scratch")}
        at.update({k: (1 << 20) + v for k, v in moved.items()})
        f.X, f.dt, g.dY, g.dX, g.scratch, g.fwd_scratch = (at[k] for k in ("X", "dt", "dY", "dX", "scratch", "fwd_scratch"))
        for where, name in ((f, "Bm"), (f, "Cm"), (f, "z"), (g, "dB"), (g, "dC"), (g, "dz")):
            p = getattr(where, name)
            p.ptr, p.sb, p.st, p.sh, p.sq = at[name], 100 * 256, 256, 64, 1
        return lib.ssm_chunk_scan_bwd_fused(ctypes.byref(g))

    assert fused() == 1 and fused(fwd_scratch=-(1 << 20)) == 1  # a missing fwd_scratch is formed again
    for name in ("X", "Bm", "Cm", "z", "dY", "dX", "dB", "dC", "dz"):
        assert fused(**{name: 4}) == 0 and fused(**{name: 8}) == 1, name
    for name in ("scratch", "fwd_scratch"):
        assert fused(**{name: 8}) == 0 and fused(**{name: 16}) == 1, name


# the rule for 148 SMs (which it assumes where there is no device): calls that a cut was measured to slow down stay whole, those that
# it speeds up are cut into the counts that were measured best or close to it
@pytest.mark.parametrize("batch,dim,length,nstate,segments", [
    (1, 4096, 512, 16, 1), (1, 4096, 1024, 16, 1), (1, 4480, 8192, 16, 1), (1, 512, 2048, 16, 16), (1, 1024, 3000, 16, 9), (2, 256, 5000, 16, 27), (3, 640, 350, 16, 6),
    (1, 4096, 512, 32, 1), (1, 3200, 4096, 32, 1), (1, 4480, 8192, 24, 1), (2, 1536, 1500, 32, 1), (1, 2048, 1024, 32, 1), (1, 512, 2048, 32, 8), (2, 256, 5000, 24, 9),
    (1, 1024, 3000, 8, 9), (1, 768, 200, 4, 4), (1, 8192, 512, 16, 1), (1, 512, 2048, 33, 1)])
def test_segments_of_a_selective_scan(batch, dim, length, nstate, segments):
    import torch

    from ssm_b200 import _lib

    if torch.cuda.is_available() and torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("stated for 148 SMs")
    assert _lib.load().ssm_scan_split_segments(batch, dim, length, nstate) == segments
