"""Packed sequences whose boundaries lie on the device (a table formed there, with room to spare) against the same boundaries on the host:
empty sequences, chunks that end with a sequence, more sequences than the table's kernel has threads; boundaries that are none."""

from __future__ import annotations

import pytest
import torch

from ssm_b200 import ops

pytestmark = pytest.mark.gpu


def _inputs(nl, nh, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    return r(1, nl, nh, 64), torch.rand(1, nl, nh, generator=g, device="cuda").bfloat16(), -torch.rand(nh, device="cuda"), r(1, nl, 1, 128) / 11, r(1, nl, 1, 128) / 11


def _cuts(nl, n, seed):
    return [0, *sorted(torch.randint(0, nl + 1, (n - 1,), generator=torch.Generator().manual_seed(seed)).tolist()), nl]


@pytest.mark.parametrize("nl,nh,cu,dtype", [(1, 2, [0, 1], torch.int32), (600, 2, [0, 0, 256, 256, 512, 600, 600], torch.int64), (1000, 4, [0, 255, 511, 512, 999, 1000], torch.int32),
                                            (3000, 2, _cuts(3000, 1500, 1), torch.int32), (4096, 3, _cuts(4096, 1024, 2), torch.int64), (2048, 4, [0, 2048], torch.int16),
                                            (5000, 2, [0] * 1100 + [5000], torch.int32), (4096, 8, _cuts(4096, 64, 3), torch.int32)])
def test_boundaries_on_the_device_match_boundaries_on_the_host(nl, nh, cu, dtype):
    X, dt, A, B, C = _inputs(nl, nh, nl)
    run = lambda c: ops.ssd_scan(X, dt, A, B, C, D=A, z=X, dt_softplus=True, cu_seqlens=c, return_final_states=True, return_varlen_states=True)  # noqa: E731
    with torch.no_grad():
        want = run(torch.tensor(cu))
        got = run(torch.tensor(cu, dtype=dtype, device="cuda"))
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    ops.ssd_check_status()


# the kernels run on a table that stays inside the tensors, then the call refuses
@pytest.mark.parametrize("cu", [[0, 300, 200, 600], [0, 600, 0, 600], [0, 300, 601], [5, 600], [0, 599], [-7, 100, 600], [0, 1 << 40, 600], [0, 600, 0, 600, 0, 600, 0, 600]])
def test_what_does_not_rise_from_zero_to_the_end_is_refused(cu):
    X, dt, A, B, C = _inputs(600, 2, 0)
    with torch.no_grad(), pytest.raises(ValueError, match="cu_seqlens must rise from 0 to L"):
        ops.ssd_scan(X, dt, A, B, C, cu_seqlens=torch.tensor(cu, device="cuda"))
    torch.cuda.synchronize()
    with torch.no_grad():
        assert ops.ssd_scan(X, dt, A, B, C, cu_seqlens=torch.tensor([0, 600], device="cuda")).isfinite().all()


# padding to a fixed number of sequences: empty ones behind the last
@pytest.mark.parametrize("entries", [64, 1024])
def test_padded_boundaries_on_the_device_take_little_more_than_on_the_host(entries):
    nl, nh = 4096, 16
    X, dt, A, B, C = _inputs(nl, nh, 1)
    cu = torch.tensor([0, 1000] + [nl] * (entries - 1), dtype=torch.int32)

    def peak(c):
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        with torch.no_grad():
            out = ops.ssd_scan(X, dt, A, B, C, dt_softplus=True, cu_seqlens=c, return_varlen_states=True)
        return torch.cuda.max_memory_allocated() - before, out

    (host, want), (device, got) = peak(cu), peak(cu.cuda())
    assert device <= host + 64 * nh * 19 * 1024
    for a, b in zip(got, want):
        assert torch.equal(a, b)
