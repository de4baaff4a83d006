"""A refused cooperative launch of the one-launch decode step, made by a stand-in for the runtime's entry point: the library says
"unsupported" for a refusal that the separate calls can serve, passes every other error on, and leaves none behind."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
OBJ = ROOT / "ssm_b200" / "lib" / "obj"

PROGRAM = r"""
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include "ssm_b200.h"
static int refusal, pending;
extern "C" cudaError_t __wrap_cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return (cudaError_t)(pending = refusal); }
extern "C" cudaError_t __wrap_cudaGetLastError() { const int e = pending; pending = 0; return (cudaError_t)e; }
int main(int argc, char** argv) {
  refusal = atoi(argv[1]);
  void* p = (void*)4096;
  ssm_mamba1_decode_args a = {};
  a.batch = 1, a.d_model = 64, a.d_inner = 128, a.nstate = 16, a.dt_rank = 4, a.width = 4, a.io_dtype = SSM_BF16;
  a.hidden = a.in_x = a.in_z = a.conv_w = a.x_proj = a.dt_proj = a.out_proj = p, a.dt_bias = a.A = a.D = (float*)p;
  a.conv_state = a.ssm_state = (float*)p, a.out = a.scratch = p;
  ssm_mamba2_decode_args b = {};
  b.batch = 1, b.d_model = 64, b.heads = 2, b.headdim = 64, b.nstate = 128, b.groups = 1, b.width = 4, b.io_dtype = SSM_F16;
  b.hidden = b.in_z = b.in_x = b.in_B = b.in_C = b.in_dt = b.conv_x_w = b.conv_B_w = b.conv_C_w = b.norm_w = b.out_proj = p;
  b.dt_bias = b.A = b.D = (float*)p, b.conv_state_x = b.conv_state_B = b.conv_state_C = b.ssm_state = (float*)p, b.out = b.scratch = p;
  const int ra = ssm_mamba1_decode(&a, 0), la = pending, rb = ssm_mamba2_decode(&b, 0), lb = pending;
  printf("%d %d %d %d\n", ra, la, rb, lb);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists() or not (OBJ / "decode_step.o").exists():
        pytest.skip("needs nvcc and the objects of the library's build")
    d = tmp_path_factory.mktemp("refused")
    (d / "refused.cu").write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", f"-I{ROOT / 'include'}", str(d / "refused.cu"), str(OBJ / "decode_step.o"), str(OBJ / "api.o"),
                    "-Xlinker", "--wrap=cudaLaunchCooperativeKernel", "-Xlinker", "--wrap=cudaGetLastError", "-o", str(d / "refused")], check=True)
    return d / "refused"


# 720 cudaErrorCooperativeLaunchTooLarge, 801 cudaErrorNotSupported; 2 cudaErrorMemoryAllocation, 700 cudaErrorIllegalAddress
@pytest.mark.parametrize("refusal,code", [(720, -5), (801, -5), (2, 2), (700, 700)])
def test_refused_cooperative_launch(program, refusal, code):
    out = subprocess.run([str(program), str(refusal)], check=True, capture_output=True, text=True).stdout.split()
    assert [int(v) for v in out] == [code, 0, code, 0]
