"""Blocks of the per-node kernels take runs of nodes across rows and planes.

The division that finds a node's row and plane, on the host; then two fused
and two subroutine steps at row lengths around a warp's and a block's, against
the oracle (1e-12, FP32 1e-5, as the other parity tests).
"""

import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import relerr
from test_gpu_parity import TOL32, TOL64, make_pair

from multiphase_flow_codes_gb300 import _capi as capi

ROOT = Path(__file__).resolve().parents[1]


def test_division_on_the_host(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc"
                                    if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "node_map_check"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2",
                    "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "multiphase_flow_codes_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "node_map_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout
    divisors, bad = map(int, out.split())
    assert divisors > 2000 and bad == 0


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.LBM_PREC_F64, capi.LBM_PREC_F32])
@pytest.mark.parametrize("preset", [capi.LBM_PRESET_BOX, capi.LBM_PRESET_CHANNEL])
@pytest.mark.parametrize("shape", [(9, 6, 7), (31, 6, 9), (33, 8, 6), (130, 7, 6), (127, 6, 8),
                                   (128, 6, 7)])
def test_row_lengths(require_gpu, oracle_mod, precision, preset, shape):
    o, box = make_pair(oracle_mod, preset=preset, shape=shape, k0=2.0, precision=precision)
    tol = TOL64 if precision == capi.LBM_PREC_F64 else TOL32
    o.step(2)
    box.step(2)
    assert relerr(box.get_f(), o.f) <= tol
    o.step(2)
    box.step_unfused(2)
    assert relerr(box.get_f(), o.f) <= tol
