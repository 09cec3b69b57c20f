"""The integer density and momentum sums over FP64's whole range, on the host.

Each population is rounded at 2^-58 of the node's largest and the exact sum
once to FP64, 2^-53 of it: 2^-52 of the sum of the magnitudes in all.  Sums that
could pass FP64's largest value are left to the FP64 form, which gives the
infinity that a diverged run is known by.
"""

import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_moments(tmp_path):
    import pytest
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc"
                                    if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "moments_check"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2",
                    "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "multiphase_flow_codes_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "moments_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout
    rows = [[float(v) for v in ln.split()] for ln in out.splitlines() if ln.strip()]
    assert len(rows) == 12
    for magnitude, states, taken, missed, worst in rows:
        assert missed == 0, magnitude
        assert worst <= 2.0 ** -52, (magnitude, worst)
        if 1e-200 <= magnitude <= 1e300:
            assert taken == states, magnitude
