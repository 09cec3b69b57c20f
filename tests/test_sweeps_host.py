"""The two forms of the nearest-image sweeps of beads_links on the host.

sweep_fast decides the shifts of a sweep in fixed point away from their ties;
the list it gives must be that of sweep_events (the reference's FP64
expressions) bit for bit wherever it takes the sweep, for even and odd box
lengths, and it must take nearly all centres inside an even box.  Built for
the host with nvcc from the header the kernels use; no GPU is needed.
"""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_fast_sweeps_equal_the_references(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc"
                                    if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "sweeps_check"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2",
                    "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "multiphase_flow_codes_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "sweeps_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout
    rows = [ln.split() for ln in out.splitlines() if ln.strip()]
    assert len(rows) == 9
    for n, taken, bad, cases in rows:
        assert int(bad) == 0 and int(cases) > 0, (n, bad, cases)
        if int(n) >= 32 and int(n) % 2 == 0:
            assert float(taken) > 0.5, (n, taken)
