"""The collision at a node's own scale keeps FP64's precision, forces included.

Against the moment matrix in long double, relative to the node's largest
population.  A node that is taken has its populations within a factor two of
the top of their range 2^-(4 + j), so the largest is at least 2^-(6 + j):
rounding them to 2^-(58 + j) is 2^-53 each, which the collision (absolute row
sums up to 3) carries to 3.3e-16, its moments' roundings add up to 20 units
of 2^-(62 + j), 2.8e-16, and the result is rounded to FP64, 1.1e-16: 8e-16
in all.  Nodes whose force or velocity would cost more take the FP64 form.
A force below twice the largest population does not, nor the velocity that goes
with them: near equilibrium six times the largest population, and half the
force.  Built for
the host with nvcc from the header the kernels use; no GPU is needed.
"""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc"
                                    if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path_factory.mktemp("scale") / "node_scale_check"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2",
                    "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "multiphase_flow_codes_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "node_scale_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout
    return [[float(v) for v in ln.split()] for ln in out.splitlines() if ln.strip()]


def test_precision_at_every_force(rows):
    assert len(rows) == 3 * 7 * 9
    for mrt, u, force, states, declined, ordinary, ordinary_declined, worst in rows:
        assert worst <= 8e-16, (mrt, u, force, worst)


def test_ordinary_nodes_are_taken(rows):
    assert sum(r[5] for r in rows) > 30000
    for mrt, u, force, states, declined, ordinary, ordinary_declined, worst in rows:
        assert ordinary_declined == 0, (mrt, u, force, ordinary_declined)
