"""The integer collision core's products on the host.

Each moment is one sum of 64-bit products by signed 32-bit halves without the
products of the low words, rounded once: against the exact sum the error is
at most half a unit of the result plus a quarter per product for a shift of
64 (twice and four times that for 63 and 62).  The splitting is exact, and the
factors of the three MRT rate sets fit their scales; a rate of exactly 2 does
not, and the kernel then takes the core with FP64 products.  Built for the
host with nvcc from the header the kernels use; no GPU is needed.
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
    exe = tmp_path_factory.mktemp("split") / "split_products_check"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2",
                    "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "multiphase_flow_codes_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "split_products_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout
    return [ln.split() for ln in out.splitlines() if ln.strip()]


def test_sums_of_products(rows):
    dots = [r[1:] for r in rows if r[0] == "dot"]
    assert len(dots) == 6
    for shift, n, worst in dots:
        assert float(worst) <= 0.5 + 0.25 * int(n) * 2 ** (64 - int(shift)) + 1e-9, (shift, n, worst)


def test_split_is_exact_and_factors_fit(rows):
    split = next(r for r in rows if r[0] == "split")
    assert int(split[1]) == 0 and int(split[2]) > 0
    assert next(r for r in rows if r[0] == "rates")[1:] == ["1", "1", "1", "0"]
