"""Roundings of the integer collision core, one step against long double.

Each population is rounded to its storage 2^-58 from 2^-61, ties up: a mean
error of 1/16 unit.  Nothing before that may add to it: a mean error has one
sign, so it adds up as mass.  Built for the host with nvcc from the header the
kernels use; no GPU is needed.
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
    exe = tmp_path_factory.mktemp("core") / "core_rounding_check"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2",
                    "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "multiphase_flow_codes_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "core_rounding_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout
    return [ln.split() for ln in out.splitlines() if ln.strip()]


def step_rows(rows):
    steps = [[float(v) for v in r] for r in rows if r[0] != "mass"]
    assert len(steps) == 15
    return steps


def test_mean_error_is_the_last_roundings(rows):
    for mrt, visc, int_ok, states, declined, mean, rms, xy in step_rows(rows):
        if int_ok:
            # (20000 states of 19 populations: the mean of their errors of 0.4
            # units is known to 0.001)
            assert abs(mean) <= 1 / 16 + 0.003, (mrt, visc, mean)


def test_stress_error_is_the_populations_roundings(rows):
    """The stress c_x c_y f sums four populations' roundings to the storage, 0.577
    units, and its moment's own at 1/8 unit, entering fourfold: a rounding and
    three products without their low words, 0.32 units rms, 0.16; 0.6 in all."""
    for mrt, visc, int_ok, states, declined, mean, rms, xy in step_rows(rows):
        if int_ok:
            # (rms of 20000 states: to 0.5 %)
            assert xy <= 0.62, (mrt, visc, xy)


def test_rates_near_two_keep_the_integer_core(rows):
    """Every rate set down to viscosities of 1e-8 (rates within 1e-7 of 2) has
    factors that fit their scales, and near-equilibrium nodes are taken with the
    error of the core: a rounding to the storage, 0.29 units, and the moments'
    roundings at 1/8 unit, less than 0.3 in all."""
    for mrt, visc, int_ok, states, declined, mean, rms, xy in step_rows(rows):
        assert int_ok == 1, (mrt, visc)
        assert declined == 0, (mrt, visc)
        assert rms <= (0.29 ** 2 + 0.3 ** 2) ** 0.5, (mrt, visc, rms)


def test_no_mass_at_a_nodes_own_scale(rows):
    """Populations are rounded to the node's scale and its results to FP64, ties
    to even: no mean error beyond five standard errors of 20000 states whose
    mass error is 2e-16 (19 + 19 roundings of at most 2^-54)."""
    mass = [r[1:] for r in rows if r[0] == "mass"]
    assert len(mass) == 9
    for mrt, u, states, mean in mass:
        assert int(states) > 19000
        assert abs(float(mean)) <= 5 * 2e-16 / 20000 ** 0.5, (mrt, u, mean)
