"""The pre-relaxation's passes where they end and over the forms they take.

Passes are enqueued sixteen at a time; with eps = 0 the last one is max_iter + 2:
14 and 30 end on the last pass of a chunk, 15 begins a chunk with the last density
update alone.  Rows of whole blocks (nx = 128), solid nodes, every arithmetic
mode and rates whose factors fit no integer scale, against the oracle's loop.
"""

import numpy as np
import pytest

from conftest import relerr
from test_gpu_parity import TOL64
from test_prerelax import oracle_prerelax

from multiphase_flow_codes_gb300 import _capi as capi
from multiphase_flow_codes_gb300 import inputs

pytestmark = pytest.mark.gpu


def pair(oracle_mod, shape, npart=0, visc=0.0036, preset=capi.LBM_PRESET_BOX, urms=0.03):
    from multiphase_flow_codes_gb300.engine import LBMBox
    nx, ny, nz = shape
    cfg = capi.config_init(preset, nx, ny, nz, npart, 3.0, 1.0)
    cfg.forcing = capi.LBM_FORCING_NONE
    cfg.visc = visc
    u = inputs.spectral_velocity(nx, 4.0, urms, ny=ny, nz=nz, seed=31)
    o = oracle_mod.OracleBox(cfg)
    box = LBMBox(cfg)
    for b in (o, box):
        b.initpop(*u)
        b.macrovar()
    if npart:
        y = inputs.initpartpos(nx, ny, nz, npart, 3.0, seed=4,
                               channel=preset == capi.LBM_PRESET_CHANNEL)
        o.release_particles(y, np.zeros((npart, 3)))
        box.release_particles(y, np.zeros((npart, 3)))
    for b in (o, box):
        b.rhoupdat()
    return o, box


def check(o, box, max_iter):
    it_o, err_o = oracle_prerelax(o, 0.0, max_iter)
    it_g, err_g = box.prerelax(0.0, max_iter)
    assert it_g == it_o
    assert abs(err_g - err_o) <= 1e-12 * float(np.abs(np.asarray(o.rho)).max())
    assert relerr(box.get_f(), o.f) <= TOL64
    assert relerr(box.get_macro()[0], o.rho) <= TOL64


@pytest.mark.parametrize("max_iter", [0, 13, 14, 15, 30])
def test_ends_of_chunks(require_gpu, oracle_mod, max_iter):
    check(*pair(oracle_mod, (36, 20, 28)), max_iter)


@pytest.mark.parametrize("preset", [capi.LBM_PRESET_BOX, capi.LBM_PRESET_CHANNEL])
@pytest.mark.parametrize("shape,npart", [((128, 12, 10), 0), ((128, 20, 18), 2), ((40, 24, 28), 2)])
def test_whole_rows_and_solid_nodes(require_gpu, oracle_mod, preset, shape, npart):
    o, box = pair(oracle_mod, shape, npart, preset=preset)
    if npart:
        assert (box.get_flags()[1] >= 0).any()
    check(o, box, 5)


@pytest.mark.parametrize("mode", [capi.LBM_SUMS_FLOAT, capi.LBM_SUMS_FIXED, capi.LBM_SUMS_INTEGER])
def test_modes(require_gpu, oracle_mod, mode):
    o, box = pair(oracle_mod, (36, 20, 28), 1)
    box.set_sums(mode)
    check(o, box, 7)


@pytest.mark.parametrize("visc", [1e-4, 1e-8, 1e-13])
def test_rates_near_two(require_gpu, oracle_mod, visc):
    """1e-13: the rates are 2 to FP64's last bits, and the three kernels run."""
    o, box = pair(oracle_mod, (36, 20, 28), visc=visc)
    check(o, box, 7)
    for b in (o, box):
        b.macrovar()
    o.step(2)
    box.step(2)
    assert relerr(box.get_f(), o.f) <= TOL64
