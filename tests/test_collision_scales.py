"""collision_MRT, macrovar and the pre-relaxation of FP64 populations over the
fields' magnitudes.

Outside the fused step these run in integer arithmetic at a scale of each
node's own; a field of any size keeps FP64's relative precision, down to ones
so quiet that a node takes the FP64 form, and up to populations that are too
large for the scales.  Against the oracle, relative to the field's largest
value (1e-12, as the other FP64 tests).
"""

import numpy as np
import pytest

from conftest import relerr
from test_gpu_parity import TOL64
from test_prerelax import oracle_prerelax

from multiphase_flow_codes_gb300 import _capi as capi
from multiphase_flow_codes_gb300 import inputs

pytestmark = pytest.mark.gpu


def pair(oracle_mod, urms, shape=(36, 20, 28), preset=capi.LBM_PRESET_BOX):
    from multiphase_flow_codes_gb300.engine import LBMBox
    nx, ny, nz = shape
    cfg = capi.config_init(preset, nx, ny, nz, 0, 4.0, 1.0)
    cfg.forcing = capi.LBM_FORCING_NONE
    u = inputs.spectral_velocity(nx, 4.0, urms, ny=ny, nz=nz, seed=31)
    u = tuple(a * (np.arange(nz)[:, None, None] >= nz // 4) for a in u)  # a quarter at rest
    o = oracle_mod.OracleBox(cfg)
    o.initpop(*u)
    box = LBMBox(cfg)
    box.initpop(*u)
    return o, box


@pytest.mark.parametrize("urms", [1e-14, 1e-7, 1e-3, 0.03, 0.25])
def test_subroutines_keep_relative_precision(require_gpu, oracle_mod, urms):
    o, box = pair(oracle_mod, urms)
    o.macrovar()
    box.macrovar()
    for a, b in zip(box.get_macro(), (o.rho, o.ux, o.uy, o.uz)):
        assert np.abs(a - b).max() <= TOL64 * np.abs(np.asarray(o.ux)).max()
    for _ in range(3):
        o.collision_MRT()
        box.collision_MRT()
        assert relerr(box.get_f(), o.f) <= TOL64
        o.streaming()
        box.streaming()
        o.macrovar()
        box.macrovar()


@pytest.mark.parametrize("preset", [capi.LBM_PRESET_BOX, capi.LBM_PRESET_CHANNEL])
@pytest.mark.parametrize("urms,max_iter", [(1e-9, 20), (0.03, 3), (0.03, 37)])
def test_prerelax_of_fields_of_any_size(require_gpu, oracle_mod, preset, urms, max_iter):
    """Counters that end inside the first chunk of enqueued iterations, at its
    end and beyond it."""
    o, box = pair(oracle_mod, urms, preset=preset)
    o.rhoupdat()
    box.rhoupdat()
    it_o, err_o = oracle_prerelax(o, 0.0, max_iter)
    it_g, err_g = box.prerelax(0.0, max_iter)
    assert it_g == it_o
    assert abs(err_g - err_o) <= 1e-12 * float(np.abs(np.asarray(o.rho)).max())
    assert relerr(box.get_f(), o.f) <= TOL64
    assert relerr(box.get_macro()[0], o.rho) <= TOL64


def test_prerelax_reports_a_non_finite_density(require_gpu):
    from multiphase_flow_codes_gb300 import LBMError
    from multiphase_flow_codes_gb300.engine import LBMBox
    cfg = capi.config_init(capi.LBM_PRESET_BOX, 16, 16, 16, 0, 4.0, 1.0)
    box = LBMBox(cfg)
    f = np.zeros((19, 16, 16, 16))
    f[3, 2, 2, 2] = np.nan
    box.set_f(f)
    with pytest.raises(LBMError) as e:
        box.prerelax(1e-9, 50)
    assert e.value.code == capi.LBM_ERR_NONFINITE
