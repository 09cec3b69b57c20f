"""rmsstat of a field that is not finite reports it, with and without spheres."""

import math

import numpy as np
import pytest

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu

VORTICITY = ("oxmn", "oymn", "ozmn", "oxrms", "oyrms", "ozrms", "omgfmn")


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("npart", [0, 1])
@pytest.mark.parametrize("prec", [capi.LBM_PREC_F64, capi.LBM_PREC_F32])
def test_vorticity_of_a_bad_node_is_nan(require_gpu, bad, npart, prec):
    from multiphase_flow_codes_gb300.engine import LBMBox
    n = 16
    cfg = capi.config_init(capi.LBM_PRESET_BOX, n, n, n, npart, 3.0, 1.0)
    cfg.precision = prec
    cfg.forcing = capi.LBM_FORCING_NONE
    box = LBMBox(cfg)
    if npart:
        box.release_particles(np.array([[4.0, 4.0, 4.0]]))
    f = np.zeros((19, n, n, n))
    # three directions: every component of the velocity is bad there
    f[[1, 3, 5], 12, 12, 12] = bad
    box.set_f(f)
    box.macrovar()
    row = box.rmsstat()
    for k in VORTICITY:
        assert math.isnan(row[k]), (k, row[k])
