"""Boxes with an odd number of nodes have no spectrum: statistics and rmsstat
refuse them, with spheres and without, and leave the context as it was."""

import numpy as np
import pytest

from multiphase_flow_codes_gb300 import LBMError
from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [capi.LBM_PREC_F64, capi.LBM_PREC_F32])
@pytest.mark.parametrize("npart", [0, 1])
def test_odd_boxes_are_refused(require_gpu, npart, prec):
    from multiphase_flow_codes_gb300.engine import LBMBox
    cfg = capi.config_init(capi.LBM_PRESET_BOX, 17, 19, 21, npart, 3.0, 1.0)
    cfg.precision = prec
    box = LBMBox(cfg)
    z = np.zeros((21, 19, 17))
    box.initpop(z + 0.01, z, z)
    box.macrovar()
    if npart:
        box.release_particles(np.array([[8.0, 9.0, 10.0]]))
    before = box.get_macro()
    for entry in (box.statistics, box.rmsstat):
        with pytest.raises(LBMError) as e:
            entry()
        assert e.value.code == capi.LBM_ERR_CUDA
    for a, b in zip(before, box.get_macro()):
        assert np.array_equal(a, b)
    assert box.diag()["vmax"] > 0
    box.step(1)
    box.synchronize()
