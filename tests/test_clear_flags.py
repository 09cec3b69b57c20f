"""The solid flags are cleared by their mask: every id of every step against
the oracle (bit for bit) with spheres that cross rows, planes, mask words and
the periodic seam, fused, by subroutines and in a batch.
"""

import numpy as np
import pytest

from test_gpu_parity import check_flags, make_pair

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset", [capi.LBM_PRESET_BOX, capi.LBM_PRESET_CHANNEL])
@pytest.mark.parametrize("shape", [(30, 27, 26), (33, 26, 29), (64, 26, 26), (130, 26, 28)])
def test_ids_of_moving_spheres(require_gpu, oracle_mod, shape, preset):
    wp = np.array([[0.31, -0.22, 0.17], [-0.27, 0.29, -0.24]])
    o, box = make_pair(oracle_mod, preset=preset, shape=shape, npart=2, rad=3.2, rhopart=5.0,
                       urms=0.01, wp=wp, omgp=np.zeros((2, 3)))
    for s in range(8):
        o.step(1)
        if s % 4 == 2:
            box.step_unfused(1)
        else:
            box.step(1)
        check_flags(o, box)


def test_ids_in_a_batch(require_gpu):
    from test_batch import make_box
    from multiphase_flow_codes_gb300.engine import LBMBatch
    spec = (0, 3, 3.5, 61)

    def box(shape):
        return make_box(*spec, precision=capi.LBM_PREC_F32, shape=shape)

    shapes = [(32, 28, 36), (44, 30, 32)]
    alone, mates = [box(s) for s in shapes], [box(s) for s in shapes]
    for b in alone:
        b.step(14)
    with LBMBatch(mates) as t:
        t.step(14)
        t.synchronize()
    for a, m in zip(alone, mates):
        for x, y in zip(a.get_flags(), m.get_flags()):
            assert np.array_equal(x, y)
