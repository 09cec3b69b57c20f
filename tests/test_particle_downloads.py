"""lbm_download_particles gives each wanted vector, whichever are asked for and
however often, the same as the whole particle state, and touches no other."""

import itertools

import numpy as np
import pytest

from test_batch import make_box

from multiphase_flow_codes_gb300 import _capi as capi
from multiphase_flow_codes_gb300._capi import dptr

pytestmark = pytest.mark.gpu

NAMES = ("ypglb", "wp", "omgp", "fHIp", "flubp", "torqp")


@pytest.mark.parametrize("prec", [capi.LBM_PREC_F64, capi.LBM_PREC_F32])
def test_every_choice_of_vectors(require_gpu, prec):
    from multiphase_flow_codes_gb300.engine import LBMBox
    cfg = capi.config_init(capi.LBM_PRESET_BOX, 32, 32, 32, 7, 3.0, 2.5)  # room for 7
    cfg.precision = prec
    box = LBMBox(cfg)
    box.init_particles(5, 3)
    rng = np.random.default_rng(8)
    st = box.get_particle_state()
    for k in box.PARTICLE_VECTORS:
        if k != "ypglb":
            st[k] = rng.standard_normal((5, 3))
    box.set_particle_state(st)
    for repeat in range(2):
        for wanted in itertools.product((False, True), repeat=6):
            outs = [np.full((5, 3), np.nan) for _ in NAMES]
            args = [dptr(o) if w else None for o, w in zip(outs, wanted)]
            assert capi.lib().lbm_download_particles(box.handle, *args) == capi.LBM_OK
            for k, o, w in zip(NAMES, outs, wanted):
                assert np.array_equal(o, st[k]) if w else np.isnan(o).all(), (k, wanted)


def test_state_keeps_its_order(require_gpu):
    a = make_box(32, 3, 3.5, 61)
    a.step(3)
    st, p = a.get_particle_state(), a.get_particles()
    for k in NAMES:
        assert np.array_equal(st[k], p[k]), k
    assert not np.array_equal(st["ypglb"], st["ypglbp"])
