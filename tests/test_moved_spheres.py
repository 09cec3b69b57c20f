"""Spheres moved by beads_move alone, without new links, before a fused step.

The lists of the step before say which links there are; the wall velocity and
the torque of the bounce-back are taken at the spheres' present centres, as the
per-subroutine entries take them.  FP32 boxes of few spheres, which form lever
arms with the lists, alone and in a batch.
"""

import numpy as np
import pytest

from test_batch import make_box

from multiphase_flow_codes_gb300 import _capi as capi
from multiphase_flow_codes_gb300.engine import LBMBatch

pytestmark = pytest.mark.gpu


def moved_box(preset, wp=0.05):
    box = make_box(32, 3, 3.5, 61, preset=preset)
    box.step(4)
    # speed the spheres up, then move them a few times: half a unit and more
    st = box.get_particle_state()
    st["wp"][:] = wp
    st["wpp"][:] = wp
    box.set_particle_state(st)
    for _ in range(12):
        box.beads_move()
    box.beads_redistribute()
    return box


def close(a, b):
    pa, pb = a.get_particles(), b.get_particles()
    assert np.abs(pb["torqp"]).max() > 0
    for k in ("fHIp", "torqp"):
        # (a thousand links of 0.02 at an arm of 4: terms of 80 in all, 1e-5 in
        # FP32, against sums of some 0.05; an arm that is half a unit off changes
        # the torque by a tenth and more)
        assert np.abs(pa[k] - pb[k]).max() <= 1e-3 * np.abs(pb[k]).max(), k


@pytest.mark.parametrize("preset", [capi.LBM_PRESET_BOX, capi.LBM_PRESET_CHANNEL])
@pytest.mark.parametrize("steps", [1, 2])
def test_fused_step_after_a_move(require_gpu, preset, steps):
    a, b = moved_box(preset), moved_box(preset)
    a.step(steps)
    b.step_unfused(steps)
    close(a, b)


def test_batch_after_a_move(require_gpu):
    a, b = moved_box(capi.LBM_PRESET_BOX), moved_box(capi.LBM_PRESET_BOX)
    with LBMBatch([a]) as t:
        t.step(1)
        t.synchronize()
    b.step_unfused(1)
    close(a, b)
