"""Single steps that are replayed, and known to be, against directly launched
ones: same bits after many idle steps in a row, in both precisions and
geometries, and across what a replay must notice."""

import numpy as np
import pytest

from test_batch import make_box
from test_step_graphs import same

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu

F64, F32 = capi.LBM_PREC_F64, capi.LBM_PREC_F32
BOX, CHANNEL = capi.LBM_PRESET_BOX, capi.LBM_PRESET_CHANNEL


def pair(prec, preset):
    boxes = [make_box(0, 3, 3.5, 61, precision=prec, preset=preset, shape=(32, 28, 36))
             for _ in range(2)]
    boxes[1].profile(True)      # direct launches
    return boxes


def idle_steps(box, n):
    for _ in range(n):
        box.synchronize()
        box.step(1)


@pytest.mark.parametrize("prec", [F64, F32])
@pytest.mark.parametrize("preset", [BOX, CHANNEL])
def test_runs_of_replays(require_gpu, prec, preset):
    a, b = pair(prec, preset)
    for box in (a, b):
        box.step(255)
        idle_steps(box, 1)
    assert a.replayed_steps() == 0
    for n in (13, 6, 1):
        before = a.replayed_steps()
        for box in (a, b):
            idle_steps(box, n)
        assert a.replayed_steps() == before + n and b.replayed_steps() == 0
        for k, v in a.get_particles().items():
            assert np.array_equal(v, b.get_particles()[k]), k
    same(a, b)
    # (in FP64 the populations have gone back to doubles to be read: the next
    # step takes them to fixed point by itself, those after it are replayed)
    before = a.replayed_steps()
    for box in (a, b):
        idle_steps(box, 8)
    assert a.replayed_steps() >= before + 7
    same(a, b)


def test_a_queued_step_is_launched(require_gpu):
    """A step whose stream is busy is not replayed."""
    a, b = pair(F32, BOX)
    for box in (a, b):
        box.step(256)
        box.step(1)
        idle_steps(box, 5)
    assert 0 < a.replayed_steps() <= 6
    same(a, b)


@pytest.mark.parametrize("prec", [F64, F32])
def test_moved_spheres_between_replays(require_gpu, prec):
    a, b = pair(prec, BOX)
    for box in (a, b):
        box.step(256)
        for _ in range(3):
            idle_steps(box, 6)
            box.beads_move()
    assert a.replayed_steps() > 0
    same(a, b)
