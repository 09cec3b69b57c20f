"""lbm_profile times every kernel group of a fused step: the solid flags and the
link lists, which run on a stream of their own, as two intervals a step."""

import pytest

from test_batch import make_box

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [capi.LBM_PREC_F64, capi.LBM_PREC_F32])
def test_intervals_of_a_step(require_gpu, prec):
    box = make_box(48, 6, 4.0, 61, precision=prec)
    box.step(4)
    box.profile(True)
    steps = 15
    box.step(steps)
    phases = box.profile_read()
    want = {"stream_collide": 1, "bounce": 1, "particles": 1, "links": 2, "filling": 1, "forcing": 1}
    for k, (ms, n) in phases.items():
        assert n == want[k] * steps, (k, n)
        assert 0 < ms < 1000, (k, ms)
    box.profile(False)
    box.step(3)
    assert box.profile_read()["links"][1] == 2 * steps


def test_read_while_the_next_forcing_runs(require_gpu):
    """Without spheres a small step ends before the next step's FORCING, which is
    timed on its own stream."""
    box = make_box(16, 0, 3.0, 61)
    box.profile(True)
    for k in range(200):
        box.step(1)
        # (the first FORCING runs in the step itself and is not timed)
        assert box.profile_read()["forcing"][1] >= k
