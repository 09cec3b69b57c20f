"""The forms of the bounce-back.

How many blocks share a sphere of the FP64 path depends on how many spheres
there are and on their radius: the smallest and a large radius, one sphere and
several, against the oracle.  The FP32 path with few spheres (kPrepParticles)
takes the links' gathers and coefficients from the link build, a batch with
more in all forms them in the bounce-back: the same bits either way, also when
a box goes from one to the other.
"""

import numpy as np
import pytest

from conftest import relerr
from test_batch import make_box, run_batch
from test_gpu_parity import TOL32, TOL64, make_pair

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npart,rad", [(1, 3.0), (1, 7.0), (5, 4.5)])
def test_fp64_split_matches_oracle(require_gpu, oracle_mod, npart, rad):
    o, box = make_pair(oracle_mod, shape=(48, 40, 44), npart=npart, rad=rad, rhopart=2.5)
    for _ in range(4):
        o.step(1)
        box.step(1)
    assert relerr(box.get_f(), o.f) <= TOL64
    p = box.get_particles()
    scale = np.abs(o.fHIp[:npart]).max()
    assert np.abs(p["fHIp"] - o.fHIp[:npart]).max() <= 1e-11 * max(scale, 1.0)


def test_fp32_gathers_from_the_link_build_give_the_same_bits(require_gpu):
    from multiphase_flow_codes_gb300.engine import LBMBatch
    few = [(32, 2, 3.5, 101), (48, 3, 6.0, 202)]
    crowd = (80, 250, 3.0, 77)                       # twice: 500 spheres
    alone = run_batch(few, 7, graph=False)
    mixed = run_batch(few + [crowd, crowd], 7, graph=False)
    for (f1, p1), (f2, p2) in zip(alone, mixed):
        assert np.array_equal(f1, f2)
        for k in ("fHIp", "torqp", "ypglb"):
            assert np.array_equal(p1[k], p2[k]), k
    # from the crowded batch to one of its own and on alone
    moved, ref = make_box(*few[0]), make_box(*few[0])
    others = [make_box(*crowd), make_box(*crowd)]
    with LBMBatch([moved] + others) as b:
        b.step(4, graph=False)
        b.synchronize()
    for box in (moved, ref):
        with LBMBatch([box]) as b:
            b.step(6 if box is moved else 10, graph=False)
            b.synchronize()
        box.step(3)
    assert np.array_equal(moved.get_f(), ref.get_f())
    assert np.array_equal(moved.get_particles()["fHIp"], ref.get_particles()["fHIp"])


def test_fp32_channel_links_at_the_walls(require_gpu, oracle_mod):
    o, box = make_pair(oracle_mod, preset=capi.LBM_PRESET_CHANNEL, shape=(28, 30, 26), npart=3,
                       rad=4.0, rhopart=1.0, precision=capi.LBM_PREC_F32, mrt_type=1)
    for _ in range(6):
        o.step(1)
        box.step(1)
    assert relerr(box.get_f(), o.f) <= TOL32
