"""The bounce-back of one sphere over several blocks.

How many blocks share a sphere of the FP64 path depends on how many spheres
there are and on their radius: the smallest and a large radius, one sphere and
several, against the oracle.
"""

import numpy as np
import pytest

from conftest import relerr
from test_gpu_parity import TOL64, make_pair

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
