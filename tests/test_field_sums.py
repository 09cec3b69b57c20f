"""rmsstat, statistics and diag at odd and even grids, with and without solid
nodes, in both precisions: against the numpy restatement on the same fields
(the tolerances of test_rmsstat), and leaving the fields as they were.
"""

import numpy as np
import pytest

from conftest import relerr
from test_gpu_parity import make_pair

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.LBM_PREC_F64, capi.LBM_PREC_F32])
@pytest.mark.parametrize("shape,npart", [((33, 20, 15), 0), ((34, 20, 19), 0), ((8, 6, 7), 0),
                                         ((33, 30, 35), 2)])
def test_sums_over_fields(require_gpu, oracle_mod, shape, npart, precision):
    from oracle import statistics as ost
    o, box = make_pair(oracle_mod, shape=shape, npart=npart, rad=4.0, rhopart=2.5, urms=0.04,
                       k0=2.0, precision=precision)
    box.step(2)
    fields = box.get_macro()
    _, isn = box.get_flags()
    _, ux, uy, uz = fields
    p = box.get_particles()
    parts = (p["wp"], p["omgp"]) if npart else (None, None)
    got = np.array(list(box.rmsstat().values()))
    want = ost.rmsstat(ux, uy, uz, isn, *parts)
    assert got[0] == want[0]
    assert np.allclose(got, want, rtol=1e-11, atol=1e-13)
    assert relerr(box.diag()["vmax"], ost.diag(ux, uy, uz, isn, *parts)[0]) <= 1e-15
    box.statistics()
    for a, b in zip(box.get_macro(), fields):
        assert np.array_equal(a, b)
