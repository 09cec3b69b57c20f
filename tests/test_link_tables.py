"""Flags and links of many small spheres, for which the flag and link kernels
take small tables and a thread a row, about the limit of their radius: against
the oracle, flags and link sets bit for bit, link fractions as elsewhere.
"""

import numpy as np
import pytest

from test_gpu_parity import check_flags, check_links

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu


def many_pair(oracle_mod, preset, shape, npart, rad):
    from multiphase_flow_codes_gb300.engine import LBMBox
    cfg = capi.config_init(preset, *shape, npart, rad, 5.0)
    still = tuple(np.zeros(shape[::-1]) for _ in range(3))
    o = oracle_mod.OracleBox(cfg)
    box = LBMBox(cfg)
    for b in (o, box):
        b.initpop(*still)
        b.macrovar()
    return o, box


@pytest.mark.parametrize("preset,rad", [(capi.LBM_PRESET_BOX, 1.2), (capi.LBM_PRESET_CHANNEL, 3.0),
                                        (capi.LBM_PRESET_BOX, 4.0), (capi.LBM_PRESET_BOX, 5.0),
                                        (capi.LBM_PRESET_BOX, 5.001)])
def test_many_spheres(require_gpu, oracle_mod, preset, rad):
    counts = (9, 9, 8)                         # 648 spheres on a jittered lattice
    d = int(np.ceil(2.0 * rad)) + 2
    shape = tuple(d * c for c in counts)
    o, box = many_pair(oracle_mod, preset, shape, 648, rad)
    rng = np.random.default_rng(int(1000 * rad))
    at = np.stack(np.meshgrid(*[np.arange(c) for c in counts], indexing="ij"), -1).reshape(-1, 3)
    y = d * (at + 0.5) + rng.uniform(-0.45, 0.45, (648, 3))
    if preset == capi.LBM_PRESET_BOX:
        y += 0.5 * d                           # the last ones wrap
    else:
        y[:, 1:] += 0.5 * d
    y %= np.array(shape)
    o.release_particles(y)
    box.release_particles(y)
    check_flags(o, box)
    check_links(o, box)
