"""Fused steps replayed from captured graphs equal directly launched ones.

A context with few nodes that has made some hundreds of fused steps captures and
replays a single step that finds its stream idle; timing phases with profile()
keeps it on direct launches.  Same bits,
for both precisions, with and without stochastic forcing, and across what
changes a step: new spheres, another kernel, another stream, statistics, a
forcing state read back, subroutine calls and a batch in between.
"""

import numpy as np
import pytest

from test_batch import make_box

from multiphase_flow_codes_gb300 import _capi as capi

pytestmark = pytest.mark.gpu

F64, F32 = capi.LBM_PREC_F64, capi.LBM_PREC_F32


def same(a, b):
    assert np.array_equal(a.get_f(), b.get_f())
    pa, pb = a.get_particle_state(), b.get_particle_state()
    for k in pa:
        assert np.array_equal(pa[k], pb[k]), k


def pair(prec, preset, npart=3):
    spec = (0, npart, 3.5, 61)
    boxes = [make_box(*spec, precision=prec, preset=preset, shape=(32, 28, 36)) for _ in range(2)]
    boxes[1].profile(True)      # direct launches
    return boxes


@pytest.mark.parametrize("prec", [F64, F32])
@pytest.mark.parametrize("preset", [capi.LBM_PRESET_BOX, capi.LBM_PRESET_CHANNEL])
def test_replayed_steps_same_bits(require_gpu, prec, preset):
    a, b = pair(prec, preset)
    for n in (254, 1, 1, 1, 1, 1, 1, 1, 1, 1, 7, 1, 1, 2, 1, 1, 1):
        a.step(n)
        b.step(n)
        same(a, b)


@pytest.mark.parametrize("prec", [F64, F32])
def test_replayed_steps_across_changes(require_gpu, prec):
    import torch
    from multiphase_flow_codes_gb300.engine import LBMBatch
    a, b = pair(prec, capi.LBM_PRESET_BOX)
    y = a.get_particles()["ypglb"]
    stream = torch.cuda.Stream()

    def batch(box):
        if prec == F64:
            return
        direct = box is b
        if direct:
            box.profile(False)      # a batch takes no profiled box
        with LBMBatch([box]) as t:
            t.step(3)
            t.synchronize()
        if direct:
            box.profile(True)

    changes = [
        lambda box: box.release_particles(y[:2] + 1.25),
        lambda box: box.set_variant(capi.LBM_VARIANT_DIRECT),
        lambda box: box.get_forcing_state(),
        lambda box: box.step_unfused(1),
        lambda box: box.mass_momentum(),
        lambda box: box.statistics(),
        batch,
        lambda box: box.set_variant(capi.LBM_VARIANT_STAGED),
        lambda box: box.set_stream(stream.cuda_stream),
    ]
    for box in (a, b):
        box.step(254)
    for change in [lambda box: None] + changes:
        for box in (a, b):
            change(box)
            for _ in range(9):
                box.synchronize()
                box.step(1)
        same(a, b)
