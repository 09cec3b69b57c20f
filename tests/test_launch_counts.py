"""Kernels of a replayed step or batch cycle, counted while another thread
launches: lbm_kernel_launches grows by the same number for a replayed step as
for a direct one, whatever ran beside its capture."""

import threading

import pytest

from test_batch import make_box

from multiphase_flow_codes_gb300 import _capi as capi
from multiphase_flow_codes_gb300.engine import LBMBatch, LBMBox

pytestmark = pytest.mark.gpu


class Busy:
    """Steps a box of its own on another thread, launching all the time."""

    def __enter__(self):
        self.box = make_box(24, 2, 3.0, 9)
        self.stop = False
        self.started = threading.Event()
        self.thread = threading.Thread(target=self.work)
        self.thread.start()
        assert self.started.wait(30)
        return self

    def work(self):
        while not self.stop:
            self.box.step(40)
            self.box.synchronize()
            self.started.set()

    def __exit__(self, *exc):
        self.stop = True
        self.thread.join()


def launches(f):
    n0 = LBMBox.kernel_launches()
    f()
    return LBMBox.kernel_launches() - n0


def single_steps(box, n):
    for _ in range(n):
        box.synchronize()
        box.step(1)


@pytest.mark.parametrize("prec", [capi.LBM_PREC_F64, capi.LBM_PREC_F32])
def test_replayed_steps(require_gpu, prec):
    a, b = (make_box(32, 3, 3.5, 61, precision=prec) for _ in range(2))
    b.profile(True)  # direct launches
    for box in (a, b):
        box.step(256)
    with Busy():
        single_steps(a, 24)
    single_steps(b, 24)
    assert launches(lambda: single_steps(a, 12)) == launches(lambda: single_steps(b, 12))


def test_replayed_batch_cycles(require_gpu):
    a = make_box(32, 3, 3.5, 61)
    with LBMBatch([a]) as t:
        with Busy():
            t.step(12)
            t.synchronize()
        direct = launches(lambda: t.step(6, False))
        assert launches(lambda: t.step(6)) == direct
        t.synchronize()
