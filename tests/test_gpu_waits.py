"""A wait that runs out is its own field's failure (GPU): an FP32 solve whose
copies never land, beside another thread's solves that issue none.  Nothing
faults or hangs: the wait's limit is a few milliseconds.
"""
import threading

import numpy as np
import pytest

import cellweave_b200 as cw
from cellweave_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def back_to_defaults():
    yield
    _lib.check(_lib.lib().cw_test_faults(0, -1, 0, 0))


def field(n):
    rng = np.random.default_rng(n)
    held = np.zeros((n, n), np.uint8)
    held[0] = 1
    f = cw.ScalarField.new(n, n, 1.0, 0.0, 0.0)
    f.set_linear_sink(np.where(rng.random(n * n) < 0.6, 0.01, 0.0))
    f.hold_where(1.0, held.reshape(-1))
    return f


def relax(f):
    f.fill(1.0)
    return f.relax(1e-7, 100_000, omega=1.9, stop=cw.STOP_RESIDUAL, precision=cw.FP32_DC, block_depth=8)


def test_an_fp32_timeout_is_its_own_fields_alone():
    wide, narrow = field(256), field(127)  # copies by TMA; plain loads
    sweeps = relax(narrow)
    relax(wide)
    _lib.check(_lib.lib().cw_test_faults(5_000_000, -1, 0, 1))
    wrong, running = [], threading.Event()
    running.set()

    def settles():
        try:
            while running.is_set():
                if relax(narrow) != sweeps:
                    wrong.append("another count")
        except Exception as e:
            wrong.append(repr(e))

    t = threading.Thread(target=settles)
    t.start()
    try:
        for _ in range(10):
            with pytest.raises(_lib.TimeoutError_):
                relax(wide)
    finally:
        running.clear()
        t.join()
    assert not wrong
