"""The FP32 solve's two ways of adding a correction (GPU): the last launch of the
blocked sweeps adds its own, and one half-sweep per launch leaves it to two passes
of update and residual, a colour each.  The same arithmetic: the same values,
counts and residuals, to the bit.
"""
import numpy as np
import pytest

import cellweave_b200 as cw

pytestmark = pytest.mark.gpu


def fields(shapes, depth, window, uptake, inner):
    g = cw.ScalarField(shapes, 1.0, 0.001, 0.0)
    for k, (w, h, d) in enumerate(shapes):
        rng = np.random.default_rng(k)
        n = w * h * d
        held = np.zeros((d, h, w), np.uint8)
        held[:, 0] = 1
        held[rng.random((d, h, w)) < 0.03] = 1
        g.set_linear_sink(np.where(rng.random(n) < 0.6, 0.01, 0.0), k)
        # (empties pixels: the floor binds)
        g.set_uptake_array(np.where(rng.random(n) < 0.5, uptake, 0.0), k)
        g.hold_where(1.0, held.reshape(-1), k)
    try:
        st = g.relax(1e-7, 1000, omega=1.8, stop=cw.STOP_RESIDUAL, precision=cw.FP32_DC, block_depth=depth,
                     window=window, inner_sweeps=inner, stats=True)
    except cw.SimulationError as e:  # (a correction that the floor cuts may turn in a cycle: so must the other's)
        st = e.stats
    return [(s["sweeps"], s["residual"], s["status"]) for s in st], [g.values(k) for k in range(len(shapes))]


@pytest.mark.parametrize("uptake", [0.0, 0.02])
@pytest.mark.parametrize("inner", [16, 5])
@pytest.mark.parametrize("shapes", [[(128, 128, 1), (200, 96, 1), (64, 70, 1)],   # rows 16-byte aligned
                                    [(127, 90, 1), (61, 61, 1), (1, 40, 1)],      # any width
                                    [(70, 37, 9), (33, 19, 6)], [(64, 48, 40)]])
def test_a_corrections_last_launch_equals_two_passes_of_update(shapes, inner, uptake):
    counts, values = fields(shapes, 1, cw.WINDOW_AUTO, uptake, inner)
    for window in (cw.WINDOW_AUTO, cw.WINDOW_TALL, cw.WINDOW_64):
        for depth in (4, 8):
            got, v = fields(shapes, depth, window, uptake, inner)
            assert got == counts, (window, depth)
            for a, b in zip(v, values):
                np.testing.assert_array_equal(a.view(np.uint64), b.view(np.uint64))
