"""The wide FP32 windows where a block takes more of them than it looks up at
once (GPU): thousands of small histories that settle after different counts,
against the 64 x 64 windows, to the bit.
"""
import numpy as np
import pytest

import cellweave_b200 as cw

pytestmark = pytest.mark.gpu


# one window each: within one look-up of every block (32 windows), past it, and
# past two of them with a ragged end (two blocks of 128 x 64, one of 128 x 128
# a multiprocessor)
@pytest.mark.parametrize("count,side", [(4_000, 16), (9_700, 12), (20_011, 8)])
def test_blocks_that_list_their_windows_more_than_once(count, side):
    held = np.zeros((side, side), np.uint8)
    held[0] = 1
    out = []
    for window in (cw.WINDOW_AUTO, cw.WINDOW_TALL, cw.WINDOW_64):
        g = cw.ScalarField([(side, side, 1)] * count, 1.0, 0.0, 0.0)
        for k in range(count):
            # every ninth history has no sink and settles first
            sink = np.full(side * side, 0.03 * (k % 9))
            g.set_linear_sink(sink, k)
            g.hold_where(1.0, held.reshape(-1), k)
        st = g.relax(1e-6, 1_000_000, omega=1.5, stop=cw.STOP_RESIDUAL, precision=cw.FP32_DC, block_depth=8,
                     window=window, stats=True)
        out.append((st, np.concatenate([g.values(k) for k in range(0, count, 7)])))
    (sa, va), *rest = out
    assert len({s["sweeps"] for s in sa}) > 1
    for sb, vb in rest:
        assert [s["sweeps"] for s in sa] == [s["sweeps"] for s in sb]
        np.testing.assert_array_equal(va.view(np.uint64), vb.view(np.uint64))
