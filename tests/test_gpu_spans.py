"""The boxes of free pixels of uneven batches (GPU): histories of less than one
block of pixels, of a few, and of more than a group of blocks, some with a box
well inside the history, some without a free pixel, each relaxed as the oracle
relaxes it (its relaxation factor and its sweeps follow from its box).
"""
import numpy as np
import pytest

import cellweave_b200 as cw
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DIMS = [(3, 3, 1), (7, 5, 6), (40, 30, 1), (2, 2, 1), (33, 20, 5), (90, 61, 1), (16, 16, 9), (1, 1, 1), (5, 200, 1),
        (24, 24, 24), (130, 3, 1)]


def problem(dims, seed):
    w, h, d = dims
    rng = np.random.default_rng(seed)
    held = np.ones((d, h, w), np.uint8)
    if seed % 4:  # a box of its own; every fourth history holds every pixel
        held[d // 3:d - d // 4, h // 4:max(h - h // 5, h // 4 + 1), w // 5:max(w - w // 6, w // 5 + 1)] = 0
        held[rng.random(held.shape) < 0.1] = 1
    return held.reshape(-1), rng.uniform(0, 1, w * h * d), np.full(w * h * d, 1e-3)


def test_each_history_relaxes_over_its_own_box():
    g = cw.ScalarField(DIMS, 0.2, 0.0, 0.0)
    for k, dims in enumerate(DIMS):
        held, values, uptake = problem(dims, k)
        g.set_held(held, k)
        g.set_values(values, k)
        g.set_uptake_array(uptake, k)
    st = g.relax(1e-9, 100_000, stats=True)
    for k, dims in enumerate(DIMS):
        o = O.Field(*dims, 0.2, 0.0, 0.0)
        o.held[:], o.values[:], o.uptake[:] = problem(dims, k)
        rc, sweeps = o.relax(1e-9, 100_000)
        assert rc == 0 and st[k]["sweeps"] == sweeps
        np.testing.assert_array_equal(g.values(k).view(np.uint64), o.values.view(np.uint64))
