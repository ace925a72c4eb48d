"""The sublattice passes' two ways against the oracle's sequence (GPU), to the
bit: by the cells' chains, and by rounds of claims where a cell has more
attempts in a pass than its list holds or records past what a chain hands on;
at row lengths and lattice sizes on either side of the proposals' segments.
"""
import numpy as np
import pytest

import cellweave_b200 as cw
from cellweave_b200 import seeding
from oracle import oracle as O

pytestmark = pytest.mark.gpu

J3 = np.array([[0, 16, 16], [16, 8, 12], [16, 12, 8]], float)
SEED = 0xC0FFEE12345


def packed(shape, side, seed=0, skip=0.2):
    """side^2 (or side^3) cells on a grid of that pitch, some left out."""
    w, h, d = shape
    grid, rec = seeding.empty(w, h, d), seeding.Records()
    rng = np.random.default_rng(seed)
    sz = side if d > 1 else 1
    for z in range(0, d - sz + 1, sz):
        for y in range(0, h - side + 1, side):
            for x in range(0, w - side + 1, side):
                if rng.random() >= skip:
                    seeding.add_block(grid, rec, 1 + int(rng.integers(2)), (x, y), side, side, lam=1.3, z=z, depth=sz)
    return grid, rec


def compare(grid, rec, order, steps, surface=False, subsweeps=1, volume=None, T=10.0):
    d, h, w = grid.shape
    o = O.Lattice(grid, (w, h, d), len(rec), J3, T, order)
    g = cw.CpmLattice.from_grids([grid], [rec], T, J3, order, seeds=[SEED])
    t, v, tg, lam = rec.arrays()
    if volume is not None:
        v = volume(v)
        g.set_cells(volume=v)
    o.type[:], o.volume[:], o.target[:], o.lam[:] = t, v, tg, lam
    if surface:
        ts, ls = np.full(len(rec), 40, np.int32), np.full(len(rec), 0.3)
        o.enable_surface(ts, ls)
        g.set_surface(ts, ls)
    if subsweeps > 1:
        g.set_subsweeps(subsweeps)
    before = g.grid().copy()
    o.mcs_checkerboard(SEED, 0, steps, subsweeps=subsweeps)
    g.monte_carlo_step(steps)
    np.testing.assert_array_equal(g.grid().reshape(-1), o.grid)
    np.testing.assert_array_equal(g.cells()["volume"][1:], o.volume[1:])
    if surface:
        np.testing.assert_array_equal(g.surfaces()[1:], o.surface[1:])
    assert (g.grid() != before).any()


# (width and height about a segment of 32, 64 or 128 pixels of a colour, one
# pixel wide, and enough pixels for the longer segments)
@pytest.mark.parametrize("shape,order", [((63, 40, 1), 2), ((129, 33, 1), 1), ((257, 70, 1), 2), ((1, 90, 1), 1),
                                         ((190, 96, 1), 3), ((1500, 1101, 1), 2), ((2305, 2203, 1), 2),
                                         ((33, 40, 21), 2), ((70, 31, 29), 3), ((66, 35, 33), 1)])
def test_passes_by_chains(shape, order):
    side = 1 if min(shape[:2]) < 5 else 7 if shape[2] == 1 else 4
    grid, rec = packed(shape, side)
    compare(grid, rec, order, 2 if shape[0] > 1000 else 5, surface=shape[2] > 1)


@pytest.mark.parametrize("shape,side,order,surface,subsweeps", [((200, 160, 1), 60, 2, False, 1),
                                                                ((200, 160, 1), 60, 1, True, 3),
                                                                ((60, 58, 50), 20, 3, True, 1)])
def test_passes_by_rounds_where_a_cell_has_many_attempts(shape, side, order, surface, subsweeps):
    # cells whose border holds more pixels of a colour than a list's 64 entries
    grid, rec = packed(shape, side, skip=0.0)
    compare(grid, rec, order, 6, surface, subsweeps, T=40.0)


def test_small_and_large_cells_side_by_side():
    # passes by rounds beside passes by chains on one lattice: the large cell
    # shrinks below a list's length as the small ones eat it
    grid, rec = packed((150, 150, 1), 6, skip=0.1)
    seeding.add_block(grid, rec, 1, (0, 0), 150, 150, lam=0.01)  # every free pixel
    compare(grid, rec, 2, 8)


@pytest.mark.parametrize("far", [1 << 27, -(1 << 27), (1 << 30) + 5])
def test_records_past_what_a_chain_hands_on(far):
    grid, rec = packed((64, 64, 1), 7)
    def volume(v):
        v = v.copy()
        v[3] = far
        return v
    compare(grid, rec, 2, 3, volume=volume)
