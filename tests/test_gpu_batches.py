"""The sublattice passes over batches and lattices of many shapes (GPU): rows
shorter than what a warp reads at once, one behind another; thousands of
histories; cells' lists of every length; passes long enough that the blocks
share out anew; and the memory that they take.  Grids and records are the
oracle's, to the bit.
"""
import numpy as np
import pytest

import cellweave_b200 as cw
from cellweave_b200 import seeding
from oracle import oracle as O

pytestmark = pytest.mark.gpu

J3 = np.array([[0, 16, 16], [16, 8, 12], [16, 12, 8]], float)


def packed(shape, side, seed, skip=0.2):
    w, h, d = shape
    grid, rec = seeding.empty(w, h, d), seeding.Records()
    rng = np.random.default_rng(seed)
    sz = min(side, d)
    for z in range(0, d - sz + 1, sz):
        for y in range(0, h - side + 1, side):
            for x in range(0, w - side + 1, side):
                if rng.random() >= skip:
                    seeding.add_block(grid, rec, 1 + int(rng.integers(2)), (x, y), side, side, lam=1.3, z=z, depth=sz)
    return grid, rec


def same_as_the_oracle(lat, k, grid, rec, order, steps, seed):
    d, h, w = grid.shape
    o = O.Lattice(grid, (w, h, d), len(rec), J3, 10.0, order)
    o.type[:], o.volume[:], o.target[:], o.lam[:] = rec.arrays()
    o.mcs_checkerboard(seed, 0, steps)
    got = lat.grid(k)
    np.testing.assert_array_equal(got.reshape(-1), o.grid)
    np.testing.assert_array_equal(lat.cells(len(rec), k)["volume"][1:], o.volume[1:])
    assert (got != grid).any()


# 1 to 128 pixels of a colour in a row, whole and cut short; more histories than
# a block keeps the plan of in shared memory
@pytest.mark.parametrize("shapes,order", [([(31, 9, 1), (64, 64, 1), (5, 70, 1), (130, 33, 1), (256, 20, 1)], 2),
                                          ([(33, 40, 1), (64, 30, 1), (7, 7, 1), (300, 21, 1)], 1),
                                          ([(48, 48, 1), (100, 30, 1), (200, 17, 1)], 3),
                                          ([(20, 24, 22), (9, 33, 8), (66, 12, 10)], 1),
                                          ([(20, 24, 22), (9, 33, 8), (70, 12, 10)], 2)])
@pytest.mark.parametrize("copies", [1, 300])
def test_batches_of_short_rows(shapes, order, copies):
    side = 4
    base = [packed(s, side, 11 + k) for k, s in enumerate(shapes)]
    n = len(shapes) * copies
    grids = [base[k % len(shapes)][0] for k in range(n)]
    recs = [base[k % len(shapes)][1] for k in range(n)]
    lat = cw.CpmLattice.from_grids(grids, recs, 10.0, J3, order, seeds=list(range(100, 100 + n)))
    lat.monte_carlo_step(3)
    for k in {0, 1, len(shapes) - 1, n // 2, n - 2, n - 1}:
        same_as_the_oracle(lat, k, grids[k], recs[k], order, 3, 100 + k)


def test_the_scratch_of_short_rows_follows_their_pixels():
    torch = pytest.importorskip("torch")
    grid, rec = packed((64, 64, 1), 7, 1)
    n = 2048
    lat = cw.CpmLattice.from_grids([grid] * n, [rec] * n, 10.0, J3, 2, seeds=list(range(n)))
    before = torch.cuda.mem_get_info()[0]
    lat.monte_carlo_step(1)
    taken = before - torch.cuda.mem_get_info()[0]
    # a colour's pixels: a quarter of the sites.  152 bytes each, an eighth for
    # chunks' ends and one chunk of 2,048 for each of up to 148 blocks; 516 + 16
    # bytes a record; 2 MB for each of six allocations
    pixels = n * 64 * 64 // 4
    assert taken <= 152 * (pixels * 9 // 8 + 148 * 2048) + 532 * n * len(rec) + (12 << 20)


# cells whose lists hold about 2 to 50 attempts a pass, side by side
@pytest.mark.parametrize("order", [1, 2, 3])
def test_lists_of_every_length(order):
    grid, rec = seeding.empty(400, 300, 1), seeding.Records()
    rng = np.random.default_rng(4)
    for x0, side in ((0, 2), (60, 4), (120, 7), (190, 12), (260, 20), (330, 30)):
        for y in range(0, 300 - side + 1, side):
            for x in range(x0, x0 + 60 - side + 1, side):
                if rng.random() < 0.9:
                    seeding.add_block(grid, rec, 1 + int(rng.integers(2)), (x, y), side, side, lam=1.0)
    lat = cw.CpmLattice.from_grids([grid], [rec], 10.0, J3, order, seeds=[77])
    lat.monte_carlo_step(4)
    same_as_the_oracle(lat, 0, grid, rec, order, 4, 77)


def test_a_pass_of_many_turns():
    # 125-voxel cells filling a volume, two colours: a quarter of a million attempts a
    # pass, and some 90 that follow one another
    shape = (128, 128, 128)
    grid, rec = packed(shape, 5, 9, skip=0.05)
    lat = cw.CpmLattice.from_grids([grid], [rec], 10.0, J3, 1, seeds=[5])
    lat.monte_carlo_step(2)
    same_as_the_oracle(lat, 0, grid, rec, 1, 2, 5)


@pytest.mark.parametrize("shape,side,order,surface", [((150, 131, 1), 7, 2, False), ((150, 131, 1), 7, 1, True),
                                                      ((40, 33, 36), 5, 2, True)])
def test_passes_without_room_for_the_cells_lists(shape, side, order, surface):
    # so many records that their lists would take a third of the device: every
    # pass by rounds, its attempts' constants read from the records
    grid, rec = packed(shape, side, 3)
    lat = cw.CpmLattice.from_grids([grid], [rec], 10.0, J3, order, seeds=[21], capacity=120_000_000)
    t, v, tg, lam = rec.arrays()
    d, h, w = grid.shape
    o = O.Lattice(grid, (w, h, d), len(rec), J3, 10.0, order)
    o.type[:], o.volume[:], o.target[:], o.lam[:] = t, v, tg, lam
    if surface:
        ts, ls = np.full(len(rec), 40, np.int32), np.full(len(rec), 0.3)
        o.enable_surface(ts, ls)
        lat.set_surface(ts, ls)
    lat.monte_carlo_step(4)
    o.mcs_checkerboard(21, 0, 4)
    np.testing.assert_array_equal(lat.grid().reshape(-1), o.grid)
    np.testing.assert_array_equal(lat.cells(len(rec))["volume"][1:], o.volume[1:])
    if surface:
        np.testing.assert_array_equal(lat.surfaces(len(rec))[1:], o.surface[1:])


# tissues that fill their box, a corner of it, or a few cells in the middle: the
# pixels a lane reads follow the spans
@pytest.mark.parametrize("order", [1, 2, 3])
def test_volumes_whose_tissue_is_a_part_of_the_box(order):
    boxes = [((200, 60, 56), (0, 0, 0), (200, 60, 56)), ((200, 60, 56), (150, 30, 20), (45, 25, 30)),
             ((130, 70, 66), (60, 30, 28), (12, 8, 8)), ((96, 96, 96), (1, 1, 1), (90, 90, 90))]
    for some in (boxes, boxes[1:2], boxes[2:3], boxes[3:]):
        grids, recs = [], []
        for (w, h, d), (x, y, z), (sw, sh, sd) in some:
            part, rec = packed((sw, sh, sd), 4, 6)
            grid = seeding.empty(w, h, d)
            grid[z:z + sd, y:y + sh, x:x + sw] = part
            grids.append(grid)
            recs.append(rec)
        lat = cw.CpmLattice.from_grids(grids, recs, 10.0, J3, order, seeds=list(range(50, 50 + len(some))))
        lat.monte_carlo_step(3)
        for k in range(len(some)):
            same_as_the_oracle(lat, k, grids[k], recs[k], order, 3, 50 + k)
