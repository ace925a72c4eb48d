"""The FP64 relax kept on chip when a meeting of its blocks runs out, when
fields are solved at once from several threads, and when a solve takes more
sweeps than one launch (GPU).  A wait that runs out is made by a block kept from
its meeting, with a limit of a few milliseconds: nothing faults or hangs.
"""
import threading

import numpy as np
import pytest

import cellweave_b200 as cw
from cellweave_b200 import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LIMIT_NS = 5_000_000


def faults(wait_ns=0, withhold=-1):
    _lib.check(_lib.lib().cw_test_faults(wait_ns, withhold, 0, 0))


@pytest.fixture(autouse=True)
def back_to_defaults():
    faults()
    yield
    faults()


def bits(a):
    return np.ascontiguousarray(a, np.float64).view(np.uint64)


def problem(shape, seed=3):
    w, h, d = shape
    rng = np.random.default_rng(seed)
    n = w * h * d
    held = np.zeros((d, h, w), np.uint8)
    held[:, 0] = 1
    held = held.reshape(-1)
    return held, np.where(held, 1.0, rng.uniform(0.0, 1.0, n)), np.where(rng.random(n) < 0.5, 1e-4, 0.0)


def field(shape, p):
    held, values, uptake = p
    g = cw.ScalarField([shape], 0.2, 0.0, 0.0)
    g.set_held(held)
    g.set_values(values)
    g.set_uptake_array(uptake)
    return g


def solved(shape, p, omega, tol=1e-7):
    held, values, uptake = p
    o = O.Field(*shape, 0.2, 0.0, 0.0)
    o.held[:], o.values[:], o.uptake[:] = held, values, uptake
    rc, sweeps = o.relax(tol, 100_000, omega=omega)
    assert rc == 0
    return o.values, sweeps


@pytest.mark.parametrize("shape", [(301, 287, 1), (33, 40, 21)])
@pytest.mark.parametrize("withhold", [0, 1])
def test_a_block_kept_from_its_meeting_times_out_and_the_next_solve_is_the_oracles(shape, withhold):
    p = problem(shape)
    g = field(shape, p)
    faults(LIMIT_NS, withhold)
    with pytest.raises(_lib.TimeoutError_):
        g.relax(1e-7, 100_000, omega=1.8)
    faults()
    g.set_values(p[1])
    want, sweeps = solved(shape, p, 1.8)
    assert g.relax(1e-7, 100_000, omega=1.8) == sweeps
    np.testing.assert_array_equal(bits(g.values()), bits(want))


def test_a_timeout_is_its_own_fields_alone():
    # one field's block 1 is kept from its meetings; the other, of one block,
    # settles every time
    wide, small = (301, 287, 1), (16, 16, 1)
    pw, ps = problem(wide), problem(small)
    a, b = field(wide, pw), field(small, ps)
    want, sweeps = solved(small, ps, 1.5)
    faults(LIMIT_NS, 1)
    wrong, running = [], threading.Event()
    running.set()

    def settles():
        try:
            while running.is_set():
                b.set_values(ps[1])
                if b.relax(1e-7, 100_000, omega=1.5) != sweeps or (bits(b.values()) != bits(want)).any():
                    wrong.append("another result")
        except Exception as e:  # the other thread's failure
            wrong.append(repr(e))

    t = threading.Thread(target=settles)
    t.start()
    try:
        for _ in range(20):
            with pytest.raises(_lib.TimeoutError_):
                a.relax(1e-7, 100_000, omega=1.8)
    finally:
        running.clear()
        t.join()
    assert not wrong


def test_fields_relaxed_at_once_from_several_threads_are_the_oracles():
    shapes = [(301, 287, 1), (33, 40, 21), (129, 67, 1)]
    ps = [problem(s, seed=k) for k, s in enumerate(shapes)]
    wants = [solved(s, p, 1.8) for s, p in zip(shapes, ps)]
    wrong = []

    def run(k):
        try:
            g = field(shapes[k], ps[k])
            for _ in range(10):
                g.set_values(ps[k][1])
                if g.relax(1e-7, 100_000, omega=1.8) != wants[k][1] or (bits(g.values()) != bits(wants[k][0])).any():
                    wrong.append(k)
        except Exception as e:
            wrong.append(repr(e))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_a_solve_of_more_sweeps_than_a_launch_takes_carries_on():
    # 16,384 sweeps a launch: one history past it, one settled long before
    shapes = [(110, 100, 1), (16, 16, 1)]
    ps = [problem(s, seed=k) for k, s in enumerate(shapes)]
    g = cw.ScalarField(shapes, 0.2, 0.0, 0.0)
    for k, (held, values, uptake) in enumerate(ps):
        g.set_held(held, k)
        g.set_values(values, k)
        g.set_uptake_array(uptake, k)
    wants = [solved(s, p, 0.5, 1e-9) for s, p in zip(shapes, ps)]
    assert wants[0][1] > 17_000 and wants[1][1] < 16_000
    st = g.relax(1e-9, 100_000, omega=0.5, stats=True)
    for k, (values, sweeps) in enumerate(wants):
        assert st[k]["sweeps"] == sweeps
        np.testing.assert_array_equal(bits(g.values(k)), bits(values))
    o = O.Field(*shapes[0], 0.2, 0.0, 0.0)
    o.held[:], o.values[:], o.uptake[:] = ps[0][0], wants[0][0], ps[0][2]
    assert st[0]["residual"] == o.residual()


def test_a_small_tissue_in_a_large_box_takes_little_beside_its_field():
    torch = pytest.importorskip("torch")

    def tissue(n, z0):
        free = np.zeros((n, n, n), bool)
        free[z0:z0 + 20, 40:60, 30:70] = True
        held = (~free).reshape(-1).astype(np.uint8)
        values = np.random.default_rng(1).uniform(0.0, 1.0, n**3)
        return held, values, np.where(held, 0.0, 1e-4)

    shape = (256, 256, 256)
    small = field((100, 100, 100), tissue(100, 40))
    small.relax(1e-6, 1000, omega=1.7)  # the kernel loaded
    p = tissue(256, 100)
    g = field(shape, p)
    before = torch.cuda.mem_get_info()[0]
    counts = [g.relax(1e-6, 1000, omega=1.7)]
    taken = before - torch.cuda.mem_get_info()[0]
    # 20 of 256 slices of 8 bytes a voxel (10.5 MB), a few allocations of 2 MB
    assert taken <= 20 * 256 * 256 * 8 + (8 << 20)
    # and the tissue moves, to slices that buffer has not held
    moved = tissue(256, 180)
    for held, values, uptake in (p, moved):
        g.set_held(held)
        g.set_values(values)
        g.set_uptake_array(uptake)
        counts.append(g.relax(1e-6, 1000, omega=1.7))
        want, sweeps = solved(shape, (held, values, uptake), 1.7, 1e-6)
        assert counts[-1] == sweeps
        np.testing.assert_array_equal(bits(g.values()), bits(want))
    assert counts[0] == counts[1]


def test_a_tissue_that_moves_through_a_plane_is_solved_as_the_oracles():
    # rows of the second buffer that no solve has held, windows cut by the box's
    # border, a larger and a smaller tissue in turn
    shape = (900, 700, 1)
    g = cw.ScalarField([shape], 0.2, 0.0, 0.0)
    rng = np.random.default_rng(2)
    for x, y, w, h in ((400, 300, 60, 40), (700, 640, 200, 60), (0, 0, 90, 30), (100, 200, 500, 160), (450, 690, 8, 10)):
        free = np.zeros((700, 900), bool)
        free[y:y + h, x:x + w] = rng.random((h, w)) < 0.97
        held = (~free).reshape(-1).astype(np.uint8)
        p = held, np.where(held, rng.uniform(0.5, 1.0, held.size), rng.uniform(0.0, 1.0, held.size)), np.where(held, 0.0, 1e-4)
        g.set_held(p[0])
        g.set_values(p[1])
        g.set_uptake_array(p[2])
        want, sweeps = solved(shape, p, 1.8)
        assert g.relax(1e-7, 100_000, omega=1.8) == sweeps
        np.testing.assert_array_equal(bits(g.values()), bits(want))
