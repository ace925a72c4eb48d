"""The FP64 relax kept on chip against the oracle (GPU), to the bit: values,
sweep counts and residuals, at the edges of its tiling (one block, many, odd
sides, windows cut by the box), with every coefficient array, both stops, a
count that ends inside a round, and a batch of uneven histories.
"""
import numpy as np
import pytest

import cellweave_b200 as cw
from cellweave_b200 import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (w, h, d): one pixel free of one block, thin strips, odd sides over many
# tiles, a plane whose tiles take the whole device, volumes of odd sides
SHAPES = [(3, 3, 1), (5, 64, 1), (200, 3, 1), (129, 67, 1), (301, 287, 1), (640, 411, 1), (7, 5, 6), (33, 40, 21),
          (64, 61, 57)]


def bits(a):
    return np.ascontiguousarray(a, np.float64).view(np.uint64)


def problem(shape, sink, production, seed=5):
    w, h, d = shape
    rng = np.random.default_rng(seed)
    n = w * h * d
    held = np.zeros((d, h, w), np.uint8)
    held[:, 0] = 1
    held[rng.random((d, h, w)) < 0.02] = 1
    held = held.reshape(-1)
    values = np.where(held, 1.0, rng.uniform(0.0, 1.0, n))
    uptake = np.where(rng.random(n) < 0.5, rng.uniform(0.0, 2e-3, n), 0.0)  # empties some pixels: the floor binds
    ks = rng.uniform(0.0, 0.02, n) if sink else None
    pr = rng.uniform(0.0, 1e-3, n) if production else None
    return held, values, uptake, ks, pr


def pair(shape, sink=False, production=False, dcoef=0.2, decay=0.0):
    held, values, uptake, ks, pr = problem(shape, sink, production)
    o = O.Field(*shape, dcoef, decay, 0.0)
    o.held[:], o.values[:], o.uptake[:] = held, values, uptake
    g = cw.ScalarField([shape], dcoef, decay, 0.0)
    g.set_held(held)
    g.set_values(values)
    g.set_uptake_array(uptake)
    if sink:
        o.lin_sink = ks.copy()
        g.set_linear_sink(ks)
    if production:
        o.production[:] = pr
        g.set_production_array(pr)
    return o, g


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("stop", [cw.STOP_MAX_CHANGE, cw.STOP_RESIDUAL])
def test_values_and_counts_are_the_oracles(shape, stop):
    o, g = pair(shape, decay=0.001)
    rc, sweeps = o.relax(1e-7, 3000, omega=1.8, stop=stop)
    assert rc == 0
    assert g.relax(1e-7, 3000, omega=1.8, stop=stop) == sweeps
    np.testing.assert_array_equal(bits(g.values()), bits(o.values))
    assert g.residual()[0] == o.residual()


@pytest.mark.parametrize("sink,production", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("shape", [(129, 67, 1), (33, 40, 21)])
def test_every_coefficient_array(shape, sink, production):
    o, g = pair(shape, sink, production, dcoef=1.0)
    rc, sweeps = o.relax(1e-8, 3000, omega=1.7)
    assert rc == 0
    st = g.relax(1e-8, 3000, omega=1.7, stats=True)[0]
    assert st["sweeps"] == sweeps and st["residual"] == o.residual()
    np.testing.assert_array_equal(bits(g.values()), bits(o.values))


@pytest.mark.parametrize("limit", [1, 2, 7, 8, 13])
@pytest.mark.parametrize("shape", [(301, 287, 1), (33, 40, 21)])
def test_a_solve_cut_short_leaves_the_oracles_field(shape, limit):
    o, g = pair(shape)
    assert o.relax(1e-12, limit, omega=1.9)[0] != 0
    with pytest.raises(cw.SimulationError) as e:
        g.relax(1e-12, limit, omega=1.9)
    assert e.value.stats[0]["sweeps"] == limit
    np.testing.assert_array_equal(bits(g.values()), bits(o.values))


def test_a_batch_of_uneven_histories_settles_each_by_itself():
    shapes = [(129, 67, 1), (16, 16, 1), (200, 90, 1), (4, 4, 1)]
    problems = [problem(s, False, False, seed=k) for k, s in enumerate(shapes)]
    problems[3][0][:] = 1  # nothing free
    g = cw.ScalarField(shapes, 0.2, 0.0, 0.0)
    for k, (held, values, uptake, _, _) in enumerate(problems):
        g.set_held(held, k)
        g.set_values(values, k)
        g.set_uptake_array(uptake, k)
    counts = g.relax(1e-8, 5000, omega=1.8)
    for k, (held, values, uptake, _, _) in enumerate(problems):
        o = O.Field(*shapes[k], 0.2, 0.0, 0.0)
        o.held[:], o.values[:], o.uptake[:] = held, values, uptake
        assert o.relax(1e-8, 5000, omega=1.8) == (0, counts[k])
        np.testing.assert_array_equal(bits(g.values(k)), bits(o.values))


def test_quotients_outside_the_corrected_range_are_divided():
    # values and sinks whose products leave 2^+-600 and denominators past
    # 2^200, beside ordinary ones; no floor
    shape = (40, 24, 1)
    o, g = pair(shape, sink=True)
    rng = np.random.default_rng(9)
    n = shape[0] * shape[1]
    v = o.values * 2.0 ** rng.choice([0, 0, 0, -1000, 700, -640], n)
    ks = o.lin_sink * 2.0 ** rng.choice([0, 0, 0, 230, -900], n)
    o.values[:], o.lin_sink = v, ks.copy()
    g.set_values(v)
    g.set_linear_sink(ks)
    o.relax(1e-9, 5, omega=1.2)
    with pytest.raises(cw.SimulationError):
        g.relax(1e-9, 5, omega=1.2)
    np.testing.assert_array_equal(bits(g.values()), bits(o.values))


def test_a_plane_too_large_for_the_chip_is_solved_by_launches():
    # a plane past what the device holds on chip takes the solve by launches
    shape = (1500, 1400, 1)
    o, g = pair(shape)
    o.relax(1e-9, 3, omega=1.9)
    before = _lib.lib().cw_launch_count()
    with pytest.raises(cw.SimulationError):
        g.relax(1e-9, 3, omega=1.9)
    assert _lib.lib().cw_launch_count() - before > 6
    np.testing.assert_array_equal(bits(g.values()), bits(o.values))
