"""The cooperative pass of the binned finders at the limits of its lists (GB300).

From sparse to very dense cells: warps whose pairs fit the pool at once,
warps that take their cells in batches, lists of more than 32 candidates a
plane, and cells with more neighbours than the lists hold, which take the
general path.  Pairs, deltas and runs have to be the oracle's bit for bit, on
cubic grids and on grids one or two bins wide (the bin numbers are divided by
the extents).  The multi-simulation engine runs the same phases: its runs have
to be the plain ones.
"""
import numpy as np
import pytest

import oracle
import tecs_gb300 as tg
from tecs_gb300 import workloads as wl
from tecs_gb300.engine import Engine, bins_needed

pytestmark = pytest.mark.gpu

FINDERS = {"binned_all_pairs": oracle.BINNED_ALL_PAIRS, "binned_gabriel": oracle.BINNED_GABRIEL}


def cells(n, density, seed, dims=3):
    x = wl.ball(n, seed, wl.ball_radius(n, density)) if dims == 3 else wl.disk(n, seed, density)
    x[n // 2] = x[n // 3]  # two cells at one place
    return x


def both(x, finder, bounds=None, integrator="heun", pol=None):
    mn, mx = bounds or wl.bounds_for(x)
    pf = tg.PairFinderSettings(min_bounds=mn, max_bounds=mx)
    s = tg.Simulation(tg.Settings(agent_count=len(x), capacity=len(x), pair_finder_settings=pf), dims=x.shape[1],
                      pair_finder=finder, integrator=integrator)
    o = oracle.Oracle(dims=x.shape[1], finder=FINDERS[finder], min_bounds=mn, max_bounds=mx,
                      integrator=tg.INTEGRATORS[integrator], capacity=len(x))
    s.set_state(x)
    o.set_state(x)
    return s, o


def check(s, o, steps=2):
    d, _, pairs = s.evaluate()
    od, _, opairs = o.evaluate()
    np.testing.assert_array_equal(tg.canonical_pairs(pairs), tg.canonical_pairs(opairs))
    np.testing.assert_array_equal(d, od)
    s.take_step(0.01, steps)
    o.step(0.01, steps)
    np.testing.assert_array_equal(s.get_state()[0], o.get_state()[0])


@pytest.mark.parametrize("density", [0.2, 1.0, 2.4, 4.5, 9.0, 30.0])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("finder", list(FINDERS))
def test_densities(density, dims, finder):
    check(*both(cells(2017, density, 3, dims), finder))


@pytest.mark.parametrize("extents", [(1, 1, 1), (1, 2, 7), (2, 1, 3), (7, 2, 1), (3, 5, 2)])
@pytest.mark.parametrize("finder", list(FINDERS))
def test_narrow_grids(extents, finder):
    rng = np.random.default_rng(9)
    e = np.asarray(extents, np.float32)
    x = (rng.random((40 * int(np.prod(extents)), 3)).astype(np.float32) * (e + 1) - 0.5).astype(np.float32)
    check(*both(x, finder, ((0.0, 0.0, 0.0), tuple(float(v) for v in e))))


@pytest.mark.parametrize("finder", list(FINDERS))
def test_engine_runs_are_the_plain_ones(finder):
    states = [cells(n, density, 5) for n, density in ((900, 1.0), (77, 2.4), (1501, 4.5), (333, 12.0))]
    settings = []
    for x in states:
        mn, mx = wl.bounds_for(x)
        settings.append(tg.Settings(agent_count=len(x), capacity=len(x),
                                    pair_finder_settings=tg.PairFinderSettings(min_bounds=mn, max_bounds=mx)))
    descs = [tg.make_desc(s, pair_finder=finder, integrator="heun") for s in settings]
    eng = Engine(cell_capacity=sum(map(len, states)), bin_capacity=sum(bins_needed(d) for d in descs) + 64, max_sims=8)
    slots = [eng.add(d, x) for d, x in zip(descs, states)]
    eng.step(0.01, 3)
    for x, st, slot in zip(states, settings, slots):
        plain = tg.Simulation(st, pair_finder=finder, integrator="heun")
        plain.set_state(x)
        plain.take_step(0.01, 3)
        np.testing.assert_array_equal(eng.download(slot)[0], plain.get_state()[0])
    eng.close()


@pytest.mark.parametrize("n,density", [(1, 1.0), (2, 1.0), (31, 1.0), (700, 0.1), (1000, 1.0), (1000, 9.0), (1200, 60.0),
                                       (1535, 1.0), (1536, 2.4)])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("finder", list(FINDERS))
def test_small_steps(n, density, dims, finder):
    # one launch, a warp a cell: few and many cells a block, more candidates
    # than lanes, more neighbours than the list holds (the general path)
    x = cells(n, density, 11, dims) if n > 2 else wl.ball(n, 11)[:, :dims].copy()
    s, o = both(x, finder, integrator="euler")
    s.take_step(0.01, 3)
    o.step(0.01, 3)
    bins = np.prod([np.ceil(s.desc.max_bounds[k] - s.desc.min_bounds[k]) for k in range(dims)])
    assert (s.kernels_per_step() == 1) == (bins <= 16384)  # a sparse grid's steps go over the grid
    np.testing.assert_array_equal(s.get_state()[0], o.get_state()[0])
    check(s, o, steps=2)


def test_small_steps_in_several_launches_and_then_over_the_grid():
    # 300 steps are two launches; links then take the steps to the grid, whose
    # rebuild needs the bin counts that small steps do not make
    x = cells(600, 1.0, 12)
    s, o = both(x, "binned_gabriel", integrator="euler")
    s.take_step(0.01, 300)
    o.step(0.01, 300)
    np.testing.assert_array_equal(s.get_state()[0], o.get_state()[0])
    plain = tg.Simulation(tg.Settings(agent_count=600, capacity=601,  # (another capacity: another simulation)
                                      pair_finder_settings=tg.PairFinderSettings(
                                          min_bounds=tuple(s.desc.min_bounds), max_bounds=tuple(s.desc.max_bounds))),
                          integrator="euler")
    plain.set_state(s.get_state()[0])
    links = np.array([[0, 5], [7, 300], [599, 1]], np.uint32)
    for sim in (s, plain):
        sim.set_links(links, 0.3)
        sim.take_step(0.01, 2)
    assert s.kernels_per_step() > 1
    np.testing.assert_array_equal(s.get_state()[0], plain.get_state()[0])
    for sim in (s, plain):
        sim.set_links(np.zeros((0, 2), np.uint32), 0.0)
        sim.take_step(0.01, 2)
    assert s.kernels_per_step() == 1
    np.testing.assert_array_equal(s.get_state()[0], plain.get_state()[0])
