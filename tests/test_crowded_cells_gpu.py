"""Cells with many neighbours and the polarity law on a GB300, one path against another.

Cells among many candidates with few of them in cutoff, against the oracle.
Densities at which a warp's pairs fill the pool several times (about 4.5
cells a unit volume), lists overflow into the general path (9 and 30) and the
small steps' lists do (64 neighbours).  Runs have to be bit-identical: small
steps to the same steps over the grid, the cooperative Gabriel pass to the
general path (which a grid more than 2^18 bins wide takes, with the cells in
the same bins and order), and the multi-simulation engine to the plain pass.
All-pairs with the polarity law is compared with 64-bit arithmetic: a pair is
within 1e-5 of its value and 1e-6 of the largest pair (test_polarity_law_gpu),
n of them and their sum within n times that.
"""
import os

import numpy as np
import pytest

import oracle
import tecs_gb300 as tg
from tecs_gb300 import workloads as wl
from tecs_gb300.engine import Engine, bins_needed
from test_polarity_law_gpu import pair_f64

pytestmark = pytest.mark.gpu

FORCES = {"none": lambda: None, "spring": tg.Spring2R, "polarity": lambda: tg.PolaritySpring(k_pol=0.2)}


def cells(n, density, dims=3, seed=3):
    return wl.ball(n, seed, wl.ball_radius(n, density)) if dims == 3 else wl.disk(n, seed, density)


def polarity(n, seed=5):
    rng = np.random.default_rng(seed)
    return np.stack([rng.random(n) * 2.6 + 0.2, rng.random(n) * 6 - 3], 1).astype(np.float32)


def sim(x, finder, integrator, force, p=None, bounds=None):
    mn, mx = bounds or wl.bounds_for(x)
    pf = tg.PairFinderSettings(min_bounds=mn, max_bounds=mx)
    s = tg.Simulation(tg.Settings(agent_count=len(x), capacity=len(x), pair_finder_settings=pf), dims=x.shape[1],
                      pair_finder=finder, integrator=integrator, force=FORCES[force](), polarity=p is not None)
    s.set_state(x, p)
    return s


def same_state(a, b):
    for u, v in zip(a.get_state(), b.get_state()):
        np.testing.assert_array_equal(u, v)


@pytest.mark.parametrize("n,density", [(1000, 4.5), (1200, 9.0), (1536, 30.0), (400, 1e6)])
@pytest.mark.parametrize("dims,force", [(3, "spring"), (2, "spring"), (3, "polarity"), (2, "none"), (3, "none")])
@pytest.mark.parametrize("finder", ["binned_all_pairs", "binned_gabriel"])
def test_small_steps(finder, dims, force, n, density):
    x = cells(n, density, dims)
    p = polarity(n) if force == "polarity" else None
    if p is None:
        x[n // 2] = x[n // 3]  # two cells at one place (the polarity law divides by the distance)
    a = sim(x, finder, "euler", force, p)
    os.environ["TECS_NO_SMALL_STEP"] = "1"
    try:
        b = sim(x, finder, "euler", force, p)
    finally:
        os.environ.pop("TECS_NO_SMALL_STEP")
    for s in (a, b):
        s.take_step(1e-4, 35)  # two launches
    assert a.kernels_per_step() == 1 < b.kernels_per_step()
    same_state(a, b)


@pytest.mark.parametrize("density", [0.5, 4.5, 9.0, 30.0])
def test_gabriel_polarity_pass_is_the_general_path(density):
    x, p = cells(2017, density), polarity(2017)
    mn, mx = wl.bounds_for(x)
    a = sim(x, "binned_gabriel", "heun", "polarity", p)
    b = sim(x, "binned_gabriel", "heun", "polarity", p, (mn, (mn[0] + float((1 << 18) + 64), mx[1], mx[2])))
    da, db = a.evaluate(), b.evaluate()
    np.testing.assert_array_equal(da[0], db[0])
    np.testing.assert_array_equal(da[1], db[1])
    np.testing.assert_array_equal(tg.canonical_pairs(da[2]), tg.canonical_pairs(db[2]))
    for s in (a, b):
        s.take_step(0.01, 2)
    same_state(a, b)


@pytest.mark.parametrize("density", [4.5, 30.0])
def test_all_pairs_polarity_pass(density):
    n = 333
    x, p = cells(n, density), polarity(n)
    force = tg.PolaritySpring(k_rep=2.0, r_rep=0.7, k_adh=0.5, r_adh=0.8, k_pol=0.2)
    mn, mx = wl.bounds_for(x)
    s = tg.Simulation(tg.Settings(agent_count=n, capacity=n, pair_finder_settings=tg.PairFinderSettings(
        min_bounds=mn, max_bounds=mx)), pair_finder="binned_all_pairs", integrator="euler", force=force, polarity=True)
    s.set_state(x, p)
    dx, dp, pairs = s.evaluate()
    ex, ep, tol = np.zeros((n, 3)), np.zeros((n, 2)), np.zeros((n, 1))
    xf, pf = x.astype(np.float64), p.astype(np.float64)
    for i, j in np.asarray(pairs).tolist():
        fx, fp = pair_f64(xf[i], xf[j], tuple(pf[i]), tuple(pf[j]))
        ex[i] += fx
        ep[i] += fp
        big = max(np.abs(fx).max(), np.abs(fp).max(), 0.2)
        tol[i] = np.maximum(tol[i], 1.1e-5 * big)
    count = np.bincount(np.asarray(pairs)[:, 0], minlength=n)[:, None]
    d = np.linalg.norm(xf[:, None] - xf[None], axis=-1)
    assert count.sum() == (d < 1.0).sum() - n and count.max() > (24 if density > 9 else 12)
    assert (np.abs(dx - ex) <= count * tol).all() and (np.abs(dp - ep) <= count * tol).all()


@pytest.mark.parametrize("finder", ["binned_all_pairs", "binned_gabriel"])
def test_engine_polarity_runs_are_the_plain_ones(finder):
    states = [(cells(n, density, seed=7), polarity(n)) for n, density in ((900, 1.0), (700, 4.5), (501, 9.0), (333, 30.0))]
    settings = []
    for x, _ in states:
        mn, mx = wl.bounds_for(x)
        settings.append(tg.Settings(agent_count=len(x), capacity=len(x),
                                    pair_finder_settings=tg.PairFinderSettings(min_bounds=mn, max_bounds=mx)))
    force = FORCES["polarity"]()
    descs = [tg.make_desc(s, pair_finder=finder, integrator="heun", force=force, polarity=True) for s in settings]
    eng = Engine(cell_capacity=sum(len(x) for x, _ in states), bin_capacity=sum(bins_needed(d) for d in descs) + 64,
                 max_sims=8)
    slots = [eng.add(d, x, p) for d, (x, p) in zip(descs, states)]
    eng.step(0.002, 3)
    for (x, p), st, slot in zip(states, settings, slots):
        plain = tg.Simulation(st, pair_finder=finder, integrator="heun", force=force, polarity=True)
        plain.set_state(x, p)
        plain.take_step(0.002, 3)
        xe, pe = eng.download(slot)
        xp, pp = plain.get_state()
        np.testing.assert_array_equal(xe, xp)
        np.testing.assert_array_equal(pe, pp)
    eng.close()


@pytest.mark.parametrize("clump", [70, 80, 170, 190, 700])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("finder", ["binned_all_pairs", "binned_gabriel"])
def test_lone_cells_beside_a_clump(finder, dims, clump):
    # a clump in the corner of one bin: the cells of the bins around it have it
    # among their candidates, out of cutoff for most
    rng = np.random.default_rng(6)
    x = np.concatenate([rng.random((clump, dims)) * 0.1, rng.random((60, dims)) * 4]).astype(np.float32)
    box = dict(min_bounds=(0.0,) * 3, max_bounds=(4.0,) * 3)
    s = tg.Simulation(tg.Settings(agent_count=len(x), capacity=len(x), pair_finder_settings=tg.PairFinderSettings(**box)),
                      dims=dims, pair_finder=finder, integrator="heun")
    o = oracle.Oracle(dims=dims, finder=getattr(oracle, finder.upper()), integrator=oracle.HEUN, capacity=len(x), **box)
    s.set_state(x)
    o.set_state(x)
    d, _, pairs = s.evaluate()
    od, _, opairs = o.evaluate()
    np.testing.assert_array_equal(tg.canonical_pairs(pairs), tg.canonical_pairs(opairs))
    np.testing.assert_array_equal(d, od)
    s.take_step(0.001, 2)
    o.step(0.001, 2)
    np.testing.assert_array_equal(s.get_state()[0], o.get_state()[0])


def test_engine_of_crowded_bins_runs_are_the_plain_ones():
    # more than 1.2 resident cells a bin take another instance of the pass; a
    # large sparse simulation that joins takes the engine back
    xs = [cells(n, density, seed=8) for n, density in ((2000, 30.0), (1500, 20.0), (900, 0.2))]
    settings = []
    for x in xs:
        mn, mx = wl.bounds_for(x)
        settings.append(tg.Settings(agent_count=len(x), capacity=len(x),
                                    pair_finder_settings=tg.PairFinderSettings(min_bounds=mn, max_bounds=mx)))
    descs = [tg.make_desc(s, pair_finder=f, integrator="heun") for s, f in
             zip(settings, ("binned_gabriel", "binned_all_pairs", "binned_gabriel"))]
    bins = [bins_needed(d) for d in descs]
    assert 3500 > 1.2 * sum(bins[:2]) and 4400 < 1.2 * sum(bins)
    eng = Engine(cell_capacity=4400, bin_capacity=sum(bins) + 64, max_sims=4)
    slots = [eng.add(d, x) for d, x in zip(descs[:2], xs)]
    eng.step(1e-4, 2)
    slots.append(eng.add(descs[2], xs[2]))
    eng.step(1e-4, 2)
    for x, st, f, slot, steps in zip(xs, settings, ("binned_gabriel", "binned_all_pairs", "binned_gabriel"), slots, (4, 4, 2)):
        plain = tg.Simulation(st, pair_finder=f, integrator="heun")
        plain.set_state(x)
        plain.take_step(1e-4, steps)
        np.testing.assert_array_equal(eng.download(slot)[0], plain.get_state()[0])
    eng.close()
