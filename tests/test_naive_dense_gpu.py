"""The naive finders' passes on a GB300 with most cells in cutoff, against the oracle.

Rounds of 32 candidates with few and with many pairs are summed in different
loops, and past 32,768 cells a warp takes four cells: pairs and deltas have to
be the oracle's bit for bit where a cutoff takes in a handful of cells, some of
a round, and all of them, up to the places past the last cell of a warp.  The
polarity law's sums have to be the same with the cells behind one that is far
away, which puts them in other places of their rounds.
"""
import numpy as np
import pytest

import oracle
import tecs_gb300 as tg
from tecs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

FINDERS = {"naive_all_pairs": oracle.NAIVE_ALL_PAIRS, "naive_gabriel": oracle.NAIVE_GABRIEL,
           "naive_delaunay": oracle.NAIVE_DELAUNAY}
BOX = dict(min_bounds=(-1e3,) * 3, max_bounds=(1e3,) * 3)


def cells(n, dims):
    x = wl.ball(n, 9) if dims == 3 else wl.disk(n, 9)
    if n > 40:
        x[n // 2] = x[n // 3]  # two cells at one place
    return x


def sim(x, finder, cutoff, **kw):
    n = len(x)
    return tg.Simulation(tg.Settings(agent_count=n, capacity=n, cutoff_distance=cutoff,
                                     pair_finder_settings=tg.PairFinderSettings(**BOX)),
                         dims=x.shape[1], pair_finder=finder, integrator="euler", **kw)


def same(x, finder, cutoff, pairs=True):
    s = sim(x, finder, cutoff)
    o = oracle.Oracle(dims=x.shape[1], finder=FINDERS[finder], cutoff=cutoff, integrator=oracle.EULER, capacity=len(x), **BOX)
    s.set_state(x)
    o.set_state(x)
    if pairs:
        d, _, p = s.evaluate()
        od, _, op = o.evaluate()
        np.testing.assert_array_equal(tg.canonical_pairs(p), tg.canonical_pairs(op))
        np.testing.assert_array_equal(d, od)
    else:
        s.take_step(0.01, 1)
        o.step(0.01, 1)
        np.testing.assert_array_equal(s.get_state()[0], o.get_state()[0])


@pytest.mark.parametrize("cutoff", [1.7, 4.0, 1e6])
@pytest.mark.parametrize("n", [2, 33, 129, 700])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("finder", ["naive_all_pairs", "naive_gabriel"])
def test_pairs_of_every_density(finder, dims, n, cutoff):
    same(cells(n, dims), finder, cutoff)


@pytest.mark.parametrize("n,cutoff", [(32_768, 1.2), (32_769, 1.2), (32_771, 3.0)])
@pytest.mark.parametrize("dims", [2, 3])
def test_four_cells_a_warp(dims, n, cutoff):
    same(cells(n, dims), "naive_all_pairs", cutoff, pairs=cutoff < 2)


def test_four_cells_a_warp_all_in_cutoff():
    same(cells(32_770, 3), "naive_all_pairs", 1e6, pairs=False)


@pytest.mark.parametrize("n", [1, 3, 17_001])
@pytest.mark.parametrize("dims", [2, 3])
def test_gabriel_sizes(dims, n):
    same(cells(n, dims), "naive_gabriel", 1.0)


@pytest.mark.parametrize("dims", [2, 3])
def test_delaunay_counts_with_every_cell_in_cutoff(dims):
    same(cells(40, dims), "naive_delaunay", 1e6)


@pytest.mark.parametrize("n,capacity", [(1, 1), (3, 3), (5, 9), (8, 8), (8, 9), (9, 9), (41, 41), (40, 43), (64, 64)])
@pytest.mark.parametrize("dims", [2, 3])
def test_delaunay_table_of_half_words(dims, n, capacity):
    # rows that start at either half of a word, up to 8 cells written by one
    # block each, and a second evaluation that finds the first one's counts
    x = cells(n, dims)
    s = tg.Simulation(tg.Settings(agent_count=n, capacity=capacity, cutoff_distance=1.5,
                                  pair_finder_settings=tg.PairFinderSettings(**BOX)),
                      dims=dims, pair_finder="naive_delaunay", integrator="euler")
    o = oracle.Oracle(dims=dims, finder=oracle.NAIVE_DELAUNAY, cutoff=1.5, integrator=oracle.EULER, capacity=capacity, **BOX)
    s.set_state(x)
    o.set_state(x)
    for _ in range(2):
        d, _, p = s.evaluate()
        od, _, op = o.evaluate()
        np.testing.assert_array_equal(tg.canonical_pairs(p), tg.canonical_pairs(op))
        np.testing.assert_array_equal(d, od)


def test_delaunay_table_takes_two_bytes_a_pair():
    import torch

    sim(cells(64, 3), "naive_delaunay", 1.0).close()
    before = torch.cuda.mem_get_info()[0]
    s = sim(np.zeros((4096, 3), np.float32), "naive_delaunay", 1.0)
    used = before - torch.cuda.mem_get_info()[0]
    s.close()
    # 33.6 MB, the cells' arrays (about 200 bytes each) and 2 MB pages; at four bytes 67 MB
    assert used < 4096 * 4096 * 2 + (16 << 20)


@pytest.mark.parametrize("cutoff", [1.5, 50.0])
@pytest.mark.parametrize("n", [40, 321])
def test_polarity_sums_do_not_depend_on_the_place_in_a_round(n, cutoff):
    x = wl.ball(n, 9)
    p = np.random.default_rng(2).random((n, 2)).astype(np.float32) * 2 + np.float32(0.3)
    out = []
    for before in (0, 1, 19):
        far = np.full((before, 3), 500.0, np.float32) + np.arange(before, dtype=np.float32)[:, None] * 60
        s = sim(np.concatenate([far, x]), "naive_all_pairs", cutoff, force=tg.PolaritySpring(k_pol=0.2), polarity=True)
        s.set_state(np.concatenate([far, x]), np.concatenate([np.ones((before, 2), np.float32), p]))
        dx, dp, _ = s.evaluate()
        out.append((dx[before:], dp[before:]))
    for dx, dp in out[1:]:
        np.testing.assert_array_equal(dx, out[0][0])
        np.testing.assert_array_equal(dp, out[0][1])
