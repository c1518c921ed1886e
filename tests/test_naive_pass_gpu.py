"""The naive finders' passes on a GB300 at the edges of their tiles, against the oracle.

Lanes take 32 candidates a round and four rounds at a time, and past 16,384
cells a warp takes four cells: pairs and deltas have to be the oracle's bit
for bit at sizes around each of these.  The naive Delaunay counts are checked
on inputs whose points-near-i list is short (a handful of cells), full
(a dense cluster beside far cells) and degenerate (a lattice, duplicates).
"""
import numpy as np
import pytest

import oracle
import tecs_gb300 as tg
from tecs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

FINDERS = {"naive_all_pairs": oracle.NAIVE_ALL_PAIRS, "naive_gabriel": oracle.NAIVE_GABRIEL,
           "naive_delaunay": oracle.NAIVE_DELAUNAY}


def both(x, finder, capacity=None):
    n, dims = x.shape
    cap = capacity or n
    pf = tg.PairFinderSettings(min_bounds=(-1e3,) * 3, max_bounds=(1e3,) * 3)
    s = tg.Simulation(tg.Settings(agent_count=n, capacity=cap, pair_finder_settings=pf), dims=dims,
                      pair_finder=finder, integrator="euler")
    o = oracle.Oracle(dims=dims, finder=FINDERS[finder], min_bounds=(-1e3,) * 3, max_bounds=(1e3,) * 3,
                      integrator=oracle.EULER, capacity=cap)
    s.set_state(x)
    o.set_state(x)
    return s, o


def same(x, finder, capacity=None):
    s, o = both(x, finder, capacity)
    d, _, pairs = s.evaluate()
    od, _, opairs = o.evaluate()
    np.testing.assert_array_equal(tg.canonical_pairs(pairs), tg.canonical_pairs(opairs))
    np.testing.assert_array_equal(d, od)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 257, 1025])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("finder", ["naive_all_pairs", "naive_gabriel"])
def test_tile_edges(n, dims, finder):
    same(wl.ball(n, 5) if dims == 3 else wl.disk(n, 5), finder, capacity=n + 7)


@pytest.mark.parametrize("n", [16_384, 16_387])
def test_cells_per_warp(n):
    same(wl.ball(n, 6), "naive_all_pairs")


def delaunay_input(kind):
    rng = np.random.default_rng(3)
    if kind == "five":
        return rng.random((5, 3)).astype(np.float32)
    if kind == "lattice":
        g = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.5
        return g.astype(np.float32)
    if kind == "cluster":  # 70 cells within a twentieth of the cutoff, and a few far away
        return np.concatenate([rng.random((70, 3)) * 0.05, rng.random((6, 3)) * 5 + 2]).astype(np.float32)
    x = wl.ball(61, 4)
    x[7] = x[8]
    return x


@pytest.mark.parametrize("kind", ["five", "lattice", "cluster", "duplicates"])
def test_naive_delaunay_counts(kind):
    same(delaunay_input(kind), "naive_delaunay")


def test_naive_delaunay_counts_2d():
    x = wl.disk(333, 8)
    x[10] = x[11]
    same(x, "naive_delaunay")
