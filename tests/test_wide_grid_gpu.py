"""Binned Gabriel passes on a GB300 where float hardly resolves the bins, against the oracle.

Millions of bins a side, or coordinates millions of cutoffs from the origin: a
cutoff spans five to eleven positions there, midpoints are rounded by a good
part of it, and a witness may lie outside the cell's cutoff or two bins away.
The inputs are triples (a pair and a third cell within the ball around its
rounded midpoint), those kept for which one of the two is so; pairs and deltas
have to be the oracle's bit for bit.
"""
import numpy as np
import pytest

import oracle
import tecs_gb300 as tg

pytestmark = pytest.mark.gpu

F = np.float32


def triples(cutoff, lo, hi, keep, seed=4):
    """Triples spread along x over [lo, hi], at y about 1.5 cutoffs."""
    rng = np.random.default_rng(seed)
    cut, out, n = F(cutoff), [], 400_000
    while len(out) < keep:
        x0 = (lo + rng.random(n) * (hi - lo)).astype(F)
        y0 = np.full(n, 1.5 * cut, F)
        d = cut * (0.95 + 0.0499 * rng.random(n))
        th = np.arccos(0.4 + 0.6 * rng.random(n))
        x1 = (x0 + d * np.cos(th)).astype(F)
        y1 = (y0 + d * np.sin(th) * rng.choice([-1, 1], n)).astype(F)
        dx, dy = x0 - x1, y0 - y1
        d2 = dx * dx + dy * dy
        mx, my = x0 - dx * F(0.5), y0 - dy * F(0.5)
        rsq = d2 * F(F(0.9) * F(0.9) * F(0.25))
        a, r = rng.random(n) * 2 * np.pi, np.sqrt(rng.random(n) * rsq)
        x2, y2 = (mx + r * np.cos(a)).astype(F), (my + r * np.sin(a)).astype(F)
        ball = (x2 - mx) ** 2 + (y2 - my) ** 2 < rsq
        b = [np.floor((v - F(lo)) / cut) for v in (x0, x1, x2)]
        odd = (np.abs(b[2] - b[0]) > 1) | ((x0 - x2) ** 2 + (y0 - y2) ** 2 >= cut * cut)
        ok = np.nonzero(ball & odd & (d2 < cut * cut) & (np.abs(b[1] - b[0]) <= 1))[0]
        out += [np.array([[x0[q], y0[q]], [x1[q], y1[q]], [x2[q], y2[q]]], F) for q in ok]
    return np.concatenate(out[:keep])


@pytest.mark.parametrize("cutoff,lo,bins", [(0.7, -1453326.25, 1 << 21), (1.0, -4152361.0, 1 << 22), (1.0, 3.0e6, 600)])
def test_witnesses_out_of_the_cells_reach(cutoff, lo, bins):
    hi = lo + bins * cutoff
    x = triples(cutoff, lo + 2, lo + min(bins - 4, 40_000) * cutoff, keep=200)
    mn, mx = (lo, 0.0, 0.0), (hi, 3.0 * cutoff, cutoff)
    pf = tg.PairFinderSettings(min_bounds=mn, max_bounds=mx, gabriel_coefficient=0.9)
    s = tg.Simulation(tg.Settings(agent_count=len(x), capacity=len(x), cutoff_distance=cutoff, pair_finder_settings=pf),
                      dims=2, pair_finder="binned_gabriel", integrator="heun")
    o = oracle.Oracle(dims=2, finder=oracle.BINNED_GABRIEL, cutoff=cutoff, gabriel_coefficient=0.9,
                      min_bounds=mn, max_bounds=mx, integrator=oracle.HEUN, capacity=len(x))
    s.set_state(x)
    o.set_state(x)
    d, _, pairs = s.evaluate()
    od, _, opairs = o.evaluate()
    np.testing.assert_array_equal(tg.canonical_pairs(pairs), tg.canonical_pairs(opairs))
    np.testing.assert_array_equal(d, od)
