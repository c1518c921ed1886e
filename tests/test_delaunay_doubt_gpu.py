"""The Delaunay finder's local search on a GB300 where its verdicts are hard to reach, against the walk in double.

Rows have to be the host walk's (tests/cpp/delaunay_star_host.cpp), pair by
pair, whichever of the searches takes a cell: hull edges that carry cells
nearly on one line (faces too thin for a float normal), cells in other units
of length than about one cell a unit, and turned lattices, whose spheres hold
eight cells but for rounding.
"""
import numpy as np
import pytest

from tecs_gb300 import workloads as wl
from test_delaunay_local_gpu import expected, found, host_search  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


def box_with_edges(jitter):
    # a box of cells whose twelve edges carry thirty cells each, off the line by the jitter
    rng = np.random.default_rng(8)
    x = [rng.random((1500, 3)) * 9.8 + 0.1]
    for d in range(3):
        for c in range(4):
            e = np.zeros((30, 3))
            e[:, d] = np.sort(rng.random(30)) * 10
            e[:, (d + 1) % 3], e[:, (d + 2) % 3] = 10.0 * (c & 1), 10.0 * (c >> 1)
            x.append(e + rng.normal(0, jitter, e.shape))
    return np.concatenate(x).astype(np.float32)


@pytest.mark.parametrize("jitter", [1e-4, 1e-5, 3e-6, 1e-6])
def test_thin_hull_faces(host_search, jitter):  # noqa: F811
    x = box_with_edges(jitter)
    assert found(x, 1.0) == expected(host_search, x, 1.0)


def scaled(kind, unit):
    rng = np.random.default_rng(13)
    if kind == "ball":
        x = wl.ball(3000, 7)
    else:
        x = np.stack(np.meshgrid(*[np.arange(11)] * 3, indexing="ij"), -1).reshape(-1, 3) + rng.normal(0, 1e-3, (1331, 3))
    return (x * unit).astype(np.float32)


@pytest.mark.parametrize("unit", [1e-9, 1e-4, 1e-3, 1e3, 5e3, 1e6])
@pytest.mark.parametrize("kind", ["ball", "near_lattice"])
def test_units_of_length(host_search, kind, unit):  # noqa: F811
    x = scaled(kind, unit)
    cutoff = float(np.float32(1.3 * unit))
    rows = found(x, cutoff)
    assert rows == expected(host_search, x, cutoff)
    assert len(rows) > 3 * len(x)


@pytest.mark.parametrize("jitter", [0.0, 1e-7, 1e-5])
def test_turned_lattices(host_search, jitter):  # noqa: F811
    rng = np.random.default_rng(3)
    turn = np.linalg.qr(rng.normal(size=(3, 3)))[0]
    x = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3) + rng.normal(0, 1.0, (1000, 3)) * jitter
    x = (x @ turn.T).astype(np.float32)
    assert found(x, 1.2) == expected(host_search, x, 1.2)


@pytest.mark.parametrize("cutoff", [0.7, 1e3])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_a_few_cells(host_search, n, dims, cutoff):  # noqa: F811
    # walked all (up to six in space, eight in the plane) or searched first
    x = np.ascontiguousarray(wl.ball(n, 3)[:, :dims])
    assert found(x, cutoff) == expected(host_search, x, cutoff)


@pytest.mark.parametrize("n", [511, 512, 513, 700])
def test_sets_with_and_without_points_tested_first(host_search, n):  # noqa: F811
    # every cell in cutoff: all are walked, in the plane with a list of points
    # to test first past 512 cells
    x = wl.disk(n, 4)
    assert found(x, 1e3) == expected(host_search, x, 1e3)
