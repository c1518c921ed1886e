"""The Delaunay finder's local search on a GB300 against the walk in double compiled for the host.

The local search keeps a cell's partners only where they are certain and hands
the others on (tecs/device/delaunay_local.cuh); whichever way a cell takes, its
row has to be that of the search of delaunay_star.cuh, pair by pair with the
multiplicities: cells on the hull and far from it, sets that are all hull,
boxes with too many points, two clusters far apart, lattices (five and more
points on a sphere), duplicates, flat sets, a handful of cells, and cutoffs
that take in many partners.
"""
import collections
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import tecs_gb300 as tg
from tecs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def host_search(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("dl") / "star"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT / 'include'}",
                    str(ROOT / "tests" / "cpp" / "delaunay_star_host.cpp"), "-o", str(out)], check=True)
    return out


def expected(binary, x, cutoff):
    n, dims = x.shape
    xx = np.zeros((n, 3), np.float32)
    xx[:, :dims] = x
    text = f"{n} {dims} {float(np.float32(cutoff))!r}\n" + "".join("%.9g %.9g %.9g\n" % tuple(r) for r in xx.tolist())
    lines = subprocess.run([str(binary)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    rows = (ln.split() for ln in lines if not ln.startswith(("err", "cellerr")))
    return {(int(a), int(b)): int(c) for a, b, c in rows}


def found(x, cutoff):
    n = len(x)
    pf = tg.PairFinderSettings(min_bounds=(-1e3,) * 3, max_bounds=(1e3,) * 3)
    s = tg.Simulation(tg.Settings(agent_count=n, capacity=n, cutoff_distance=cutoff, pair_finder_settings=pf),
                      dims=x.shape[1], pair_finder="delaunay", integrator="euler")
    s.set_state(x)
    return dict(collections.Counter(map(tuple, s.evaluate()[2].tolist())))


def inputs(kind, dims):
    rng = np.random.default_rng(21)
    if kind == "interior":
        x = wl.ball(6000, 4) if dims == 3 else wl.disk(6000, 4)
    elif kind == "shell":
        d = rng.normal(size=(900, dims))
        x = d / np.linalg.norm(d, axis=1)[:, None] * (9.0 + rng.normal(0, 0.05, (900, 1)))
    elif kind == "clusters":
        x = np.concatenate([rng.normal(0, 0.5, (500, dims)), rng.normal(0, 0.05, (300, dims)) + 30,
                            rng.random((200, dims)) * 40 - 20])
    elif kind == "lattice":
        x = np.stack(np.meshgrid(*[np.arange(8 if dims == 3 else 24)] * dims, indexing="ij"), -1).reshape(-1, dims) * 0.75
    elif kind == "near_lattice":
        x = np.stack(np.meshgrid(*[np.arange(9 if dims == 3 else 24)] * dims, indexing="ij"), -1).reshape(-1, dims) * 0.75
        x = x + rng.normal(0, 2e-4, x.shape)
    elif kind == "flat":
        x = rng.random((600, dims)) * 12
        x[:, -1] = 0.25
    elif kind == "duplicates":
        x = wl.ball(800, 6) if dims == 3 else wl.disk(800, 6)
        x[10], x[20], x[21] = x[11], x[22], x[22]
    elif kind == "far":
        x = (wl.ball(2000, 5) if dims == 3 else wl.disk(2000, 5)) + 150.0
    else:
        x = rng.random((int(kind), dims)) * 0.9
    return np.ascontiguousarray(x, np.float32)


KINDS = ["interior", "shell", "clusters", "lattice", "near_lattice", "flat", "duplicates", "far", "1", "2", "3", "4", "5",
         "9"]


@pytest.mark.parametrize("cutoff", [0.8, 1.7])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("kind", KINDS)
def test_rows_are_those_of_the_walk(host_search, kind, dims, cutoff):
    x = inputs(kind, dims)
    assert found(x, cutoff) == expected(host_search, x, cutoff)
