"""The Delaunay finder's local search on a GB300 where its verdicts are hard to reach, against the walk in double.

Rows have to be the host walk's (tests/cpp/delaunay_star_host.cpp), pair by
pair, whichever of the searches takes a cell: hull edges that carry cells
nearly on one line (faces too thin for a float normal).
"""
import numpy as np
import pytest

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
