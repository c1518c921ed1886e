"""The margins of the Delaunay finder's local search (tecs/device/delaunay_local.cuh), on the CPU.

Its verdicts stand only where they are certain: each margin is compared here
with 64-bit arithmetic on inputs made to be doubtful
(tests/cpp/delaunay_margins_host.cpp includes the headers that the kernels do).
"""
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def margins(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("dl") / "margins"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-ffp-contract=off",
                    f"-I{ROOT / 'include'}", str(ROOT / "tests" / "cpp" / "delaunay_margins_host.cpp"), "-o", str(out)],
                   check=True)
    return lambda what: [ln.split() for ln in subprocess.run([str(out), what], capture_output=True, text=True,
                                                             check=True).stdout.splitlines()]


def test_rows_of_an_open_face_hold_its_open_side(margins):
    # two cells nearly on one line with the third: no cell on the open side
    # may be left out, and only faces thinner than 1e-5 may be refused
    for angle, faces, refused, points, missed in margins("normals"):
        assert int(missed) == 0, (angle, missed)
        assert int(faces) == 60 and (int(points) > 0 or int(refused) == 60)
        assert int(refused) == 0 or float(angle) < 1e-4


def test_a_line_called_without_rest_has_none(margins):
    # near-ties and lines far from the cell: nothing certain may be wrong in
    # more bits, in any unit of length; one that is a power of two changes no
    # verdict (but for lines too short to be formed); among random cells next
    # to nothing is looked at in double (the set of 1e-6 jitter has exact ties)
    rows = [(int(s), float(u)) + tuple(map(int, c)) for s, u, *c in margins("lines")]
    assert len(rows) == 30
    for s, unit, none, again, doubtful, wrong in rows:
        assert none > 1000 and wrong == 0, (s, unit, wrong)
        same = next(r for r in rows if r[0] == s and r[1] == 1.0)
        if unit == 1024.0 or (unit == 1.0 / 8192.0 and s != 3):
            assert (none, again, doubtful) == same[2:5]
        assert s > 0 or (doubtful <= again < 0.01 * none), (s, unit, again, doubtful, none)


def sphere(p):
    """The fifth point's power in the sphere of the first four, and (|a| |b| |c| / det)^2, exactly (None: no sphere)."""
    v = [[Fraction(float(np.float32(p[3 * k + d]))) - Fraction(float(np.float32(p[d]))) for d in range(3)] for k in range(1, 5)]
    h = [sum(c * c for c in u) for u in v]
    a, b, c, e = v

    def cross(s, t):
        return [s[1] * t[2] - s[2] * t[1], s[2] * t[0] - s[0] * t[2], s[0] * t[1] - s[1] * t[0]]

    bc, ca, ab = cross(b, c), cross(c, a), cross(a, b)
    det = sum(s * t for s, t in zip(a, bc))
    if det == 0:
        return None, None
    x2 = [(h[0] * bc[d] + h[1] * ca[d] + h[2] * ab[d]) / det for d in range(3)]
    return h[3] - sum(s * t for s, t in zip(x2, e)), h[0] * h[1] * h[2] / det ** 2


def test_a_point_called_outside_of_a_sphere_is(margins):
    # ... and only spheres of a thinness past 10^6 are refused (its square is
    # formed in double, off by far less than a tenth there)
    certain = 0
    for refused, outside, *p in margins("spheres"):
        if refused == "1" or outside == "1":
            pw, thin2 = sphere([float(c) for c in p])
            assert pw > 0 if refused == "0" else (thin2 is None or thin2 > 0.9e12), p
            certain += refused == "0"
    assert certain > 1500
