"""The margins of the Delaunay finder's local search (tecs/device/delaunay_local.cuh), on the CPU.

Its verdicts stand only where they are certain: each margin is compared here
with 64-bit arithmetic on inputs made to be doubtful
(tests/cpp/delaunay_margins_host.cpp includes the headers that the kernels do).
"""
import shutil
import subprocess
from pathlib import Path

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
