"""The near-axis element maps (csrc/bgt_near.cuh) and the branch-free
quotients, square roots and transcendentals under them (csrc/bgt_fastmath.cuh),
built for the host (tests/near_maps_check.cpp).

Every result is compared for equality: the arithmetic with the IEEE square
root and quotient and with libquadmath rounded to double wherever the rounding
test holds (which it must for all but 1 in 1000 arguments), the maps with the
general maps on particles inside, at and outside the near-axis region, on
axis, past apertures and limits, for every record form that has a near-axis
form (multipole orders 0 to 7, offsets and roll, both apertures at both ends,
zero and negative lengths, edges at one end, bend angles up to the limit),
alone and with the drift that follows taken along.
"""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent / "near_maps_check.cpp"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("near") / "near_maps_check"
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-o", str(exe), str(SRC), "-lquadmath"],
                   check=True, capture_output=True)
    return exe


def run(checker, what, n, seed):
    r = subprocess.run([str(checker), what, str(n), str(seed)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    return [(f[0], int(f[1]), int(f[2]), int(f[3])) for f in (ln.split() for ln in r.stdout.splitlines())]


@pytest.mark.parametrize("seed", [1, 2])
def test_arithmetic_is_correctly_rounded(checker, seed):
    rows = run(checker, "math", 40000, seed)
    assert len(rows) == 9
    for name, bad, passed, total in rows:
        assert bad == 0, name
        assert passed >= 0.999 * total, name


@pytest.mark.parametrize("seed", [1, 2])
def test_near_axis_maps_equal_the_general_maps(checker, seed):
    rows = run(checker, "maps", 8000, seed)
    assert len(rows) == 82
    for name, bad, passed, total in rows:
        assert bad == 0, name
        assert 0.2 * total < passed < 0.9 * total, name  # both sides of the region's edge are covered
