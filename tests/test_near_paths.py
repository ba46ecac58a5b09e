"""Which way particles take through a record (csrc/bgt_near.cuh,
track1_finish): the near-axis form in line, body_near, or the general maps --
and that each gives the general maps' values, time included, bit for bit.

Built for the host (tests/near_paths_check.cpp).  Particles well inside the
near-axis region, on axis, off momentum, of the smallest numbers, past
apertures, on the region's edges and outside; every record with the quadrupole
memo empty and filled, alone and with a following drift of ordinary, zero,
negative and large length.
"""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent / "near_paths_check.cpp"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("paths") / "near_paths_check"
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-o", str(exe), str(SRC), "-lquadmath"],
                   check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_every_way_through_a_record(checker, seed):
    r = subprocess.run([str(checker), "4500", str(seed)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    rows = [ln.split() for ln in r.stdout.splitlines()]
    assert len(rows) == 732 and {row[1] for row in rows} == {"plain", "time"}
    for name, kernel, *counts in rows:
        wrong, in_line, body, total = (int(c) for c in counts)
        assert wrong == 0, (name, kernel)
        form = name.split("+")[0]
        assert total == 2000
        if form == "quad_offset":  # no order above 1: the general map
            assert in_line == body == 0, (name, kernel)
            continue
        # a sextupole of the sextupole order alone is a plain one
        in_body = form.startswith(("quad_poles", "quad_mis", "sext_poles", "sext_mis")) and form != "sext_poles22"
        way, other = (body, in_line) if in_body else (in_line, body)
        assert other == 0, (name, kernel)
        if form.startswith("quad"):
            # the exact low-energy correction is the general map's: |pz| above
            # 0.054, two thirds of a quarter of the particles
            assert way > 0.79 * total, (name, kernel)
        elif form.startswith("bend"):
            # its 12 rounding tests, each of which may fail for 1 in 1000
            # arguments (test_near_maps.py), leave a particle to the general map
            assert way > 0.988 * total, (name, kernel)
        else:
            assert way == total, (name, kernel)
