"""The launch fitted to a call (csrc/bgt_launch_fit.h), built for the host
(tests/launch_fit_check.cpp): a named placement is launched as given, and with
table_mode 0 the shape and the placement follow the sizes of the call.  148 SMs;
a table of 20 KB (the ideal ring) and of 150 KB (a ring with errors)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent / "launch_fit_check.cpp"
SMALL, LARGE, SMS = 20000, 150000, 148


@pytest.fixture(scope="module")
def fit(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("fit") / "launch_fit_check"
    subprocess.run([gxx, "-O1", "-std=c++17", "-o", str(exe), str(SRC)], check=True, capture_output=True)

    def run(threads, per_sm, mode, table, *groups, compact=0):
        r = subprocess.run([str(exe)] + [str(a) for a in (threads, per_sm, mode, table, compact) + groups],
                           capture_output=True, text=True, check=True, timeout=60)
        return tuple(int(x) for x in r.stdout.split())

    return run


@pytest.mark.parametrize("mode", [1, 2, 3])
@pytest.mark.parametrize("shape", [(256, 2), (256, 3), (128, 4), (64, 8)])
@pytest.mark.parametrize("table", [SMALL, LARGE])
@pytest.mark.parametrize("n", [1, 8064, 40000, 1000000])
def test_a_named_placement_is_launched_as_given(fit, mode, shape, table, n):
    assert fit(*shape, mode, table, n) == (*shape, mode)


@pytest.mark.parametrize("n, want", [
    (0, (128, 4, 0)), (1, (128, 4, 0)), (512 * SMS - 256, (128, 4, 0)),  # all tiles resident at once
    (512 * SMS - 255, (256, 2, 0)), (1000000, (256, 2, 0)),              # one wave or more
])
def test_small_table(fit, n, want):
    assert fit(256, 2, 0, SMALL, n) == want
    assert fit(128, 4, 0, SMALL, n) == (128, 4, 0)


@pytest.mark.parametrize("n, want", [
    (1, (128, 4, 0)), (128 * SMS, (128, 4, 0)),          # one CTA per SM, table staged
    (128 * SMS + 1, (256, 2, 0)), (256 * SMS, (256, 2, 0)),
    (256 * SMS + 1, (128, 4, 2)), (384 * SMS, (128, 4, 2)),
    (384 * SMS + 1, (256, 2, 2)), (1000000, (256, 2, 2)),
])
def test_large_table(fit, n, want):
    assert fit(256, 2, 0, LARGE, n) == want
    assert fit(128, 4, 0, LARGE, n) == (128, 4, 0 if n <= 128 * SMS else 2)


def test_tiles_are_counted_per_group(fit):
    assert fit(256, 2, 0, LARGE, *[1] * SMS) == (128, 4, 0)
    assert fit(256, 2, 0, LARGE, *[1] * (SMS + 1)) == (128, 4, 2)


def test_a_shape_without_a_global_instance_stays(fit):
    assert fit(64, 8, 0, LARGE, 1000000) == (64, 8, 0)
    assert fit(256, 4, 0, LARGE, 1000000) == (256, 4, 0)
    assert fit(256, 4, 0, LARGE, 100) == (128, 8, 0)


def test_the_compaction_stage_counts(fit):
    # three CTAs of 48 KB of table and 27 KB of memo fit 228 KB, with 9 KB of stage each two
    assert fit(128, 4, 0, 48000, 384 * SMS) == (128, 4, 0)
    assert fit(128, 4, 0, 48000, 384 * SMS, compact=1) == (128, 4, 2)
