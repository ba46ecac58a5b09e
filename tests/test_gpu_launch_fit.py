"""The launch shape and table placement fitted to a call (bgt_track.cu,
fit_tuning): results do not depend on them.  Sizes around the rule's edges --
one CTA per SM, one full wave, one more -- with the small table of the ideal
ring and the 150 KB tables of error rings, against the shape taken as given
(64 threads with the table staged, which the rule never changes)."""
from __future__ import annotations

import numpy as np
import pytest

from bgt import rings
from bgt.track import Tracker

pytestmark = pytest.mark.gpu

SMS = 148


def tracked(tr, v0, variant, with_time=False, **tuning):
    tr.set_tuning(**tuning)
    b = tr.make_bunch(v0.copy(), with_time=with_time)
    tr.track_turns(b, 1, variant=variant)
    return b


def same(a, b):
    assert np.array_equal(a.state, b.state)
    assert np.array_equal(a.ix_ele_lost, b.ix_ele_lost) and np.array_equal(a.ix_turn_lost, b.ix_turn_lost)
    assert np.array_equal(a.vec6, b.vec6) and np.array_equal(a.beta, b.beta)
    if a.t is not None:
        assert np.array_equal(a.t, b.t)


@pytest.mark.parametrize("n", [1, 129, 128 * SMS, 128 * SMS + 1, 512 * SMS - 255, 512 * SMS + 1])
@pytest.mark.parametrize("rings_of", ["ideal", "errors"])
def test_results_do_not_depend_on_the_fitted_launch(n, rings_of):
    v0 = rings.gaussian_beam(rings.CONFIG1_BEAM, n=n)
    v0[:4] *= 3
    if rings_of == "ideal":
        tr, variant = Tracker(rings.fodo_ring(apertures=True)), None
    else:
        tr = Tracker(rings.error_variants(3))
        variant = np.sort(np.arange(n) * 7 % 3).astype(np.int32)
    want = tracked(tr, v0, variant, threads_per_block=64, blocks_per_sm=8, table_mode=1)
    for tuning in (dict(), dict(threads_per_block=256, blocks_per_sm=2),
                   dict(threads_per_block=256, blocks_per_sm=2, compact_every=1),
                   dict(threads_per_block=256, blocks_per_sm=2, table_mode=2),
                   dict(threads_per_block=256, blocks_per_sm=2, table_mode=3),
                   dict(threads_per_block=128, blocks_per_sm=5)):
        same(tracked(tr, v0, variant, **tuning), want)


def test_with_particle_times():
    v0 = rings.gaussian_beam(rings.CONFIG1_BEAM, n=300)
    tr = Tracker(rings.error_variants(1), absolute_time=True)
    want = tracked(tr, v0, None, True, threads_per_block=64, blocks_per_sm=8, table_mode=1)
    for tuning in (dict(), dict(threads_per_block=256, blocks_per_sm=2, compact_every=1)):
        same(tracked(tr, v0, None, True, **tuning), want)
