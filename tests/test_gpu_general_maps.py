"""Elements and particles without a near-axis form (csrc/bgt_kernel.cuh,
track_warp_turn): what they cost beside a drift, and that a particle's result
does not depend on the loop its neighbours in the warp are in."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import helpers
from bgt import lattice as L
from bgt import rings
from bgt.track import Tracker

pytestmark = pytest.mark.gpu


def line(els, n, name="line"):
    out = [els[k % len(els)].copy() for k in range(n)]
    return L.Lattice(out, L.Species("electron", L.M_ELECTRON, -1), rings.p0c(), rings.E_TOT, name).finalize()


def milliseconds(els, px=0.0, n=606208):
    v = rings.gaussian_beam(rings.CONFIG1_BEAM, n=n) * 0.1
    v[1] += px
    tr = Tracker(line(els, 64))
    b = tr.make_bunch(v)
    src = [torch.from_numpy(a).cuda() for a in (b.vec6, b.beta, b.state, b.ix_ele_lost, b.ix_turn_lost)]
    times = []
    for _ in range(5):
        d = [a.clone() for a in src]
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        e[0].record()
        tr.track_turns_device(*d, 1)
        e[1].record()
        e[1].synchronize()
        times.append(e[0].elapsed_time(e[1]))
    assert int((d[2] != 1).sum()) == 0
    return sorted(times)[2]


DRIFT = L.Element("drift", "D", {"l": 0.2})
QUADS = [L.Element("quadrupole", n, {"l": 0.1, "k1": k, "x_offset": 1e-5, "tilt": 1e-4}) for n, k in
         (("QF", 0.5), ("QD", -0.5))]


# The factors are half-way between these forms in a loop of general maps of
# their own and the same maps called out of line, where a call cost more than
# any of them: marker 0.7 (3.2), kicker 1.3 (3.9), monitor 1.2 (3.4), thin
# multipole 1.7 (3.8), misaligned quadrupole 2.4 (4.0), wide drift 1.5 (3.6).
@pytest.mark.parametrize("els, px, factor", [
    ([L.Element("marker", "M")], 0.0, 1.9),
    ([L.Element("hkicker", "K", {"l": 0.2, "kick": 1e-7})], 0.0, 2.5),
    ([L.Element("monitor", "B", {"l": 0.2})], 0.0, 2.3),
    ([L.Element("multipole", "T", {}, a_pole={2: 0.1})], 0.0, 2.7),
    (QUADS, 0.0, 3.2),
    ([DRIFT], 0.01, 2.5),
], ids=["marker", "kicker", "monitor", "multipole", "quads_misaligned", "drift_wide"])
def test_cost_beside_a_drift(els, px, factor):
    assert milliseconds(els, px) < factor * milliseconds([DRIFT])


def tracked(tr, v, with_time, turns):
    b = tr.make_bunch(v, with_time=with_time)
    tr.track_turns(b, turns)
    return [b.vec6.T, b.beta, b.state, b.ix_ele_lost, b.ix_turn_lost] + ([b.t.reshape(v.shape[1], -1)] if with_time else [])


@pytest.mark.parametrize("with_time", [False, True])
@pytest.mark.parametrize("ring", ["zoo", "rare_zoo", "cells"])
def test_results_do_not_depend_on_the_neighbours(ring, with_time):
    """Particles well inside the near-axis region, on its edge (2^-7), outside,
    with a large pz, and past apertures: dealt over the warps, and sorted by
    kind, so that the warps are of one kind each."""
    if ring == "cells":
        cell = [e for e in helpers.zoo_lattice().elements if e.name in ("Q0", "QERR", "S", "SERR", "B", "BE", "MK", "HK")]
        els = []
        for k, e in enumerate(cell + cell[::-1]):
            els += [e, L.Element("drift", "D%d" % k, {"l": 0.1 + 0.05 * (k % 3)})]
        lat = line(els, len(els), "cells")
    else:
        lat = helpers.zoo_lattice() if ring == "zoo" else helpers.rare_zoo_lattice()
    n, kinds = 640, 5
    rng = np.random.default_rng(5)
    v = rng.standard_normal((6, n)) * np.array([[1e-4], [2e-5], [1e-4], [2e-5], [1e-3], [1e-3]])
    kind = np.arange(n) % kinds
    v[1] += np.where(kind == 1, 2.0 ** -7 * rng.uniform(0.9, 1.1, n), 0)
    v[3] += np.where(kind == 2, 0.012, 0)
    v[5] += np.where(kind == 3, 0.2, 0)
    v[0] += np.where(kind == 4, rng.uniform(5e-3, 3e-2, n), 0)
    order = np.argsort(kind, kind="stable")
    tr = Tracker(lat)
    turns = 3 if ring == "cells" else 1
    dealt = tracked(tr, v.copy(), with_time, turns)
    by_kind = tracked(tr, np.ascontiguousarray(v[:, order]), with_time, turns)
    assert 0 < (dealt[2] == 1).sum() < n
    for a, b in zip(dealt, by_kind):
        assert np.array_equal(a[order], b, equal_nan=a.dtype.kind == "f")
