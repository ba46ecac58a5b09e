"""Performance cases of the tracker and of its survival classifier.

What a user of this package has it do, through its public entry points: track
a bunch through one element or around the ring, from host or device buffers;
find the closed orbit and optics of error rings; scan their dynamic aperture;
track with particle times (absolute-time RF); and train and run the classifier
that prunes those scans.  Ring, beams, errors and grids are those of
``bgt.rings``, at sizes from a handful of particles to the 1M-particle beam.

``exact`` restates the ring in plain torch FP64 (the same physics, none of the
package's code), and the classifier in FP64 from its FP32 parameters.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "bmad-ecosystem_b200"))

# the FODO ring of bgt.rings, in numbers (used by `exact` and the errors)
N_CELL, ANGLE = 64, 2 * math.pi / 128
K1, K2_SF, K2_SD = 0.8, 3.51108791627275, -5.132216700784618
E_TOT, MC2, C_LIGHT = 5e9, 0.51099895069e6, 2.99792458e8
HARMONIC, RF_VOLTAGE = 748, 5e6
TWISS = dict(ba=11.887244599751257, aa=-1.8074579900510381, bb=3.7441933691886216, ab=0.47324178195194055,
             ex=0.7913233223685988, epx=0.127872130259893)
N_FEATURES, N_IN, HIDDEN, N_PARAMS = 30, 64, 256, 148481
# FP64 operations per particle and turn: the ideal ring, an error ring
FLOPS_IDEAL, FLOPS_ERRORS = 98807, 902775


def listed():
    return [
        # track1: a few particles through one element, as a host program's own tracking loop calls it
        dict(name="track1_bend", kind="element", element="sbend", n=101),
        # closed orbit, Twiss and dispersion of error rings: 19 probes a ring, launch and turn latency
        dict(name="optics", kind="optics", variants=5),
        # the 10,000-particle beam on the ring without apertures, host buffers
        dict(name="bunch_10k_host", kind="host", n=10000, turns=16, apertures=False, shape=0),
        # a large odd-sized bunch for one turn, host buffers: the copies are part of the call
        dict(name="bunch_300k_host", kind="host", n=300001, turns=1, apertures=True, shape=256),
        # the 1M-particle beam on the ring with apertures, device buffers, the benchmark's launch shape
        dict(name="bunch_1M_device", kind="device", n=1000000, turns=2, apertures=True, shape=256),
        # bunches on rings with misaligned, rolled magnets and multipole errors (16 kicks a quadrupole)
        dict(name="error_rings", kind="errors", n=60000, variants=6, turns=1, shape=0),
        # dynamic-aperture scan of error rings: most probes are lost early, the rest live on
        dict(name="da_scan", kind="da", variants=4, deltas=3, angles=21, radii=32, turns=24, shape=256),
        # absolute-time RF with binary128 particle times (the dynamic-aperture program's setting)
        dict(name="absolute_time", kind="time", n=40000, turns=1),
        # classifier inputs of a large scan's surviving probes
        dict(name="features", kind="features", n=500001, variants=128, raw=False),
        # classifier on a whole scan's probes, and on one ring's
        dict(name="classify_262k", kind="forward", n=262144),
        dict(name="classify_1k", kind="forward", n=1152),
        # one epoch of training: shuffled batches of forward, backward and Adam
        dict(name="fit", kind="fit", n=40960, batch=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["element", "optics", "host", "device", "errors", "da", "time", "features", "forward", "fit",
                       "gradients"])
    if kind == "element":
        el = rng.choice(["sbend", "quadrupole", "sextupole", "drift", "rfcavity"])
        return dict(kind=kind, element=el, n=_log(rng, 1, 20000))
    if kind == "optics":
        return dict(kind=kind, variants=rng.randint(1, 12))
    if kind in ("host", "device"):
        n = _log(rng, 200, 1000000 if kind == "device" else 300000)
        turns = max(1, min(_log(rng, 1, 40), 2000000 // n, 24))
        return dict(kind=kind, n=n, turns=turns, apertures=rng.random() < 0.6, shape=rng.choice([0, 128, 256]))
    if kind == "errors":
        nv = rng.randint(1, 10)
        return dict(kind=kind, n=max(nv, _log(rng, 300, 100000)), variants=nv, turns=1, shape=rng.choice([0, 256]))
    if kind == "da":
        return dict(kind=kind, variants=rng.randint(1, 4), deltas=rng.choice([1, 3]), angles=rng.randint(1, 24),
                    radii=rng.randint(9, 40), turns=rng.randint(2, 24), shape=rng.choice([0, 256]))
    if kind == "time":
        return dict(kind=kind, n=_log(rng, 100, 40000), turns=1)
    if kind == "features":
        return dict(kind=kind, n=_log(rng, 1000, 1000000), variants=rng.randint(1, 256), raw=rng.random() < 0.3)
    if kind == "forward":
        return dict(kind=kind, n=128 * _log(rng, 1, 2048))
    if kind == "gradients":
        return dict(kind=kind, n=128 * _log(rng, 1, 64))
    batch = 128 * rng.choice([8, 16, 32, 64])
    return dict(kind=kind, n=batch * rng.randint(1, 5) + rng.randint(0, 1000), batch=batch)


# ---------------------------------------------------------------------------
# inputs

def _rng(case, seed):
    return np.random.default_rng([seed, case["n"] if "n" in case else case["variants"]])


def _beam(case, seed):
    """A matched Gaussian beam at three times the design emittances."""
    n, t = case["n"], TWISS
    u = _rng(case, seed).standard_normal((6, n))
    v = np.zeros((6, n))
    v[5] = 1e-3 * math.sqrt(3) * u[5]
    v[4] = 3e-3 * math.sqrt(3) * u[4]
    v[0] = math.sqrt(3e-9 * t["ba"]) * u[0] + t["ex"] * v[5]
    v[1] = math.sqrt(3e-9 / t["ba"]) * (u[1] - t["aa"] * u[0]) + t["epx"] * v[5]
    v[2] = math.sqrt(3e-11 * t["bb"]) * u[2]
    v[3] = math.sqrt(3e-11 / t["bb"]) * (u[3] - t["ab"] * u[2])
    return v


def _errors(case, seed):
    """Per variant and magnet (128 quadrupoles, 128 sextupoles, interleaved):
    x and y offset, roll, a_3..a_6, b_3..b_6."""
    r = np.random.default_rng([seed, 7, case["variants"]])
    e = np.clip(r.standard_normal((case["variants"], 256, 11)), -3, 3)
    return e * np.array([50e-6, 50e-6, 100e-6] + [1e-4] * 8)


def _error_rings(case, seed):
    from bgt import rings

    out = []
    for ev in _errors(case, seed):
        lat = rings.fodo_ring(apertures=True)
        for e, row in zip([e for e in lat.elements if e.key in ("quadrupole", "sextupole")], ev):
            e.values.update(x_offset=float(row[0]), y_offset=float(row[1]), tilt=float(row[2]), r0_mag=0.01)
            e.a_pole = {k: float(row[k]) for k in range(3, 7)}
            e.b_pole = {k: float(row[k + 4]) for k in range(3, 7)}
            e.num_steps = 0
            e.values.pop("ds_step", None)
        out.append(lat.finalize())
    return out


def _tuning(case):
    return {256: dict(threads_per_block=256, blocks_per_sm=2),
            128: dict(threads_per_block=128, blocks_per_sm=4)}.get(case["shape"])


def _device_bunch(tr, v):
    b = tr.make_bunch(v)
    return [torch.from_numpy(a).cuda() for a in (b.vec6, b.beta, b.state, b.ix_ele_lost, b.ix_turn_lost)], b


def _variant_ids(case):
    """Particles dealt to the variants in contiguous, uneven groups."""
    n, nv = case["n"], case["variants"]
    edges = [round(n * (k / nv) ** 1.2) for k in range(nv + 1)]
    return np.repeat(np.arange(nv, dtype=np.int32), np.diff(edges))


def _mlp_params(seed):
    r = np.random.default_rng([seed, 11])
    p = np.zeros(N_PARAMS, np.float32)
    o = 0
    for rows, cols, used in ((HIDDEN, N_IN, N_FEATURES), (HIDDEN, HIDDEN, HIDDEN), (HIDDEN, HIDDEN, HIDDEN),
                             (1, HIDDEN, HIDDEN)):
        w = np.zeros((rows, cols), np.float32)
        w[:, :used] = r.uniform(-1, 1, (rows, used)) * math.sqrt(6.0 / used)
        p[o:o + w.size] = w.ravel()
        o += w.size
        p[o:o + rows] = 0.05 * r.standard_normal(rows)
        o += rows
    return p


def _mlp_inputs(case, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    x = torch.zeros((case["n"], N_IN), dtype=torch.bfloat16)
    x[:, :N_FEATURES] = torch.randn((case["n"], N_FEATURES), generator=g).clamp(-4, 4)
    y = (torch.rand(case["n"], generator=g) < torch.sigmoid(2 * x[:, 0].float() - 1)).float()
    return x, y


def _feature_inputs(case, seed):
    v0 = _beam(case, seed)
    v1 = _beam(case, seed + 1000003)
    r = np.random.default_rng([seed, 13])
    t = np.concatenate([1e-5 * r.standard_normal((case["variants"], 6)), 0.1 * r.standard_normal((case["variants"], 4)),
                        np.tile([TWISS["ba"], TWISS["aa"], TWISS["bb"], TWISS["ab"]], (case["variants"], 1)),
                        np.abs(1 + 0.2 * r.standard_normal((case["variants"], 16)))], axis=1)
    var = np.sort(r.integers(0, case["variants"], case["n"])).astype(np.int32)
    mean = 1e-3 * r.standard_normal(N_FEATURES)
    std = np.concatenate([np.full(6, 1e-3), np.full(16, 0.3), np.full(6, 1e-3), np.full(2, 1e-4)])
    return v0, v1, t, var, mean, std


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind in ("element", "host", "device", "time"):
        from bgt import rings
        from bgt.track import Tracker

        lat = rings.fodo_ring(apertures=case.get("apertures", True))
        s["tr"] = Tracker(lat, tuning=_tuning(case) if "shape" in case else None, absolute_time=kind == "time")
        v = _beam(case, seed)
        if kind == "element":
            s["pos"] = [e.key for e in lat.elements].index(case["element"])
        if kind in ("element", "host"):
            s["bunch"] = s["tr"].make_bunch(v)
        else:
            s["dev"], b = _device_bunch(s["tr"], v)
            s["t"] = torch.from_numpy(b.t.view(np.int64)).cuda() if kind == "time" else None
    elif kind in ("optics", "errors", "da"):
        from bgt import da
        from bgt.track import Tracker

        s["tr"] = Tracker(_error_rings(case, seed), tuning=_tuning(case) if "shape" in case else None)
        if kind == "errors":
            s["dev"], _ = _device_bunch(s["tr"], _beam(case, seed))
            s["var"] = torch.from_numpy(_variant_ids(case)).cuda()
        if kind == "da":
            ref = np.zeros((case["variants"], case["deltas"], 6))
            for d, pz in enumerate([0.0] if case["deltas"] == 1 else [-0.01, 0.0, 0.01]):
                ref[:, d, 0], ref[:, d, 1], ref[:, d, 5] = TWISS["ex"] * pz, TWISS["epx"] * pz, pz
            s["ref"], s["ys"] = ref, da.y_scale(TWISS["ba"], TWISS["bb"])
    else:
        from bgt import mlp

        s["mlp"] = mlp.SurvivalMLP(max_batch=65536 if kind in ("forward", "features") else 8192)
        if kind == "features":
            v0, v1, t, var, mean, std = _feature_inputs(case, seed)
            s["mlp"].set_normalization(mean, std)
            s["args"] = [torch.from_numpy(a).cuda() for a in (v0, v1, var, t)]
        else:
            s["mlp"].set_params(_mlp_params(seed))
            s["x"], s["y"] = (a.cuda() for a in _mlp_inputs(case, seed))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "element":  # a bunch of its own each call: one element again and again would lose it
        b = s["bunch"].copy()
        s["tr"].track1(b, s["pos"])
        return [b.vec6, b.beta, b.state, b.ix_ele_lost]
    if kind == "host":  # in place, pass after pass, as a long-term tracking loop
        b = s["tr"].track_turns(s["bunch"], case["turns"])
        return [b.vec6, b.beta, b.state, b.ix_ele_lost, b.ix_turn_lost]
    if kind in ("device", "time"):
        s["tr"].track_turns_device(*s["dev"], case["turns"], t=s["t"])
        return s["dev"] + ([s["t"]] if kind == "time" else [])
    if kind == "errors":
        s["tr"].track_turns_device(*s["dev"], case["turns"], variant=s["var"])
        return s["dev"]
    if kind == "optics":
        from bgt import da

        o = da.variant_optics(da.tracker_one_turn(s["tr"]), case["variants"])
        return [o.closed_orbit, o.eta, o.beta_a, o.alpha_a, o.beta_b, o.alpha_b, o.tune_a, o.tune_b]
    if kind == "da":
        return list(s["tr"].da_scan_grid(s["ref"], case["angles"], 0.0, math.pi, case["radii"], 0.025, s["ys"],
                                         case["turns"], return_survival=True))
    if kind == "features":
        v0, v1, var, t = s["args"]
        return [a for a in s["mlp"].features(v0, v1, var, t, raw=case["raw"]) if a is not None]
    if kind == "forward":
        return s["mlp"].forward(s["x"])
    if kind == "gradients":
        return list(s["mlp"].gradients(s["x"], s["y"]))
    s["mlp"].fit(s["x"], s["y"], epochs=1, batch=case["batch"])
    return s["mlp"].get_params()


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    weights = 2 * (HIDDEN * N_IN + 2 * HIDDEN * HIDDEN + HIDDEN)
    if kind == "element":
        return {"bytes": 136 * n, "flops": 300 * n}
    if kind in ("host", "device", "time"):
        return {"bytes": (168 if kind == "time" else 136) * n, "flops": FLOPS_IDEAL * n * case["turns"]}
    if kind == "errors":
        return {"bytes": 140 * n, "flops": FLOPS_ERRORS * n * case["turns"]}
    if kind == "optics":  # five or so Newton turns of 7 probes, one of 12
        return {"bytes": 136 * 47 * case["variants"], "flops": FLOPS_ERRORS * 47 * case["variants"]}
    if kind == "da":  # about a third of the probes live on
        p = case["variants"] * case["deltas"] * case["angles"] * case["radii"]
        return {"bytes": 4 * p, "flops": FLOPS_ERRORS * p * (1 + case["turns"] / 3)}
    if kind == "features":
        return {"bytes": n * (96 + 4 + 2 * N_IN + (120 if case["raw"] else 0)), "flops": 100 * n}
    if kind == "forward":
        return {"bytes": n * (2 * N_IN + 4) + weights, "flops": n * weights}
    steps = case["n"] // case["batch"] if kind == "fit" else 1
    rows = steps * case["batch"] if kind == "fit" else n
    return {"bytes": rows * (2 * N_IN + 4) + steps * 4 * N_PARAMS * (7 if kind == "fit" else 2),
            "flops": 3 * rows * weights}


# ---------------------------------------------------------------------------
# the same in plain FP64

def _sqrt_one(x):
    return x / (torch.sqrt(1 + x) + 1)


def _drift(p, length):
    x, px, y, py, z, pz, beta = p
    rel = 1 + pz
    u, w = px / rel, py / rel
    ps = torch.sqrt(1 - u * u - w * w)
    p0c2, m2 = E_TOT ** 2 - MC2 ** 2, MC2 ** 2
    lead = _sqrt_one(m2 * (2 * pz + pz * pz) / (p0c2 * rel * rel + m2))
    z = z + length * (lead + _sqrt_one(-(u * u + w * w)) / ps)
    return [x + length * u / ps, px, y + length * w / ps, py, z, pz, beta]


def _kick(p, an, bn, scale):
    """Thin magnetic kicks: px - i py gets -sum (b_n + i a_n)(x + i y)^n."""
    x, px, y, py, z, pz, beta = p
    re, im = torch.ones_like(x), torch.zeros_like(x)
    fx, fy = torch.zeros_like(x), torch.zeros_like(x)
    top = max(list(an) + list(bn))
    for n in range(top + 1):
        if n in bn:
            fx, fy = fx - bn[n] * re, fy + bn[n] * im
        if n in an:
            fx, fy = fx + an[n] * im, fy + an[n] * re
        re, im = re * x - im * y, re * y + im * x
    return [x, px + scale * fx, y, py + scale * fy, z, pz, beta]


def _quad_mat(k, length, rel):
    sk = torch.sqrt(k.abs())
    a = sk * length
    c, s = (torch.cos(a), torch.sin(a) / sk) if float(k.flatten()[0]) < 0 else (torch.cosh(a), torch.sinh(a) / sk)
    return c, s, k * (length - c * s) / 4, -k * s * s / (2 * rel), -(length + c * s) / (4 * rel * rel)


def _quad(p, k1, steps, an, bn):
    step = 0.4 / steps
    rel = 1 + p[5]
    mats = [_quad_mat(f * k1 / rel, step, rel) for f in (-1, 1)]
    b0 = math.sqrt(E_TOT ** 2 - MC2 ** 2) / E_TOT
    if an:
        p = _kick(p, an, bn, 0.5 / steps)
    for i in range(steps):
        x, px, y, py, z, pz, beta = p
        (cx, sx, a0, a1, a2), (cy, sy, d0, d1, d2) = mats
        z = z + a0 * x * x + a1 * x * px + a2 * px * px + d0 * y * y + d1 * y * py + d2 * py * py
        x, px = cx * x + sx / rel * px, -k1 * sx * x + cx * px
        y, py = cy * y + sy / rel * py, k1 * sy * y + cy * py
        # (beta - beta0) / beta0 as its series in pz: step pz (1 - 3/2 beta0^2 pz + ...) (mc2 / E)^2
        z = z + step * pz * (1 - 1.5 * pz * b0 ** 2 + pz ** 2 * b0 ** 2 * (2 * b0 ** 2 - 0.5 * (MC2 / E_TOT) ** 2)) * \
            (MC2 / E_TOT) ** 2
        p = [x, px, y, py, z, pz, beta]
        if an:
            p = _kick(p, an, bn, (0.5 if i == steps - 1 else 1.0) / steps)
    return p


def _bend(p):
    """Exact sector bend (length 2, no edge angles) with its hard edges."""
    g, length = ANGLE / 2, 2.0
    p = _bend_edge(p, g, 1.0)
    x, px, y, py, z, pz, beta = p
    rel = 1 + pz
    pt = torch.sqrt(rel * rel - py * py)
    phi = torch.asin(px / pt)
    gp = g / pt
    sa, ca = math.sin(ANGLE), math.cos(ANGLE)
    sinc = sa / ANGLE
    cosc = 0.5 * (math.sin(ANGLE / 2) / (ANGLE / 2)) ** 2
    alpha = 2 * (1 + g * x) * torch.sin(ANGLE + phi) * length * sinc - gp * ((1 + g * x) * length * sinc) ** 2
    cp = torch.cos(ANGLE + phi)
    xi = alpha / (torch.sqrt(cp * cp + gp * alpha) + cp)
    x1 = x * ca - length * length * g * cosc + xi
    lv = -(length * sinc + x * sa)
    th = 2 * (ANGLE + phi - torch.atan2(xi, -lv))
    lp = torch.sqrt(lv * lv + xi * xi) / (torch.sin(th / 2) / (th / 2))
    b0 = math.sqrt(E_TOT ** 2 - MC2 ** 2) / E_TOT
    p = [x1, pt * torch.sin(phi + ANGLE - th), y + py * lp / pt, py, z + beta * length / b0 - rel * lp / pt, pz, beta]
    return _bend_edge(p, g, -1.0)


def _bend_edge(p, g, sign):
    """Second-order hard edge of a sector bend, pole faces normal to the orbit."""
    x, px, y, py, z, pz, beta = p
    f = 1 / (1 + pz)
    return [x + sign * g * y * y * f / 2, px, y, py - sign * g * px * y * f, z - sign * g * px * y * y * f * f / 2, pz,
            beta]


def _rf(p):
    p0c = math.sqrt(E_TOT ** 2 - MC2 ** 2)
    circ = N_CELL * 7.0 + 0.5
    f = HARMONIC * (p0c / E_TOT) * C_LIGHT / circ
    phase = 2 * math.pi * f * p[4] / (p[6] * C_LIGHT)
    phase = torch.remainder(phase + math.pi, 2 * math.pi) - math.pi
    for i in range(11):
        de = RF_VOLTAGE * torch.sin(phase) / (20 if i in (0, 10) else 10)
        x, px, y, py, z, pz, beta = p
        pc = (1 + pz) * p0c
        e_old = pc / beta
        pz1 = pz + (1 + pz) * _sqrt_one((2 * e_old * de + de * de) / (pc * pc))
        b1 = p0c * (1 + pz1) / (e_old + de)
        p = [x, px, y, py, z * b1 / beta, pz1, b1]
        if i < 10:
            z0 = p[4]
            p = _drift(p, 0.05)
            phase = phase + 2 * math.pi * f * (p[4] - z0) / (C_LIGHT * p[6])
    return p


def _magnet(p, kind, focus, err):
    """A quadrupole or sextupole; err: its 11 errors, one value a particle, or None."""
    k = (K1 if focus else -K1) if kind == "quad" else (K2_SF if focus else K2_SD)
    length, order = (0.4, 1) if kind == "quad" else (0.2, 2)
    if err is None:
        an, bn, steps = {}, {} if kind == "quad" else {2: k * length / 2}, 1
    else:
        # relative multipoles at 10 mm, scaled by the main integrated strength
        main = k * length
        an = {n: err[n] * main * 0.01 ** (order - n) for n in range(3, 7)}
        bn = {n: err[n + 4] * main * 0.01 ** (order - n) for n in range(3, 7)}
        if kind == "sext":
            bn[2] = main / 2
        steps = 16 if kind == "quad" else 1
        c, s = torch.cos(err[2]), torch.sin(err[2])
        x, px, y, py = p[0] - err[0], p[1], p[2] - err[1], p[3]
        p = [c * x + s * y, c * px + s * py, c * y - s * x, c * py - s * px] + p[4:]
    if kind == "quad":
        p = _quad(p, torch.full_like(p[0], k), steps, an, bn)
    else:
        p = _kick(_drift(_kick(p, an, bn, 0.5), length), an, bn, 0.5)
    if err is not None:
        x, px, y, py = p[:4]
        p = [c * x - s * y + err[0], c * px - s * py, c * y + s * x + err[1], c * py + s * px] + p[4:]
    return p


def _turn(p, err=None, variant=None):
    for cell in range(N_CELL):
        for half, focus in ((0, True), (1, False)):
            for slot, kind in ((0, "quad"), (1, "sext")):
                e = None if err is None else [c for c in err[variant, 4 * cell + 2 * half + slot].T]
                p = _drift(_magnet(p, kind, focus, e), 0.3)
            p = _drift(_bend(p), 0.3)
    return _rf(p)


def _probe(v):
    """The phase-space columns and beta of an FP64 array [6, n]."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.as_tensor(v, dtype=torch.float64, device=dev)
    pc = (1 + v[5]) * math.sqrt(E_TOT ** 2 - MC2 ** 2)
    return [v[k] for k in range(6)] + [pc / torch.sqrt(pc * pc + MC2 ** 2)]


def _mlp64(case, seed, grad):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.from_numpy(_mlp_params(seed)).double().to(dev).requires_grad_(grad)
    x, y = (a.double().to(dev) for a in _mlp_inputs(case, seed))
    o, a = 0, x
    for k, (rows, cols) in enumerate(((HIDDEN, N_IN), (HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (1, HIDDEN))):
        w, b = p[o:o + rows * cols].view(rows, cols), p[o + rows * cols:o + rows * cols + rows]
        o += rows * cols + rows
        a = a @ w.T + b
        a = torch.relu(a) if k < 3 else a[:, 0]
    if not grad:
        return torch.sigmoid(a)
    loss = torch.nn.functional.binary_cross_entropy_with_logits(a, y)
    loss.backward()
    return [p.grad, float(loss.detach())]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("element", "host", "device", "errors", "time"):
        if kind != "element" and case["turns"] * (8 if kind == "errors" else 1) > 24:
            return None
        p = _probe(_beam(case, seed))
        if kind == "element":
            one = {"sbend": _bend, "rfcavity": _rf, "drift": lambda q: _drift(q, 0.3),
                   "quadrupole": lambda q: _magnet(q, "quad", True, None),
                   "sextupole": lambda q: _magnet(q, "sext", True, None)}
            p = one[case["element"]](p)
        else:
            err = var = None
            if kind == "errors":
                err = torch.from_numpy(_errors(case, seed)).to(p[0].device)
                var = torch.from_numpy(_variant_ids(case)).long().to(p[0].device)
            for _ in range(case["turns"]):
                p = _turn(p, err, var)
        out = [torch.stack(p[:6]), p[6], None, None, None]
        return out[:4] if kind == "element" else out + ([None] if kind == "time" else [])
    if kind == "features":
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        v0, v1, t, var, mean, std = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in
                                     _feature_inputs(case, seed))
        T = t[var.long()].T
        d = v1 - T[:6]
        xb, pxb, yb, pyb = (d[k] - T[6 + k] * d[5] for k in range(4))
        act = [torch.sqrt(0.5 * ((1 + a * a) / b * q * q + 2 * a * q * r + b * r * r))
               for q, r, b, a in ((xb, pxb, T[10], T[11]), (yb, pyb, T[12], T[13]))]
        f = torch.cat([v0 - T[:6], T[14:30], d, torch.stack(act)]).T
        x = torch.zeros((-(-case["n"] // 128) * 128, N_IN), dtype=torch.float64, device=dev)
        x[:case["n"], :N_FEATURES] = (f - mean) / std
        return [x] + ([f] if case["raw"] else [])
    if kind == "forward":
        return _mlp64(case, seed, False)
    if kind == "gradients":
        return _mlp64(case, seed, True)
    # optics: differences over 1e-8 steps; a scan's radii: counts of whole outcomes; a fit: steps of Adam,
    # which turn on the signs of gradients near zero
    return None
