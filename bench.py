"""Benchmark: FP64 particle.turns/s of bmad_standard ring tracking on B200.

Workload (the configuration the metric is quoted on): the 64-cell FODO ring
with apertures (elliptical 20 x 10 mm on every quadrupole, rectangular
30 x 15 mm at the RF), 1,000,000 particles from a seeded 6D Gaussian at 3x the
base emittances, FP64.  One step = one persistent-kernel pass of
`--turns-per-step` turns over the whole bunch (a segment of the 10,000-turn
run).  value = particle.turns tracked (particles alive at the start of each
turn) / device time, summed over ranks.

Usage:
    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]
Multi-GPU: launched by torch.distributed.run, one rank per GPU; each rank
tracks its own 1M-particle bunch (weak scaling, no data-path collective).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT / "bmad-ecosystem_b200"))
sys.path.insert(0, str(ROOT))

METRIC = "FP64 particle*turns/s, bmad_standard ring tracking (1M particles, apertures)"
UNIT = "particle*turns/s"
N_PARTICLES = 1_000_000
# FP64 operations per particle.turn on this ring (add/sub/mul/div/sqrt = 1
# each) and libm calls per particle.turn, counted by the instrumented oracle
# build over the config-1 beam (tests/test_flop_count.py pins them to that count).
FLOPS_PER_PARTICLE_TURN = 98807.0
LIBM_PER_PARTICLE_TURN = 2315.0


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="bgt", choices=["bgt", "reference"])
    ap.add_argument("--turns-per-step", type=int, default=20)
    ap.add_argument("--particles", type=int, default=N_PARTICLES)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-autotune", action="store_true", help="use the library's default launch shape")
    ap.add_argument("--tuning", default="", help="threads_per_block,blocks_per_sm (skips the autotuner); DA "
                    "workloads also take ,table_mode[,compact_every]")
    ap.add_argument("--workload", default="track", choices=["track", "da", "learned-da", "sext-scan", "mlp"],
                    help="track: the headline tracking metric (default); da: batched DA scan of error variants; "
                         "learned-da: classifier-pruned vs plain DA scan; sext-scan: pruned sextupole-setting scan; "
                         "mlp: the survival classifier's tensor-core forward pass and training step")
    ap.add_argument("--mlp-rows", type=int, default=262144, help="mlp: rows of one forward pass")
    ap.add_argument("--variants", type=int, default=0, help="DA workloads: number of lattice variants")
    ap.add_argument("--da-turns", type=int, default=0, help="DA workloads: turns per probe (default 20000)")
    ap.add_argument("--repack-turn", type=int, default=64, help="da: plain scan in two launches, the probes alive "
                    "after this many turns packed densely for the second (0: one launch for all turns)")
    ap.add_argument("--jitter", action="store_true", help="learned-da: add one jittered probe per grid cell")
    ap.add_argument("--boundary-cells", default="", help="pruned scans: grid cells either side of the predicted "
                    "DA boundary tracked in full; comma list (learned-da default 0,2; sext-scan 2)")
    ap.add_argument("--p-lo", default="", help="pruned scans: retire probes with p(lost) < p_lo as surviving; 0 "
                    "(default) follows the method's rule (only confidently lost probes retired early); a comma "
                    "list (e.g. 0,0.02) adds measured comparisons outside the rule")
    ap.add_argument("--epochs", type=int, default=6)
    ap.add_argument("--seed", type=int, default=1)
    ap.add_argument("--model", default="", help="sext-scan: start from this saved classifier (fine-tune)")
    ap.add_argument("--save-model", default="", help="learned-da / sext-scan: save the trained classifier")
    return ap.parse_args()


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    def __init__(self, index: int):
        self.index = index
        self.samples = []
        self.proc = None

    def __enter__(self):
        q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 7:
                self.samples.append(parts)

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(s[0]) for s in self.samples if s[0].replace(".", "").isdigit()]
        mx = [float(s[1]) for s in self.samples if s[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for s in self.samples for i in range(4) if s[3 + i].lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.samples)}


def turns_tracked(state0_alive, ix_turn_lost, state, t0, t1):
    """particle.turns with the particle alive at the start of each turn in [t0, t1)."""
    alive_end = state == 1
    tracked = np.where(alive_end, t1 - t0, np.clip(ix_turn_lost + 1, t0, t1) - t0)
    return int(np.sum(np.where(state0_alive, tracked, 0)))


def run_reference(args, rank, world):
    """Reference arm: the reference's CPU path for this workload -- the C
    restatement of Bmad's bmad_standard track1 in the reference's loop
    structure (element-outer, OpenMP over particles), on all host threads."""
    if rank != 0:
        return
    from bgt import rings
    from oracle import oracle as O

    lat = rings.fodo_ring(apertures=True)
    eles = O.to_eles(lat)
    param = O.make_param(lat.species.mass, lat.species.charge)
    threads = os.cpu_count() or 1
    n_sample, t_sample = 2000, 10
    v0 = rings.gaussian_beam(rings.CONFIG1_BEAM, n=n_sample)

    def step():
        v = v0.copy()
        b = O.beta_of(lat.p0c, v[5], lat.species.mass)
        st = np.ones(n_sample, np.int32)
        ie = np.full(n_sample, -1, np.int32)
        it = np.full(n_sample, -1, np.int32)
        t = time.perf_counter()
        O.track_turns(eles, lat.p0c, param, v, b, st, ie, it, t_sample, n_threads=threads, element_outer=True)
        return time.perf_counter() - t, turns_tracked(np.ones(n_sample, bool), it, st, 0, t_sample)

    for _ in range(args.warmup):
        step()
    tot_t, tot_u = 0.0, 0
    for _ in range(args.steps):
        dt, u = step()
        tot_t += dt
        tot_u += u
    val = tot_u / tot_t
    sample = f"{n_sample} particles x {t_sample} turns of the config-1 ring per step"
    line = {"impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * tot_t / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": "fodo64 ring (770 elements) + apertures, config-1 beam",
                       "particles_per_step_sample": n_sample, "turns_per_step": t_sample,
                       "parallelism": f"openmp x{threads}"},
            "cpu_baseline": {"value": val, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample},
            "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def cpu_baseline():
    """Oracle (C restatement) on the host cores, a bounded sample."""
    from bgt import rings
    from oracle import oracle as O

    lat = rings.fodo_ring(apertures=True)
    eles = O.to_eles(lat)
    param = O.make_param(lat.species.mass, lat.species.charge)
    threads = os.cpu_count() or 1
    n, turns = 4000, 20
    v = rings.gaussian_beam(rings.CONFIG1_BEAM, n=n)
    b = O.beta_of(lat.p0c, v[5], lat.species.mass)
    st = np.ones(n, np.int32)
    ie = np.full(n, -1, np.int32)
    it = np.full(n, -1, np.int32)
    v2, b2, st2, ie2, it2 = v.copy(), b.copy(), st.copy(), ie.copy(), it.copy()
    t = time.perf_counter()
    O.track_turns(eles, lat.p0c, param, v, b, st, ie, it, turns, n_threads=threads, element_outer=True)
    dt = time.perf_counter() - t
    # the stronger CPU bound: OpenMP over particles, turns and elements inside
    t = time.perf_counter()
    O.track_turns(eles, lat.p0c, param, v2, b2, st2, ie2, it2, turns, n_threads=threads, element_outer=False)
    dt2 = time.perf_counter() - t
    return {"value": turns_tracked(np.ones(n, bool), it, st, 0, turns) / dt, "unit": UNIT, "cores": threads,
            "kind": "port", "sample": f"{n} particles x {turns} turns, element-outer OpenMP (reference loop order)",
            "particle_major_value": turns_tracked(np.ones(n, bool), it2, st2, 0, turns) / dt2}


# ---------------------------------------------------------------------------
# Dynamic-aperture workloads: the batched scan of error variants, the
# classifier-pruned scan against the plain one, and the pruned
# sextupole-setting scan.  Each prints one JSON line (rank 0).  Under
# torchrun the variants are sharded over ranks (bgt.da.sharded_scan: one
# contiguous block of variants per GPU, DA radii all-gathered, wall time the
# max over ranks); the classifier's training samples are all-gathered so that
# every rank trains the same network (bgt.learned_da.gather_rows).

class Ranks:
    """rank / world / device of this process, and the reductions the DA
    workloads need (NCCL under torchrun; identity on one GPU)."""

    def __init__(self):
        import torch

        self.rank = int(os.environ.get("RANK", "0"))
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.local = int(os.environ.get("LOCAL_RANK", "0"))
        torch.cuda.set_device(self.local)
        self.dev = torch.device("cuda", self.local)
        self.dist = None
        if self.world > 1:
            import datetime

            import torch.distributed as dist

            dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))
            self.dist = dist

    def _red(self, x, op):
        if not self.dist:
            return x
        import torch

        t = torch.tensor([float(x)], dtype=torch.float64, device=self.dev)
        self.dist.all_reduce(t, op=op)
        return float(t.item())

    def sum(self, x):
        return self._red(x, self.dist.ReduceOp.SUM if self.dist else None)

    def max(self, x):
        return self._red(x, self.dist.ReduceOp.MAX if self.dist else None)

    def all(self, flag: bool) -> bool:
        return self._red(1.0 if flag else 0.0, self.dist.ReduceOp.MIN if self.dist else None) > 0.5

    def gather_rows(self, t):
        from bgt import learned_da as LD

        return LD.gather_rows(t) if self.dist else t

    def barrier(self):
        if self.dist:
            self.dist.barrier()

    def close(self):
        if self.dist:
            self.dist.barrier()
            self.dist.destroy_process_group()


def _da_problem(lats, grid, turns, device=0):
    import dataclasses

    from bgt import da, rings
    from bgt import learned_da as LD
    from bgt.track import Tracker

    g = dataclasses.replace(grid, n_turns=turns)
    ys = da.y_scale(rings.TWISS0["beta_a"], rings.TWISS0["beta_b"])
    return LD.setup(Tracker(lats, device=device), lats, g, (rings.K2_SF, rings.K2_SD), yscale=ys)


def _autotune_da(pb, turns=2, fixed=""):
    from bgt import autotune
    from bgt import da

    if fixed:
        # threads_per_block,blocks_per_sm[,table_mode[,compact_every]]: no sweep
        f = [int(x) for x in fixed.split(",")] + [0, 0]
        pb.tracker.set_tuning(threads_per_block=f[0], blocks_per_sm=f[1], table_mode=f[2], compact_every=f[3])
        return pb.tracker.get_tuning()

    v6 = da.grid_initial_conditions(pb.ref, pb.n_angle, pb.angle_min, pb.angle_max, pb.n_radius, pb.r_max,
                                    pb.yscale)
    var = np.repeat(np.arange(pb.n_variants, dtype=np.int32), pb.per_variant)
    autotune.tune(pb.tracker, v6, turns=turns, sample=min(v6.shape[1], 262_144), variant=var,
                  compact_options=(0, 16))
    return pb.tracker.get_tuning()


def _mm(x):
    return float(np.mean(x)) * 1e3


def da_cpu_baseline(lat, pb, n_probe=512, turns=20):
    """The oracle in the reference's loop order (element-outer OpenMP) on all
    host cores, tracking a sample of one error variant's DA probes (spread
    over its grid) for a few turns: particle.turns/s of the plain scan on the
    CPU."""
    from bgt import da
    from oracle import oracle as O

    eles = O.to_eles(lat)
    param = O.make_param(lat.species.mass, lat.species.charge)
    threads = os.cpu_count() or 1
    v6 = da.grid_initial_conditions(pb.ref[:1], pb.n_angle, pb.angle_min, pb.angle_max, pb.n_radius, pb.r_max,
                                    pb.yscale)
    pick = np.linspace(0, v6.shape[1] - 1, n_probe).astype(np.int64)
    v = np.ascontiguousarray(v6[:, pick])
    b = O.beta_of(lat.p0c, v[5], lat.species.mass)
    st = np.ones(n_probe, np.int32)
    ie = np.full(n_probe, -1, np.int32)
    it = np.full(n_probe, -1, np.int32)
    t = time.perf_counter()
    O.track_turns(eles, lat.p0c, param, v, b, st, ie, it, turns, n_threads=threads, element_outer=True)
    dt = time.perf_counter() - t
    return {"value": turns_tracked(np.ones(n_probe, bool), it, st, 0, turns) / dt, "unit": "particle*turns/s",
            "cores": threads, "kind": "port",
            "sample": f"{n_probe} grid probes of variant 0 x {turns} turns, element-outer OpenMP"}


def run_da(args):
    """Batched DA scan of error variants (per GPU: its block of variants).
    Plain FP64 tracking of every probe to the full turn count, either in one
    launch (--repack-turn 0) or in two: every probe --repack-turn turns, then
    the probes still alive packed densely (bit-identical outcomes)."""
    import torch

    from bgt import da, rings
    from bgt import learned_da as LD

    R = Ranks()
    nv = args.variants or 256
    if nv < R.world:
        raise SystemExit("more GPUs than variants")
    turns = args.da_turns or rings.CONFIG2_GRID.n_turns
    t0 = time.perf_counter()
    lats = rings.error_variants(nv)
    info = {}

    def scan(b, e):
        pb = _da_problem(lats[b:e], rings.CONFIG2_GRID, turns, R.local)
        info["setup_s"] = time.perf_counter() - t0
        info["tuning"] = _autotune_da(pb, fixed=args.tuning)
        info["pb"] = pb
        launches0 = pb.tracker.launch_count
        R.barrier()
        if args.repack_turn > 0:
            res = LD.compacted_scan(pb, 0, pb.n_variants, early=args.repack_turn)
        else:
            res = da.plain_scan(pb.tracker, pb.ref, **pb.grid())
        info["launches"] = pb.tracker.launch_count - launches0
        return res

    with ClockSampler(R.local) as clk:
        sh = da.sharded_scan(scan, nv, R.rank, R.world)
    pb = info["pb"]
    if R.rank == 0:
        n = nv * pb.per_variant
        line = {"metric": "DA scan wall time, error variants x polar grid, plain FP64 tracking of every probe",
                "value": sh.wall_s, "unit": "s", "higher_is_better": False, "n_gpus": R.world,
                "scaling": "strong", "dtype": "f64", "data": "synthetic",
                "config": {"workload": "batched DA scan of error variants", "variants": nv, "probes": n,
                           "probes_per_variant": pb.per_variant, "turns": turns, "angles": pb.n_angle,
                           "radii": pb.n_radius, "r_max_m": pb.r_max, "deltas": list(pb.deltas),
                           "repack_turn": args.repack_turn, "parallelism": f"variants x{R.world} GPUs"},
                "particle_turns": sh.particle_turns, "particle_turns_per_s": sh.particle_turns / sh.wall_s,
                "da_radius_mm_mean": _mm(sh.radius),
                "da_radius_mm_mean_per_delta": [_mm(sh.radius[:, d]) for d in range(len(pb.deltas))],
                "setup_s": info["setup_s"], "tuning": info["tuning"], "gpu_launches": info["launches"],
                "clocks": clk.summary()}
        if not args.no_cpu_baseline and R.world == 1:
            cpu = da_cpu_baseline(lats[0], pb)
            line["cpu_baseline"] = cpu
            line["cpu_estimate_s"] = sh.particle_turns / cpu["value"]
        print(json.dumps(line), flush=True)
    R.close()


def _train_classifier(args, R, pb, scans, net, fine_tune=False):
    from bgt import learned_da as LD

    raw, lab = LD.training_set(pb, scans, net)
    raw, lab = R.gather_rows(raw), R.gather_rows(lab)
    hist, t_train = LD.train(net, raw, lab, epochs=args.epochs if not fine_tune else max(2, args.epochs // 2),
                             batch=8192, lr=2e-3 if not fine_tune else 1e-3, seed=args.seed,
                             set_normalization=not fine_tune)
    n = (raw.shape[0] // 128) * 128
    b = min(8192, n)
    steps = len(hist) * (n // b)
    flops = 852_000.0 * b * steps  # GEMM flops per sample (forward + backward) x samples
    return {"samples": int(raw.shape[0]), "lost_fraction": float(lab.float().mean().item()), "epochs": len(hist),
            "loss_per_epoch": hist, "wall_s": t_train, "samples_per_s": b * steps / t_train,
            "gemm_tflops": flops / t_train / 1e12}


def _staged_scan_sharded(R, lats, grid, turns, n, jitter_seeds=(None,), tun=None):
    """Staged plain scans (turn-64 snapshot) of this rank's block of the
    variants lats[:n]: (ScanProblem, [StagedScan], wall max over ranks)."""
    from bgt import da
    from bgt import learned_da as LD

    b, e = da.shard_range(n, R.rank, R.world)
    pb = _da_problem(lats[b:e], grid, turns, R.local)
    if tun:
        pb.tracker.set_tuning(**tun)
    R.barrier()
    scans = [LD.staged_scan(pb, 0, e - b, jitter_seed=j) for j in jitter_seeds]
    return pb, scans, R.max(sum(s.wall_s for s in scans))


def run_learned_da(args):
    """Classifier-pruned DA scan vs the plain scan on held-out variants."""
    from bgt import da, rings
    from bgt import learned_da as LD
    from bgt.mlp import SurvivalMLP

    R = Ranks()
    nv = args.variants or 256
    turns = args.da_turns or rings.CONFIG2_GRID.n_turns
    half = nv // 2
    if half < R.world:
        raise SystemExit("more GPUs than held-out variants")
    lats = rings.error_variants(nv)
    held = lats[half:]
    bh, eh = da.shard_range(nv - half, R.rank, R.world)
    pb_te = _da_problem(held[bh:eh], rings.CONFIG2_GRID, turns, R.local)
    tun = _autotune_da(pb_te, fixed=args.tuning)
    p_los = [float(x) for x in (args.p_lo or "0").split(",")]
    bcs = [int(c) for c in (args.boundary_cells or "0,2").split(",")]
    with ClockSampler(R.local) as clk:
        jit = (None, args.seed) if args.jitter else (None,)
        pb_tr, scans, train_scan_s = _staged_scan_sharded(R, lats, rings.CONFIG2_GRID, turns, half, jit, tun)
        net = SurvivalMLP(max_batch=65536, seed=args.seed)
        train = _train_classifier(args, R, pb_tr, scans, net)
        R.barrier()
        plain = da.sharded_scan(lambda b, e: da.plain_scan(pb_te.tracker, pb_te.ref, **pb_te.grid()), nv - half,
                                R.rank, R.world)
        R.barrier()
        # the same plain tracking with the probes alive at the snapshot turn
        # packed densely for the rest: the faster plain scan
        plain_c = da.sharded_scan(lambda b, e: LD.compacted_scan(pb_te, 0, e - b), nv - half, R.rank, R.world)
        runs = []
        for pl in p_los:
            for c in bcs:
                R.barrier()
                pr = da.sharded_scan(lambda b, e: LD.pruned_scan(pb_te, net, 0, e - b, seed=args.seed + R.rank,
                                                                 boundary_cells=c, p_lo=pl),
                                     nv - half, R.rank, R.world)
                runs.append((pl, c, pr))
    if args.save_model and R.rank == 0:
        net.save(args.save_model)
    plain_surv = (plain.local.survive_turns >= turns).reshape(-1)
    dr = pb_te.r_max / (pb_te.n_radius - 1)
    plain_best_s = min(plain.wall_s, plain_c.wall_s)
    compacted_equal = R.all(bool(np.array_equal(plain_c.local.survive_turns, plain.local.survive_turns)))

    def summary(pl, c, sh):
        pr = sh.local
        cells = np.abs(sh.radius - plain.radius) / dr
        return {"p_lo": pl, "boundary_cells": c,
                "rule": "the method's rule: only confidently lost probes retired early" if pl == 0 else
                        "retires confident survivors too (outside the method's rule; comparison only)",
                "speedup": plain_best_s / sh.wall_s, "speedup_vs_one_launch_plain": plain.wall_s / sh.wall_s,
                "pruned_s": sh.wall_s,
                "da_error": da.da_error(sh.radius, plain.radius), "rays_exact_fraction": float(np.mean(cells < 0.5)),
                "max_error_cells": float(np.max(cells)), "pruned_particle_turns": sh.particle_turns,
                "particle_turns_ratio": plain.particle_turns / max(1, sh.particle_turns),
                "tracked_fraction": R.sum(pr.n_tracked) / R.sum(pr.n_probes),
                "retired_lost": int(R.sum(pr.n_retired_lost)), "retired_survive": int(R.sum(pr.n_retired_survive)),
                "audit_probes": int(R.sum(pr.audit_n)), "audit_errors": int(R.sum(pr.audit_errors)),
                "tracked_outcomes_equal_plain": R.all(bool(np.array_equal(pr.survive_label[pr.tracked],
                                                                           plain_surv[pr.tracked]))),
                "da_radius_mm_mean": _mm(sh.radius)}

    runs = [summary(pl, c, sh) for pl, c, sh in runs]
    # the headline: the fastest rule-following setting whose DA error is within 2 %
    rule = [r for r in runs if r["p_lo"] == 0] or runs
    ok = [r for r in rule if r["da_error"] <= 0.02] or rule
    best = max(ok, key=lambda r: r["speedup"])
    train_pt = R.sum(sum(s.particle_turns for s in scans[:1]))
    if R.rank == 0:
        line = {"metric": "DA-scan wall time, faster plain scan / classifier-pruned, held-out variants",
                "value": best["speedup"], "unit": "x", "higher_is_better": True, "n_gpus": R.world,
                "scaling": "strong", "dtype": "f64 tracking, bf16/fp32 classifier", "data": "synthetic",
                "config": {"workload": "learned DA scan of error variants", "variants_train": half,
                           "variants_heldout": nv - half, "probes_per_variant": pb_te.per_variant, "turns": turns,
                           "early_turns": 64, "p_hi": 0.98, "p_lo": best["p_lo"], "audit": 0.02,
                           "boundary_cells": best["boundary_cells"], "jitter": bool(args.jitter),
                           "parallelism": f"variants x{R.world} GPUs"},
                "plain_s": plain.wall_s, "plain_compacted_s": plain_c.wall_s, "plain_best_s": plain_best_s,
                "compacted_plain_equals_one_launch": compacted_equal,
                "pruned_s": best["pruned_s"], "da_error": best["da_error"],
                "plain_particle_turns": plain.particle_turns, "pruned": runs,
                "all_variants_plain": {"wall_s": train_scan_s + plain.wall_s,
                                       "launches": "2 x 128 variants (training scan staged at turn 64)",
                                       "particle_turns": int(train_pt) + plain.particle_turns},
                "train_scan_s": train_scan_s, "train": train,
                "da_radius_mm_mean_plain": _mm(plain.radius), "tuning": tun, "clocks": clk.summary()}
        if not args.no_cpu_baseline and R.world == 1:
            cpu = da_cpu_baseline(lats[half], pb_te)
            line["cpu_baseline"] = cpu
            line["cpu_estimate_plain_s"] = plain.particle_turns / cpu["value"]
        print(json.dumps(line), flush=True)
    R.close()


def run_sext_scan(args):
    """Sextupole-setting scan: fine-tune on the first 256 variants' tracking,
    prune the rest with the boundary verified by the tracker, rank all
    variants by DA, and compare the ranking of 256 audited variants with a
    plain-tracking ranking of the same variants."""
    from bgt import da, rings
    from bgt import learned_da as LD
    from bgt.mlp import SurvivalMLP

    R = Ranks()
    nv = args.variants or 4096
    turns = args.da_turns or rings.CONFIG4_GRID.n_turns
    first = min(256, nv // 4)
    t0 = time.perf_counter()
    lats = rings.sextupole_variants(nv)
    rest = lats[first:]
    rng = np.random.default_rng(args.seed)
    n_audit = min(256, nv - first)
    audit_idx = np.sort(rng.choice(nv - first, n_audit, replace=False))
    audited = [rest[i] for i in audit_idx]
    br, er = da.shard_range(nv - first, R.rank, R.world)
    ba, ea = da.shard_range(n_audit, R.rank, R.world)
    pb_rest = _da_problem(rest[br:er], rings.CONFIG4_GRID, turns, R.local)
    pb_aud = _da_problem(audited[ba:ea], rings.CONFIG4_GRID, turns, R.local)
    t_setup = time.perf_counter() - t0
    tun = _autotune_da(pb_rest, fixed=args.tuning)
    pb_aud.tracker.set_tuning(**tun)
    net = SurvivalMLP(max_batch=65536, seed=args.seed)
    fine = bool(args.model)
    if fine:
        net.load(args.model)
    bc = int((args.boundary_cells or "2").split(",")[0])
    pl = float((args.p_lo or "0").split(",")[0])
    with ClockSampler(R.local) as clk:
        pb_ft, fts, ft_s = _staged_scan_sharded(R, lats, rings.CONFIG4_GRID, turns, first, (None,), tun)
        ft = fts[0]
        train = _train_classifier(args, R, pb_ft, [ft], net, fine_tune=fine)
        R.barrier()
        pr = da.sharded_scan(lambda b, e: LD.pruned_scan(pb_rest, net, 0, e - b, seed=args.seed + R.rank,
                                                         boundary_cells=bc, p_lo=pl), nv - first, R.rank, R.world)
        R.barrier()
        plain = da.sharded_scan(lambda b, e: da.plain_scan(pb_aud.tracker, pb_aud.ref, **pb_aud.grid()), n_audit,
                                R.rank, R.world)
    if args.save_model and R.rank == 0:
        net.save(args.save_model)
    ft_surv = (ft.survive >= turns).cpu().numpy()
    da_ft_local = LD.radius_of(pb_ft, ft_surv, pb_ft.n_variants)
    da_ft = da.sharded_radii(da_ft_local, first, R.rank, R.world) if R.dist else da_ft_local
    da_ft = da_ft.mean(axis=(1, 2))
    da_rest = pr.radius.mean(axis=(1, 2))
    da_all = np.concatenate([da_ft, da_rest])
    order = np.argsort(-da_all, kind="stable")
    ranking = LD.ranking_mismatches(da_rest[audit_idx], plain.radius.mean(axis=(1, 2)))
    if R.rank == 0:
        line = {"metric": "sextupole scan: ranking mismatches of pruned vs plain DA, audited variants",
                "value": ranking["discordant_pairs"], "unit": "discordant pairs", "higher_is_better": False,
                "n_gpus": R.world, "scaling": "strong", "dtype": "f64 tracking, bf16/fp32 classifier",
                "data": "synthetic",
                "config": {"workload": "pruned sextupole-setting scan", "variants": nv, "fine_tune_variants": first,
                           "probes_per_variant": pb_rest.per_variant, "turns": turns, "audited_variants": n_audit,
                           "boundary_cells": bc, "p_lo": pl, "start_model": args.model or None,
                           "parallelism": f"variants x{R.world} GPUs"},
                "ranking": ranking, "da_error_audited": da.da_error(pr.radius[audit_idx], plain.radius),
                "pruned_s": pr.wall_s, "fine_tune_scan_s": ft_s, "audit_plain_s": plain.wall_s,
                "audit_plain_s_per_variant": plain.wall_s / n_audit, "pruned_s_per_variant": pr.wall_s / (nv - first),
                "tracked_fraction": R.sum(pr.local.n_tracked) / R.sum(pr.local.n_probes), "train": train,
                "top10_variants_by_da": [[int(i), _mm(da_all[i])] for i in order[:10]],
                "setup_s": t_setup, "tuning": tun, "clocks": clk.summary()}
        print(json.dumps(line), flush=True)
    R.close()


def run_mlp(args):
    """The survival classifier on its own: one step = 200 forward passes over
    --mlp-rows probes each (three tcgen05 layers and the output layer in one
    kernel; 200 passes so the clock sampler sees the timed region)
    and, separately, 200 Adam training steps on an 8,192-sample batch; CUDA
    events on the launching stream.  Beside it the same three layers as torch
    bf16 matmuls (cuBLAS) with ReLU, for context."""
    import torch

    from bgt.mlp import SurvivalMLP

    dev = torch.device("cuda", 0)
    rows = args.mlp_rows
    net = SurvivalMLP(max_batch=65536, seed=args.seed)
    g = torch.Generator(device="cpu").manual_seed(args.seed)
    x = (torch.randn(rows, 64, generator=g) * 0.5).to(dev).to(torch.bfloat16)
    xb = x[:8192].contiguous()
    yb = (torch.rand(8192, generator=g) < 0.3).float().to(dev)

    passes = 200

    def timed(fn, steps, warmup):
        """ms per pass"""
        for _ in range(warmup):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(steps * passes):
            fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / (steps * passes)

    fwd_flops = 2.0 * rows * (64 * 256 + 2 * 256 * 256)
    train_flops = 852_000.0 * 8192  # forward + backward GEMM flops per sample x batch
    l0 = net.launch_count
    with ClockSampler(0) as clk:
        ms_fwd = timed(lambda: net.forward(x), args.steps, args.warmup)
        l1 = net.launch_count
        ms_train = timed(lambda: net.train_step(xb, yb, 1e-4), args.steps, args.warmup)
    per_pass = (l1 - l0) // max(1, args.steps * passes + args.warmup)  # the library's kernels in one forward pass
    w = [(torch.randn(256, k, generator=g) * 0.05).to(dev).to(torch.bfloat16) for k in (64, 256, 256)]

    def torch_fwd():
        a = x
        for wi in w:
            a = torch.relu(a @ wi.T)
        return a

    ms_torch = timed(torch_fwd, args.steps, args.warmup)
    peaks = {}
    try:
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
    except Exception:
        pass
    peak = peaks.get("bf16_tflops", 1590.0)
    tf = fwd_flops / (ms_fwd * 1e-3) / 1e12
    line = {"metric": "survival-classifier forward pass, tcgen05 BF16 GEMMs (FP32 accumulation)",
            "value": tf, "unit": "TFLOP/s", "higher_is_better": True, "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_fwd * passes, "ms_per_forward": ms_fwd, "dtype": "bf16",
            "data": "synthetic",
            "config": {"workload": "64-256-256-256-1 MLP forward", "rows": rows,
                       "passes_per_step": passes},
            "roofline": {"bound": "tensor", "achieved": tf, "peak": peak, "unit": "TFLOP/s", "frac": tf / peak,
                         "peak_source": "MEASURED_PEAKS.json bf16_tflops (burst)" if peaks else "fallback"},
            "train_step": {"batch": 8192, "ms": ms_train,
                           "tflops": train_flops / (ms_train * 1e-3) / 1e12},
            "torch_cublas_forward_ms": ms_torch, "gpu_launches": per_pass * passes * args.steps,
            "clocks": clk.summary()}
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    if args.workload != "track":
        {"da": run_da, "learned-da": run_learned_da, "sext-scan": run_sext_scan,
         "mlp": run_mlp}[args.workload](args)
        return
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
        return

    import torch

    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))

    from bgt import lattice as L
    from bgt import rings
    from bgt.track import Tracker, fp64_peak_tflops

    lat = rings.fodo_ring(apertures=True)
    tr = Tracker(lat, device=local)
    n = args.particles
    spec = rings.CONFIG1_BEAM
    spec = rings.BeamSpec(n, spec.emit_x, spec.emit_y, spec.sigma_z, spec.sigma_pz, spec.seed + 1000 * rank)
    v0 = rings.gaussian_beam(spec)
    dev = torch.device("cuda", local)
    vec = torch.tensor(v0, dtype=torch.float64, device=dev).contiguous()
    beta = torch.tensor(L.beta_of(lat.p0c, v0[5], lat.species.mass), device=dev)
    state = torch.ones(n, dtype=torch.int32, device=dev)
    ixe = torch.full((n,), -1, dtype=torch.int32, device=dev)
    ixt = torch.full((n,), -1, dtype=torch.int32, device=dev)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream(dev)
    T = args.turns_per_step
    tune_info = None
    if args.tuning:
        tpb, bps = (int(x) for x in args.tuning.split(","))
        tr.set_tuning(threads_per_block=tpb, blocks_per_sm=bps)
    elif not args.no_autotune:
        from bgt import autotune

        autotune.tune(tr, v0, turns=2, sample=min(n, 300_000))
        res = autotune.last_results(tr, n)
        tune_info = {"sample": res["sample"], "turns": res["turns"],
                     "candidates_ms": [[round(ms, 3), t["threads_per_block"], t["blocks_per_sm"]]
                                       for ms, t in res["all"]]}

    def barrier():
        if dist:
            dist.barrier()

    turn = 0
    for _ in range(args.warmup):
        tr.track_turns_device(vec, beta, state, ixe, ixt, T, turn0=turn, stream=stream)
        turn += T
    torch.cuda.synchronize()

    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    units = 0
    launches0 = tr.launch_count
    barrier()
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        for k in range(args.steps):
            flush.fill_(float(k))  # evict L2 between timed steps (outside the events)
            alive0 = (state == 1).cpu().numpy()
            t0 = turn
            ev[k][0].record(stream)
            tr.track_turns_device(vec, beta, state, ixe, ixt, T, turn0=turn, stream=stream)
            ev[k][1].record(stream)
            turn += T
            torch.cuda.synchronize()
            units += turns_tracked(alive0, ixt.cpu().numpy(), state.cpu().numpy(), t0, turn)
        torch.cuda.synchronize()
    barrier()
    launches = tr.launch_count - launches0
    ms = sum(a.elapsed_time(b) for a, b in ev)
    t_local = ms / 1e3
    t_max = t_local
    units_all = units
    if dist:
        tt = torch.tensor([t_local], dtype=torch.float64, device=dev)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        t_max = float(tt.item())
        uu = torch.tensor([units], dtype=torch.float64, device=dev)
        dist.all_reduce(uu, op=dist.ReduceOp.SUM)
        units_all = int(uu.item())
    value = units_all / t_max

    # ---- end to end through the public API with host buffers ----
    e2e = None
    if not args.no_e2e:
        hb = tr.make_bunch(v0.copy())
        tr.track_turns(hb, 1)  # warm-up (staging buffers)
        hb = tr.make_bunch(v0.copy())
        e2e_units, e2e_t = 0, 0.0
        for k in range(max(1, min(args.steps, 5))):
            alive0 = hb.state == 1
            t0k = T * k
            barrier()
            ts = time.perf_counter()
            tr.track_turns(hb, T, turn0=t0k)
            e2e_t += time.perf_counter() - ts
            e2e_units += turns_tracked(alive0, hb.ix_turn_lost, hb.state, t0k, t0k + T)
        if dist:
            tt = torch.tensor([e2e_t], dtype=torch.float64, device=dev)
            dist.all_reduce(tt, op=dist.ReduceOp.MAX)
            e2e_t = float(tt.item())
            uu = torch.tensor([e2e_units], dtype=torch.float64, device=dev)
            dist.all_reduce(uu, op=dist.ReduceOp.SUM)
            e2e_units = int(uu.item())
        per = 6 * 8 + 8 + 3 * 4
        e2e = {"value": e2e_units / e2e_t, "unit": UNIT, "h2d_bytes_per_step": per * n,
               "d2h_bytes_per_step": per * n}

    if rank == 0:
        peak = fp64_peak_tflops(local)
        units_per_launch = units / max(1, launches)
        launch_s = t_local / max(1, launches)
        achieved = FLOPS_PER_PARTICLE_TURN * units_per_launch / launch_s / 1e12
        # DRAM bytes per launch: 68.5 B per particle (dram__bytes_read.sum +
        # dram__bytes_write.sum of one ncu capture of this kernel on 400k
        # particles; the written records stay in L2 at kernel end), scaled to
        # this launch's particle count
        roofline = {"bound": "fp64", "achieved": achieved, "peak": peak, "unit": "TFLOP/s",
                    "frac": achieved / peak, "traffic": 68.52 * n,
                    "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum, 400k-particle launch "
                                      "scaled by particle count",
                    "peak_source": "measured: DFMA throughput probe (bgt_fp64_peak_tflops) on this GPU; "
                                   "MEASURED_PEAKS.json has no FP64 figure",
                    "flops_per_unit": FLOPS_PER_PARTICLE_TURN, "libm_calls_per_unit": LIBM_PER_PARTICLE_TURN}
        cpu = None if args.no_cpu_baseline or world > 1 else cpu_baseline()
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak",
                "vs_baseline": None, "dtype": "f64", "data": "synthetic",
                "config": {"workload": "fodo64 ring (770 elements) + apertures, config-1 beam",
                           "particles_per_gpu": n, "turns_per_step": T, "parallelism": f"particles x{world} GPUs",
                           "l2": "flushed between timed steps (256 MB write)"},
                "roofline": roofline, "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches,
                "clocks": clk.summary(), "tuning": tr.get_tuning(), "autotune": tune_info}
        print(json.dumps(line), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
