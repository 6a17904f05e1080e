#!/usr/bin/env python
"""Benchmark of the trajectory hot path on GB300.

Workload: the electrostatic-lens beamline (aperture r = 6 mm at 0.30 m,
hexapole lens 0.80-1.40 m with a 4096-knot Stark spline and RK4 at dt = 1 us,
detection plane at 3 m), 1e7 molecules per GPU, FP32, initial conditions drawn
on the device from x, y ~ N(0, 1.5 mm), vx, vy ~ N(0, 20 m/s), vz ~ N(184, 16).
One step = one full propagation of all molecules (ctraj_run).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Metric: molecule-steps/s = sum over molecules of len(trajectory.t) - 1 (the
reference's trajectory rows after the initial one), counted on the device.

`value` times the K runs as one pipelined ctraj_run_batch with CUDA events on
the engine's stream (runs alternate between two lanes, so one run's ballistic
front overlaps the previous run's lens pass; L2 flushed before every run
inside the timed region); `sequential` times the same runs one ctraj_run at a
time (L2 flushed between them), and those runs give the front / lens split
and the roofline.  `e2e` times the public drop-in TrajectorySimulator
(host Beamline / Distribution objects in, Counters out) with perf_counter:
run_simulations over the K batches, and (run_simulation_loop) one
run_simulation per batch.
`cpu_baseline` and --impl reference time the FP64 C restatement of the
reference (oracle/) on the host cores on a bounded sample of the same workload.
For N > 1 (torchrun) every rank propagates its own 1e7 molecules on disjoint
Philox counters (replicas, weak scaling); time is the max over ranks.

`sweep` (rank 0) times the batched lens sweep -- 256 voltages x 4 Stark
tables, 2.1e8 molecules -- as one graph-replayed ctraj_run_sweep and as the
loop of one plain run per configuration, and checks their counts agree.
`adjoint` (rank 0) times full gradients of the soft transmission at 1e6
molecules (grads/s) against one soft forward and one plain run.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT / "centrex-molecule-trajectories_gb300"))
sys.path.insert(0, str(ROOT))

METRIC = "molecule-steps/s (1e7 lens beamline)"
UNIT = "molecule-steps/s"
# Algorithmic FP32 work per molecule-step, FMA counted as 2 (the lens RK4 step:
# four table-driven force evaluations, stage points, RK4 combination, bore test).
FLOP_PER_RK4_STEP = 114
FLOP_PER_BALLISTIC_STEP = 12
# dram__bytes_read.sum + dram__bytes_write.sum of a grouped k_lens_persist
# launch per 1e7 molecules of the group, from the ncu capture summarised in
# profiles/k_lens_persist_grouped_lens_beamline.md (the queue is read once;
# the table and the molecule state stay on chip)
LENS_DRAM_BYTES_PER_1E7 = 9.72e6
# Shared-memory wavefronts per warp table lookup (the bench table goes to the
# kernels in the 8-byte linear form: one LDS.64 per lane, random intervals,
# bank-conflicted), from l1tex__data_pipe_lsu_wavefronts_mem_shared_op_ld of the
# k_lens_persist capture in profiles/k_lens_persist_lens_beamline_1e7.md:
# 1.14e8 wavefronts for 1.43e8 lane-steps x 4 lookups at 27.15 lanes per warp
# instruction (the 16-byte quadratic form took 9.1).  One wavefront per cycle
# per SM is the roof for the throughput-bound phases of a lens pass.
SHARED_WAVEFRONTS_PER_LOOKUP = 5.4
LOOKUPS_PER_RK4_STEP = 4


def shared_roof(lens_steps_per_s: float, sms: int, mhz: float) -> dict:
    roof = sms * mhz * 1e6 * 32 / (LOOKUPS_PER_RK4_STEP * SHARED_WAVEFRONTS_PER_LOOKUP)
    return {"bound": "shared-memory wavefronts (force-table lookups)", "unit": "RK4 lane-steps/s",
            "wavefronts_per_lookup": SHARED_WAVEFRONTS_PER_LOOKUP, "lookups_per_step": LOOKUPS_PER_RK4_STEP,
            "roof": roof, "achieved": lens_steps_per_s, "frac": lens_steps_per_s / roof,
            "note": "1 shared-memory wavefront per cycle per SM; wavefronts per lookup from ncu"}
L2_NOTE = ("GPU arm: 160 MiB (1.3 x the 126 MiB L2) written before every run on the run's stream inside the timed region; "
           "CPU arm: not applicable")


def bench_config(n: int) -> dict:
    """The workload both arms (this engine and --impl reference) time."""
    return {"workload": WORKLOAD, "molecules_per_step": n, "l2": L2_NOTE}


WORKLOAD = ("lens beamline: aperture r=6mm@0.30m, hexapole lens z0=0.80m L=0.60m R=17.5mm V=30kV "
            "(4096-knot Stark spline, a=h*6.7GHz, d=4.2D), RK4 dt=1us, detection@3.0m; "
            "x,y~N(0,1.5mm) vx,vy~N(0,20m/s) vz~N(184,16m/s)")


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=40)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--molecules", type=float, default=1e7)
    p.add_argument("--cpu-sample", type=float, default=0,
                   help="molecules of the CPU-baseline sample (default: --molecules, the GPU arm's step)")
    p.add_argument("--no-parity", action="store_true", help="skip the full-size parity checks")
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--no-sweep", action="store_true", help="skip the batched-sweep measurement")
    p.add_argument("--no-adjoint", action="store_true", help="skip the gradient measurement")
    p.add_argument("--no-large", action="store_true", help="skip the 1e9-molecule streamed run and the Adam tuning")
    p.add_argument("--profile", nargs="?", const="lens", default=None,
                   choices=["lens", "sweep", "adjoint", "ring", "batch"],
                   help="only run one workload --steps times with the default launch knobs (the commands "
                        "the ncu captures under profiles/ use): the lens beamline (--molecules), the "
                        "batched sweep (counts scaled by --sweep-scale), the gradient at 1e6 molecules, "
                        "a ring-recording run (--molecules), or (batch) --steps lens-beamline runs as one "
                        "pipelined ctraj_run_batch")
    p.add_argument("--sweep-scale", type=float, default=1.0, help="molecule counts of --profile sweep x this")
    p.add_argument("--lens-mode", choices=["persistent", "chunked"], default="persistent",
                   help="--profile lens/sweep: the FP32 lens pass to run (ctraj_tuning.lens_mode)")
    p.add_argument("--batch-group", type=int, default=10, help="--profile batch: runs per shared lens pass")
    p.add_argument("--front-threads", type=int, default=128, help="--profile: threads per front block")
    p.add_argument("--batch-lens-threads", type=int, default=0,
                   help="--profile batch: threads per CTA of the shared lens pass (0: by the queue's length)")
    p.add_argument("--lens-interval", type=int, default=256,
                   help="--profile: RK4 steps between the persistent pass's compactions once its queue is empty")
    p.add_argument("--lens-threads", type=int, default=0,
                   help="--profile lens/sweep: threads per CTA of a run's or a sweep's persistent lens pass "
                        "(0: by the queue's length)")
    return p.parse_args()


def run_profile(args):
    """Plain runs of the workload: no autotuning, probes, flushes or CPU leg."""
    from __graft_entry__ import build
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import device_spec
    from ctraj.engine import Engine
    from ctraj.workloads import lens_beamline, source

    build()
    cb = compile_beamline(lens_beamline())
    xd, vd = source()
    xs, vs = device_spec(xd, "position"), device_spec(vd, "velocity")
    eng = Engine(0)
    eng.set_tuning(lens_mode=0 if args.lens_mode == "persistent" else 1, batch_group=args.batch_group,
                   front_threads=args.front_threads, batch_lens_threads=args.batch_lens_threads,
                   lens_interval=args.lens_interval, lens_threads=args.lens_threads)
    n = int(args.molecules)
    for k in range(args.steps):
        if args.profile == "sweep":
            import numpy as np

            from ctraj.sweep import run_sweep
            from ctraj.workloads import sweep_configs

            if k == 0:
                cfg = sweep_configs()
                cfg.n_molecules = np.maximum(1, np.rint(cfg.n_molecules * args.sweep_scale)).astype(np.int64)
            r = run_sweep(cb, cfg, xdist=xs, vdist=vs, seed=k, timing=True, engine=eng)
            out = {"molecules": cfg.total, "kernels": r.kernels, **r.extra, "molecule_steps": r.molecule_steps}
        elif args.profile == "adjoint":
            from ctraj.adjoint import SoftProblem, soft_transmission

            prob = SoftProblem.from_beamline(lens_beamline(), n=1_000_000, aperture="A1", seed=k)
            o = soft_transmission(prob, prob.initial_params(), engine=eng, timing=True)
            out = {"loss": o.loss, "grad": o.grad.tolist(), "kernels": o.kernels, **o.extra}
        elif args.profile == "batch":  # the headline: --steps runs as one pipelined batch
            rs = eng.run_batch(cb, n, list(range(args.steps)), xdist=xs, vdist=vs)
            for j, r in enumerate(rs):
                print(json.dumps({"run": j, "profile": "batch", "kernels": r.kernels,
                                  "molecule_steps": r.molecule_steps, "counts": r.counter_dict()}), flush=True)
            break
        else:
            ring = None
            if args.profile == "ring":
                from ctraj.ring import HBMRing

                ring = HBMRing(capacity_rows=50_000_000, capacity_molecules=5_000_000, stride=50)
            r = eng.run(cb, n, xdist=xs, vdist=vs, seed=k, timing=True, ring=ring)
            out = {"kernels": r.kernels, **r.extra, "molecule_steps": r.molecule_steps,
                   "lens_steps": r.lens_steps, "counts": r.counter_dict()}
            if ring is not None:
                out["ring"] = ring.counts()
        print(json.dumps({"run": k, "profile": args.profile, **out}), flush=True)
    eng.close()


# ---------------------------------------------------------------------------
def cpu_sample(n: int, threads: int, seed: int):
    """The oracle (FP64 C restatement of the reference) on n molecules: host draw + propagation."""
    import ctraj
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import host_draw
    from ctraj.workloads import lens_beamline, source
    from oracle import oracle

    cb = compile_beamline(lens_beamline())
    xd, vd = source()
    t0 = time.perf_counter()
    ics = host_draw(xd, vd, n, seed=seed)
    r = oracle.run(cb, ics, threads=threads, outputs=False)
    dt = time.perf_counter() - t0
    return r["steps"], dt


def reference_python_rate():
    """The reference's own Python run_simulation(n_jobs=cores) on this workload,
    measured where the reference is installed (oracle/measure_reference_python.py
    wrote the file); labelled, never part of the GPU/CPU ratio."""
    path = ROOT / "oracle" / "reference_python_rate.json"
    try:
        r = json.loads(path.read_text())
    except (OSError, ValueError):
        return None
    return {"value": r["value"], "unit": UNIT, "cores": r["cores"], "machine": r["machine"],
            "molecules": r["molecules"], "steps_per_molecule": r["steps_per_molecule"], "api": r["api"],
            "recipe": r["recipe"], "when": r["when"],
            "note": "measured in the container holding the reference (not the GPU machine, where the reference "
                    "is not installed); reported for reference only, not used in any ratio"}


def config0_oracle_check(gpu):
    """Config 0 (ballistic beamline, 1e5 molecules, numpy default_rng(0) initial
    conditions): the oracle on the same initial conditions as the GPU FP64 run
    `gpu` (from config0_gpu), labels and final rows compared bit for bit."""
    import numpy as np

    from ctraj.compiler import compile_beamline
    from ctraj.workloads import ballistic_beamline
    from oracle import oracle

    cb = compile_beamline(ballistic_beamline())
    o = oracle.run(cb, gpu["ics"], threads=os.cpu_count() or 1)
    fin = np.isfinite(o["final"]).all(0) & np.isfinite(gpu["final"]).all(0)
    return {"labels_equal": bool(np.array_equal(o["label"], gpu["label"])),
            "final_rows_equal": bool(np.array_equal(o["final"][:, fin], gpu["final"][:, fin])
                                     and np.array_equal(fin, np.isfinite(o["final"]).all(0))),
            "counts_equal": bool(np.array_equal(o["counts"], gpu["counts"])),
            "molecule_steps_equal": bool(o["steps"] == gpu["molecule_steps"])}


def cpu_baseline(n: int, config0=None):
    """The oracle on all host cores on one sample of n molecules of the bench
    workload, plus (config0) the oracle side of the config-0 parity check."""
    threads = os.cpu_count() or 1
    cpu_sample(min(n, 100_000), threads, seed=99)  # warm-up: library load, page-in
    steps, secs = cpu_sample(n, threads, seed=100)
    out = {"value": steps / secs, "unit": UNIT, "cores": threads, "kind": "port",
           "sample": f"{n} molecules of the same workload (one run), ICs drawn on the host (numpy), "
                     f"FP64 oracle/ctraj_oracle.c on {threads} threads, {secs:.2f} s",
           "reference_python": reference_python_rate()}
    if config0 is not None:
        out["config0_check"] = config0_oracle_check(config0)
    return out


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    n = int(args.molecules)
    threads = os.cpu_count() or 1
    for k in range(args.warmup):
        cpu_sample(min(n, 100_000), threads, seed=k)
    steps = secs = 0
    for k in range(args.steps):
        s, dt = cpu_sample(n, threads, seed=1000 + k)
        steps += s
        secs += dt
    v = steps / secs
    line = {"metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": secs / args.steps * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded numpy draws)",
            "impl": "reference", "config": bench_config(n),
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
                             "sample": f"{n} molecules per step (the GPU arm's step), {args.warmup} warm-up "
                                       f"steps of {min(n, 100_000)}; the reference is pure Python and "
                                       f"cannot run on the GPU machine, so its FP64 C restatement "
                                       f"(oracle/) is timed on {threads} threads",
                             "reference_python": reference_python_rate()},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
class Clocks:
    """nvidia-smi samples of SM clock and throttle reasons during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=self.file, stderr=subprocess.DEVNULL)
            time.sleep(0.3)
        except OSError:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc:
            time.sleep(0.2)
            self.proc.terminate()
            self.proc.wait()

    def summary(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.file.seek(0)
        rows = [r.split(",") for r in self.file.read().strip().splitlines() if r.count(",") >= 8]
        os.unlink(self.file.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows]
        mx = max(float(r[2]) for r in rows)
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].strip() == "Active"})
        busy = [s for s in sm if s > 0.5 * mx] or sm
        return {"sm_mhz": statistics.median(busy), "sm_max_mhz": mx, "reasons": reasons,
                "samples": len(rows), "power_w_max": max(float(r[3]) for r in rows)}


def fp32_peak(device: int):
    from bench_kernels.build import build as build_probes

    lib = ctypes.CDLL(str(build_probes()))
    lib.ctraj_peak_fp32.restype = ctypes.c_int
    lib.ctraj_peak_fp32.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_double),
                                    ctypes.POINTER(ctypes.c_double)]
    best = 0.0
    for _ in range(3):
        tf, ms = ctypes.c_double(), ctypes.c_double()
        if lib.ctraj_peak_fp32(device, 20000, ctypes.byref(tf), ctypes.byref(ms)) == 0:
            best = max(best, tf.value)
    return best


def step_probe(device: int, bl):
    """The production FP32 lens step in a loop: cycles per step of a lone warp
    (latency floor) and lane-steps/s at 512 threads per SM, as the persistent
    lens pass runs (throughput without queue, compaction or loss effects)."""
    import numpy as np
    import torch

    from bench_kernels.build import build as build_probes

    lens = [e for e in bl.elements if type(e).__name__ == "ElectrostaticLens"][0]
    F = lens.a_interp
    h = (F.knots[-1] - F.knots[0]) / (len(F.knots) - 1)
    kappa = 2.0 * F.alpha / F.mass
    # the lens kernels' layout for this table (kForceStark2Lin): per knot
    # interval four linear quarter-interval pieces (w, dw) in two float4
    a = -kappa * F.coef[:, 2]
    b = -kappa * 2.0 * F.coef[:, 1] * h
    c = -kappa * 3.0 * F.coef[:, 0] * h * h
    w = [a + (k / 4) * (b + (k / 4) * c) for k in range(5)]
    pieces = np.stack([x for k in range(4) for x in (w[k], w[k + 1] - w[k])], axis=1)  # (n_int, 8)
    q = np.ascontiguousarray(pieces.astype(np.float32).reshape(-1, 4))  # 2 float4 per interval
    qd = torch.from_numpy(q).to(f"cuda:{device}")
    # the exact quadratic form (kForceStark2), for the latency comparison
    qq = np.zeros((len(F.coef), 4), np.float32)
    qq[:, 0], qq[:, 1], qq[:, 2] = a, b, c
    qqd = torch.from_numpy(qq).to(f"cuda:{device}")
    lib = ctypes.CDLL(str(build_probes()))
    lib.ctraj_peak_step.restype = ctypes.c_int
    lib.ctraj_peak_step.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_int, ctypes.c_int,
                                    ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_double),
                                    ctypes.POINTER(ctypes.c_double)]
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    out = {}
    runs = (("one_warp", qd, len(q), 4.0, 1, 1, 32), ("full", qd, len(q), 4.0, 1, sms, 512),
            ("one_warp_quadratic", qqd, len(qq), 1.0, 0, 1, 32))
    for key, table, n_int, scale, linear, blocks, threads in runs:
        cyc, lps = ctypes.c_double(), ctypes.c_double()
        rc = lib.ctraj_peak_step(ctypes.c_void_p(table.data_ptr()), n_int, ctypes.c_float(scale * F.alpha / h),
                                 linear, 4096, blocks, threads, ctypes.byref(cyc), ctypes.byref(lps))
        out[key] = (cyc.value, lps.value) if rc == 0 else (None, None)
    return {"one_warp_cycles_per_step": out["one_warp"][0],
            "one_warp_cycles_per_step_quadratic_table": out["one_warp_quadratic"][0],
            "isolated_lane_steps_per_s": out["full"][1],
            "isolated_tflops": None if out["full"][1] is None else out["full"][1] * FLOP_PER_RK4_STEP / 1e12}


def bench_sweep(eng, stream, flush, steps: int, warmup: int, device_name: str):
    """The batched lens sweep (256 voltages x 4 Stark tables, log-uniform
    molecules per configuration) as one graph-replayed ctraj_run_sweep, against
    the same configurations looped through the plain path (ctraj_run each)."""
    import numpy as np
    import torch

    from ctraj.distributions import device_spec
    from ctraj.sweep import config_beamlines, loop_sweep, run_sweep, sweep_beamline
    from ctraj.tuning import autotune
    from ctraj.workloads import lens_beamline, source, sweep_configs

    cfg = sweep_configs()
    bl = lens_beamline()
    cb = sweep_beamline(bl)
    xd, vd = source()
    xs, vs = device_spec(xd, "position"), device_spec(vd, "velocity")
    plain_tuning = eng.get_tuning()

    def sweep(seed, timing=False):
        return run_sweep(cb, cfg, xdist=xs, vdist=vs, seed=seed, use_graph=True, timing=timing, engine=eng)

    def measure():
        r = sweep(5, timing=True)
        return r.extra["front_ms"] + r.extra["lens_ms"]

    for k in range(warmup):
        sweep(k)
    tuned = autotune(eng, cb, cfg.total, {}, device_name=device_name, measure=measure, key_extra="|sweep")
    for k in range(warmup):
        sweep(k)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times, res = [], []
    for k in range(steps):
        flush.zero_()
        ev0.record(stream)
        r = sweep(100 + k, timing=True)
        ev1.record(stream)
        ev1.synchronize()
        times.append(ev0.elapsed_time(ev1))
        res.append(r)
    sweep_ms = sum(times) / steps
    msteps = sum(r.molecule_steps for r in res) / steps
    lsteps = sum(r.lens_steps for r in res) / steps
    lens_ms = sum(r.extra["lens_ms"] for r in res) / steps
    # the loop of plain runs, on the same seed as the last sweep: counts must agree
    eng.set_tuning(**plain_tuning)
    cbs = config_beamlines(bl, cfg)
    for cbx in cbs[:8]:  # warm-up: first runs of each kernel
        eng.run(cbx, 10_000, xdist=xs, vdist=vs, seed=0)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    loop = loop_sweep(cbs, cfg, xdist=xs, vdist=vs, seed=100 + steps - 1, engine=eng)
    loop_ms = (time.perf_counter() - t0) * 1e3
    diff = np.abs(loop - res[-1].counts).sum(-1)
    return {"workload": "256 lens voltages U[0,30kV] x 4 Stark tables (a=h*{6.7,13.3,20.0,26.6}GHz), "
                        "molecules per configuration log-uniform [1e4,1e6] (numpy default_rng(0))",
            "configs": cfg.n_configs, "molecules": cfg.total, "molecule_steps": msteps,
            "ms_per_sweep": sweep_ms, "molecule_steps_per_s": msteps / (sweep_ms / 1e3),
            "gpu_launches_per_sweep": res[-1].kernels, "cuda_graph": True,
            "loop_of_plain_runs_ms": loop_ms, "speedup_vs_loop": loop_ms / sweep_ms,
            "loop_count_difference": {"max_per_config": int(diff.max()), "total": int(diff.sum())},
            "tuning": tuned["tuning"], "tuning_cached": tuned.get("cached", False),
            "lens_ms": lens_ms, "lens_steps": lsteps,
            # at the GB300's maximum SM clock (the sweep runs outside the sampled region)
            "roofline": shared_roof(lsteps / (lens_ms / 1e3), torch.cuda.get_device_properties(0).multi_processor_count,
                                    2070.0),
            "timing": "CUDA events on the launching stream around ctraj_run_sweep (counts back on the host), "
                      "L2 flushed before each; loop timed with perf_counter"}


def bench_adjoint(eng, stream, flush, steps: int, warmup: int):
    """Full gradients of the soft transmission (sigmoid edges of width 0.2 mm)
    of the lens beamline with respect to (V, lens z0, r_A1, r_bore, sigma_vx,
    sigma_vy) at 1e6 molecules, FP32 discrete adjoint (checkpoint every 64
    steps), against one soft forward and one plain (hard-count) run of the same
    molecules; plus a central-difference check (h = 1e-4 relative) of the
    gradient on 1e5 molecules with the FP64 forward."""
    import numpy as np
    import torch

    from ctraj.adjoint import PARAM_NAMES, SoftProblem, soft_transmission
    from ctraj.distributions import device_spec
    from ctraj.workloads import lens_beamline, source

    n = 1_000_000
    prob = SoftProblem.from_beamline(lens_beamline(), n=n, aperture="A1", precision=32, checkpoint=64)
    p0 = prob.initial_params()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def timed(fn):
        ts = []
        for k in range(warmup):
            fn(k)
        for k in range(steps):
            flush.zero_()
            ev0.record(stream)
            out = fn(100 + k)
            ev1.record(stream)
            ev1.synchronize()
            ts.append(ev0.elapsed_time(ev1))
        return sum(ts) / len(ts), out

    def grad(seed):
        prob.seed = seed
        return soft_transmission(prob, p0, want_grad=True, engine=eng)

    def fwd(seed):
        prob.seed = seed
        return soft_transmission(prob, p0, want_grad=False, engine=eng)

    xd, vd = source()
    xs, vs = device_spec(xd, "position"), device_spec(vd, "velocity")

    def hard(seed):
        return eng.run(prob.cb, n, xdist=xs, vdist=vs, seed=seed)

    grad_ms, g = timed(grad)
    fwd_ms, f = timed(fwd)
    hard_ms, h = timed(hard)
    # finite-difference check on 1e5 molecules
    small = SoftProblem.from_beamline(lens_beamline(), n=100_000, aperture="A1", precision=64, seed=3)
    small32 = SoftProblem.from_beamline(lens_beamline(), n=100_000, aperture="A1", precision=32, seed=3)
    fd = np.zeros(6)
    for k in range(6):
        hk = 1e-4 * abs(p0[k])
        pp, pm = p0.copy(), p0.copy()
        pp[k] += hk
        pm[k] -= hk
        fd[k] = (soft_transmission(small, pp, want_grad=False, engine=eng).loss
                 - soft_transmission(small, pm, want_grad=False, engine=eng).loss) / (2 * hk)
    ga = soft_transmission(small32, p0, engine=eng).grad
    rel = np.abs(ga - fd) / np.maximum(np.abs(fd), 1e-300)
    return {"workload": "soft transmission of the lens beamline (sigmoid edges, width 0.2 mm), 1e6 molecules, "
                        "FP32, gradient w.r.t. " + ", ".join(PARAM_NAMES),
            "grads_per_s": 1e3 / grad_ms, "ms_per_gradient": grad_ms, "soft_forward_ms": fwd_ms,
            "plain_run_ms": hard_ms, "gradient_over_soft_forward": grad_ms / fwd_ms,
            "gradient_over_plain_run": grad_ms / hard_ms, "checkpoint_steps": 64,
            "loss": g.loss, "gradient": dict(zip(PARAM_NAMES, map(float, g.grad))),
            "lens_molecules": g.lens_molecules, "lens_steps": g.lens_steps,
            "gpu_launches_per_gradient": g.kernels,
            "fd_check": {"molecules": 100_000, "h": "1e-4 relative, central, FP64 forward",
                         "max_rel_error_fp32_adjoint": float(rel.max())},
            "timing": "CUDA events on the launching stream around the call (result on the host), L2 flushed before each"}


EDGE_BAND = 1e-6   # m: molecules nearer than this to an edge (FP64 margin) may change label in FP32
POS_TOL = 1e-6     # m: FP32 final positions against FP64


def parity_config1(eng, cb, n: int, seed: int, xs, vs, timed_counts=None) -> dict:
    """The bench workload at its full size: the FP32 run (the timed path, with
    per-molecule outputs) against the FP64 run of the same Philox stream.  Every
    molecule farther than 1 um from an edge (FP64 margin) must get the same
    label, and the same-label molecules' final x, y must agree within 1 um."""
    import torch

    outs, runs = {}, {}
    for prec in (32, 64):
        o = {"label": torch.empty(n, dtype=torch.int32, device="cuda"),
             "final": torch.empty((10, n), dtype=torch.float64, device="cuda"),
             "margin": torch.empty(n, dtype=torch.float64, device="cuda")}
        runs[prec] = eng.run(cb, n, precision=prec, xdist=xs, vdist=vs, seed=seed, device_outputs=o, timing=True)
        outs[prec] = o
    o32, o64 = outs[32], outs[64]
    far = o64["margin"] >= EDGE_BAND
    same = (o32["label"] == o64["label"]) & far
    d = (o32["final"][:, same] - o64["final"][:, same]).abs()
    m = lambda t: float(t.max()) if t.numel() else 0.0  # noqa: E731
    r32, r64 = runs[32], runs[64]
    out = {"workload": "the bench workload (lens beamline, FP32) against FP64 on the same Philox stream",
           "molecules": n, "seed": seed,
           "edge_band": int((~far).sum()),
           "label_mismatch_off_band": int(((o32["label"] != o64["label"]) & far).sum()),
           "label_mismatch_in_band": int(((o32["label"] != o64["label"]) & ~far).sum()),
           "max_abs_dx_m": m(d[0]), "max_abs_dy_m": m(d[1]), "max_abs_dv_m_per_s": m(d[3:6]),
           "max_abs_dt_s": m(d[9]), "position_tolerance_m": POS_TOL,
           "counts_fp32": r32.counter_dict(), "counts_fp64": r64.counter_dict(),
           "detected_fraction_fp32": float(r32.counts[-1]) / n, "detected_fraction_fp64": float(r64.counts[-1]) / n,
           "fp64_ms": r64.extra.get("front_ms", 0.0) + r64.extra.get("lens_ms", 0.0)}
    if timed_counts is not None:
        out["fp32_counts_equal_timed_run"] = bool(list(timed_counts) == list(r32.counts))
    out["pass"] = (out["label_mismatch_off_band"] == 0 and out["max_abs_dx_m"] <= POS_TOL
                   and out["max_abs_dy_m"] <= POS_TOL)
    del outs, o32, o64, d
    torch.cuda.empty_cache()
    return out


def config0_gpu(eng, n: int = 100_000, seed: int = 0) -> dict:
    """Config 0: the plain ballistic beamline (apertures r = 6 mm at 0.30 m,
    10 x 8 mm at 1.00 m, r = 10 mm at 2.00 m, detection plane at 3.00 m) in FP64,
    n molecules drawn on the host with numpy default_rng(seed) from the bench's
    distributions; per-element counts and the detected fraction."""
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import host_draw
    from ctraj.workloads import ballistic_beamline, source

    cb = compile_beamline(ballistic_beamline())
    xd, vd = source()
    ics = host_draw(xd, vd, n, seed=seed)
    r = eng.run(cb, n, precision=64, ics=ics, outputs=True)
    return {"ics": ics, "label": r.label, "final": r.final, "counts": r.counts, "molecule_steps": r.molecule_steps,
            "report": {"workload": "ballistic beamline (config 0), FP64, initial conditions numpy "
                                   f"default_rng({seed})", "molecules": n, "seed": seed,
                       "counts": r.counter_dict(), "detected_fraction": float(r.counts[-1]) / n,
                       "molecule_steps": int(r.molecule_steps)}}


def bench_large(eng, stream, flush, n_total: int = 1_000_000_000, chunk: int = 134_000_000):
    """The lens beamline at 1e9 molecules, streamed in runs of 1.34e8 with the
    molecules lost on the lens recorded every 50 RK4 steps into an HBM ring,
    then 200 Adam steps on (lens V, lens z0) through the adjoint at 1e6
    molecules per step."""
    import numpy as np
    import torch

    from ctraj.adjoint import SoftProblem, soft_transmission
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import device_spec
    from ctraj.ring import HBMRing, HostRingStore
    from ctraj.stream import adam_tune, run_streamed
    from ctraj.workloads import lens_beamline, source

    cb = compile_beamline(lens_beamline())
    xd, vd = source()
    xs, vs = device_spec(xd, "position"), device_spec(vd, "velocity")
    eng.set_tuning()  # default knobs (persistent lens pass), not the sweep's
    # sized for one run's records (~4e7 rows of a 1.34e8-molecule run) and
    # drained to pinned host memory after every run: nothing is overwritten
    ring = HBMRing(capacity_rows=64_000_000, capacity_molecules=6_000_000, stride=50)
    store = HostRingStore(keep=False)
    run_streamed(cb, 2_000_000, chunk=chunk, xdist=xs, vdist=vs, seed=1, ring=ring, engine=eng, drain=store)  # warm-up
    ring.reset()
    store = HostRingStore(keep=False)
    torch.cuda.synchronize()
    flush.zero_()
    t0 = time.perf_counter()
    st = run_streamed(cb, n_total, chunk=chunk, xdist=xs, vdist=vs, seed=2, ring=ring, engine=eng, drain=store)
    torch.cuda.synchronize()
    wall = time.perf_counter() - t0
    rows, mols = st.ring_rows, st.ring_molecules
    # Adam on V and z0, focusing onto a detector aperture: the config-1
    # geometry with a 10 mm aperture at 3.0 m and the Stark curve's
    # low-field-seeking sign (the hexapole defocuses the workload's
    # high-field-seeking state, for which switching the lens off is optimal)
    det_bl = dict(detector_d=10e-3, low_field_seeker=True)
    prob = SoftProblem.from_beamline(lens_beamline(**det_bl), n=1_000_000, aperture="A1", precision=32)
    p0 = prob.initial_params()
    p0[0] = 10e3  # a detuned lens (10 kV) for Adam to tune
    adam_tune(prob, steps=3, params0=p0, engine=eng)  # warm-up
    opt = adam_tune(prob, which=("V", "lens_z0"), steps=200, lr=0.01, params0=p0, engine=eng, seed0=1000)
    prob.seed = 99
    before = soft_transmission(prob, p0, want_grad=False, engine=eng).loss
    after = soft_transmission(prob, opt["params"], want_grad=False, engine=eng).loss
    lim = prob.param_bounds()

    def hard_detected(V, z0, n=10_000_000):
        r = eng.run(compile_beamline(lens_beamline(V=V, z0=z0, **det_bl)), n, xdist=xs, vdist=vs, seed=4242)
        return int(r.counts[-1])

    hard_before = hard_detected(p0[0], p0[1])
    hard_design = hard_detected(30e3, 0.80)
    hard_after = hard_detected(opt["params"][0], opt["params"][1])
    return {"workload": f"lens beamline, {n_total:.0e} molecules streamed in runs of {chunk:.3g}, "
                        "molecules lost on the lens recorded every 50 RK4 steps into an HBM ring "
                        "drained to host memory after every run; then 200 Adam steps on (lens V, lens z0) "
                        "at 1e6 molecules per step, focusing the low-field-seeking state onto a 10 mm "
                        "detector aperture at 3.0 m",
            "molecules": n_total, "runs": st.chunks, "molecule_steps": st.molecule_steps,
            "seconds": wall, "molecule_steps_per_s": st.molecule_steps / wall,
            "kernel_ms_sum": float(sum(st.chunk_ms)), "gpu_launches": st.kernels,
            "counts": st.counter_dict(), "ring_rows": rows, "ring_molecules": mols,
            "ring_capacity_rows": ring.capacity_rows, "ring_capacity_molecules": ring.capacity_molecules,
            "rows_drained_to_host": store.rows_total, "molecules_drained_to_host": store.molecules_total,
            "rows_lost": st.rows_lost, "molecules_lost": st.molecules_lost,
            "ring_drain": "after every run the ring's records are copied to pinned host memory and the ring "
                          "is emptied (inside the timed wall clock)",
            "adam": {"steps": 200, "seconds": opt["seconds"], "steps_per_s": 200 / opt["seconds"],
                     "beamline": "A1 r=6mm@0.30m, hexapole lens (low-field-seeking two-level curve), "
                                 "detector aperture r=5mm@3.0m",
                     "V_start": float(p0[0]), "V_end": float(opt["params"][0]),
                     "z0_start": float(p0[1]), "z0_end": float(opt["params"][1]),
                     "z0_bounds": [float(lim[1, 0]), float(lim[1, 1])],
                     "soft_transmission_start": before, "soft_transmission_end": after,
                     "hard_detected_start": hard_before, "hard_detected_end": hard_after,
                     "hard_detected_design_30kV_0.80m": hard_design,
                     "hard_molecules": 10_000_000},
            "timing": "wall clock (perf_counter) around the streamed runs incl. host syncs between runs"}


def main():
    args = parse()
    if args.impl == "reference":
        return run_reference(args)
    if args.profile:
        return run_profile(args)

    import numpy as np
    import torch
    import torch.distributed as dist

    from __graft_entry__ import build
    from ctraj.compiler import compile_beamline
    from ctraj.distributions import device_spec
    from ctraj.engine import default_engine
    from ctraj.trajectory_simulator import TrajectorySimulator
    from ctraj.tuning import autotune, batch_measure
    from ctraj.workloads import lens_beamline, source

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    torch.cuda.set_device(local)
    if rank == 0:
        build()
    if world > 1:
        dist.barrier()

    n = int(args.molecules)
    bl = lens_beamline()
    cb = compile_beamline(bl)
    xdist, vdist = source()
    xs, vs = device_spec(xdist, "position"), device_spec(vdist, "velocity")
    eng = default_engine(local)  # the engine the drop-in TrajectorySimulator uses too
    stream = torch.cuda.current_stream()
    eng.set_stream(stream.cuda_stream)
    flush = torch.empty(160 << 20, dtype=torch.uint8, device="cuda")  # 1.3 x the 126 MiB (129 MB) L2

    def step(seed):
        return eng.run(cb, n, precision=32, xdist=xs, vdist=vs, seed=seed, offset=rank * n, timing=True)

    for k in range(args.warmup):
        step(seed=k)
    # launch knobs picked on this workload (outside the timed region), then re-warm
    run_kw = dict(precision=32, xdist=xs, vdist=vs, seed=7, offset=rank * n)
    tuned = autotune(eng, cb, n, run_kw, device_name=torch.cuda.get_device_name(local),
                     batch=batch_measure(eng, cb, n, run_kw, runs=args.steps, l2_flush_bytes=flush.numel()))
    for k in range(args.warmup):
        step(seed=k)
    # a batch of as many runs as the timed one: its groups' buffers are sized
    # before the timed region (with cached knobs the tuner runs no batch)
    eng.run_batch(cb, n, list(range(max(2, args.steps))), precision=32, xdist=xs, vdist=vs, offset=rank * n,
                  l2_flush_bytes=flush.numel())
    peak = fp32_peak(local)
    probe = step_probe(local, bl)

    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    seeds = [1000 + k for k in range(args.steps)]
    times, results = [], []
    with Clocks(local) as clk:
        # the K runs one at a time: the front / lens-pass split and the roofline
        for k in range(args.steps):
            flush.zero_()
            ev0.record(stream)
            r = step(seed=seeds[k])
            ev1.record(stream)
            ev1.synchronize()
            times.append(ev0.elapsed_time(ev1))
            results.append(r)
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        # the headline: the same K runs as one pipelined batch, the L2 flush
        # written on the lane's stream before every run inside the timed region
        ev0.record(stream)
        batch = eng.run_batch(cb, n, seeds, precision=32, xdist=xs, vdist=vs, offset=rank * n,
                              l2_flush_bytes=flush.numel(), timing=True)
        ev1.record(stream)
        ev1.synchronize()
        batch_ms = ev0.elapsed_time(ev1)
        tun = eng.get_tuning()  # the headline's knobs (the sweep and adjoint below set their own)
        # the dominant kernel alone: one group of batch_group runs (one lane,
        # nothing beside it); its lens pass (ordering, k_lens_persist,
        # k_lens_finish) timed with CUDA events on the lane's stream
        iso = []
        for rep in range(3):
            flush.zero_()
            rs = eng.run_batch(cb, n, seeds[:tun["batch_group"]], precision=32, xdist=xs, vdist=vs,
                               offset=rank * n, timing=True)
            iso.append((sum(r.extra.get("lens_ms", 0.0) for r in rs), sum(r.lens_steps for r in rs), len(rs)))
        torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    for a, b in zip(results, batch):  # the batch must reproduce the single runs
        if list(a.counts) != list(b.counts) or a.molecule_steps != b.molecule_steps:
            raise RuntimeError("ctraj_run_batch differs from ctraj_run on the same seeds")
    clocks = clk.summary()
    seq_ms = sum(times)
    total_ms = batch_ms
    steps = sum(r.molecule_steps for r in batch)
    lens_steps = sum(r.lens_steps for r in results)
    lens_ms = sum(r.extra["lens_ms"] for r in results)
    front_ms = sum(r.extra["front_ms"] for r in results)
    if world > 1:
        t = torch.tensor([total_ms, seq_ms], dtype=torch.float64, device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        s = torch.tensor([steps], dtype=torch.float64, device="cuda")
        dist.all_reduce(s, op=dist.ReduceOp.SUM)
        total_ms, seq_ms, steps_all = float(t[0].item()), float(t[1].item()), float(s.item())
    else:
        steps_all = float(steps)
    value = steps_all / (total_ms / 1e3)
    sequential = {"value": steps_all / (seq_ms / 1e3), "ms_per_step": seq_ms / args.steps,
                  "api": "ctraj_run once per step (Engine.run), L2 flushed between steps outside the events"}

    # end to end through the public drop-in API
    e2e = None
    if not args.no_e2e:
        sim = TrajectorySimulator(device=local)
        names = [f"run{k}" for k in range(args.steps)]
        for k in range(max(1, args.warmup)):
            sim.run_simulation(bl, "warm", vdist=vdist, xdist=xdist, N_traj=n, seed=k)
        sim.run_simulations(bl, names[:2], vdist=vdist, xdist=xdist, N_traj=n, seeds=[0, 1])
        tab = cb.tables[0]
        upload = (tab.knots.nbytes + tab.coef.nbytes + (tab.knots.size - 1) * 16
                  + ctypes.sizeof(cb.elements))
        d2h = 8 * (len(cb.labels) + 1) + 64

        def timed(fn):
            torch.cuda.synchronize()
            if world > 1:
                dist.barrier()
            t0 = time.perf_counter()
            got = fn()
            el = time.perf_counter() - t0
            if world > 1:
                t = torch.tensor([el], dtype=torch.float64, device="cuda")
                dist.all_reduce(t, op=dist.ReduceOp.MAX)
                el = float(t.item())
                s = torch.tensor([got], dtype=torch.float64, device="cuda")
                dist.all_reduce(s, op=dist.ReduceOp.SUM)
                got = float(s.item())
            return got / el, el

        def loop():  # the L2 flushed before every call, inside the timed region
            tot = 0
            for k in range(args.steps):
                flush.zero_()
                torch.cuda.synchronize()
                sim.run_simulation(bl, names[k], vdist=vdist, xdist=xdist, N_traj=n, seed=2000 + k)
                tot += sim.last_run.molecule_steps
            return tot

        def pipelined():  # the L2 flushed before every batch on its lane, as in the headline
            sim.run_simulations(bl, names, vdist=vdist, xdist=xdist, N_traj=n,
                                seeds=[2000 + k for k in range(args.steps)], l2_flush_bytes=flush.numel())
            return sum(r.molecule_steps for r in sim.last_runs)

        v_loop, s_loop = timed(loop)
        v_pipe, s_pipe = timed(pipelined)
        # run_simulations compiles and uploads the beamline once per call for
        # each of the two lanes; run_simulation once per call
        e2e = {"value": v_pipe, "unit": UNIT, "h2d_bytes_per_step": int(round(2 * upload / args.steps)),
               "d2h_bytes_per_step": int(d2h),
               "api": "ctraj.TrajectorySimulator.run_simulations(beamline, run_names, vdist, xdist, N_traj=1e7): "
                      "the loop of run_simulation over K batches as one pipelined call",
               "l2": "160 MiB written before every batch on its lane's stream, inside the timed region",
               "ms_per_step": s_pipe / args.steps * 1e3,
               "run_simulation_loop": {"value": v_loop, "ms_per_step": s_loop / args.steps * 1e3,
                                       "h2d_bytes_per_step": int(upload), "d2h_bytes_per_step": int(d2h),
                                       "api": "ctraj.TrajectorySimulator.run_simulation once per batch",
                                       "l2": "160 MiB written (and synchronized) before every call, inside the "
                                             "timed region"}}

    if rank != 0:
        return
    # parity at the quoted sizes (outside the timed region): config 1 on the
    # last timed step's Philox stream, config 0 at 1e5 (its oracle check runs
    # in the CPU-baseline leg below)
    parity = None
    cfg0 = None
    if not args.no_parity:
        parity = {"config1": parity_config1(eng, cb, n, seeds[-1], xs, vs, timed_counts=batch[-1].counts)}
        cfg0 = config0_gpu(eng)
        parity["config0"] = cfg0["report"]
    sweep = None if args.no_sweep else bench_sweep(eng, stream, flush, args.steps, args.warmup,
                                                   torch.cuda.get_device_name(local))
    adjoint = None if args.no_adjoint else bench_adjoint(eng, stream, flush, args.steps, args.warmup)
    large = None if args.no_large else bench_large(eng, stream, flush)
    # the headline's dominant kernel: the lens pass a batch group shares (one
    # k_lens_persist launch per group, after its three ordering launches),
    # timed with CUDA events on the lane's stream inside the timed batch
    groups = -(-args.steps // tun["batch_group"]) if tun["lens_mode"] == 0 else args.steps
    g_lens_ms = sum(r.extra.get("lens_ms", 0.0) for r in batch)
    g_lens_steps = sum(r.lens_steps for r in batch)
    iso_ms = sum(t for t, _, _ in iso) / len(iso)
    iso_steps, iso_runs = iso[-1][1], iso[-1][2]
    achieved = iso_steps * FLOP_PER_RK4_STEP / (iso_ms / 1e3) / 1e12
    mhz = clocks.get("sm_mhz") if clocks else None
    sms = torch.cuda.get_device_properties(local).multi_processor_count
    roofline = {"bound": "fp32",
                "kernel": f"k_lens_persist, grouped: the lens pass {tun['batch_group']} runs of the batch share "
                          f"({tun['batch_lens_threads'] or 'by the queue 512, 768 or 1024'} threads per CTA, one CTA "
                          f"per SM; with its entrant "
                          f"ordering and k_lens_finish, timed together)",
                "achieved": achieved, "peak": peak, "unit": "TFLOP/s", "frac": achieved / peak if peak else None,
                "peak_source": "measured in this run: FMA-chain kernel (bench_kernels/fp32_peak.cu), "
                               "MEASURED_PEAKS.json has no FP32 CUDA-core figure",
                "flop_per_step": FLOP_PER_RK4_STEP, "runs_per_launch": iso_runs,
                "lens_steps_per_launch": iso_steps, "lens_ms_per_launch": iso_ms,
                "timing": "CUDA events on the lane's stream around one group's lens pass, the group run alone "
                          "(a batch of batch_group runs) right after the timed region, mean of 3",
                "in_batch": {"launches": groups, "lens_span_ms_per_launch": g_lens_ms / groups,
                             "lens_steps_per_launch": g_lens_steps / groups,
                             "front_span_ms_per_run": sum(r.extra.get("front_ms", 0.0) for r in batch) / args.steps,
                             "note": "event spans on each lane's stream inside the timed batch: a lens pass's span "
                                     "includes waiting for SMs the other lane's kernels hold"},
                "traffic": LENS_DRAM_BYTES_PER_1E7 * n * iso_runs / 1e7,
                "traffic_unit": "bytes per grouped lens pass: ncu DRAM bytes of one grouped k_lens_persist launch "
                                "on a 1e7-molecule group, scaled by molecules per launch",
                "step_probe": probe}
    if mhz:
        roofline["shared_memory"] = shared_roof(iso_steps / (iso_ms / 1e3), sms, mhz)
    # the single-run lens pass (one ctraj_run at a time): bound by its critical
    # path, the molecule with the most RK4 steps, which cannot finish before
    # that many steps of one-warp latency (the step probe)
    single = {"kernel": "k_lens_persist of one run (512 threads per CTA)",
              "achieved": lens_steps * FLOP_PER_RK4_STEP / (lens_ms / 1e3) / 1e12,
              "lens_steps_per_launch": lens_steps / args.steps, "lens_ms_per_launch": lens_ms / args.steps,
              "front_ms_per_launch": front_ms / args.steps}
    single["frac"] = single["achieved"] / peak if peak else None
    max_steps = max(r.extra.get("max_lens_steps", 0) for r in results)
    cyc = probe.get("one_warp_cycles_per_step") if probe else None
    if max_steps and cyc and mhz:
        floor_ms = max_steps * cyc / (mhz * 1e3)
        single["critical_path"] = {
            "max_lens_steps": int(max_steps), "one_warp_cycles_per_step": cyc, "sm_mhz": mhz,
            "floor_ms": floor_ms, "frac": floor_ms / (lens_ms / args.steps),
            "note": "latency floor of the slowest molecule (max_lens_steps x one-warp step latency); "
                    "frac = floor / measured lens pass"}
    roofline["single_run"] = single
    cpu = None if args.no_cpu or world > 1 else cpu_baseline(int(args.cpu_sample or n), config0=cfg0)
    if parity is not None and cpu is not None and "config0_check" in cpu:
        parity["config0"]["oracle"] = cpu["config0_check"]
    r0 = results[-1]
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "fp32",
            "data": "synthetic: Philox-4x32-10 initial conditions drawn on the device",
            "config": bench_config(n),
            "engine": {"molecules_per_gpu": n, "precision": "fp32",
                       "pipelining": "ctraj_run_batch: the K runs alternate between two lanes (contexts with "
                                     "their own streams and buffers, one host thread each); a run's front "
                                     "overlaps the other lane's lens pass",
                       "l2": "flushed before every run: 160 MiB written on the run's lane stream inside the "
                             "timed region (pipelined batch); between steps outside the events (sequential)",
                       "parallelism": f"replicas x{world}",
                       "tuning": tuned["tuning"], "tuning_cached": tuned.get("cached", False)},
            "e2e": e2e, "sequential": sequential, "roofline": roofline, "cpu_baseline": cpu, "clocks": clocks,
            "parity": parity, "sweep": sweep, "adjoint": adjoint, "large": large,
            "gpu_launches": int(sum(r.kernels for r in batch)),
            "molecule_steps_per_step": steps / args.steps, "counts_last_step": r0.counter_dict()}
    print(json.dumps(line), flush=True)
    eng.close()
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
