"""Benchmark of the GB300 AVBD step: body-steps/s on the batched workload.

Workload (default): batched_4096 — 4096 independent scenes of log-uniform
8..1024 bodies (boxes and spheres dropped into a 20x20 bin), dt 1/120 s,
2 substeps, 8 iterations, f32, 240 steps.  A "step" is one 1/60 s frame =
2 substeps of every scene.  body-steps/s = dynamic bodies x steps / seconds.
Every rate below covers the same steps of the workload's 240-step
trajectory: all 240 by default; with --steps K < 240, K steps spread evenly
over the trajectory (step i of the sample is trajectory step
floor((i + 1/2) 240 / K); the steps between them run untimed), so the cheap
falling phase and the contact-heavy piles at the end weigh as they do in the
workload; --start S times the contiguous window [S, S + K) instead.

  value        device time of the K graph-replayed steps, state resident in
               HBM (CUDA events on the world's stream around each timed step).
  e2e          the same K steps through the C ABI with host buffers: every
               step uploads all body records, steps, downloads all body
               records and drains the contact events (host wall clock
               around synchronised calls).
  plain        a bounded sample of the same scenes, each stepped alone (one
               world per scene, plain launches) over the same K steps; the
               batched/plain ratio is the batching speed-up.
  roofline     the primal kernel in one profiled substep at the end of the
               trajectory: algorithmic bytes per launch (byte model in
               ornis_gb300/roofline.py) / its CUDA-event time per launch,
               against the measured HBM copy bandwidth.
  cpu_baseline the oracle's Reference-mode step (the reference's own serial
               algorithm restated in C++) on the host cores, a bounded sample
               of the same scenes over the same K steps, one process per core.
  parity       part of the oracle leg: sampled scenes of the batch at the end
               of the trajectory, each stepped from the device's state by the
               oracle (Coloured order, f32 and f64) while the device steps the
               whole batch in the benchmarked configuration; integer outputs
               compared exactly, poses relative to max(1, |x|).

Warm-up steps run from the initial state and the world is then reset to it,
so the timed trajectory starts at step 0.  The primal launch shape is
autotuned at step --tune-at (piles formed), then the state is reset.
--impl reference times the CPU path alone (the reference itself is Rust and
cannot be built here).  Under a multi-process launcher (N > 1: RANK,
WORLD_SIZE, LOCAL_RANK, MASTER_ADDR, MASTER_PORT) scenes are sharded across
ranks (scene s -> rank s mod N), no data-path collective; the barrier and
the max-over-ranks timing go over plain sockets (SocketRanks); rank 0
prints.
"""
import argparse
import atexit
import json
import math
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from ornis_gb300 import abi, scenes  # noqa: E402

METRIC = "AVBD body-steps/s: batched vs one-scene launches @<=1e-5 err; adjoint steps/s"
PEAKS = os.path.join(ROOT, "MEASURED_PEAKS.json")
FALLBACK_HBM_GBS = 6800.0


def hbm_peak():
    try:
        with open(PEAKS) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


class Clocks:
    """nvidia-smi sampling around the timed region.

    The sampler starts before the warm-up steps (nvidia-smi needs a moment
    before its first row) and every row carries its host arrival time;
    `mark(t0, t1)` bounds the timed region and the summary keeps the rows
    inside it.  When the region is shorter than a few sampling periods, the
    rows within one period of its ends are kept too (stated in `window`).
    """

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    PERIOD_MS = 100

    def __init__(self, device=0):
        self.rows = []
        self.proc = None
        self.device = device
        self.t0 = self.t1 = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", str(self.PERIOD_MS)],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append((time.perf_counter(), [x.strip() for x in line.split(",")]))

    def wait_first(self, timeout=5.0):
        end = time.perf_counter() + timeout
        while self.proc and not self.rows and time.perf_counter() < end:
            time.sleep(0.02)

    def mark(self, t0, t1):
        self.t0, self.t1 = t0, t1

    def __exit__(self, *a):
        if self.proc and self.proc.poll() is None:
            time.sleep(2 * self.PERIOD_MS / 1e3)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        rows = list(self.rows)
        window = "timed region"
        if self.t0 is not None:
            inside = [r for t, r in rows if self.t0 <= t <= self.t1]
            if len(inside) < 3:
                pad = self.PERIOD_MS / 1e3
                inside = [r for t, r in rows if self.t0 - pad <= t <= self.t1 + pad]
                window = f"timed region +- {self.PERIOD_MS} ms ({(self.t1 - self.t0) * 1e3:.0f} ms long)"
            rows = inside
        else:
            rows = [r for _, r in rows]
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            try:
                sm.append(float(r[1]))
                mx = max(mx, float(r[2]))
                for k, nm in enumerate(names):
                    if r[5 + k].lower() == "active":
                        reasons.add(nm)
            except (ValueError, IndexError):
                continue
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": mx or None,
                "reasons": sorted(reasons), "samples": len(sm), "window": window}


class SocketRanks:
    """The N>1 barrier and reductions over plain sockets (no PyTorch): rank 0
    serves on MASTER_ADDR at MASTER_PORT + 1 (the launcher keeps MASTER_PORT
    for its own store), the other ranks connect, and every collective is one
    line of JSON each way (floats round-trip exactly).  Scenes are sharded,
    so these carry only the timing and the body counts."""

    def __init__(self, rank, world, addr, port, timeout=300.0):
        import socket

        self.rank, self.world = rank, world
        self.peers = []
        if rank == 0:
            srv = socket.create_server((addr, port))
            srv.settimeout(timeout)
            try:
                for _ in range(world - 1):
                    conn, _ = srv.accept()
                    conn.settimeout(timeout)
                    f = conn.makefile("rw")
                    self.peers.append((int(f.readline()), conn, f))
            finally:
                srv.close()
            self.peers.sort(key=lambda p: p[0])
        else:
            deadline = time.monotonic() + timeout
            while True:
                try:
                    conn = socket.create_connection((addr, port), timeout=5.0)
                    break
                except OSError:
                    if time.monotonic() > deadline:
                        raise
                    time.sleep(0.2)
            conn.settimeout(timeout)
            self.conn, self.f = conn, conn.makefile("rw")
            self.f.write(f"{rank}\n")
            self.f.flush()

    def allreduce(self, vals, op):
        """Element-wise max or sum of each rank's list; every rank gets it."""
        vals = [float(v) for v in vals]
        if self.rank != 0:
            self.f.write(json.dumps(vals) + "\n")
            self.f.flush()
            return json.loads(self.f.readline())
        rows = [vals] + [json.loads(f.readline()) for _, _, f in self.peers]
        red = [max(c) if op == "max" else sum(c) for c in zip(*rows)]
        for _, _, f in self.peers:
            f.write(json.dumps(red) + "\n")
            f.flush()
        return red

    def barrier(self):
        self.allreduce([0.0], "sum")

    def close(self):
        for _, conn, _ in self.peers:
            conn.close()
        if self.rank != 0:
            self.conn.close()


def dist_init(n_gpus):
    """The N>1 rendezvous (rank, world size and local GPU from the launcher's
    environment); None on one GPU."""
    if n_gpus <= 1 or int(os.environ.get("WORLD_SIZE", "1")) <= 1:
        return None
    rank = int(os.environ["RANK"])
    world = int(os.environ["WORLD_SIZE"])
    local = int(os.environ.get("LOCAL_RANK", rank))
    port = int(os.environ.get("AVBD_BENCH_PORT", int(os.environ["MASTER_PORT"]) + 1))
    return SocketRanks(rank, world, os.environ.get("MASTER_ADDR", "127.0.0.1"), port), rank, world, local


def combine_ranks(ranks, worst=(), total=()):
    """The job-wide view of per-rank numbers: the max over ranks of each of
    `worst` (times) and the sum of each of `total` (counts)."""
    return (ranks.allreduce(worst, "max") if worst else []), (ranks.allreduce(total, "sum") if total else [])


def workload(args):
    """(bodies, scene offsets, joints, params, substeps) of the chosen workload."""
    if args.workload == "ragdoll_8192":
        # 8192 ragdolls of 15 capsules in two scenes of 3000 and 5192
        counts = (3000, 5192) if args.scenes == 4096 else (args.scenes // 3, args.scenes - args.scenes // 3)
        bodies, offs, joints = scenes.ragdolls(counts)
        params, nsub = scenes.params_for("ragdoll_8192")
        return bodies, offs, joints, params, nsub
    if args.workload in SINGLE_SCENE:
        # one scene: 100,000 bodies dropped over a 200 x 200 m ground plane,
        # or the 210-cube pyramid on a ground plane
        bodies = single_scene_bodies(args.workload)
        params, nsub = scenes.params_for(args.workload)
        return bodies, np.array([0, len(bodies)], dtype=np.uint32), [], params, nsub
    bodies, offs, _ = scenes.batched(args.scenes)
    params, nsub = scenes.params_for("batched_4096")
    return bodies, offs, [], params, nsub


def shard(bodies, offs, rank, world):
    """Scenes s with s % world == rank, repacked with their own offsets."""
    parts, new_offs = [], [0]
    for s in range(rank, len(offs) - 1, world):
        sc = bodies[offs[s]:offs[s + 1]]
        parts.append(sc)
        new_offs.append(new_offs[-1] + len(sc))
    return np.concatenate(parts), np.asarray(new_offs, dtype=np.uint32)


TRAJECTORY_STEPS = 240  # the batched and articulated workloads' trajectories
TRAJECTORY = {"batched_4096": 240, "ragdoll_8192": 240, "large_100k": 300, "pyramid_210": 600}
SINGLE_SCENE = ("large_100k", "pyramid_210")  # one-scene workloads: one GPU, L2 flushed per timed step


def single_scene_bodies(name):
    return scenes.large_100k() if name == "large_100k" else scenes.pyramid_210()


def trajectory_len(args):
    return TRAJECTORY.get(getattr(args, "workload", "batched_4096"), TRAJECTORY_STEPS)


def timed_steps(args, total=None):
    """Trajectory steps the timed region covers (the state before each)."""
    total = total or trajectory_len(args)
    if args.start is not None:
        return list(range(args.start, args.start + args.steps))
    if args.steps >= total:
        return list(range(args.steps))
    return [int((i + 0.5) * total / args.steps) for i in range(args.steps)]


def describe_steps(steps, total=TRAJECTORY_STEPS):
    if steps == list(range(steps[0], steps[0] + len(steps))):
        return f"steps {steps[0]}..{steps[0] + len(steps)} from the initial drop"
    stride = steps[1] - steps[0] if len(steps) > 1 else 0
    return (f"{len(steps)} single steps spread over the {total}-step trajectory (steps {steps[0]}, "
            f"{steps[0] + stride}, ..., {steps[-1]}; the steps between them run untimed)")


def run_sampled(step_untimed, step_timed, steps):
    """Advance through `steps` (sorted trajectory indices): untimed steps up to
    each, then one timed step; returns the summed timed quantity.  A
    contiguous window is timed by one call."""
    if steps == list(range(steps[0], steps[0] + len(steps))):
        if steps[0]:
            step_untimed(steps[0])
        return step_timed(len(steps))
    total, cur = 0.0, 0
    for t in steps:
        if t > cur:
            step_untimed(t - cur)
        total += step_timed(1)
        cur = t + 1
    return total


# ---------------------------------------------------------------------------
# CPU baseline: the oracle's Reference-mode step, one process per core.
# ---------------------------------------------------------------------------
def _cpu_scene_worker(args):
    """Step one scene through the trajectory, timing the oracle on the sampled steps."""
    bodies, params_tuple, nsub, steps = args
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_api as O

    p = abi.default_params(step_dt=params_tuple[0], iterations=params_tuple[1])
    w = O.OracleWorld(p, mode=O.REFERENCE)
    w.add_bodies(bodies)

    def timed(k):
        t0 = time.perf_counter()
        w.step_fixed(nsub * k)
        return time.perf_counter() - t0

    secs = run_sampled(lambda k: w.step_fixed(nsub * k), timed, steps)
    return secs, scenes.dynamic_count(bodies) * len(steps)


def cpu_baseline(bodies, offs, params, nsub, steps, per_core=3):
    """Body-steps/s of the oracle's Reference step on a seeded sample of scenes.

    Each sampled scene runs its trajectory and is timed on `steps` (the
    trajectory steps the device is timed on); scenes run one process per
    core and the rate is sampled body-steps over the summed per-scene seconds
    divided by cores.  The spread of the per-scene rates is reported too.
    """
    import multiprocessing as mp

    cores = os.cpu_count() or 1
    S = len(offs) - 1
    rng = np.random.default_rng(12345)
    chosen = [int(s) for s in rng.permutation(S)[: min(S, cores * per_core)]]
    jobs = [(bodies[offs[s]:offs[s + 1]], (params.step_dt, params.iterations), nsub, steps) for s in chosen]
    ctx = mp.get_context("spawn")
    t0 = time.perf_counter()
    with ctx.Pool(cores) as pool:
        res = pool.map(_cpu_scene_worker, jobs, chunksize=1)
    wall = time.perf_counter() - t0
    busy = sum(r[0] for r in res)
    body_steps = sum(r[1] for r in res)
    mean_n = float(np.mean([offs[s + 1] - offs[s] for s in chosen]))
    # the sample's own spread: the rate of each half of the sampled scenes
    halves = [res[0::2], res[1::2]]
    half_rates = [sum(r[1] for r in h) / (sum(r[0] for r in h) / cores) for h in halves if h]
    return {
        "value": body_steps / (busy / cores),
        "unit": "body-steps/s",
        "cores": cores,
        "kind": "port",
        "half_sample_rates": half_rates,
        "sample": f"{len(chosen)} of {S} scenes (seeded random, mean {mean_n:.0f} bodies incl. 5 planes), "
                  f"timed on {describe_steps(steps)} x {nsub} substeps per scene; one process per core; "
                  f"rate = body-steps / (summed scene seconds / cores); wall {wall:.1f} s",
    }


def _cpu_adjoint_worker(args):
    """One tower scene's gradients by the f64 dual-number oracle: the ball's
    initial velocity (3 directions) and the scene friction (1), frozen
    frames, `steps` steps timed (values and derivatives in one pass)."""
    bodies, ball, params_tuple, nsub, steps = args
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_api as O

    p = abi.default_params(step_dt=params_tuple[0], iterations=params_tuple[1])
    w = O.OracleWorld(p, mode=O.REFERENCE, use_double=O.DUAL)
    w.add_bodies(bodies)
    for c in range(3):
        w.seed(ball, O.F_VEL, c, c)
    for i in range(len(bodies)):
        w.seed(i, O.F_FRICTION, 0, 3)
    w.freeze_frames(7)
    t0 = time.perf_counter()
    w.step_fixed(nsub * steps)
    w.tangents()
    return time.perf_counter() - t0, steps


def adjoint_cpu_baseline(bodies, offs, ball, params, nsub, steps, per_core=1):
    """Scene-steps/s of the differentiable batch's gradients on the host
    cores: the dual-number oracle (forward mode, the four directions the
    workload asks for) on a seeded sample of scenes, one process per core."""
    import multiprocessing as mp

    cores = os.cpu_count() or 1
    S = len(offs) - 1
    rng = np.random.default_rng(54321)
    chosen = [int(s) for s in rng.permutation(S)[: min(S, cores * per_core)]]
    jobs = [(bodies[offs[s]:offs[s + 1]], int(ball[s] - offs[s]), (params.step_dt, params.iterations), nsub, steps)
            for s in chosen]
    ctx = mp.get_context("spawn")
    t0 = time.perf_counter()
    with ctx.Pool(cores) as pool:
        res = pool.map(_cpu_adjoint_worker, jobs, chunksize=1)
    wall = time.perf_counter() - t0
    busy = sum(r[0] for r in res)
    scene_steps = sum(r[1] for r in res)
    return {
        "value": scene_steps / (busy / cores),
        "unit": "gradient scene-steps/s",
        "cores": cores,
        "kind": "port",
        "sample": f"{len(chosen)} of {S} scenes (seeded random), {steps} steps each by the f64 dual-number "
                  f"oracle (reference order, frozen frames; ball velocity and friction directions seeded: 4 of "
                  f"the 8 tangents the dual type always carries, so the host does about twice the tangent "
                  f"arithmetic the 4 directions need, in f64 where the device computes in f32); one "
                  f"process per core; rate = scene-steps / (summed scene seconds / cores); wall {wall:.1f} s",
    }


def _large_cpu_worker(job):
    """One oracle step of the large scene in the reference's order, timed."""
    st, params_tuple, nsub, cores = job
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_api as O

    p = abi.default_params(step_dt=params_tuple[0], iterations=params_tuple[1])
    o = O.OracleWorld(p, mode=O.REFERENCE, threads=cores)
    o.add_bodies(st["bodies"])
    o.import_state(st)
    t0 = time.perf_counter()
    o.step_fixed(nsub)
    return time.perf_counter() - t0


def large_cpu_baseline(states, params, nsub, ndyn, at, limit_s=90.0):
    """The oracle's Reference step of the one-scene 100k workload on the host
    cores, from the device's state at a few of the timed trajectory steps.
    The reference's CPU step is quadratic here (all-pairs discovery, a linear
    pair lookup per discovered pair), so the sample is a few steps, each
    timed alone in a child process and given at most limit_s seconds; a
    step that runs out counts as limit_s, which makes the rate an upper
    bound of the reference's."""
    import multiprocessing as mp

    cores = os.cpu_count() or 1
    secs, capped = [], 0
    ctx = mp.get_context("spawn")
    for st in states:
        pool = ctx.Pool(1)
        try:
            r = pool.apply_async(_large_cpu_worker, ((st, (params.step_dt, params.iterations), nsub, cores),))
            secs.append(r.get(timeout=limit_s))
        except mp.TimeoutError:
            secs.append(limit_s)
            capped += 1
        finally:
            pool.terminate()
            pool.join()
        print(f"[large] cpu step {len(secs)}: {secs[-1]:.1f} s", file=sys.stderr, flush=True)
    return {"value": ndyn * len(secs) / sum(secs), "unit": "body-steps/s", "cores": cores, "kind": "port",
            "per_step_s": secs, "steps_cut_at_limit": capped, "upper_bound": capped > 0,
            "sample": f"{len(secs)} of the timed steps (trajectory steps {at}), each one oracle step in the "
                      f"reference's order (all-pairs discovery split over {cores} threads as the reference splits "
                      f"it with rayon, linear pair lookup, serial sweep) from the device's state at that step, "
                      f"in a child process given {limit_s:.0f} s (a step cut there counts as {limit_s:.0f} s, so the "
                      f"rate is then an upper bound); rate = body-steps / summed seconds"}


def oracle_parity(w, offs, params, nsub, nscenes=8, steps=3, split=True, threads=1):
    """Part of the oracle leg: per-substep parity of the benchmarked world
    against the oracle on a seeded sample of its scenes, at the world's
    current state, for `steps` steps.  Before every substep, each sampled
    scene's state is exported from the device and loaded into an f32 and an
    f64 oracle world (Coloured order; rows summed per pair when the device
    does); the device steps the whole batch one
    substep (the reference's step_inner) in the benchmarked configuration
    and the oracles step their scene.  Integer outputs (pair sets, points per
    pair, contact IDs, colours) are compared exactly; poses relative to
    max(1, |x|), velocities x dt."""
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_api as O
    import parity as P

    S = len(offs) - 1
    rng = np.random.default_rng(2468)
    sizes = np.diff(offs)
    # half the sample from the largest scenes (the deepest piles), half random
    big = [int(x) for x in np.argsort(-sizes, kind="stable")[: nscenes // 2]]
    rest = [int(x) for x in rng.permutation(S) if int(x) not in big][: nscenes - len(big)]
    chosen = big + rest
    worst = {"f32": 0.0, "f64": 0.0, "f32_oracle_vs_f64": 0.0, "vel_f32": 0.0}
    same = True
    st = w.export_state()
    for _ in range(steps * nsub):
        ors = []
        for sc in chosen:
            sub = P.scene_state(st, offs, sc)
            pair = []
            for dbl in (False, True):
                o = O.OracleWorld(params, mode=O.COLOURED, use_double=dbl, threads=threads)
                o.split_sums(split)
                o.add_bodies(sub["bodies"])
                o.import_state(sub)
                o.step_fixed(1)
                pair.append(o)
            ors.append(pair)
        w.step_graph(1)
        st = w.export_state()
        cols = w.colours()
        for sc, (o32, o64) in zip(chosen, ors):
            sg = P.scene_state(st, offs, sc)
            a0, a1 = int(offs[sc]), int(offs[sc + 1])
            ok, pe, ve = P.scene_step_errors(o32.export_state(), sg, o32.colours(), cols[a0:a1], params.step_dt)
            same &= ok
            worst["f32"] = max(worst["f32"], pe)
            worst["vel_f32"] = max(worst["vel_f32"], ve)
            s64 = o64.export_state()
            worst["f64"] = max(worst["f64"], P.pose_errors(sg["bodies"], s64["bodies"], params.step_dt)[0])
            worst["f32_oracle_vs_f64"] = max(worst["f32_oracle_vs_f64"],
                                             P.pose_errors(o32.export_state()["bodies"], s64["bodies"],
                                                           params.step_dt)[0])
    return {"max_pose_rel_err": worst["f32"], "max_vel_err_x_dt": worst["vel_f32"], "vs_f64": worst["f64"],
            "oracle_f32_vs_f64": worst["f32_oracle_vs_f64"], "integers_identical": bool(same),
            "bar": P.POSE_RTOL, "scenes": chosen, "bodies": [int(sizes[c]) for c in chosen],
            "substeps": steps * nsub,
            "how": "per substep from the device's state: the device steps the whole batch (benchmarked launch "
                   "shape, precision and graph replay), f32 and f64 oracles (Coloured order, per-pair row "
                   "sums) step each sampled scene; pose error relative to max(1, |x|)"}


# ---------------------------------------------------------------------------
def run_reference_large(args):
    """The reference's CPU step on a one-scene workload: the oracle in the
    reference's order from the initial drop, at least three steps timed and
    more while they take under 20 s together (a step of the 100k scene is
    quadratic in bodies: its rate is extrapolated from three)."""
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_api as O

    bodies = single_scene_bodies(args.workload)
    params, nsub = scenes.params_for(args.workload)
    cores = os.cpu_count() or 1
    o = O.OracleWorld(params, mode=O.REFERENCE, threads=cores)
    o.add_bodies(bodies)
    secs = []
    while len(secs) < 3 or (sum(secs) < 20.0 and len(secs) < trajectory_len(args)):
        t0 = time.perf_counter()
        o.step_fixed(nsub)
        secs.append(time.perf_counter() - t0)
    ndyn = scenes.dynamic_count(bodies)
    v = ndyn * len(secs) / sum(secs)
    cb = {"value": v, "unit": "body-steps/s", "cores": cores, "kind": "port", "per_step_s": secs,
          "sample": f"steps 0..{len(secs)} of the {trajectory_len(args)}-step trajectory from the initial drop, the "
                    f"oracle in the reference's order (all-pairs discovery over {cores} threads, linear pair lookup, "
                    f"serial sweep); rate from those steps"}
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "body-steps/s", "n_gpus": args.gpus,
            "steps": len(secs), "warmup": 0, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic (seeded scene)",
            "config": {"workload": args.workload, "scenes": 1, "dynamic_bodies": ndyn, "dt": params.step_dt,
                       "substeps": nsub, "iterations": params.iterations, "trajectory": f"steps 0..{len(secs)}"},
            "cpu_baseline": cb, "e2e": {"value": v, "unit": "body-steps/s", "h2d_bytes_per_step": 0,
                                        "d2h_bytes_per_step": 0}}
    print(json.dumps(line))
    return 0


def run_reference(args):
    d = dist_init(args.gpus)
    if d is not None and d[1] != 0:
        return 0
    if args.workload in SINGLE_SCENE:
        return run_reference_large(args)
    bodies, offs, counts = scenes.batched(args.scenes)
    params, nsub = scenes.params_for("batched_4096")
    steps = timed_steps(args)
    cb = cpu_baseline(bodies, offs, params, nsub, steps, per_core=args.cpu_per_core)
    v = cb["value"]
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "body-steps/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded scenes)",
            "config": {"workload": "batched_4096", "scenes": args.scenes, "dt": 1 / 120, "substeps": nsub,
                       "iterations": params.iterations, "trajectory": describe_steps(steps)},
            "cpu_baseline": cb, "e2e": {"value": v, "unit": "body-steps/s", "h2d_bytes_per_step": 0,
                                        "d2h_bytes_per_step": 0}}
    print(json.dumps(line))
    return 0


def run_ours(args):
    from ornis_gb300 import roofline
    from ornis_gb300.avbd import AvbdWorld

    d = dist_init(args.gpus)
    rank, world = (d[1], d[2]) if d else (0, 1)
    device = d[3] if d else 0
    bodies_all, offs_all, joints_all, params, nsub = workload(args)
    if world > 1 and joints_all:
        raise SystemExit("the articulated workload runs on one GPU (two scenes)")
    if world > 1 and args.workload in SINGLE_SCENE:
        raise SystemExit("a one-scene workload runs on one GPU")
    large = args.workload in SINGLE_SCENE
    bodies, offs = shard(bodies_all, offs_all, rank, world) if world > 1 else (bodies_all, offs_all)
    ndyn = scenes.dynamic_count(bodies)
    w = AvbdWorld(params, device=device, bodies=bodies, scene_offsets=offs)
    for j in joints_all:
        w.add_joint(j)
    w.set_precision(args.fast)
    w.set_events(nsub)  # contact events every step, as the reference's step(dt) reports them
    s0 = w.export_state()  # the initial drop: no contacts yet
    tuned = None
    if args.lanes is not None:
        w.set_tuning(args.lanes, args.block)
    elif args.autotune:
        from ornis_gb300.tune import autotune

        w.step_graph(nsub * args.tune_at)  # piles formed: where the primal costs most
        tuned = autotune(w, substeps_per_trial=2 * nsub)
    steps = timed_steps(args)
    clk = Clocks(device).__enter__()
    atexit.register(clk.__exit__)
    clk.wait_first()
    for _ in range(args.warmup):
        w.step_graph(nsub)
    w.import_state(s0)
    if args.profile_region:
        if steps[0]:
            w.step_graph(nsub * steps[0])
        w.sync()
        # only the kernels of these steps are collected by `ncu --profile-from-start off`;
        # they run from the state the timed region starts at, which is restored afterwards
        from ornis_gb300.avbd import lib as _lib

        snap = w.export_state()
        _lib().avbd_profiler(1)
        w.step_graph(nsub * args.profile_region)
        w.sync()
        _lib().avbd_profiler(0)
        w.import_state(snap)
        w.import_state(s0)
    w.sync()
    # ---- timed region: K steps of the trajectory, device time --------------
    if d:
        d[0].barrier()
    t0 = time.perf_counter()
    if large:
        # the one scene's state is about L2's size: evict it before every timed step
        def timed_one(k):
            total = 0.0
            for _ in range(k):
                w.flush_cache()
                total += w.step_timed(nsub, use_graph=True)
            return total

        ms = run_sampled(lambda k: w.step_graph(nsub * k), timed_one, steps)
    else:
        ms = run_sampled(lambda k: w.step_graph(nsub * k), lambda k: w.step_timed(nsub * k, use_graph=True), steps)
    clk.mark(t0, time.perf_counter())
    clk.__exit__()
    if large:
        print(f"[large] timed {len(steps)} steps: {ms:.1f} ms", file=sys.stderr, flush=True)
    if d:
        (ms,), (nd,) = combine_ranks(d[0], worst=[ms], total=[ndyn])
        ndyn_total = int(nd)
    else:
        ndyn_total = ndyn
    value = ndyn_total * args.steps / (ms / 1e3)
    launches_per_step = w.graph_nodes() * (nsub - 1) + w.graph_nodes_emit()
    c = w.counters()
    # ---- parity of the benchmarked configuration at the end of the trajectory
    par = None
    if args.parity_scenes > 0 and not joints_all:
        lanes = tuned[0][0] if tuned else (args.lanes if args.lanes is not None else 1)
        if large:
            print("[large] oracle parity", file=sys.stderr, flush=True)
        par = oracle_parity(w, offs, params, nsub, nscenes=args.parity_scenes,
                            steps=min(args.parity_steps, 1) if large else args.parity_steps,
                            split=lanes <= 0, threads=(os.cpu_count() or 1) if large else 1)
    # ---- per-phase profile at the end of the trajectory: primal roofline ---
    phases, info = w.profile_substep()
    lanes = tuned[0][0] if tuned else (args.lanes if args.lanes is not None else 1)
    kind = "engine" if lanes <= 1 else "lanes"
    roof = roofline.primal_roofline(phases, info, hbm_peak(), kind=kind, iterations=params.iterations)
    roof["state"] = "one profiled substep at the end of the trajectory"
    # ---- e2e through the C ABI with host buffers, same trajectory steps ----
    e2e_steps = steps if args.e2e_steps is None else timed_steps(argparse.Namespace(
        start=args.start, steps=args.e2e_steps))
    w.import_state(s0)
    w.contact_events()
    io = {"host": None, "ev": 0}

    def e2e_untimed(k):
        w.step_graph(nsub * k)
        w.contact_events()

    def e2e_timed(k):
        io["host"] = w.bodies()  # the state the caller holds (untimed)
        t0 = time.perf_counter()
        for _ in range(k):
            w.set_bodies(io["host"])
            w.step_graph(nsub)
            io["host"] = w.bodies()
            io["ev"] += w.contact_events().nbytes
        return time.perf_counter() - t0

    if d:
        d[0].barrier()
    e2e_s = run_sampled(e2e_untimed, e2e_timed, e2e_steps)
    h2d = d2h = io["host"].nbytes
    d2h += io["ev"] // max(1, len(e2e_steps))
    e2e = ndyn * len(e2e_steps) / e2e_s
    if d:
        (e2e_max,), _ = combine_ranks(d[0], worst=[e2e_s])
        e2e = ndyn_total * len(e2e_steps) / e2e_max
    cb = None
    if large and args.cpu_per_core > 0:
        # the device's state at three of the timed steps (early, middle, late)
        at = sorted({steps[len(steps) // 6], steps[len(steps) // 2], steps[-1]})
        w.import_state(s0)
        states, cur = [], 0
        for t in at:
            if t > cur:
                w.step_graph(nsub * (t - cur))
            cur = t
            states.append(w.export_state())
        cb = large_cpu_baseline(states, params, nsub, ndyn, at)
    w.close()
    if rank != 0:
        return 0
    # ---- plain: one scene per world, same trajectory, bounded sample --------
    plain = None
    # the one-scene and CPU comparisons belong to the batched workload (the
    # ragdoll scenes are 45k and 78k bodies: the oracle's all-pairs discovery
    # does not finish a step in bounded time)
    if args.plain_scenes > 0 and not joints_all and not large:
        plain = plain_rate(bodies_all, offs_all, params, nsub, args)
    adj = None
    if args.adjoint_scenes > 0 and world == 1 and not joints_all and not large:
        adj = adjoint_rate(args)
    rag = None
    if args.ragdoll_adjoint_steps > 0 and world == 1 and not large:
        rag = ragdoll_adjoint_rate(args)
    if args.cpu_per_core > 0 and world == 1 and not joints_all and not large:
        cb = cpu_baseline(bodies_all, offs_all, params, nsub, steps, per_core=args.cpu_per_core)
    line = {
        "metric": METRIC, "value": value, "unit": "body-steps/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded scenes, no dataset)",
        "config": {"workload": args.workload, "scenes": len(offs_all) - 1, "dynamic_bodies": ndyn_total,
                   "joints": len(joints_all),
                   "dt": params.step_dt, "substeps": nsub, "iterations": params.iterations,
                   "trajectory": describe_steps(steps, trajectory_len(args)),
                   "l2": ("256 MB write before every timed step (the scene's state is about L2's size)" if large
                          else "state larger than L2 (GB-scale pair/point arrays), no flush"),
                   "graph": True, "precision": "fast" if args.fast else "exact",
                   "primal_launch": {"lanes": tuned[0][0], "block": tuned[0][1], "min_blocks_per_sm": tuned[0][2],
                                     "by_work": tuned[0][3], "tuned_at_step": args.tune_at,
                                     "trials_ms": [[list(cd), round(m, 3)] for cd, m in tuned[1]]}
                   if tuned else {"lanes": args.lanes if args.lanes is not None else 1, "block": args.block}},
        "e2e": {"value": e2e, "unit": "body-steps/s", "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h),
                "steps": len(e2e_steps)},
        "gpu_launches": int(launches_per_step * args.steps),
        "roofline": roof,
        "cpu_baseline": cb,
        "parity": par,
        "clocks": clk.summary(),
        "plain_one_scene": plain,
        "batched_over_plain": (value / plain["value"]) if plain else None,
        "adjoint": adj,
        "adjoint_articulated": rag,
        "phases_ms_per_substep": phases,
        "counters_at_end": {"candidates": c.candidates, "pairs": c.pairs, "points": c.points, "colours": c.colours,
                            "sleeping": c.sleeping, "breakdowns": c.breakdowns, "ccd_hits": c.ccd_hits,
                            "ccd_left": c.timeouts},
    }
    print(json.dumps(line))
    return 0


def finite(x):
    """A JSON-safe float: None for NaN and infinities."""
    x = float(x)
    return x if math.isfinite(x) else None


def adjoint_rate(args):
    """The differentiable batch (diff_1024): recorded forward with checkpoints,
    then the reverse sweep, against the plain graph-replayed forward."""
    from ornis_gb300.avbd import AvbdWorld

    bodies, offs, ball, tower = scenes.diff_towers(nscenes=args.adjoint_scenes)
    params, nsub = scenes.params_for("diff_1024")
    steps, every = args.adjoint_steps, 10
    ndyn = scenes.dynamic_count(bodies)
    w = AvbdWorld(params, bodies=bodies, scene_offsets=offs)
    w.set_precision(True)
    w.set_events(-1)
    s0 = w.export_state()
    fwd = {}
    for lanes in (1, 0):  # rows in the reference's order ("thread"), then per pair ("split"), which the rollout runs
        w.set_tuning(lanes, 128)
        w.step_graph(nsub * 3)  # warm-up: graphs captured
        w.import_state(s0)
        w.sync()
        t0 = time.perf_counter()
        dev_ms = w.step_timed(nsub * steps, use_graph=True)
        fwd[lanes] = (time.perf_counter() - t0, dev_ms)
        w.import_state(s0)
    best = min(fwd, key=lambda k: fwd[k][0])  # the faster forward is the reference cost
    fwd_s, fwd_dev_ms = fwd[best]
    first_s = None
    for rep in range(2):  # the first rollout sets up frames and recording graphs; the second is timed
        w.import_state(s0)
        w.sync()
        t0 = time.perf_counter()
        w.adjoint_forward(steps, nsub, every)
        rec_s = time.perf_counter() - t0
        end = w.bodies()
        g = np.zeros((len(bodies), 13), dtype=np.float32)
        g[tower, 0:3] = 2.0 * end["position"][tower]
        loss = float(np.sum(end["position"][tower].astype(np.float64) ** 2))
        t0 = time.perf_counter()
        g0, gmu = w.adjoint_backward(g)
        bwd_s = time.perf_counter() - t0
        first_s = bwd_s if first_s is None else first_s
    rec_ms, rev_ms = w.adjoint_timing()
    amax, _ = w.adjoint_trace()
    w.close()
    gv = g0[ball, 7:10]
    cpu = None
    if args.adjoint_cpu_per_core > 0:
        cpu = adjoint_cpu_baseline(bodies, offs, ball, params, nsub, steps, per_core=args.adjoint_cpu_per_core)
    return {"workload": "diff_1024", "scenes": int(len(offs) - 1), "dynamic_bodies": ndyn, "steps": steps,
            "checkpoint_every": every, "dt": 1 / 60, "iterations": params.iterations, "precision": "fast",
            "forward_ms_per_step": 1e3 * fwd_s / steps, "forward_device_ms_per_step": fwd_dev_ms / steps,
            "forward_ms_per_step_by_primal": {"thread": 1e3 * fwd[1][0] / steps, "split": 1e3 * fwd[0][0] / steps},
            "record_ms_per_step": 1e3 * rec_s / steps, "backward_ms_per_step": 1e3 * bwd_s / steps,
            "backward_first_call_ms_per_step": 1e3 * first_s / steps,
            "adjoint_steps_per_s": steps / bwd_s, "adjoint_body_steps_per_s": ndyn * steps / bwd_s,
            "backward_over_forward": bwd_s / fwd_s, "loss": loss,
            "backward_split_ms_per_step": {"recompute": rec_ms / steps, "reverse": rev_ms / steps},
            "grad_ball_velocity_mean": [finite(x) for x in gv.mean(axis=0)],
            "grad_friction_mean": finite(np.mean(gmu)),
            "adjoint_max_abs": finite(np.max(amax)) if len(amax) else None,
            "gradient_scene_steps_per_s": (len(offs) - 1) * steps / (rec_s + bwd_s),
            "cpu_baseline": cpu,
            "how": "wall time with the host waiting; backward = per-segment recompute from the checkpoint "
                   "plus the reverse sweep; forward = the same rollout by CUDA-graph replay with the faster "
                   "of the two row orders (the rollout itself adds rows up per pair); the second of two "
                   "rollouts from the same start is timed (the first sets up the frames and recording graphs, "
                   "as the forward's warm-up captures its graphs)"}


RAGDOLL_STIFFNESS = 2.0e4  # N/m (anchor rows), N m/rad (hinge rows)


def ragdoll_adjoint_rate(args):
    """The articulated batch (8192 ragdolls in scenes of 3000 and 5192) with
    joints of finite stiffness: recorded forward with checkpoints, then the
    reverse sweep for d(final centre-of-mass height of each scene)/d(joint
    stiffness), against the plain graph-replayed forward."""
    from ornis_gb300.avbd import AvbdWorld

    bodies, offs, joints = scenes.ragdolls(counts=tuple(int(c) for c in args.ragdoll_counts.split(",")))
    params, nsub = scenes.params_for("ragdoll_8192")
    steps, every = args.ragdoll_adjoint_steps, 10
    ndyn = scenes.dynamic_count(bodies)
    w = AvbdWorld(params, bodies=bodies, scene_offsets=offs)
    for j in joints:
        w.add_joint(j)
    w.set_joint_stiffness(RAGDOLL_STIFFNESS)
    w.set_precision(True)
    w.set_events(-1)
    s0 = w.export_state()
    fwd = {}
    for lanes in (1, 0):
        w.set_tuning(lanes, 128)
        w.step_graph(nsub * 3)
        w.import_state(s0)
        w.sync()
        t0 = time.perf_counter()
        dev_ms = w.step_timed(nsub * steps, use_graph=True)
        fwd[lanes] = (time.perf_counter() - t0, dev_ms)
        w.import_state(s0)
    best = min(fwd, key=lambda k: fwd[k][0])
    fwd_s, fwd_dev_ms = fwd[best]
    first_s = None
    for rep in range(2):  # as the differentiable batch: the second rollout is timed
        w.import_state(s0)
        w.sync()
        t0 = time.perf_counter()
        w.adjoint_forward(steps, nsub, every)
        rec_s = time.perf_counter() - t0
        end = w.bodies()
        dyn = end["inv_mass"] > 0
        mass = np.where(dyn, 1.0 / np.where(dyn, end["inv_mass"], 1.0), 0.0)
        g = np.zeros((len(bodies), 13), dtype=np.float32)
        com = []
        for s in range(len(offs) - 1):
            a, b = offs[s], offs[s + 1]
            m = mass[a:b]
            g[a:b, 1] = m / m.sum()
            com.append(float(np.sum(m * end["position"][a:b, 1]) / m.sum()))
        t0 = time.perf_counter()
        w.adjoint_backward(g)
        bwd_s = time.perf_counter() - t0
        first_s = bwd_s if first_s is None else first_s
    gk = w.adjoint_grad_joint_stiffness()
    rec_ms, rev_ms = w.adjoint_timing()
    amax, _ = w.adjoint_trace()
    w.close()
    return {"workload": "ragdoll_8192" if args.ragdoll_counts == "3000,5192" else f"ragdolls_{args.ragdoll_counts}",
            "scenes": int(len(offs) - 1), "dynamic_bodies": ndyn, "joints": len(joints),
            "joint_stiffness": RAGDOLL_STIFFNESS, "steps": steps, "checkpoint_every": every, "dt": 1 / 120,
            "substeps": nsub, "iterations": params.iterations, "precision": "fast",
            "forward_ms_per_step": 1e3 * fwd_s / steps, "forward_device_ms_per_step": fwd_dev_ms / steps,
            "forward_ms_per_step_by_primal": {"thread": 1e3 * fwd[1][0] / steps, "split": 1e3 * fwd[0][0] / steps},
            "record_ms_per_step": 1e3 * rec_s / steps, "backward_ms_per_step": 1e3 * bwd_s / steps,
            "backward_first_call_ms_per_step": 1e3 * first_s / steps,
            "adjoint_steps_per_s": steps / bwd_s, "adjoint_body_steps_per_s": ndyn * steps / bwd_s,
            "backward_over_forward": bwd_s / fwd_s,
            "backward_split_ms_per_step": {"recompute": rec_ms / steps, "reverse": rev_ms / steps},
            "com_height": com, "grad_com_height_wrt_stiffness": [finite(x) for x in gk],
            "adjoint_max_abs": finite(np.max(amax)) if len(amax) else None,
            "how": "as the differentiable batch: wall time with the host waiting; loss per scene = final "
                   "centre-of-mass height of its dynamic bodies"}


def plain_rate(bodies, offs, params, nsub, args):
    """Body-steps/s stepping sampled scenes one world (one launch sequence) at a time."""
    from ornis_gb300.avbd import AvbdWorld

    S = len(offs) - 1
    rng = np.random.default_rng(777)
    pick = rng.choice(S, size=min(args.plain_scenes, S), replace=False)
    tot_ms = 0.0
    body_steps = 0
    steps = timed_steps(args)
    for s in pick:
        sc = bodies[offs[s]:offs[s + 1]]
        wd = AvbdWorld(params, bodies=sc)
        tot_ms += run_sampled(lambda k: wd.step_fixed(nsub * k), lambda k: wd.step_timed(nsub * k, use_graph=False),
                              steps)
        body_steps += scenes.dynamic_count(sc) * len(steps)
        wd.close()
    return {"value": body_steps / (tot_ms / 1e3), "unit": "body-steps/s", "scenes_sampled": int(len(pick)),
            "steps": len(steps),
            "how": "one world per scene, plain launches, each scene over the same trajectory steps, device time "
                   "summed"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=240)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--scenes", type=int, default=4096)
    ap.add_argument("--workload", default="batched_4096",
                    choices=["batched_4096", "ragdoll_8192", "large_100k", "pyramid_210"],
                    help="ragdoll_8192: 8192 15-capsule ragdolls with ball/hinge joints in two scenes; "
                         "large_100k: one scene of 100,000 bodies, dt 1/60, 1 substep, 10 iterations, 300 steps; "
                         "pyramid_210: the 210-cube pyramid on a plane, dt 1/60, 1 substep, 10 iterations, 600 steps")
    ap.add_argument("--start", type=int, default=None,
                    help="time the contiguous window [start, start + steps) instead of steps spread over the "
                         "trajectory")
    ap.add_argument("--parity-scenes", type=int, default=8,
                    help="scenes of the oracle parity check at the end of the trajectory (0: skip)")
    ap.add_argument("--parity-steps", type=int, default=3)
    ap.add_argument("--tune-at", type=int, default=150, help="step at which the primal launch is autotuned")
    ap.add_argument("--e2e-steps", type=int, default=None, help="default: --steps")
    ap.add_argument("--plain-scenes", type=int, default=16)
    ap.add_argument("--cpu-per-core", type=int, default=3)
    ap.add_argument("--lanes", type=int, default=None, help="fixed primal launch shape instead of autotuning")
    ap.add_argument("--block", type=int, default=128)
    ap.add_argument("--fast", action="store_true",
                    help="fast build of the iteration kernels (contracted multiply-adds, approximate division: "
                         "not held to the 1e-5 per-step bar at the piles); default: the exact build, which "
                         "computes the oracle's arithmetic")
    ap.add_argument("--profile-region", type=int, default=0,
                    help="steps bracketed by cudaProfilerStart/Stop before the timed region")
    ap.add_argument("--no-autotune", dest="autotune", action="store_false")
    ap.add_argument("--adjoint-scenes", type=int, default=1024, help="differentiable batch size (0: skip)")
    ap.add_argument("--adjoint-steps", type=int, default=120)
    ap.add_argument("--adjoint-cpu-per-core", type=int, default=1,
                    help="differentiable-batch scenes per host core for the dual-number CPU baseline (0: skip)")
    ap.add_argument("--ragdoll-adjoint-steps", type=int, default=240,
                    help="steps of the articulated forward+adjoint measurement (0: skip)")
    ap.add_argument("--adjoint-only", action="store_true",
                    help="print only the differentiable-batch measurement (for profiling)")
    ap.add_argument("--ragdoll-counts", default="3000,5192",
                    help="ragdolls per scene of the articulated forward+adjoint measurement")
    ap.add_argument("--ragdoll-adjoint-only", action="store_true",
                    help="print only the articulated forward+adjoint measurement")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    if args.impl == "reference":
        return run_reference(args)
    if args.adjoint_only:
        print(json.dumps(adjoint_rate(args)))
        return 0
    if args.ragdoll_adjoint_only:
        print(json.dumps(ragdoll_adjoint_rate(args)))
        return 0
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
