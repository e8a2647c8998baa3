#!/usr/bin/env python
"""Map-integration benchmark: batched, plain and served forms on one B200.

Headline ("value", "e2e"): the batched form at README scale.  K maps (robots,
default 8) of 701 x 701 x 151 voxels (74.2M) at 0.1 m, FP32 log-odds from the
yaml probabilities; per step every map integrates one 64-beam x 1024-azimuth
scan (65,536 points, 50 m max range, sigma 0.02 m, seeded scene of a ground
plane and 400 boxes over +-60 m, robot m at trajectory offset 25 m along a
circle of radius 25 m at 1.5 m/s, 10 Hz) and recenters with the 4 m
threshold.  All K scans of a step go through one cublox_batch_update (one
walk and one fold launch, replayed from a CUDA graph; the launch shape is
chosen by the batch's tuner in a separate pass before warm-up, so no timed
step runs a candidate shape).

Metric: voxel-steps/s, the reference's own work unit (DDA iterations that
did not break + 1 endpoint per ray, counted for every scan against the
window it was integrated in), with p50/p99 per-step latency.

  value  device time, scans already resident in HBM, CUDA events on the
         batch's stream, L2 flushed (512 MiB write) between steps
  e2e    through the public API from pinned host memory: each step copies
         its K scans host->device, integrates, recenters and reads 4 bytes of
         the last map back (one stream orders every map's work before it)
  --impl reference  the reference's own kernels (oracle/_ref, its
         src/kernels.cu built for sm_100a) on the same K maps, one map after
         another in its OccupancyGrid call sequence; that process maps no
         library of this package (its scans and work-unit counts come from
         oracle/_ref/libcublox_refinputs.so)

Beside the headline (one GPU only): "plain" (one README map through the
drop-in OccupancyGrid), "batching" (32 maps of 257x257x65 / 401x401x81 /
513x513x129, 8,192-131,072 points each), "serving" (16 robots, Poisson
scans at 400/s and fetches at 100/s, 60 s, p50/p99 scan-to-map latency), and
"cpu_baseline" (the CPU oracle on the host cores).

Under torchrun every rank integrates its own replica of the headline
workload (maps shard across GPUs with no exchange); value = all ranks'
voxel-steps / the slowest rank's time.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "voxel-steps/s & p50/p99 scan latency, batched/served vs plain on 1 B200"
UNIT = "voxel-steps/s"
TRAJ_OFFSET = 25  # scans between consecutive robots on the shared trajectory


def _peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.path = None
        self.skip = 0

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}", "--format=csv,noheader,nounits",
                 "-lms", "50"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
            # nvidia-smi takes a moment to start: let its first sample land
            # before the timed region begins, so that the region's own
            # samples follow
            t0 = time.perf_counter()
            while time.perf_counter() - t0 < 3.0 and os.path.getsize(self.path) == 0:
                time.sleep(0.01)
            with open(self.path) as f:
                self.skip = sum(1 for _ in f)  # samples taken before the region
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                pass

    def summary(self):
        rows = []
        try:
            with open(self.path) as f:
                for line in f:
                    parts = [p.strip() for p in line.split(",")]
                    if len(parts) >= 9:
                        rows.append(parts)
        except Exception:
            pass
        finally:
            try:
                os.unlink(self.path)
            except Exception:
                pass
        if len(rows) > self.skip:
            rows = rows[self.skip:]  # keep the region's own samples when there are any
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        reasons = sorted({names[i] for r in rows for i in range(4) if "Active" in r[5 + i]
                          and "Not" not in r[5 + i]})
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": float(max(mx)) if mx else None, "reasons": reasons,
                "samples": len(rows)}


# ---------------------------------------------------------------------------
# workloads and accounting
# ---------------------------------------------------------------------------
def readme_batch(n_maps: int, n_steps: int):
    """Scans of the README-scale batch: scans[k][m], origins[k][m]."""
    from cublox_b200 import synth
    w = synth.readme_scale(n_steps + TRAJ_OFFSET * n_maps)
    scans = [[w.scan(k + TRAJ_OFFSET * m) for m in range(n_maps)] for k in range(n_steps)]
    origins = [[w.sensor_origin(k + TRAJ_OFFSET * m) for m in range(n_maps)] for k in range(n_steps)]
    return w, scans, origins


def count_steps(half, res, max_range, threshold, scans, origins):
    """The reference's voxel-steps of one map's scan sequence, each counted
    against the window it is integrated in (first scan snaps the window,
    recenter after every scan)."""
    import cublox_b200 as C
    g = C.OccupancyGrid(half, res, False, threshold, origin=tuple(float(v) for v in origins[0]))
    g.setMaxRaycastRange(max_range)
    out = []
    for s, o in zip(scans, origins):
        out.append(g.reference_steps(s, o))
        g.recenter(o)
    g.close()
    return np.asarray(out, dtype=np.int64)


def cpu_baseline(w, scans, origins, steps, budget_s=12.0):
    """The oracle (CPU restatement of the reference's path) on the host cores."""
    import oracle as O
    import cublox_b200 as C
    threads = os.cpu_count() or 1
    g = O.OracleGrid(w.half, w.resolution, False, w.threshold)
    g.set_log_odds(*C.yaml_log_odds())
    g.set_max_range(w.sensor.max_range)
    t0 = time.perf_counter()
    done = 0
    vs = 0
    while done < len(scans) and (done < 2 or time.perf_counter() - t0 < budget_s):
        g.update(scans[done], origins[done], threads=threads)
        g.recenter(origins[done])
        vs += int(steps[done])
        done += 1
    dt = time.perf_counter() - t0
    return {"value": vs / dt, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": f"first {done} scans of one README-scale map (update + recenter), "
                      f"{threads} threads, {dt:.1f} s"}


def profiled_traffic(n_maps: int, key: str = "update_bytes_per_map"):
    """DRAM bytes of one batched step per map (walk + fold, or the kernel
    `key` names), from the ncu capture recorded in profiles/traffic.json,
    scaled to n_maps (each map's walk and fold touch only its own voxels).
    Returns (bytes, source)."""
    try:
        with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
            t = json.load(f)
        return float(t[key]) * n_maps, t.get("source")
    except (OSError, KeyError, ValueError):
        return None, None


def headline_config(K: int) -> dict:
    """The headline workload, identical in both arms' lines."""
    return {"workload": f"batch{K}_readme_701x701x151_64x1024", "maps": K,
            "grid": [701, 701, 151], "resolution_m": 0.1, "points_per_scan": 65536,
            "max_range_m": 50.0, "recenter_threshold_m": 4.0,
            "l2": "flushed between steps (512 MiB write)"}


def pct(a, q):
    return float(np.percentile(np.asarray(a, dtype=np.float64), q)) if len(a) else None


# ---------------------------------------------------------------------------
# headline: batched README-scale maps
# ---------------------------------------------------------------------------
def tune_shape(new_batch, dev, sensors, offsets, fixed=-1, max_updates=256):
    """The launch shape and voxel layout the batch's tuner picks for this
    workload, from a throw-away batch that integrates the step scans in
    order (wrapping around) until the tuner has timed every candidate.
    Returns ((shape, layout), updates the tuner took); a fixed shape (>= 0)
    is returned as is, with the default layout."""
    import cublox_b200 as C
    if fixed >= 0:
        return (fixed, C.LAYOUTS[0]), 0
    b, gs = new_batch(graphs=False)
    k = 0
    while b.tuning() and k < max_updates:
        j = k % len(dev)
        b.update(gs, dev[j], sensors[j], offsets=offsets[j])
        b.recenter(gs, sensors[j])
        k += 1
    choice = (b.get_option(C.BATCH_OPT_SHAPE), b.get_option(C.BATCH_OPT_LAYOUT))
    b.close()
    return choice, k


def run_headline(args, rank, world, dist):
    import torch
    import cublox_b200 as C
    from cublox_b200 import replicas

    K = args.maps
    n_steps = args.warmup + args.steps
    w, scans, origins = readme_batch(K, n_steps)
    steps = np.stack([count_steps(w.half, w.resolution, w.sensor.max_range, w.threshold,
                                  [scans[k][m] for k in range(n_steps)],
                                  [origins[k][m] for k in range(n_steps)]) for m in range(K)], axis=1)
    lo = C.yaml_log_odds()
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    flush = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")

    def new_batch(graphs=True, shape=None):
        b = C.Batch(stream=stream.cuda_stream)
        b.set_option(C.BATCH_OPT_GRAPHS, int(graphs))
        if shape is not None:  # (launch shape, voxel layout)
            b.set_option(C.BATCH_OPT_SHAPE, shape[0])
            b.set_option(C.BATCH_OPT_LAYOUT, shape[1])
        gs = []
        for _ in range(K):
            g = b.add_grid(w.half, w.resolution, False, w.threshold)
            g.setLogOddsParams(*lo)
            g.setMaxRaycastRange(w.sensor.max_range)
            gs.append(g)
        return b, gs

    offsets = []
    for k in range(n_steps):
        off = np.zeros(K + 1, np.int64)
        off[1:] = np.cumsum([s.shape[0] for s in scans[k]])
        offsets.append(off)
    sensors = [np.stack(origins[k]).astype(np.float32) for k in range(n_steps)]
    dev = [torch.from_numpy(np.concatenate(scans[k])).cuda() for k in range(n_steps)]
    # ---- launch shape: the batch's tuner, in its own pass before warm-up ---
    shape, tune_updates = tune_shape(new_batch, dev, sensors, offsets, args.shape)
    # ---- value: device-resident scans ------------------------------------
    b, gs = new_batch(shape=shape)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(n_steps)]
    actions = []
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    with Clocks(torch.cuda.current_device()) as clk:
        for k in range(n_steps):
            flush.zero_()
            ev[k][0].record(stream)
            b.update(gs, dev[k], sensors[k], offsets=offsets[k])
            a = b.recenter(gs, sensors[k])
            ev[k][1].record(stream)
            if k >= args.warmup:
                actions.extend(int(x) for x in a)
        torch.cuda.synchronize()
    if dist:
        dist.barrier()
    step_ms = np.asarray([ev[k][0].elapsed_time(ev[k][1]) for k in range(args.warmup, n_steps)])
    timed_vs = int(steps[args.warmup:].sum())
    own_ms = float(step_ms.sum())
    value = replicas.job_rate(timed_vs, own_ms / 1e3, dist, device="cuda")
    tot_ms = replicas.max_over_ranks(own_ms, dist, device="cuda")
    assert b.get_option(C.BATCH_OPT_SHAPE) == shape[0] and not b.tuning()
    for g in gs:
        assert g.check() == 0, "device error word set"
    b.close()

    # ---- kernel split, touched voxels: a separate pass with timing + stats --
    b, gs = new_batch(graphs=False, shape=shape)
    b.set_option(C.BATCH_OPT_TIMING, 1)
    for g in gs:
        g.enable_stats(True)
        g.enable_timing(True)
    walk_ms, fold_ms, touched, incs = [], [], [], []
    clear_ms, cleared = [], []  # recenters that fired (every step, warm-up included)
    for k in range(n_steps):
        flush.zero_()
        b.update(gs, dev[k], sensors[k], offsets=offsets[k])
        wm, fm = b.last_timing()
        acts = b.recenter(gs, sensors[k])
        for g, a in zip(gs, acts):
            if a == 1:
                clear_ms.append(g.last_timing()[2])
                cleared.append(g.last_clear())
        if k >= args.warmup:
            walk_ms.append(wm)
            fold_ms.append(fm)
            st = [g.last_stats() for g in gs]
            touched.append(sum(s["touched"] for s in st))
            incs.append(sum(s["op_incs"] + s["hit_incs"] for s in st))
    # a served-style fetch on the last map after the drive: 256 centres
    # within 3 m of the robot, r 1.5 m, the driver's OCCUPIED filter
    rng = np.random.default_rng(9)
    so = sensors[-1][-1]
    cen = (so + np.stack([rng.uniform(-3, 3, 256), rng.uniform(-3, 3, 256),
                          rng.uniform(-1.5, 1.5, 256)], axis=1)).astype(np.float32)
    fetch_ms, n_samples = [], 0
    for _ in range(6):
        t0 = time.perf_counter()
        off_f, _, _ = gs[-1].fetch_batch(cen, 1.5, C.VoxelState.OCCUPIED)
        fetch_ms.append((time.perf_counter() - t0) * 1e3)
        n_samples = int(off_f[-1])
    b.close()
    del dev

    # ---- e2e: public API from pinned host memory ---------------------------
    pinned = [torch.from_numpy(np.concatenate(scans[k])).pin_memory() for k in range(n_steps)]
    b, gs = new_batch(shape=shape)
    wall = []
    for k in range(n_steps):
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        b.update(gs, pinned[k].numpy(), sensors[k], offsets=offsets[k])
        b.recenter(gs, sensors[k])
        _ = gs[-1].storedAt(0)  # 4 bytes back; the stream orders every map's work before it
        t1 = time.perf_counter()
        if k >= args.warmup:
            wall.append(t1 - t0)
    b.close()
    e2e = replicas.job_rate(timed_vs, float(np.sum(wall)), dist, device="cuda")
    n_points = int(offsets[0][-1])

    peak, peak_kind = _peaks()
    upd_ms = np.asarray(walk_ms) + np.asarray(fold_ms)
    alg_bytes = 12.0 * n_points + 8.0 * np.asarray(touched, dtype=np.float64)
    achieved = float(np.mean(alg_bytes) / (np.mean(upd_ms) / 1e3) / 1e9)
    launches = 2 * args.steps + sum(1 for a in actions if a == 1)
    return {
        "value": value, "tot_ms": tot_ms, "step_ms": step_ms, "e2e": e2e, "wall": wall,
        "workload": f"batch{K}_readme_701x701x151_64x1024", "K": K, "n_points": n_points,
        "shape": shape, "tune_updates": tune_updates, "walk_ms": walk_ms, "fold_ms": fold_ms, "touched": touched, "incs": incs,
        "achieved": achieved, "peak": peak, "peak_kind": peak_kind, "launches": launches,
        "recenters": sum(1 for a in actions if a), "clocks": clk.summary(), "w": w,
        "clear_ms": clear_ms, "cleared": cleared, "fetch_ms": fetch_ms[1:],
        "fetch_samples": n_samples,
        "scans": scans, "origins": origins, "steps": steps,
    }


# ---------------------------------------------------------------------------
# plain drop-in: one README-scale map
# ---------------------------------------------------------------------------
def run_plain(args, hw):
    import torch
    import cublox_b200 as C
    w = hw["w"]
    assert torch.cuda.current_stream().cuda_stream != 0, "run_headline sets a dedicated stream"
    scans = [hw["scans"][k][0] for k in range(len(hw["scans"]))]
    origins = [hw["origins"][k][0] for k in range(len(hw["origins"]))]
    steps = hw["steps"][:, 0]
    stream = torch.cuda.current_stream()
    flush = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    lo = C.yaml_log_odds()
    g = C.OccupancyGrid(w.half, w.resolution, False, w.threshold, stream=stream.cuda_stream)
    g.setLogOddsParams(*lo)
    g.setMaxRaycastRange(w.sensor.max_range)
    dev = [torch.from_numpy(np.ascontiguousarray(s.T)).cuda() for s in scans]
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in scans]
    torch.cuda.synchronize()
    for k in range(len(scans)):
        flush.zero_()
        ev[k][0].record(stream)
        g.update(dev[k], origins[k])
        g.recenter(origins[k])
        ev[k][1].record(stream)
    torch.cuda.synchronize()
    ms = np.asarray([ev[k][0].elapsed_time(ev[k][1]) for k in range(args.warmup, len(scans))])
    vs = int(steps[args.warmup:].sum())
    g.close()
    pinned = [torch.from_numpy(s).pin_memory() for s in scans]
    g = C.OccupancyGrid(w.half, w.resolution, False, w.threshold, stream=stream.cuda_stream)
    g.setLogOddsParams(*lo)
    g.setMaxRaycastRange(w.sensor.max_range)
    wall = []
    for k in range(len(scans)):
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        g.update_ptr(pinned[k].data_ptr(), scans[k].shape[0], origins[k], C.LAYOUT_AOS)
        g.recenter(origins[k])
        _ = g.storedAt(0)
        if k >= args.warmup:
            wall.append(time.perf_counter() - t0)
    g.close()
    return {"workload": "readme_701x701x151_64x1024 (one map, OccupancyGrid drop-in)",
            "value": vs / (ms.sum() / 1e3), "unit": UNIT, "p50_ms": pct(ms, 50), "p99_ms": pct(ms, 99),
            "e2e": {"value": vs / float(np.sum(wall)), "unit": UNIT, "p50_ms": pct(wall, 50) * 1e3,
                    "p99_ms": pct(wall, 99) * 1e3}}


# ---------------------------------------------------------------------------
# batching: 32 maps of mixed sizes, uneven point counts
# ---------------------------------------------------------------------------
def run_batching(args):
    import torch
    import cublox_b200 as C
    from cublox_b200 import synth
    n_steps = args.warmup + args.batch_steps
    bw = synth.batching(n_steps=n_steps)
    steps = np.zeros((n_steps, bw.n_maps), np.int64)
    data = [bw.step(k) for k in range(n_steps)]
    for m in range(bw.n_maps):
        steps[:, m] = count_steps(bw.halves[m], bw.resolution, bw.max_range, bw.threshold,
                                  [data[k][0][m] for k in range(n_steps)],
                                  [data[k][1][m] for k in range(n_steps)])
    stream = torch.cuda.current_stream()
    assert stream.cuda_stream != 0, "run_headline sets a dedicated stream"
    flush = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")

    def new_batch(graphs=True, shape=None):
        b = C.Batch(stream=stream.cuda_stream)
        b.set_option(C.BATCH_OPT_GRAPHS, int(graphs))
        if shape is not None:  # (launch shape, voxel layout)
            b.set_option(C.BATCH_OPT_SHAPE, shape[0])
            b.set_option(C.BATCH_OPT_LAYOUT, shape[1])
        gs = []
        for m in range(bw.n_maps):
            g = b.add_grid(bw.halves[m], bw.resolution, False, bw.threshold)
            g.setLogOddsParams(*C.yaml_log_odds())
            g.setMaxRaycastRange(bw.max_range)
            gs.append(g)
        return b, gs

    dev, offs = [], []
    for clouds, _ in data:
        off = np.zeros(bw.n_maps + 1, np.int64)
        off[1:] = np.cumsum([c.shape[0] for c in clouds])
        offs.append(off)
        dev.append(torch.from_numpy(np.concatenate(clouds)).cuda())
    shape, _ = tune_shape(new_batch, dev, [d[1] for d in data], offs, args.shape)
    b, gs = new_batch(shape=shape)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in data]
    torch.cuda.synchronize()
    for k in range(n_steps):
        flush.zero_()
        ev[k][0].record(stream)
        b.update(gs, dev[k], data[k][1], offsets=offs[k])
        b.recenter(gs, data[k][1])
        ev[k][1].record(stream)
    torch.cuda.synchronize()
    ms = np.asarray([ev[k][0].elapsed_time(ev[k][1]) for k in range(args.warmup, n_steps)])
    vs = int(steps[args.warmup:].sum())
    b.close()
    pts = np.mean([o[-1] for o in offs[args.warmup:]])
    return {"workload": bw.name, "maps": bw.n_maps, "steps": args.batch_steps,
            "mean_points_per_step": float(pts), "value": vs / (ms.sum() / 1e3), "unit": UNIT,
            "rays_per_s": float(pts * len(ms) / (ms.sum() / 1e3)),
            "p50_ms": pct(ms, 50), "p99_ms": pct(ms, 99), "launch_shape": shape[0],
            "voxel_layout": shape[1],
            "l2": "flushed between steps (512 MiB write)"}


# ---------------------------------------------------------------------------
# serving: 16 robots, Poisson arrivals
# ---------------------------------------------------------------------------
def run_serving(args, budget_gb=None, seconds=None):
    import cublox_b200 as C
    from cublox_b200 import synth
    seconds = args.serve_seconds if seconds is None else seconds
    budget_gb = args.serve_budget_gb if budget_gb is None else budget_gb
    sw = synth.serving(seconds=seconds)
    # the reference's work units of each pooled scan, against a window
    # centred at its pose
    pool_steps = [[[count_steps(sw.halves[r], sw.resolution, sw.max_range, None, [p], [o])[0]
                    for (p, o) in cls] for cls in sw.pool[r]] for r in range(sw.n_robots)]
    s = C.Server(hbm_budget_bytes=int(budget_gb * (1 << 30)), max_tick_points=1 << 20,
                 graphs=True)
    lo = C.yaml_log_odds()
    ids = [s.add_map(sw.halves[r], sw.resolution, False, sw.threshold, max_range=sw.max_range,
                     log_odds=lo) for r in range(sw.n_robots)]
    reqs = []
    t_start = time.perf_counter()
    for i, (t, kind, r, c, j) in enumerate(sw.events):
        while True:
            now = time.perf_counter() - t_start
            if now >= t:
                break
            if t - now > 0.002:
                time.sleep(t - now - 0.001)
        if kind == "scan":
            pts, origin = sw.pool[r][c][j]
            reqs.append((t, kind, r, c, j, s.submit_scan(ids[r], pts, origin, True)))
        else:
            cen = sw.fetch_centres(i, r, sw.pool[r][0][0][1])
            reqs.append((t, kind, r, c, j, s.submit_fetch(ids[r], cen, sw.fetch_radius,
                                                          C.VoxelState.OCCUPIED)))
    s.drain()
    wall = time.perf_counter() - t_start
    warm = min(3.0, 0.1 * seconds)
    lat = {0: [], 1: [], 2: [], "fetch": []}
    vs = 0
    for t, kind, r, c, j, rid in reqs:
        if t < warm:
            continue
        _, l = s.times(rid)
        if kind == "scan":
            lat[c].append(l)
            vs += int(pool_steps[r][c][j])
        else:
            lat["fetch"].append(l)
    st = s.stats()
    s.close()
    # throughput over the time the work took: from the end of the warm-up
    # window to the last completion (drain), not the arrival window
    span = max(wall - warm, seconds - warm)
    names = {0: "16384", 1: "65536", 2: "262144"}
    out = {"workload": sw.name, "robots": sw.n_robots, "seconds": seconds,
           "arrivals": "Poisson, scans 400/s (16,384 / 65,536 / 262,144 points, p = .5/.35/.15), "
                       "fetches 100/s (256 centres, r 1.5 m, OCCUPIED filter as the driver uses)",
           "hbm_budget_gb": budget_gb, "warmup_excluded_s": warm,
           "scans_per_s": sum(len(lat[c]) for c in range(3)) / span,
           "voxel_steps_per_s": vs / span,
           "drain_s_after_last_arrival": wall - seconds,
           "ticks": st["ticks"], "scans_per_tick": st["scans"] / max(st["ticks"], 1),
           "evictions": st["evictions"], "peak_resident_gb": st["peak_resident_bytes"] / 2**30}
    for c in range(3):
        out[f"latency_ms_{names[c]}"] = {"p50": pct(lat[c], 50), "p99": pct(lat[c], 99),
                                         "n": len(lat[c])}
    out["latency_ms_fetch"] = {"p50": pct(lat["fetch"], 50), "p99": pct(lat["fetch"], 99),
                               "n": len(lat["fetch"])}
    return out


# ---------------------------------------------------------------------------
# reference arm
# ---------------------------------------------------------------------------
def run_reference(args):
    """The reference's own kernels (oracle/_ref/libcublox_ref.so) on the
    headline maps.  Scans and work-unit counts come from
    oracle/_ref/libcublox_refinputs.so (the same synthesiser source and the
    oracle's exact step count), so this process maps no library of the
    product."""
    import oracle as O
    from cublox_b200 import synth
    from cublox_b200 import yaml_log_odds  # pure Python (libm's logf)

    if not (O.ref_available() and os.path.exists(O.REF_INPUTS_SO)):
        return {"impl": "reference", "unavailable": "reference harness oracle/_ref was not built "
                                                     "(needs the reference tree)"}
    synth.use_library(O.REF_INPUTS_SO)
    import torch
    K = args.maps
    n_steps = args.warmup + args.steps
    w, scans, origins = readme_batch(K, n_steps)
    steps = np.asarray([[O.count_steps(scans[k][m], origins[k][m], w.resolution, False,
                                       w.sensor.max_range, lib_path=O.REF_INPUTS_SO)
                         for m in range(K)] for k in range(n_steps)], dtype=np.int64)
    flush = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    refs = []
    for m in range(K):
        r = O.RefGrid(w.half, w.resolution, False, w.threshold)
        r.set_log_odds(*yaml_log_odds())
        r.set_max_range(w.sensor.max_range)
        refs.append(r)
    soa = [[tuple(np.ascontiguousarray(s[:, a]) for a in range(3)) for s in row] for row in scans]
    wall = []
    fired = 0
    with Clocks(torch.cuda.current_device()) as clk:
        for k in range(n_steps):
            flush.zero_()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            acts = []
            for m in range(K):
                refs[m].update(None, origins[k][m], xyz=soa[k][m])
                acts.append(refs[m].recenter(origins[k][m]))
            t1 = time.perf_counter()
            if k >= args.warmup:
                wall.append(t1 - t0)
                fired += sum(1 for a in acts if not a["host_skip"])
    for r in refs:
        r.close()
    tot = float(np.sum(wall))
    value = int(steps[args.warmup:].sum()) / tot
    n_points = int(sum(s.shape[0] for s in scans[0]))
    # the harness's copies, as the reference's OccupancyGrid issues them:
    # x, y, z (pageable, 4 B each) and the 68-byte RayCastCfg per update; the
    # 28-byte RecenterResult back per recenter that passes the host gate
    h2d = 12 * n_points + 68 * K
    d2h = 28.0 * fired / max(args.steps, 1)
    loaded = sorted({ln.split()[-1] for ln in open("/proc/self/maps") if ln.rstrip().endswith(".so")
                     and os.path.realpath(ln.split()[-1]).startswith(ROOT)})
    return {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": tot * 1e3 / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded ray-cast LiDAR scans)", "impl": "reference",
        "config": headline_config(K),
        "form": "the reference's OccupancyGrid call sequence (three pageable copies, raycast, "
                "sync, apply, sync; recenter plan with a D2H round trip), one map after another",
        "p50_ms": pct(wall, 50) * 1e3, "p99_ms": pct(wall, 99) * 1e3,
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": 1, "kind": "reference",
                         "sample": "the reference's src/kernels.cu (sm_100a build) driven by one host "
                                   f"thread in its OccupancyGrid sequence, {args.steps} steps of {K} "
                                   "maps on the B200 (the reference has no CPU path)"},
        "repo_libraries_mapped": [os.path.relpath(p, ROOT) for p in loaded],
        "clocks": clk.summary(),
    }


# ---------------------------------------------------------------------------
# per-config suite (configs 1, 3, 4, 5 beside the headline), both arms
# ---------------------------------------------------------------------------
def _time_dev(fn, stream):
    import torch
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    fn()
    e1.record(stream)
    torch.cuda.synchronize()
    return e0.elapsed_time(e1)


def _fetch_centres(w, g_origin_f, n, seed):
    """n centres uniform inside the window (x, y) at z in [0, 3] m."""
    rng = np.random.default_rng(seed)
    half = np.asarray(w.half, dtype=np.float64) * w.resolution
    c = np.empty((n, 3), dtype=np.float32)
    c[:, 0] = g_origin_f[0] + rng.uniform(-half[0], half[0], n)
    c[:, 1] = g_origin_f[1] + rng.uniform(-half[1], half[1], n)
    c[:, 2] = rng.uniform(0.0, 3.0, n)
    return c


def suite_cublox(args):
    import torch
    import cublox_b200 as C
    from cublox_b200 import synth
    # a dedicated stream shared by the grids and the timing events (handle 0
    # would make every grid create its own stream)
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    lo = C.yaml_log_odds()
    out = {}
    # config 1: plain small
    w = synth.plain_small(threshold=1.0)
    pts, s0 = w.scan(0), w.sensor_origin(0)
    g = C.OccupancyGrid(w.half, w.resolution, False, 1.0, stream=stream.cuda_stream)
    g.setLogOddsParams(*lo)
    g.setMaxRaycastRange(w.sensor.max_range)
    g.enable_timing(True)
    dev = torch.from_numpy(np.ascontiguousarray(pts.T)).cuda()
    g.update(dev, s0)
    ms = [_time_dev(lambda: g.update(dev, s0), stream) for _ in range(30)]
    cnt = C.OccupancyGrid(w.half, w.resolution, False, None, origin=tuple(float(v) for v in s0))
    cnt.setMaxRaycastRange(w.sensor.max_range)
    vs = cnt.reference_steps(pts, s0)
    cnt.close()
    oi, of = g.getOriginIndex(), g.getOriginPosition()
    pos = (np.float32(of) + np.float32(w.extra["recenter_shift"]) * np.float32(w.resolution))
    g.last_timing()
    g.recenter(pos)
    clear_ms = g.last_timing()[2]
    cleared = g.last_clear()
    cen = _fetch_centres(w, g.getOriginPosition(), 1000, 0)
    g.fetch_batch(cen, 1.0)
    t0 = time.perf_counter()
    off, fp_, fs = g.fetch_batch(cen, 1.0)
    fetch_s = time.perf_counter() - t0
    g.close()
    out["config1_plain_small"] = {
        "update_ms_median": float(np.median(ms)), "rays_per_s": pts.shape[0] / (np.median(ms) / 1e3),
        "voxel_steps_per_s": vs / (np.median(ms) / 1e3),
        "recenter": {"shift_vox": list(w.extra["recenter_shift"]), "threshold_m": 1.0,
                     "cleared_voxels": cleared, "clear_ms": clear_ms,
                     "gb_per_s": 4.0 * cleared / (clear_ms / 1e3) / 1e9},
        "fetch_1000_centres_r1m": {"us": fetch_s * 1e6, "samples": int(off[-1]),
                                   "mode": "cublox_grid_fetch_batch (one call, samples to host)"}}
    # config 5: stress
    n_scans = args.stress_scans
    sw = synth.stress(n_scans)
    scans = [sw.scan(k) for k in range(n_scans)]
    origins = [sw.sensor_origin(k) for k in range(n_scans)]
    steps = count_steps(sw.half, sw.resolution, sw.sensor.max_range, sw.threshold, scans, origins)
    g = C.OccupancyGrid(sw.half, sw.resolution, False, sw.threshold, stream=stream.cuda_stream)
    g.setLogOddsParams(*lo)
    g.setMaxRaycastRange(sw.sensor.max_range)
    g.enable_timing(True)
    devs = [torch.from_numpy(np.ascontiguousarray(p.T)).cuda() for p in scans]
    upd, clr, cleared, fetch_occ, fetch_cnt, samples = [], [], [], [], [], []
    for k in range(n_scans):
        def step():
            g.update(devs[k], origins[k])
            g.recenter(origins[k])
        t = _time_dev(step, stream)
        tm = g.last_timing()
        if k >= 1:
            upd.append(t)
            if tm[2] >= 0:
                clr.append(tm[2])
                cleared.append(g.last_clear())
        if k >= n_scans - 3:
            cen = _fetch_centres(sw, g.getOriginPosition(), sw.fetch_centres, k)
            t0 = time.perf_counter()
            cts = g.fetch_counts(cen, sw.fetch_radius)
            fetch_cnt.append(time.perf_counter() - t0)
            t0 = time.perf_counter()
            off, _, _ = g.fetch_batch(cen, sw.fetch_radius, C.VoxelState.OCCUPIED)
            fetch_occ.append(time.perf_counter() - t0)
            samples.append((int(cts.sum()), int(off[-1])))
    g.close()
    # the batched/graph form of the same drive: a batch of one map
    b = C.Batch(stream=stream.cuda_stream)
    b.set_option(C.BATCH_OPT_GRAPHS, 1)
    gb = b.add_grid(sw.half, sw.resolution, False, sw.threshold)
    gb.setLogOddsParams(*lo)
    gb.setMaxRaycastRange(sw.sensor.max_range)
    aos = [torch.from_numpy(p).cuda() for p in scans]
    bt = []
    for k in range(n_scans):
        so = origins[k].reshape(1, 3)
        off = np.array([0, scans[k].shape[0]], np.int64)

        def bstep():
            b.update([gb], aos[k], so, offsets=off)
            b.recenter([gb], so)
        t = _time_dev(bstep, stream)
        if k >= 1:
            bt.append(t)
    b.close()
    out["next_rows"] = _next_rows_cublox(stream)
    out["config5_stress"] = {
        "scans": n_scans - 1, "voxel_steps_per_s": float(steps[1:].sum() / (np.sum(upd) / 1e3)),
        "update_recenter_ms_p50": pct(upd, 50), "update_recenter_ms_p99": pct(upd, 99),
        "recenter_gb_per_s": float(4.0 * np.sum(cleared) / (np.sum(clr) / 1e3) / 1e9) if clr else None,
        "recenters": len(clr),
        "batched_graph_form": {"voxel_steps_per_s": float(steps[1:].sum() / (np.sum(bt) / 1e3)),
                               "update_recenter_ms_p50": pct(bt, 50),
                               "note": "same drive through a one-map Batch with CUDA-graph "
                                       "replay (the first updates tune the launch shape)"},
        "fetch_10000_centres_r2m": {"all_states_counts_only_ms": float(np.mean(fetch_cnt) * 1e3),
                                    "occupied_samples_to_host_ms": float(np.mean(fetch_occ) * 1e3),
                                    "samples_all_states": samples[-1][0],
                                    "samples_occupied": samples[-1][1]}}
    return out


def _next_rows_inputs():
    """A README-scale scan in its sensor frame (yawed pose), a 640x480
    16-bit depth image and the robot's position, for the driver-side steps."""
    from cublox_b200 import synth
    w = synth.readme_scale(2)
    world, t = w.scan(0), w.sensor_origin(0)
    yaw = 0.4
    R = np.array([[np.cos(yaw), -np.sin(yaw), 0], [np.sin(yaw), np.cos(yaw), 0], [0, 0, 1]],
                 dtype=np.float32)
    local = ((world.astype(np.float64) - t) @ R.astype(np.float64)).astype(np.float32)
    rng = np.random.default_rng(5)
    depth = rng.integers(400, 8000, size=(480, 640)).astype(np.uint16)
    depth[rng.random((480, 640)) < 0.05] = 0
    K = np.float32([525.0, 525.0, 319.5, 239.5])
    return w, local, R, t, depth, K


def _next_rows_cublox(stream):
    import torch
    import cublox_b200 as C
    w, local, R, t, depth, K = _next_rows_inputs()
    g = C.OccupancyGrid(w.half, w.resolution, False, None, stream=stream.cuda_stream)
    g.setLogOddsParams(*C.yaml_log_odds())
    g.setMaxRaycastRange(w.sensor.max_range)
    dl = torch.from_numpy(local).cuda()
    g.update_pose(dl, R, t)
    pose_ms = [_time_dev(lambda: g.update_pose(dl, R, t), stream) for _ in range(10)]
    world = torch.from_numpy(np.ascontiguousarray(
        (local.astype(np.float64) @ R.T.astype(np.float64) + t).astype(np.float32).T)).cuda()
    plain_ms = [_time_dev(lambda: g.update(world, t), stream) for _ in range(10)]
    dd = torch.from_numpy(depth.view(np.int16)).cuda()
    depth_ms = [_time_dev(lambda: g.update_depth(dd, K, np.eye(3, dtype=np.float32), t), stream)
                for _ in range(10)]
    g.fetch_viz(t, 25.0, C.VoxelState.OCCUPIED, 0, 1, 25.0, 200000)
    t0 = time.perf_counter()
    for _ in range(10):
        v = g.fetch_viz(t, 25.0, C.VoxelState.OCCUPIED, 0, 1, 25.0, 200000)
    viz_ms = (time.perf_counter() - t0) / 10 * 1e3
    g.close()
    return {"update_pose_65536_points_ms": float(np.median(pose_ms)),
            "update_world_cloud_same_scan_ms": float(np.median(plain_ms)),
            "update_depth_640x480_ms": float(np.median(depth_ms)),
            "fetch_viz_occupied_r25m_ms": viz_ms, "viz_points": int(v.shape[0]),
            "note": "device time of update from a sensor-frame cloud (filter + transform fused "
                    "ahead of the walk) beside update of the same scan already in the world "
                    "frame; fetch_viz wall time with samples to host"}


def _next_rows_reference():
    """The driver's own host loops for the same steps (restated in the oracle,
    single thread): buildCloudInOdomFrame, depthCallback, the viz loop."""
    import oracle as O
    import cublox_b200 as C
    w, local, R, t, depth, K = _next_rows_inputs()
    O.build()
    t0 = time.perf_counter()
    for _ in range(5):
        O.ingest(local, R, t, w.sensor.max_range)
    ingest_ms = (time.perf_counter() - t0) / 5 * 1e3
    t0 = time.perf_counter()
    for _ in range(5):
        O.depth_cloud(depth, K)
    depth_ms = (time.perf_counter() - t0) / 5 * 1e3
    g = C.OccupancyGrid(w.half, w.resolution, False, None)
    g.setMaxRaycastRange(w.sensor.max_range)
    g.setLogOddsParams(*C.yaml_log_odds())
    g.update_pose(local, R, t)
    pos, _ = g.fetchOccupancyAround(t, 25.0, C.VoxelState.OCCUPIED, 200000)
    g.close()
    t0 = time.perf_counter()
    for _ in range(5):
        O.viz(pos, w.resolution, False, 1, 25.0, 200000, t)
    viz_ms = (time.perf_counter() - t0) / 5 * 1e3
    return {"build_cloud_in_odom_frame_65536_points_ms": ingest_ms,
            "depth_to_cloud_640x480_ms": depth_ms,
            "viz_loop_ms": viz_ms, "viz_points_in": int(pos.shape[0]),
            "kind": "port", "cores": 1,
            "note": "the reference's driver does these on the host; timed here as their "
                    "single-threaded CPU restatement (oracle)"}


def suite_reference(args):
    import oracle as O
    import cublox_b200 as C
    from cublox_b200 import synth
    if not O.ref_available():
        return {"impl": "reference", "unavailable": "oracle/_ref was not built"}
    lo = C.yaml_log_odds()

    def ref(half, res, thr, mr):
        r = O.RefGrid(half, res, False, thr)
        r.set_log_odds(*lo)
        r.set_max_range(mr)
        return r

    def soa(p):
        return tuple(np.ascontiguousarray(p[:, a]) for a in range(3))

    out = {"next_rows": _next_rows_reference()}
    w = synth.plain_small(threshold=1.0)
    pts, s0 = w.scan(0), w.sensor_origin(0)
    r = ref(w.half, w.resolution, 1.0, w.sensor.max_range)
    x = soa(pts)
    r.update(None, s0, xyz=x)
    ms = []
    for _ in range(30):
        t0 = time.perf_counter()
        r.update(None, s0, xyz=x)
        ms.append((time.perf_counter() - t0) * 1e3)
    cnt = C.OccupancyGrid(w.half, w.resolution, False, None, origin=tuple(float(v) for v in s0))
    cnt.setMaxRaycastRange(w.sensor.max_range)
    vs = cnt.reference_steps(pts, s0)
    cnt.close()
    oi, of = r.origin()
    pos = (np.float32(of) + np.float32(w.extra["recenter_shift"]) * np.float32(w.resolution))
    t0 = time.perf_counter()
    r.recenter(pos)
    rec_ms = (time.perf_counter() - t0) * 1e3
    cen = _fetch_centres(w, r.origin()[1], 1000, 0)
    t0 = time.perf_counter()
    ns = sum(r.fetch(c, 1.0)[0].shape[0] for c in cen)
    fetch_s = time.perf_counter() - t0
    r.close()
    out["config1_plain_small"] = {
        "update_ms_median": float(np.median(ms)), "rays_per_s": pts.shape[0] / (np.median(ms) / 1e3),
        "voxel_steps_per_s": vs / (np.median(ms) / 1e3), "recenter_wall_ms": rec_ms,
        "fetch_1000_centres_r1m": {"us": fetch_s * 1e6, "samples": ns,
                                   "mode": "fetchOccupancyAround once per centre"}}
    # config 3: 32 maps, one update call per map per step
    bw = synth.batching(n_steps=args.batch_steps + 3)
    refs = [ref(bw.halves[m], bw.resolution, bw.threshold, bw.max_range) for m in range(bw.n_maps)]
    data = [bw.step(k) for k in range(args.batch_steps + 3)]
    steps = np.zeros((len(data), bw.n_maps), np.int64)
    for m in range(bw.n_maps):
        steps[:, m] = count_steps(bw.halves[m], bw.resolution, bw.max_range, bw.threshold,
                                  [d[0][m] for d in data], [d[1][m] for d in data])
    wall = []
    for k, (clouds, sensors) in enumerate(data):
        xs = [soa(c) for c in clouds]
        t0 = time.perf_counter()
        for m in range(bw.n_maps):
            refs[m].update(None, sensors[m], xyz=xs[m])
            refs[m].recenter(sensors[m])
        if k >= 3:
            wall.append(time.perf_counter() - t0)
    for rr in refs:
        rr.close()
    out["config3_batching"] = {"maps": bw.n_maps, "steps": len(wall),
                               "voxel_steps_per_s": float(steps[3:].sum() / np.sum(wall)),
                               "step_ms_p50": pct(wall, 50) * 1e3, "mode": "32 sequential update calls"}
    # config 4: the same request stream served one scan at a time
    sw = synth.serving(seconds=args.serve_seconds)
    refs = [ref(sw.halves[rb], sw.resolution, sw.threshold, sw.max_range) for rb in range(sw.n_robots)]
    svc = {0: [], 1: [], 2: []}
    busy = 0.0
    n_done = 0
    t_start = time.perf_counter()
    for t, kind, rb, c, j in sw.events:
        if kind != "scan":
            continue
        p, o = sw.pool[rb][c][j]
        xs = soa(p)
        t0 = time.perf_counter()
        refs[rb].update(None, o, xyz=xs)
        refs[rb].recenter(o)
        dt = time.perf_counter() - t0
        busy += dt
        svc[c].append(dt * 1e3)
        n_done += 1
        if time.perf_counter() - t_start > args.serve_seconds:
            break
    for rr in refs:
        rr.close()
    out["config4_serving"] = {
        "mode": "each scan's update + recenter alone, back to back (no batching, no overlap)",
        "scans": n_done, "max_scans_per_s": n_done / busy,
        "offered_scans_per_s": 400.0,
        **{f"service_ms_{k}": {"p50": pct(v, 50), "p99": pct(v, 99)}
           for k, v in zip(("16384", "65536", "262144"), (svc[0], svc[1], svc[2]))}}
    # config 5: stress
    n_scans = args.stress_scans
    sw5 = synth.stress(n_scans)
    scans = [sw5.scan(k) for k in range(n_scans)]
    origins = [sw5.sensor_origin(k) for k in range(n_scans)]
    steps5 = count_steps(sw5.half, sw5.resolution, sw5.sensor.max_range, sw5.threshold, scans, origins)
    r = ref(sw5.half, sw5.resolution, sw5.threshold, sw5.sensor.max_range)
    upd, rec = [], []
    for k in range(n_scans):
        xs = soa(scans[k])
        t0 = time.perf_counter()
        r.update(None, origins[k], xyz=xs)
        t1 = time.perf_counter()
        r.recenter(origins[k])
        t2 = time.perf_counter()
        if k >= 1:
            upd.append(t2 - t0)
            rec.append(t2 - t1)
    cen = _fetch_centres(sw5, r.origin()[1], 100, n_scans)
    t0 = time.perf_counter()
    for c in cen:
        r.fetch(c, sw5.fetch_radius, state_filter=2)
    f_occ = (time.perf_counter() - t0) / len(cen)
    r.close()
    out["config5_stress"] = {
        "scans": n_scans - 1, "voxel_steps_per_s": float(steps5[1:].sum() / np.sum(upd)),
        "update_recenter_ms_p50": pct(upd, 50) * 1e3, "recenter_wall_ms_p50": pct(rec, 50) * 1e3,
        "fetch_10000_centres_r2m_occupied_ms": f_occ * 1e4 * 1e3,
        "fetch_note": "100 centres timed one call each, scaled to 10,000"}
    return out


def main():
    ap = argparse.ArgumentParser(description=__doc__.split("\n")[0])
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=30)
    ap.add_argument("--warmup", type=int, default=20, help=">= 3; the launch-shape tuner "
                    "uses the first 16 updates")
    ap.add_argument("--maps", type=int, default=8)
    ap.add_argument("--shape", type=int, default=-1, help="fix the batch launch shape "
                    "(default: tuned online during warm-up)")
    ap.add_argument("--impl", choices=["cublox", "reference"], default="cublox")
    ap.add_argument("--batch-steps", type=int, default=20)
    ap.add_argument("--serve-seconds", type=float, default=60.0)
    ap.add_argument("--serve-budget-gb", type=float, default=120.0)
    ap.add_argument("--only-headline", action="store_true")
    ap.add_argument("--suite", choices=["headline", "configs", "plain"], default="headline",
                    help="configs: the per-config numbers (1, 3, 4, 5) instead of the headline; "
                         "plain: only the one-map drop-in run")
    ap.add_argument("--stress-scans", type=int, default=12)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    args = ap.parse_args()
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    import torch
    torch.cuda.set_device(local)
    if args.suite == "plain":
        if rank == 0:
            stream = torch.cuda.Stream()
            torch.cuda.set_stream(stream)
            n_steps = args.warmup + args.steps
            w, scans, origins = readme_batch(1, n_steps)
            steps = count_steps(w.half, w.resolution, w.sensor.max_range, w.threshold,
                                [sc[0] for sc in scans], [o[0] for o in origins])
            hw = {"w": w, "scans": scans, "origins": origins, "steps": steps[:, None]}
            print(json.dumps({"suite": "plain", **run_plain(args, hw)}), flush=True)
        return 0
    if args.suite == "configs":
        if rank == 0:
            fn = suite_reference if args.impl == "reference" else suite_cublox
            print(json.dumps({"impl": args.impl, "suite": "configs", **fn(args)}), flush=True)
        return 0
    if args.impl == "reference":
        if rank != 0:
            return 0
        print(json.dumps(run_reference(args)), flush=True)
        return 0
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as tdist
        tdist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
        dist = tdist
    h = run_headline(args, rank, world, dist)
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if rank != 0:
        return 0
    out = {
        "metric": METRIC, "value": h["value"], "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": h["tot_ms"] / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded ray-cast LiDAR scans)",
        "config": headline_config(h["K"]),
        "form": "batched: one walk + one fold launch per step over all maps, CUDA graph replay",
        "launch_shape": h["shape"][0], "voxel_layout": h["shape"][1],
        "tuning": f"separate pass before warm-up ({h['tune_updates']} updates of a throw-away "
                  "batch); no timed step runs a candidate shape",
        "parallelism": f"replicas x{world} (map-sharded, no collective)",
        "p50_ms": pct(h["step_ms"], 50), "p99_ms": pct(h["step_ms"], 99),
        "kernel_ms": {"walk": float(np.mean(h["walk_ms"])), "fold": float(np.mean(h["fold_ms"]))},
        "recenters": h["recenters"],
        "e2e": {"value": h["e2e"], "unit": UNIT, "h2d_bytes_per_step": 12 * h["n_points"],
                "d2h_bytes_per_step": 4, "p50_ms": pct(h["wall"], 50) * 1e3,
                "p99_ms": pct(h["wall"], 99) * 1e3},
        "roofline": {"bound": "hbm", "kernel": "update = batch walk + batch fold",
                     "achieved": h["achieved"], "peak": h["peak"], "unit": "GB/s",
                     "frac": h["achieved"] / h["peak"], "peak_source": h["peak_kind"],
                     "traffic": profiled_traffic(h["K"])[0],
                     "traffic_source": profiled_traffic(h["K"])[1],
                     "algorithmic_bytes": "12 B per point + 8 B per touched voxel (occ read+write); "
                                          "the fold reads and writes whole 128-byte lines of the "
                                          "lines the walk flagged",
                     },
        "recenter": ({"fired": len(h["clear_ms"]),
                      "clear_ms_mean": float(np.mean(h["clear_ms"])),
                      "cleared_voxels_mean": float(np.mean(h["cleared"])),
                      "gb_per_s": float(4.0 * np.sum(h["cleared"]) / (np.sum(h["clear_ms"]) / 1e3)
                                        / 1e9),
                      "peak_gbs": h["peak"],
                      "note": "device time of the slab clear of each recenter that fired "
                              "(4 m threshold, about every 27 scans; 4 B written per cleared "
                              "voxel); the reference publishes 4.822 ms per recenter on an "
                              "RTX 3090 (README.md:35)"}
                     if h["clear_ms"] else {"fired": 0}),
        "fetch": {"centres": 256, "radius_m": 1.5, "filter": "OCCUPIED",
                  "wall_ms_median": float(np.median(h["fetch_ms"])),
                  "samples": h["fetch_samples"],
                  "note": "cublox_grid_fetch_batch on one README map after the drive, samples "
                          "copied to host, wall time"},
        "gpu_launches": h["launches"],
        "clocks": h["clocks"],
    }
    import cublox_b200 as C
    red_l2 = C.red_rate(64 << 20, 1 << 30)      # buffer in L2
    red_hbm = C.red_rate(4 << 30, 1 << 30)      # buffer far beyond L2
    ach = float(np.mean(h["incs"]) / (np.mean(h["walk_ms"]) / 1e3))
    fold_bytes = profiled_traffic(h["K"], "fold_bytes_per_map")[0]
    if fold_bytes:
        fold_gbs = fold_bytes / (float(np.mean(h["fold_ms"])) / 1e3) / 1e9
        out["roofline"]["fold"] = {
            "kernel": "batch fold (flagged lines)", "achieved": fold_gbs, "unit": "GB/s",
            "peak": h["peak"], "frac": fold_gbs / h["peak"], "peak_source": h["peak_kind"],
            "basis": "the fold's ncu DRAM bytes per map x maps / its live device time: the "
                     "bytes it must move (256 B read and up to 256 B written per flagged line)"}
    requests = profiled_traffic(h["K"], "walk_red_requests_per_map")[0]
    if requests:
        rate = requests / (float(np.mean(h["walk_ms"])) / 1e3)
        out["roofline"]["l2_atomic"] = {
            "kernel": "batch walk", "achieved": rate, "unit": "reduction requests/s",
            "peak": red_l2, "frac": rate / red_l2, "peak_beyond_l2": red_hbm,
            "peak_source": "cublox_probe_red_rate on this GPU, this run (distinct pseudo-random "
                           "addresses; 64 MiB buffer in L2, and 4 GiB beyond it)",
            "increments_per_s": ach,
            "basis": "the walk's ncu reduction requests at L2 per map (default launch shape) x maps "
                     "/ its live device time; a request adds for all lanes on one voxel or in one "
                     "sector, so the U + H in-window increments are about three a request"}
    if world == 1 and not args.only_headline:
        out["plain"] = run_plain(args, h)
        out["batching"] = run_batching(args)
        out["serving"] = run_serving(args)
        # admission queuing: a budget that holds about half of the 16 maps (5.8 GB in all)
        out["serving_small_budget"] = run_serving(args, budget_gb=3.0, seconds=0.5)
        if not args.no_cpu_baseline:
            w = h["w"]
            scans = [h["scans"][k][0] for k in range(len(h["scans"]))]
            origins = [h["origins"][k][0] for k in range(len(h["origins"]))]
            out["cpu_baseline"] = cpu_baseline(w, scans, origins, h["steps"][:, 0])
    print(json.dumps(out), flush=True)
    return 0


if __name__ == "__main__":
    sys.exit(main())
