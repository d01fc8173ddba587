#!/usr/bin/env python3
"""Throughput of the MOLOCH dynamical-core step on GB300, in grid-point-steps/s.

Workload (the 512 x 512 x 60 single-domain case): the reference's idealized
state (param + fill_atmosphere) on a 512 x 512 x 60 grid, a Gaussian hill of
500 m and 20-gridpoint e-folding radius at the domain centre, and a seeded
U(-0.5, +0.5) K theta perturbation on the lowest 10 levels (seed 1234).
Synthetic seeded inputs: the reference has no dataset.

A step is one moloch() call: dt = 30 s = 3 advection steps and 15 acoustic
substeps.  value = jx*iy*kz*steps / time of the timed steps (device time,
CUDA events on the library's stream), summed over replicas for --gpus N
(one independent domain per GPU, "replicas only": the path has no exchange
between domains).  The headline path is FP32 storage with the FP64
tridiagonal solve and the learned acoustic-cycle surrogate attached under
its judge: the surrogate is trained first (pairs collected from plain steps
of a scratch domain, outside the timed region), and every sound() call of
the timed steps runs it or the plain sound loop as the on-device judge
decides.  The plain FP32 step and the plain FP64 step are timed beside it
on the same state, and the errors against the FP64 step are reported.
--workload surrogate runs the 256 x 256 x 40 surrogate case instead.

--impl reference times the CPU restatement of the reference (the reference
itself is Fortran and no Fortran compiler exists on these machines) on the
host cores, on bounded samples of the same workload.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "grid-pt-steps/s on 1 GB300: FP32+surrogate vs plain FP64 GPU at stated error"
UNIT = "grid-point-steps/s"
JX, IY, KZ = 512, 512, 60
HILLS = ((500.0, (JX + 1) / 2.0, (IY + 1) / 2.0, 20.0),)
SEED = 1234

# Algorithmic words (one bulk-type element each) per grid point per launch:
# the distinct global arrays each kernel must read or write.  Intermediates
# that an ideal kernel would keep on chip (zdiv2b, the FP64 Thomas stash) are
# not counted; their traffic shows up as measured traffic above algorithmic.
ALG_WORDS = {
    "k_prediag": 13,          # r: pai t q(5) | w: p qsat tvirt qwltot qwitot tetav
    "k_sound_div": 7,         # r: u v fmz rfw rfs | w: s zdiv2a
    "k_sound_damp": 8,        # r: zdiv2a u v fmz s | w: u v zdiv2b
    "k_sound_divdamp": 9,     # r: u v fmz rfw rfs | w: u v s zdiv2b (fused div + damp)
    "k_sound_column": 16,     # r: w fmzf qv tetav pai qsat t zdiv2b fmz qc qwltot qwitot | w: w deltaw tetav pai
    "k_sound_column_tw": 16,  # the same arrays (the TMA-staged column solve)
    "k_sound_column_tm": 16,  # its name in earlier result lines
    "k_sound_momentum": 7,    # r: u v deltaw tetav pai | w: u v
    "k_waf_vertical": 26,     # r: 7 fields u v w s wafu wafd | w: 10 wz ux vx wx
    "k_waf_horizontal": 36,   # r: 10 wz 10 pp u v wafn wafs wafe wafw | w: 10 pp
    "k_stag_from_x": 6,       # r: ux vx wx | w: u v w
    "k_postdiag": 12,         # r: pai tetav q(5) | w: tvirt t p rho qsat
}
# DRAM traffic (dram__bytes_read.sum + dram__bytes_write.sum) of one launch
# from an ncu capture of the kernel, and the grid points of that capture;
# scaled by the point count to the benchmarked size (traffic grows in
# proportion: one pass over each array per launch)
_STAGED = (1055.7e6, 512 * 512 * 60)
NCU_TRAFFIC = {"k_sound_column": (847.0e6, 384 * 384 * 60), "k_sound_column_tw": _STAGED}
# sm__pipe_fp64_cycles_active (% of peak, active) from the same captures
_STAGED_PIPE = {"pipe_fp64_active_pct": 53.9, "capture": "512x512x60", "fp64_operations_per_level": 4}
NCU_FP64_PIPE = {"k_sound_column": {"pipe_fp64_active_pct": 35.7, "capture": "384x384x60",
                                    "fp64_operations_per_level": 4},
                 "k_sound_column_tw": _STAGED_PIPE}
# the names earlier result lines gave the staged column solve, once three kernels
for _name in ("k_sound_column_tm", "k_sound_column_tw12"):
    NCU_TRAFFIC[_name], NCU_FP64_PIPE[_name] = _STAGED, _STAGED_PIPE


def column_variant(name, tuning):
    """Name an earlier result line gives the staged column solve, whose
    profile kind was k_sound_column_tm, under a tuning: for reading those
    lines.  Profiles now name the one kernel there is, k_sound_column_tw."""
    if name != "k_sound_column_tm" or len(tuning) < 2:
        return name
    return "k_sound_column_tw12" if tuning[1] & 128 else "k_sound_column_tw16" if tuning[1] & 256 else name


# the FP64 step's kernels are bound by GB300's FP64 rate, not HBM: their
# FP64-pipe activity from one-launch ncu captures at 256x256x60, in the shapes
# a handle of that size starts with (strips of 32 rows, k-marching, five fields
# a thread), which the autotuner picks as well
NCU_FP64_STEP = {"k_sound_column": {"pipe_fp64_active_pct": 84.5, "dram_pct": 20.7},
                 "k_waf_vertical": {"pipe_fp64_active_pct": 78.7, "dram_pct": 7.3},
                 "k_waf_horizontal": {"pipe_fp64_active_pct": 87.6, "dram_pct": 12.2},
                 "k_sound_momentum": {"pipe_fp64_active_pct": 76.9, "dram_pct": 10.6},
                 "k_sound_div": {"pipe_fp64_active_pct": 86.9, "dram_pct": 23.1},
                 "k_sound_damp": {"pipe_fp64_active_pct": 85.1, "dram_pct": 26.7}}
# whole-step algorithmic words per grid point of the fused design target
# (pre-diag 11 + 3 sound cycles x 91 + 3 advection steps x 23 + post-diag 11)
B_ALG_WORDS = 364


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu=0):
        self.gpu = gpu
        self.proc = None
        self.out = None

    def start(self):
        try:
            path = os.environ.get("MOLOCH_CLOCKS_CSV")  # optional copy of the raw samples
            self.out = open(path, "w") if path else None
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.lines = []
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())
            if self.out:
                self.out.write(line)

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.t.join(timeout=2)
        if self.out:
            self.out.close()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def dist_setup():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if ws > 1:
        import torch.distributed as dist
        backend = "nccl" if os.environ.get("MOLOCH_BENCH_BACKEND", "nccl") == "nccl" else "gloo"
        dist.init_process_group(backend)
        return dist, rank, ws
    return None, 0, 1


def reduce_max(dist, x, device=None):
    """Maximum of a float over ranks (identity without a process group)."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def reduce_sum(dist, x, device=None):
    if dist is None:
        return x
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.SUM)
    return float(t.item())


def barrier(dist, device=None):
    if dist is not None:
        if device is not None:
            dist.barrier(device_ids=[device.index])
        else:
            dist.barrier()


def rmse(a, b):
    return float(np.sqrt(np.mean((np.asarray(a) - np.asarray(b)) ** 2)))


def cpu_sample(steps, jx=256, iy=256, kz=KZ, threads=None):
    """Oracle throughput on the host cores: a bounded sample of the workload."""
    from oracle import oracle
    threads = threads or os.cpu_count() or 1
    L = oracle.lib()
    L.oracle_set_threads(threads)
    hills = ((500.0, (jx + 1) / 2.0, (iy + 1) / 2.0, 20.0 * jx / JX),)
    o = oracle.Oracle(oracle.make_cfg(jx, iy, kz, hills=hills, seed=SEED))
    t0 = time.perf_counter()
    for s in range(steps):
        o.step(s + 1)
    dt = time.perf_counter() - t0
    o.close()
    return jx * iy * kz * steps / dt, dt, threads


def run_reference(args, dist, rank, ws):
    if rank != 0:
        return 0
    per_step = []
    for _ in range(args.warmup):
        cpu_sample(1)
    for _ in range(args.steps):
        v, dt, threads = cpu_sample(1)
        per_step.append(dt)
    total = sum(per_step)
    gp = 256 * 256 * KZ
    value = gp * args.steps / total
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1e3 * total / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic", "impl": "reference",
        "config": {"workload": f"{JX}x{IY}x{KZ} idealized state, 500 m hill, seeded theta noise",
                   "sample": "each step: one moloch() step on a 256x256x60 sample of the workload"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": "256x256x60, 1 step per timed step; C restatement of nompi/mod_moloch.F90 "
                                   "(reference build unavailable: no Fortran compiler on the host)"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def make_domain(dm, mode, stream):
    d = dm.Moloch(JX, IY, KZ, mode=mode, stream=stream)
    d.setup_idealized(hills=HILLS, pert_amp=0.5, pert_levels=10, seed=SEED, device=True)
    return d


def tuned(dm, mode, stream):
    """Launch shapes picked by the project's autotuner on a scratch domain of
    the same size (autotuning advances the state it runs on)."""
    scratch = make_domain(dm, mode, stream)
    choice = scratch.autotune()
    scratch.close()
    d = make_domain(dm, mode, stream)
    d.set_tuning(choice)
    return d, choice


def time_steps(torch, d, stream, steps, graph=True):
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    d.sync()
    torch.cuda.synchronize()
    e0.record(stream)
    k0 = d.kernel_count
    d.run(steps, graph=graph)
    e1.record(stream)
    e1.synchronize()
    d.sync()
    return e0.elapsed_time(e1), d.kernel_count - k0


def e2e_steps(torch, dm, d, stream, steps, warmup=3, reps=5):
    """Through the reference-facing C ABI with host arrays, as a driver time
    loop does it: every step uploads the prognostic state (u, v, w, pai, t,
    qx), runs one moloch() call and reads back the output fields t and ps
    (the fields the reference driver writes, regcm_dynamical_core.F90:203-216)
    with the asynchronous output path, whose copy overlaps the next step.
    The host arrays are registered (pinned) once before the loop, as a
    driver does with its module arrays: each upload is then a DMA that
    overlaps the step still running."""
    names_in = ("u", "v", "w", "pai", "t", "qx")
    host = {n: d.download(n) for n in names_in}
    for n in names_in:
        d.host_register(host[n])
    t_out, ps_out = d.download("t"), d.download("ps")  # the driver's output arrays
    d.host_register(t_out)
    d.host_register(ps_out)
    # untimed iterations: the upload staging buffers are allocated on first
    # use, and the first DMAs from newly registered ranges run slower
    for _ in range(max(1, warmup)):
        for n in names_in:
            d.upload(n, host[n])
        d.moloch(1)
        d.output_start()
        d.output_finish(t_out, ps_out)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    runs = []
    split = []  # (device ms, host wall ms) of each loop
    out = None
    for rep in range(reps):  # the host side of the copies varies with the machine's other work
        d.sync()
        e0.record(stream)
        t0 = time.perf_counter()
        for s in range(steps):
            for n in names_in:
                d.upload(n, host[n])
            d.moloch(s + 1)
            if s > 0:
                out = d.output_finish(t_out, ps_out)
            d.output_start()
        out = d.output_finish(t_out, ps_out)
        e1.record(stream)
        e1.synchronize()
        wall = time.perf_counter() - t0
        runs.append(max(e0.elapsed_time(e1), 1e3 * wall))
        split.append((round(e0.elapsed_time(e1), 2), round(1e3 * wall, 2)))
    # the raw DMA rate from one registered host array in the same process,
    # for reading a slow run
    src = torch.from_numpy(host["t"].reshape(-1))
    dst = torch.empty(src.numel(), dtype=src.dtype, device=torch.device("cuda", torch.cuda.current_device()))
    dma = 0.0
    for _ in range(3):
        with torch.cuda.stream(stream):
            e0.record(stream)
            dst.copy_(src, non_blocking=True)
            e1.record(stream)
        e1.synchronize()
        dma = max(dma, src.numel() * src.element_size() / (e0.elapsed_time(e1) / 1e3) / 1e9)
    for a in list(host.values()) + [t_out, ps_out]:
        d.host_unregister(a)
    h2d = sum(host[n].nbytes for n in names_in)
    d2h = out[0].nbytes + out[1].nbytes
    return runs, h2d, d2h, dma, split


def ensemble_members(dm, stream, n=64, seed=2024):
    """64 members of uneven size: (jx, iy) uniform in [64, 256] x [64, 192],
    kz drawn from {30, 40, 60}, +-1 K theta noise on every level (own seed),
    background u uniform in [0, 10] m/s; FP32 storage with FP64 solve."""
    rng = np.random.default_rng(seed)
    out = []
    for m in range(n):
        jx = int(rng.integers(64, 257))
        iy = int(rng.integers(64, 193))
        kz = int(rng.choice([30, 40, 60]))
        u0 = float(rng.uniform(0.0, 10.0))
        d = dm.Moloch(jx, iy, kz, mode="fp32_mixed", stream=stream)
        d.setup_idealized(pert_amp=1.0, pert_levels=kz, seed=seed + m, u0=u0, v0=1.0, device=True)
        out.append(d)
    return out


# surrogate training: pairs from plain steps of a scratch domain of the same
# workload (another seed), in `windows` windows of collect_steps steps with
# `gap` uncollected steps between them, so the training states come from
# across the run and not only from its start
SUR = {"collect_steps": 6, "windows": 3, "gap": 12, "cols_per_cycle": 1024, "iters": 4000, "lr": 1e-3,
       "batch": 256, "threshold": 4.0, "judge_every": 6, "tol": 0.3}


def train_surrogate(dm, mode, stream, jx, iy, kz, hills, cfg=SUR):
    """Collect (state, post-sound-cycle state) pairs from plain steps of a
    scratch domain and train the surrogate on the GPU."""
    t0 = time.perf_counter()
    scratch = dm.Moloch(jx, iy, kz, mode=mode, stream=stream)
    scratch.setup_idealized(hills=hills, pert_amp=0.5, pert_levels=10, seed=SEED + 7, device=True)
    nwin = cfg.get("windows", 1)
    cap = nwin * cfg["collect_steps"] * scratch.params.mo_nadv * cfg["cols_per_cycle"]
    sur = dm.Surrogate(kz, capacity=cap, batch=cfg["batch"], seed=1)
    for w in range(nwin):
        pairs = sur.collect(scratch, cfg["collect_steps"], cols_per_cycle=cfg["cols_per_cycle"], seed=3 + w)
        if w + 1 < nwin:
            scratch.run(cfg.get("gap", 0), graph=True)
    sur.prepare(0.1)
    _, v0 = sur.train(0)
    tl, vl = sur.train(cfg["iters"], lr=cfg["lr"])
    scratch.close()
    info = {"pairs": pairs, "windows": f"{nwin} x {cfg['collect_steps']} steps, {cfg.get('gap', 0)} between",
            "iters": cfg["iters"], "batch": cfg["batch"], "val_loss_untrained": v0,
            "val_loss": vl, "train_loss": tl, "seconds": time.perf_counter() - t0,
            "mlp": f"{45 * kz}->256->256->256->{5 * kz}, SiLU, BF16 operands, FP32 accumulate (tcgen05)"}
    return sur, info


def surrogate_forced_error(torch, dm, sur, stream, jx, iy, kz, hills, ref_fields, steps, tuning):
    """The surrogate committed on every cycle (no judge, no envelope check),
    from the same initial state as the FP64 reference: its error after
    `steps` steps and its time per step.  Shows what the judge protects
    against and what a committed cycle costs."""
    d = dm.Moloch(jx, iy, kz, mode="fp32_mixed", stream=stream)
    d.setup_idealized(hills=hills, pert_amp=0.5, pert_levels=10, seed=SEED, device=True)
    d.set_tuning(tuning)
    sur.attach(d, threshold=1e30, judge_every=0)
    d.run(2, graph=True)
    ms, _ = time_steps(torch, d, torch.cuda.ExternalStream(stream), steps - 2)
    out = {"steps": steps, "ms_per_step": ms / (steps - 2),
           "theta_rmse_K": rmse(d.get("t") / d.get("pai"), ref_fields["theta"]),
           "u_rmse_ms": rmse(d.get("u"), ref_fields["u"]),
           "v_rmse_ms": rmse(d.get("v"), ref_fields["v"])}
    sur.detach()
    d.close()
    return out


def run_accuracy(args, torch, dm, stream):
    """Long-run error of the FP32 paths against the FP64 GPU step (which
    matches the FP64 oracle to <= 1e-9 relative L2 after 100 steps): the
    512 x 512 x 60 workload (--workload accuracy) or the 1024 x 1024 x 60
    full-stack workload with two 1 km hills (--workload accuracy1024)
    advanced --steps steps, RMSE checkpoints every --steps/10 steps, all
    three paths with their autotuned launch shapes."""
    sptr = stream.cuda_stream
    sur, sur_train = train_surrogate(dm, "fp32_mixed", sptr, JX, IY, KZ, HILLS)
    d64, tune_64 = tuned(dm, "fp64", sptr)
    dmix, tune_mix = tuned(dm, "fp32_mixed", sptr)
    dsur = make_domain(dm, "fp32_mixed", sptr)
    dsur.set_tuning(tune_mix)
    sur.attach(dsur, threshold=SUR["threshold"], judge_every=SUR["judge_every"], tol=SUR["tol"])
    every = max(1, args.steps // 10)
    curve = []
    done = 0
    t0 = time.perf_counter()
    while done < args.steps:
        n = min(every, args.steps - done)
        for d in (d64, dmix, dsur):
            d.run(n, graph=True)
        done += n
        th64 = d64.get("t") / d64.get("pai")
        u64, v64 = d64.get("u"), d64.get("v")
        row = {"step": done}
        for name, d in (("fp32", dmix), ("fp32_surrogate", dsur)):
            row[name] = {"theta_rmse_K": rmse(d.get("t") / d.get("pai"), th64),
                         "u_rmse_ms": rmse(d.get("u"), u64), "v_rmse_ms": rmse(d.get("v"), v64),
                         "w_rmse_ms": rmse(d.get("w"), d64.get("w"))}
        curve.append(row)
    line = {"metric": "RMSE against the FP64 GPU step", "workload": f"{JX}x{IY}x{KZ}", "steps": args.steps,
            "hills": HILLS, "autotuned": {"fp64": tune_64, "fp32_mixed": tune_mix},
            "target": {"theta_rmse_K": 0.05, "u_v_rmse_ms": 0.05}, "curve": curve,
            "surrogate": {"training": sur_train, "judge": sur.stats_counts()},
            "seconds": time.perf_counter() - t0}
    print(json.dumps(line), flush=True)
    sur.close()
    for d in (d64, dmix, dsur):
        d.close()
    return 0


def persistent_tuning(choice):
    """The nearest tuning the persistent ensemble kernel carries: horizontal
    WAF tiles (1-8 levels), 1 or 2 vertical-WAF fields per thread, no FP32
    k-marching momentum, the one-thread column solve."""
    hz, km, vf = choice[0], choice[1], choice[2]
    hz = hz if hz < 16 else 4
    vf = vf if vf in (1, 2) else 1
    if km & 4 and not km & 8:
        km &= ~4
    km &= ~(32 | 512)  # the staged column solve and the two-level strips run only as their own launches
    return [hz, km, vf]


def run_ensemble(args, dist, rank, ws):
    import torch
    import dynamical_model_gb300 as dm
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    device = torch.device("cuda", local)
    stream = torch.cuda.Stream(device=device)
    # autotune on a scratch ensemble (tuning advances the state); it also
    # times one launch per kernel against the persistent kernel
    scratch = dm.Ensemble(ensemble_members(dm, stream.cuda_stream))
    choice = scratch.autotune()
    picked_persistent = scratch.persistent
    for m in scratch.members:
        m.close()
    scratch.close()
    mem = ensemble_members(dm, stream.cuda_stream)
    ens = dm.Ensemble(mem)
    gp = sum(m.jx * m.iy * m.kz for m in mem)
    total_gp = reduce_sum(dist, gp, device)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)

    def timed(persistent, tuning):
        ens.set_tuning(tuning)
        ens.set_persistent(persistent)
        ens.run(args.warmup, graph=True)
        ens.sync()
        clk = ClockSampler(local)
        barrier(dist, device)
        clk.start()
        torch.cuda.synchronize()
        k0 = ens.kernel_count
        e0.record(stream)
        ens.run(args.steps, graph=True)
        e1.record(stream)
        e1.synchronize()
        clocks = clk.stop()
        ens.sync()
        ms = reduce_max(dist, e0.elapsed_time(e1), device)
        launches = ens.kernel_count - k0
        prof = ens.profile_step()  # one more step, timed per kernel kind (outside the timed region)
        return {"ms_per_step": ms / args.steps, "value": total_gp * args.steps / (ms / 1e3),
                "gpu_launches": launches, "tuning": list(tuning), "clocks": clocks,
                "kernels_ms": {k: round(v[0], 4) for k, v in prof.items()},
                "kernels_launches": {k: v[1] for k, v in prof.items()}}

    modes = {"per_kernel": timed(0, choice)}
    for b in (2, 3, 4):  # persistent kernel built for b resident blocks per SM
        modes[f"persistent_{b}"] = timed(b, persistent_tuning(choice))
    head = modes[f"persistent_{picked_persistent}" if picked_persistent else "per_kernel"]
    finite = all(np.isfinite(m.get("ps")).all() for m in mem)
    if rank == 0:
        print(json.dumps({
            "metric": "grid-pt-steps/s, 64-member uneven ensemble on 1 GB300", "value": head["value"],
            "unit": UNIT, "n_gpus": ws, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": head["ms_per_step"], "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32 (f64 tridiagonal pivots)", "data": "synthetic",
            "config": {"workload": "64 members, jx in [64,256], iy in [64,192], kz in {30,40,60}, +-1 K noise, u0 in [0,10]",
                       "grid_points": gp, "autotuned": choice, "graph": True,
                       "launch": ("persistent: one cooperative launch per step, phases between grid barriers, "
                                  "(member, tile) items from a device-side work queue") if picked_persistent else
                                 "one batched launch per kernel over all members, one graph per step",
                       "autotuner_picked": f"persistent_{picked_persistent}" if picked_persistent else "per_kernel"},
            "modes": modes,
            "gpu_launches": head["gpu_launches"], "all_finite": bool(finite), "clocks": head["clocks"]}), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--size", default=None, help="JXxIYxKZ override (profiling a smaller case)")
    ap.add_argument("--only", default=None, choices=["mixed", "fp64"], help="time one path only (profiling)")
    ap.add_argument("--tuning", default=None,
                    help="comma-separated launch shapes for --only instead of autotuning (profiling runs under a "
                         "profiler, whose timings would mislead the autotuner), e.g. 32,24,1")
    ap.add_argument("--workload", default="single",
                    choices=["single", "ensemble", "full1024", "surrogate", "accuracy", "accuracy1024"],
                    help="single: 512x512x60 (headline); ensemble: 64 uneven members; full1024: 1024x1024x60; "
                         "surrogate: 256x256x40 surrogate case; accuracy: --steps-long error run vs FP64; "
                         "accuracy1024: the same on the 1024x1024x60 two-hill workload")
    args = ap.parse_args()
    global JX, IY, KZ, HILLS
    if args.size:
        JX, IY, KZ = (int(x) for x in args.size.lower().split("x"))
        HILLS = ((500.0, (JX + 1) / 2.0, (IY + 1) / 2.0, 20.0 * JX / 512.0),)
    if args.warmup < 3:
        args.warmup = 3
    dist, rank, ws = dist_setup()
    if args.impl == "reference":
        return run_reference(args, dist, rank, ws)

    import torch
    import dynamical_model_gb300 as dm
    if args.workload == "ensemble":
        return run_ensemble(args, dist, rank, ws)
    if args.workload == "surrogate":
        # learned acoustic-cycle surrogate case: 256 x 256 x 40, 20k training pairs
        JX, IY, KZ = 256, 256, 40
        HILLS = ((500.0, (JX + 1) / 2.0, (IY + 1) / 2.0, 10.0),)
        SUR.update(collect_steps=7, windows=1, cols_per_cycle=1024, iters=4000)
    if args.workload in ("full1024", "accuracy1024"):
        JX, IY = 1024, 1024
        HILLS = ((1000.0, (JX + 1) / 3.0, (IY + 1) / 2.0, 20.0), (1000.0, 2.0 * (JX + 1) / 3.0, (IY + 1) / 2.0, 20.0))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    device = torch.device("cuda", local)
    stream = torch.cuda.Stream(device=device)
    sptr = stream.cuda_stream

    if args.workload in ("accuracy", "accuracy1024"):
        return run_accuracy(args, torch, dm, stream) if rank == 0 else 0
    # ---- headline path: FP32 storage + FP64 solve --------------------------
    if args.only:
        mode = "fp32_mixed" if args.only == "mixed" else "fp64"
        if args.tuning:
            d = make_domain(dm, mode, sptr)
            d.set_tuning([int(x) for x in args.tuning.split(",")])
        else:
            d, _ = tuned(dm, mode, sptr)
        d.run(args.warmup, graph=True)
        ms, launches = time_steps(torch, d, stream, args.steps)
        if rank == 0:
            print(json.dumps({"only": args.only, "size": [JX, IY, KZ], "ms_per_step": ms / args.steps,
                              "value": JX * IY * KZ * args.steps / (ms / 1e3), "gpu_launches": launches}))
        d.close()
        return 0
    return run_single(args, dist, rank, ws, torch, dm, stream, local, device)


def run_single(args, dist, rank, ws, torch, dm, stream, local, device):
    sptr = stream.cuda_stream
    gp = JX * IY * KZ
    # ---- the surrogate: trained on the GPU outside the timed region --------
    sur, sur_train = train_surrogate(dm, "fp32_mixed", sptr, JX, IY, KZ, HILLS)
    dsur, tune_mix = tuned(dm, "fp32_mixed", sptr)
    sur.attach(dsur, threshold=SUR["threshold"], judge_every=SUR["judge_every"], tol=SUR["tol"])
    dmix = make_domain(dm, "fp32_mixed", sptr)
    dmix.set_tuning(tune_mix)
    d64, tune_64 = tuned(dm, "fp64", sptr)
    for d in (dsur, dmix, d64):
        d.run(args.warmup, graph=True)
        d.sync()

    # ---- timed: FP32 + surrogate (headline), plain FP32, plain FP64 ---------
    clk = ClockSampler(local)
    barrier(dist, device)
    clk.start()
    ms_sur, launches_sur = time_steps(torch, dsur, stream, args.steps)
    barrier(dist, device)
    clocks = clk.stop()
    ms_sur = reduce_max(dist, ms_sur, device)
    ms_mix, launches_mix = time_steps(torch, dmix, stream, args.steps)
    ms_mix = reduce_max(dist, ms_mix, device)
    ms_64, launches_64 = time_steps(torch, d64, stream, args.steps)
    ms_64 = reduce_max(dist, ms_64, device)
    n_dom = reduce_sum(dist, 1.0, device)
    value = n_dom * gp * args.steps / (ms_sur / 1e3)
    value_mix = n_dom * gp * args.steps / (ms_mix / 1e3)
    value64 = n_dom * gp * args.steps / (ms_64 / 1e3)

    # ---- errors against the FP64 GPU step after warmup + steps steps --------
    ref = {"theta": d64.get("t") / d64.get("pai"), "u": d64.get("u"), "v": d64.get("v"), "w": d64.get("w"),
           "ps": d64.get("ps")}

    def errors(d):
        return {"steps": args.warmup + args.steps,
                "theta_rmse_K": rmse(d.get("t") / d.get("pai"), ref["theta"]),
                "u_rmse_ms": rmse(d.get("u"), ref["u"]), "v_rmse_ms": rmse(d.get("v"), ref["v"]),
                "w_rmse_ms": rmse(d.get("w"), ref["w"]), "ps_rmse_Pa": rmse(d.get("ps"), ref["ps"])}

    err_sur = errors(dsur)
    err_mix = errors(dmix)
    judge = sur.stats_counts()
    inference_ms = sur.profile(dsur)
    forced = surrogate_forced_error(torch, dm, sur, sptr, JX, IY, KZ, HILLS, ref, args.warmup + args.steps, tune_mix)
    sur.attach(dsur, threshold=SUR["threshold"], judge_every=SUR["judge_every"], tol=SUR["tol"])

    # ---- per-kernel CUDA-event profile of one step (roofline) ---------------
    prof = dmix.profile_step()
    prof64 = d64.profile_step()
    peak, peak_kind = peaks()
    top = max(prof.items(), key=lambda kv: kv[1][0])
    tkind, (tms, tcount) = top
    words = ALG_WORDS.get(tkind, 0)
    esz = 4
    alg_bytes = words * esz * gp  # per launch
    avg_ms = tms / max(tcount, 1)
    achieved = alg_bytes / (avg_ms / 1e3) / 1e9
    roofline = {"bound": "hbm", "kernel": tkind, "achieved": achieved, "peak": peak,
                "unit": "GB/s", "frac": achieved / peak, "peak_kind": peak_kind,
                "alg_bytes_per_launch": alg_bytes, "avg_launch_ms": avg_ms,
                "traffic": (NCU_TRAFFIC[tkind][0] * gp / NCU_TRAFFIC[tkind][1]) if tkind in NCU_TRAFFIC else None,
                "traffic_note": "ncu dram bytes of one launch (512x512x60; the one-thread solve 384x384x60), scaled "
                                "by grid points (part of the writes is still in L2 when it ends)",
                # second roof of the top kernel: its FP64 pivot recurrence (4
                # FP64 operations per level) keeps the FP64 pipe this busy in
                # the ncu capture of the same kernel
                "fp64_pipe": NCU_FP64_PIPE.get(tkind),
                "step_alg_GBps": B_ALG_WORDS * esz * value_mix / n_dom / 1e9}
    kernels = {k: {"ms": round(v[0], 4), "launches": v[1],
                   "GBps_alg": (ALG_WORDS.get(k, 0) * esz * gp * v[1] / (v[0] / 1e3) / 1e9) if v[0] > 0 else None}
               for k, v in sorted(prof.items(), key=lambda kv: -kv[1][0])}
    kernels64 = {k: {"ms": round(v[0], 4), "launches": v[1]} for k, v in sorted(prof64.items(), key=lambda kv: -kv[1][0])}
    top64 = max(prof64.items(), key=lambda kv: kv[1][0])[0]
    roofline_fp64 = {"bound": "fp64 pipe", "kernel": top64, "unit": "fraction of the FP64 pipe",
                     "frac": NCU_FP64_STEP.get(top64, {}).get("pipe_fp64_active_pct", float("nan")) / 100.0,
                     "kernels": NCU_FP64_STEP, "capture": "ncu, one launch each, 256x256x60 FP64",
                     "share_of_step": sum(v[0] for k, v in prof64.items() if k in NCU_FP64_STEP) /
                     sum(v[0] for v in prof64.values())}

    # ---- end to end through the C ABI with host arrays ----------------------
    e2e = None
    if not args.no_e2e:
        n_e2e = max(2, args.steps)
        runs, h2d, d2h, dma, split = e2e_steps(torch, dm, dsur, stream, n_e2e, args.warmup)
        ms_e2e = reduce_max(dist, sorted(runs)[len(runs) // 2], device)
        e2e = {"value": n_dom * gp * n_e2e / (ms_e2e / 1e3), "unit": UNIT, "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": d2h, "steps": n_e2e,
               "repeats": "median of %d timed loops of %d steps" % (len(runs), n_e2e),
               "ms_per_step_runs": [round(r / n_e2e, 3) for r in runs],  # in the order they ran
               "loop_device_and_wall_ms": split,
               "h2d_dma_GBps": round(dma, 1),
               "path": "moloch_gpu_upload(u,v,w,pai,t,qx) from registered (pinned) FP64 host arrays + "
                       "moloch_gpu_step + moloch_gpu_output_start/finish(t,ps) into registered arrays, "
                       "FP32 + surrogate handle"}

    cpu = None
    if rank == 0 and not args.no_cpu_baseline:
        v, dt, threads = cpu_sample(2, kz=KZ)
        cpu = {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
               "sample": f"2 steps of a 256x256x{KZ} sample of the workload, {dt:.1f} s, OpenMP C restatement "
                         f"of nompi/mod_moloch.F90 (no Fortran compiler: reference build unavailable)"}

    if rank == 0:
        n_cyc = judge["cycles"]
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_sur / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32 (f64 tridiagonal solve; bf16/f32 surrogate)",
            "data": "synthetic",
            "config": {"workload": f"{JX}x{IY}x{KZ} idealized state, hill {HILLS[0][0]:.0f} m r={HILLS[0][3]:.0f} gp, "
                                   f"seeded +-0.5 K theta noise",
                       "jx": JX, "iy": IY, "kz": KZ,
                       "path": "fp32_mixed + acoustic-cycle surrogate under the plain-loop judge",
                       "graph": True, "parallelism": f"replicas x{ws}",
                       "autotuned": {"fp32_mixed": tune_mix, "fp64": tune_64},
                       "l2": "inputs larger than L2 (state > 1 GB per domain)"},
            "speedup_vs_fp64": value / value64,
            "error_vs_fp64": err_sur,
            "fp32_plain": {"value": value_mix, "ms_per_step": ms_mix / args.steps, "gpu_launches": launches_mix,
                           "speedup_vs_fp64": value_mix / value64, "error_vs_fp64": err_mix},
            "fp64_plain": {"value": value64, "ms_per_step": ms_64 / args.steps, "dtype": "f64",
                           "gpu_launches": launches_64},
            "surrogate": {"training": sur_train, "attach": {k: SUR[k] for k in ("threshold", "judge_every", "tol")},
                          "judge": judge,
                          "committed_cycles": n_cyc - judge["plain"],
                          "inference_ms_per_cycle": inference_ms,
                          "forced_on_error_vs_fp64": forced},
            "roofline": roofline,
            "roofline_fp64_step": roofline_fp64,
            "kernels": kernels,
            "kernels_fp64": kernels64,
            "cpu_baseline": cpu,
            "e2e": e2e,
            "gpu_launches": launches_sur,
            "clocks": clocks,
        }
        print(json.dumps(line), flush=True)
    sur.close()
    for d in (dsur, dmix, d64):
        d.close()
    if dist is not None:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
