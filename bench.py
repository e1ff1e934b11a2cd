#!/usr/bin/env python
"""Benchmark of the fused GB300 fit: sources/s of fit_parametric (PSO model
selection over the eight flux models with three restarts, L-BFGS polish, BIC
selection, profile t0 search, SVI uncertainty, profile refinements,
magnitude chi2 and MultiBazin) on 10,000 synthetic sources x 3 bands of
uneven length (counts round(lognormal(ln 40, 0.9)) clipped to [5, 500]).

One JSON line on rank 0:
  value     sources/s with the inputs resident in HBM (the device entry point
            lcf_fit_parametric_device), CUDA events on the library's stream,
            L2 flushed (256 MB write) between timed steps;
  e2e       the same metric through lcf_fit_parametric_batch with host
            buffers (pinned staging, H2D copies, pipeline, D2H of the results
            all inside the timed region);
  roofline  the dominant kernel, the model-selection swarm (pso_kernel<7>),
            against the measured SFU (MUFU) and FP32 pipe peaks (the kernel
            is bound by those pipes, not by HBM or the tensor cores); the
            L-BFGS polish beside it with its pipe shares from ncu;
  cpu_baseline  the FP64 C++ restatement of the reference's CPU path
            (oracle/, "port") on a bounded sample with all host threads, a
            1-thread sample, and a calibration on the reference's published
            CPU case (100 sources x 3 bands x 30 points, Laplace);
  basic, precision  side legs on the basic (100 x 3 x 30, Laplace) and
            precision (1,000 x 3 x 2,000, Laplace) workloads;
  plain_gpu the plain FP64 GPU form (lcf_fit_plain_device: one thread per
            particle, FP64, global-memory observations, one launch per model
            per stage, no graph) on the same 10,000 sources, and the fused
            pipeline's ratio to it — over the whole fused pipeline and over
            the stages the plain form runs (PSO, L-BFGS, selection, SVI);
  full_scale  sources/s on 100,000 sources (counts clipped at 1,000, 15 M
            observations) in one call, device-resident, one timed step.

``--impl reference`` times that CPU path alone (rank 0) on the same workload.
Under torchrun the ranks partition one workload of N x 10,000 sources by
estimated work (lightcurve_fitting_gb300.shard, weak scaling, no collective
on the data path) and value = all sources / the slowest rank's time.
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

METRIC = "sources/s, fit_parametric PSO+SVI, 10k uneven sources: fused vs plain GPU"
WORKLOAD = ("uneven-10000x3: counts round(lognormal(ln 40, 0.9)) clipped [5, 500] per band, t in [0, 300] d "
            "with 20% of nights dropped, generators Bazin/Villar/TDE/Arnett/Magnetar, sigma = 0.05|F| + 5; "
            "fit_all_models=true, SVI uncertainty, MultiBazin on the most populated band")

# Algorithmic SFU (MUFU) operations per particle x observation evaluation of
# each task kind, counted from the FP32 model forms in csrc/models_f32.cuh:
# exp/log/log1p/expm1 = 1 each, a reciprocal or division = 1, rsqrt = 1, plus
# the Gaussian term's rsqrt and log (2).  MetzgerKN also spends ~14 per Euler
# step of its 200-step ODE (counted through ode_steps), MultiBazin K spends
# 3 per component.
MUFU_PER_EVAL = {0: 5, 1: 7, 2: 8, 3: 7, 4: 6, 5: 8, 6: 8, 7: 2, 8: 5, 9: 8, 10: 11, 11: 14}
MUFU_PER_ODE_STEP = 14
# FP32 pipe operations per evaluation (adds, multiplies, FMAs, compares,
# including the Kahan update of 4 adds); MetzgerKN ~60 per ODE step.
FP32_PER_EVAL = {0: 24, 1: 34, 2: 30, 3: 30, 4: 26, 5: 30, 6: 32, 7: 16, 8: 24, 9: 34, 10: 44, 11: 54}
FP32_PER_ODE_STEP = 60
# DRAM traffic (dram__bytes_read.sum + dram__bytes_write.sum) per unit of
# work of the two reported kernels, from ncu captures: the model-selection
# swarm of 1,000 uneven sources moved 86.5 MB for 6.372e9 particle-observation
# evaluations, the polish of 5,000 moved 261.7 MB for 7.538e8 observation-term
# evaluations (its bands, its swarm results, its fits and a few spills).  A launch's traffic is scaled from these by its own
# units of work.
DRAM_BYTES_PER_PSO_OBS_EVAL = 86.54e6 / 6.372e9
DRAM_BYTES_PER_LB_OBS_EVAL = 261.7e6 / 7.538e8
# The polish's pipe shares in that capture (% of peak sustained): FMA 18.9,
# FP64 46.7, issue slots 27.5, instruction-cache hit rate 85.4 %, with 0.83 "no
# instruction" stall cycles per issued instruction and 6.1 at the round's barrier.
LBFGS_NCU = {"fma_pipe_pct": 18.9, "fp64_pipe_pct": 46.7, "issue_active_pct": 27.5, "icache_hit_pct": 85.4,
             "no_instruction_stall_per_issue": 0.83}
# The reference's published CPU figure for its benchmark case (100 sources x
# 3 bands x 30 points, fit_parametric(.., false, Laplace), one thread, Skylake
# Xeon): 113-116 sources/s (benchmarks/parametric_sources.csv:2-8).
PUBLISHED_CPU_SRC_S = (113.0, 116.0)


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="fused", choices=["fused", "reference"])
    ap.add_argument("--sources", type=int, default=10000)
    ap.add_argument("--cpu-sample", type=int, default=512, help="sources in the all-threads CPU-baseline sample")
    ap.add_argument("--cpu-sample-1t", type=int, default=12, help="sources in the 1-thread CPU-baseline sample")
    ap.add_argument("--basic-steps", type=int, default=2, help="timed steps of the basic-workload leg (0: skip)")
    ap.add_argument("--precision-steps", type=int, default=1,
                    help="timed steps of the precision-workload leg (0: skip)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true", help="skip the host entry-point measurement (profiling runs)")
    ap.add_argument("--plain-steps", type=int, default=1, help="timed steps of the plain FP64 GPU form (0: skip)")
    ap.add_argument("--scale-sources", type=int, default=100_000,
                    help="sources of the full-scale leg (counts clipped at 1000; 0: skip)")
    ap.add_argument("--finalize-sources", type=int, default=10000,
                    help="sources whose (band, model) pairs the finalisation leg runs (0: skip)")
    ap.add_argument("--joint-sources", type=int, default=2000,
                    help="sources of the fit_parametric multi-band (joint Villar) measurement (0: skip)")
    return ap.parse_args()


def dist_setup():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import torch.distributed as dist
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        import torch
        backend = "nccl" if torch.cuda.is_available() else "gloo"
        dist.init_process_group(backend=backend)
    return ws, rank, local


def rank_workload(n_sources: int, rank: int, ws: int = 1):
    """This rank's shard of one workload of ws x n_sources uneven sources
    (seed 2): the partition by estimated work of lightcurve_fitting_gb300.
    shard, fitted with no exchange between ranks (weak scaling)."""
    from lightcurve_fitting_gb300 import shard, synth
    full = synth.config_uneven(n_sources * ws, seed=2)
    if ws == 1:
        return full
    return full.subset(shard.partition(full, ws)[rank])


def job_value(n_sources_per_rank: int, ws: int, max_ms: float) -> float:
    """Whole-job sources/s: all ranks' sources over the slowest rank's time."""
    return ws * n_sources_per_rank / (max_ms * 1e-3)


def dist_max(x: float, ws: int, device) -> float:
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def dist_barrier(ws: int):
    if ws > 1:
        import torch.distributed as dist
        dist.barrier()


class ClockSampler:
    """nvidia-smi SM clocks and throttle reasons during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        os.unlink(self.path)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def _oracle_rate(batch, threads: int, **kw):
    """Sources/s of the oracle (FP64 port of the reference CPU path) fitting
    `batch` on `threads` host threads (0: all), OpenMP over sources with
    dynamic scheduling."""
    from lightcurve_fitting_gb300 import abi
    from oracle import oracle as O
    O.build()
    opts = dict(fit_all_models=True, method=abi.METHOD_SVI, run_multi_bazin=True)
    opts.update(kw)
    t = time.perf_counter()
    O.fit_batch(batch, n_threads=threads, **opts)
    dt = time.perf_counter() - t
    return batch.n_sources / dt, dt


def cpu_baseline(batch, args):
    """The reference's CPU path (the oracle port) on this workload: a sample of
    `cpu_sample` sources on all host threads (the reported value), a sample
    of `cpu_sample_1t` sources on one thread, and a calibration on the
    reference's own published CPU case."""
    from lightcurve_fitting_gb300 import abi, synth
    from oracle import oracle as O
    O.build()
    cores = O.max_threads()
    n = min(args.cpu_sample, batch.n_sources)
    v, dt = _oracle_rate(batch.subset(np.arange(n)), 0)
    n1 = min(args.cpu_sample_1t, batch.n_sources)
    v1, dt1 = _oracle_rate(batch.subset(np.arange(n1)), 1)
    # the published case: 100 x 3 x 30, fit_parametric(.., false, Laplace),
    # one thread.  The current reference routes three bands with
    # fit_all_models = false to its joint multi-band fit; per-band
    # fit_parametric_model with the Bazin gate is the published case's
    # per-band path.  Both are timed (the joint fit on a smaller sample).
    basic = synth.config_basic(100, seed=1)
    vg, _ = _oracle_rate(basic, 1, fit_all_models=False, method=abi.METHOD_LAPLACE)
    vj, _ = _oracle_rate(basic.subset(np.arange(4)), 1, fit_all_models=False, method=abi.METHOD_LAPLACE,
                         joint_multiband=True)
    return {
        "value": v, "unit": "sources/s", "cores": cores, "kind": "port",
        "sample": f"first {n} sources of the workload, all {cores} host threads, OpenMP over sources "
                  f"({dt:.1f} s wall); FP64 C++ restatement of the reference CPU path (PSO + SVI, "
                  f"fit_all_models, MultiBazin)",
        "single_thread": {"value": v1, "unit": "sources/s", "cores": 1,
                          "sample": f"first {n1} sources of the workload ({dt1:.1f} s wall)"},
        "calibration": {
            "case": "100 sources x 3 bands x 30 points, fit_parametric(.., false, Laplace), one thread",
            "published_reference_src_s": list(PUBLISHED_CPU_SRC_S),
            "published_host": "Skylake Xeon, an earlier version of the reference crate",
            "port_per_band_gated_src_s": vg,
            "port_joint_multiband_src_s": vj,
            "note": "the current reference routes this case to its joint multi-band fit (port: "
                    f"{vj:.2f} src/s), so the published figure predates that routing; the per-band path "
                    "with 3 restarts and MultiBazin runs at the port figure above",
        },
    }


def run_reference(args, ws, rank):
    """The reference's CPU path (the oracle port, all host threads) on the
    workload: each step fits a bounded sample of its sources (a window that
    moves by step)."""
    if rank != 0:
        return
    from lightcurve_fitting_gb300 import synth
    from oracle import oracle as O
    O.build()
    batch = synth.config_uneven(args.sources, seed=2)
    n = min(256, batch.n_sources)
    dts = []
    for i in range(args.warmup + args.steps):
        start = (i * n) % max(batch.n_sources - n, 1)
        _, dt = _oracle_rate(batch.subset(np.arange(start, start + n)), 0)
        if i >= args.warmup:
            dts.append(dt)
    value = args.steps * n / sum(dts)
    cores = O.max_threads()
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "sources/s", "n_gpus": 0,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * sum(dts) / len(dts),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": WORKLOAD, "sample_sources_per_step": n},
        "cpu_baseline": {"value": value, "unit": "sources/s", "cores": cores, "kind": "port",
                         "sample": f"{n} sources of the workload per step (a window moving by step), all "
                                   f"{cores} host threads, OpenMP over sources (dynamic)"},
        "e2e": {"value": value, "unit": "sources/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_fused(args, ws, rank, local):
    import torch
    from lightcurve_fitting_gb300 import abi, build, synth
    build.build()
    from lightcurve_fitting_gb300.lib import Context
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    batch = rank_workload(args.sources, rank, ws)
    ctx = Context(local)
    stream = torch.cuda.ExternalStream(ctx.stream, device=dev)
    peaks = ctx.probe_peaks()
    peaks64 = ctx.probe_fp64()
    peaks_ff = ctx.probe_ff()
    # device-resident inputs
    d = {
        "times": torch.from_numpy(batch.times).to(dev),
        "flux": torch.from_numpy(batch.flux).to(dev),
        "flux_err": torch.from_numpy(batch.flux_err).to(dev),
        "band_obs_offsets": torch.from_numpy(batch.band_obs_offsets).to(dev),
        "source_band_offsets": torch.from_numpy(batch.source_band_offsets).to(dev),
    }
    ptrs = {k: v.data_ptr() for k, v in d.items()}
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    torch.cuda.synchronize()

    def fit_dev():
        ctx.fit_device(ptrs, batch.n_sources, batch.n_bands, fit_all_models=True, method=abi.METHOD_SVI)

    for _ in range(args.warmup):
        fit_dev()
    torch.cuda.synchronize()
    clocks = ClockSampler(local)
    dist_barrier(ws)
    clocks.start()
    times, stage = [], []
    for _ in range(args.steps):
        flush.fill_(1.0)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        fit_dev()
        e1.record(stream)
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
        stage.append(ctx.stats())
    torch.cuda.synchronize()
    ck = clocks.stop()
    dist_barrier(ws)
    ms = float(np.mean(times))
    ms_max = dist_max(ms, ws, dev)
    value = job_value(args.sources, ws, ms_max)
    # end-to-end through the host entry point
    e2e_t = []
    if not args.no_e2e:
        ctx.fit_batch(batch, fit_all_models=True, method=abi.METHOD_SVI)
    for _ in range(0 if args.no_e2e else args.steps):
        flush.fill_(1.0)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        res = ctx.fit_batch(batch, fit_all_models=True, method=abi.METHOD_SVI)
        e2e_t.append(time.perf_counter() - t0)
    st_e2e = ctx.stats()
    if e2e_t:
        e2e_s = dist_max(float(np.mean(e2e_t)), ws, dev)
        e2e = {"value": ws * args.sources / e2e_s, "unit": "sources/s",
               "h2d_bytes_per_step": int(st_e2e["h2d_bytes"]), "d2h_bytes_per_step": int(st_e2e["d2h_bytes"])}
    else:
        e2e = None
    # the launch autotuner explored its candidates during the warm-up fits of
    # this workload's shape bucket; the other legs pin the candidate it chose
    tune_table = ctx.autotune_table()
    tuned = ctx.last_launch()
    plain = None
    if args.plain_steps > 0:
        plain = run_plain(args, batch, ptrs, dev, flush, stage, ws)
    joint = run_joint(args, batch, dev, flush, ws, tuned["candidate"]) if args.joint_sources > 0 else None
    scale = run_scale(args, dev, flush, ws, rank, tuned["candidate"]) if args.scale_sources > 0 else None
    final = run_finalize(args, batch, res, flush, dev, ws, rank) if args.finalize_sources > 0 and e2e_t else None
    basic = run_side(args, "basic", dev, flush, ws, rank) if args.basic_steps > 0 else None
    basic_joint = run_side(args, "basic_joint", dev, flush, ws, rank) if args.basic_steps > 0 else None
    precision = run_side(args, "precision", dev, flush, ws, rank) if args.precision_steps > 0 else None
    if rank != 0:
        ctx.close()
        return
    # roofline of the model-selection PSO launch
    s0 = stage[-1]
    ev = s0["pso0_evals_by_kind"]
    npart = s0["pso0_particles_by_kind"]
    mufu = sum(ev[k] * MUFU_PER_EVAL[k] for k in range(12)) + npart[7] * 200 * MUFU_PER_ODE_STEP
    fp32 = sum(ev[k] * FP32_PER_EVAL[k] for k in range(12)) + npart[7] * 200 * FP32_PER_ODE_STEP
    pso_ms = float(np.mean([s["ms_pso"] for s in stage]))
    mufu_rate = mufu / (pso_ms * 1e-3) * 1e-9          # Gop/s
    fp32_rate = 2.0 * fp32 / (pso_ms * 1e-3) * 1e-12   # TFLOP/s counting an op as 2 for FMA parity
    frac_mufu = mufu_rate / peaks["mufu_gops"] if peaks["mufu_gops"] else None
    frac_fp32 = fp32_rate / peaks["fp32_tflops"] if peaks["fp32_tflops"] else None
    bound_sfu = (frac_mufu or 0) >= (frac_fp32 or 0)
    roofline_pso = {
        "bound": "sfu" if bound_sfu else "fp32",
        "achieved": mufu_rate if bound_sfu else fp32_rate,
        "peak": peaks["mufu_gops"] if bound_sfu else peaks["fp32_tflops"],
        "unit": "Gop/s" if bound_sfu else "TFLOP/s",
        "frac": frac_mufu if bound_sfu else frac_fp32,
        "traffic": float(sum(ev)) * DRAM_BYTES_PER_PSO_OBS_EVAL,
        "traffic_source": "ncu DRAM bytes per particle-observation evaluation of the 1,000-source launch, "
                          "scaled by this launch's evaluations",
        "kernel": "pso_kernel<7> (model-selection swarm launch)",
        "peak_source": "measured live by lcf_probe_peaks (dependent ex2 / FMA chains over a full grid)",
        "other_pipe": ({"bound": "fp32", "achieved": fp32_rate, "peak": peaks["fp32_tflops"], "unit": "TFLOP/s",
                        "frac": frac_fp32} if bound_sfu else
                       {"bound": "sfu", "achieved": mufu_rate, "peak": peaks["mufu_gops"], "unit": "Gop/s",
                        "frac": frac_mufu}),
        "launch_ms": pso_ms,
        "particle_obs_evals": float(sum(ev)),
    }
    # the L-BFGS polish beside it: its observation-term evaluations per second
    # of the launch, its pipe shares from ncu (the FP64 pipe half busy, the
    # rest the wait for the block's slowest warp), and
    # the rate its own observation terms reach streamed at full occupancy (the
    # double-float term for the evaluations it ran, the FP64 term for the range
    # fallbacks, weighted by this launch's per-model evaluations)
    lb_ev = s0["lbfgs_obs_evals_by_model"]
    lb_fb = s0["lbfgs_fp64_obs_evals_by_model"]
    lb_ms = float(np.mean([s["ms_lbfgs"] for s in stage]))
    pk64, pkff = peaks64["obs_evals_per_s"], peaks_ff["obs_evals_per_s"]
    ideal_s = sum((lb_ev[m] - lb_fb[m]) / pkff[m] + lb_fb[m] / pk64[m] for m in range(7) if pk64[m] > 0 and pkff[m] > 0)
    lb_rate = sum(lb_ev[:7]) / (lb_ms * 1e-3)
    lb_term_peak = sum(lb_ev[:7]) / ideal_s if ideal_s > 0 else None
    polish = {
        "kernel": "lbfgs_kernel (L-BFGS polish)",
        "launch_ms": lb_ms,
        "lbfgs_obs_evals": float(sum(lb_ev[:7])),
        "achieved": lb_rate,
        "unit": "observation-term evaluations/s (value + gradient + cost, double-float; FP64 where out of range)",
        "ncu_pipes_pct_of_peak": LBFGS_NCU,
        "own_term_rate_at_full_occupancy": lb_term_peak,
        "frac_of_own_term_rate": lb_rate / lb_term_peak if lb_term_peak else None,
        "traffic": float(sum(lb_ev[:7])) * DRAM_BYTES_PER_LB_OBS_EVAL,
        "traffic_source": "ncu DRAM bytes per observation-term evaluation of the 1,000-source launch, scaled by "
                          "this launch's evaluations",
        "ff_term_rate_by_model": pkff,
        "fp64_term_rate_by_model": pk64[:7],
        "ff_vs_fp64_worst_rel_by_model": peaks_ff["worst_rel"],
        "fp64_fallback_share": float(sum(lb_fb[:7]) / max(sum(lb_ev[:7]), 1.0)),
        "fp64_dfma_tflops": peaks64["fp64_tflops"],
    }
    roofline = dict(roofline_pso)
    roofline["lbfgs_kernel"] = polish
    cpu = None
    if not args.no_cpu_baseline:
        cpu = cpu_baseline(batch, args)
    line = {
        "metric": METRIC, "value": value, "unit": "sources/s", "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_max, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": WORKLOAD, "n_sources_per_gpu": args.sources, "n_sources_rank0": batch.n_sources,
                   "n_bands_rank0": batch.n_bands, "n_obs_rank0": batch.n_obs,
                   "l2": "flushed between timed steps (256 MB write)",
                   "parallelism": f"one workload of {ws} x {args.sources} sources partitioned by estimated work "
                                  f"over {ws} rank(s)" if ws > 1 else "one GPU"},
        "stage_ms": {k: float(np.mean([s[k] for s in stage])) for k in
                     ["ms_total", "ms_pso", "ms_lbfgs", "ms_t0_search", "ms_uncertainty", "ms_refine",
                      "ms_multi_bazin"]},
        "e2e": e2e,
        "roofline": roofline,
        "cpu_baseline": cpu,
        "plain_gpu": plain,
        "fit_parametric_multiband": joint,
        "full_scale": scale,
        "finalize_all_models": final,
        "basic": basic,
        "basic_fit_parametric": basic_joint,
        "precision": precision,
        "autotune": {"candidates_block_staging_blocks_per_sm": ctx.autotune_candidates().tolist(),
                     "chosen": tuned,
                     "table_bucket_best_next_ms": tune_table.tolist(),
                     "note": "explored during the warm-up fits; bit-identical results under every candidate"},
        "clocks": ck,
        "gpu_launches": int(s0["kernel_launches"]) * args.steps,
        "peaks": {**peaks, "fp64_tflops": peaks64["fp64_tflops"]},
    }
    print(json.dumps(line), flush=True)
    ctx.close()


def run_plain(args, batch, ptrs, dev, flush, fused_stats, ws):
    """The plain FP64 GPU form on the same device-resident workload."""
    import torch
    from lightcurve_fitting_gb300.lib import Context
    pctx = Context(dev.index)
    pstream = torch.cuda.ExternalStream(pctx.stream, device=dev)
    # warm-up: one plain fit of the first 100 sources (module load)
    sub = batch.subset(np.arange(min(100, batch.n_sources)))
    keep = {k: torch.from_numpy(getattr(sub, k)).to(dev) for k in
            ["times", "flux", "flux_err", "band_obs_offsets", "source_band_offsets"]}
    pctx.fit_plain_device({k: v.data_ptr() for k, v in keep.items()}, sub.n_sources, sub.n_bands)
    torch.cuda.synchronize()
    times, st = [], None
    for _ in range(args.plain_steps):
        flush.fill_(1.0)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(pstream)
        pctx.fit_plain_device(ptrs, batch.n_sources, batch.n_bands, fit_all_models=True)
        e1.record(pstream)
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
        st = pctx.stats()
    pctx.close()
    ms = dist_max(float(np.mean(times)), ws, dev)
    value = ws * batch.n_sources / (ms * 1e-3)
    f_ms = lambda k: float(np.mean([s[k] for s in fused_stats]))
    fused_total = dist_max(f_ms("ms_total"), ws, dev)
    # the fused stages the plain form also runs (model-selection swarms, polish
    # + selection, SVI); MultiBazin runs on a branch beside the polish, so the
    # polish time includes its contention
    fused_same = dist_max(f_ms("ms_pso") + f_ms("ms_lbfgs") + f_ms("ms_uncertainty"), ws, dev)
    return {
        "value": value, "unit": "sources/s", "ms_per_step": ms, "steps": args.plain_steps,
        "warmup": "one plain fit of the first 100 sources",
        "stages": "PSO (8 models x 3 restarts, synchronous global best), L-BFGS polish, BIC selection, SVI; "
                  "no profile t0 search, refinements, magnitude chi2 or MultiBazin",
        "stage_ms": {"ms_pso": st["ms_pso"], "ms_lbfgs_select": st["ms_lbfgs"], "ms_svi": st["ms_uncertainty"]},
        "kernel_launches": int(st["kernel_launches"]),
        "fused_over_plain": (ws * batch.n_sources / (fused_total * 1e-3)) / value,
        "fused_over_plain_same_stages": (ws * batch.n_sources / (fused_same * 1e-3)) / value,
    }


def run_joint(args, batch, dev, flush, ws, candidate):
    """fit_parametric with fit_all_models = false (the reference's default):
    every source of this workload has 3 non-empty bands, so all take the
    joint multi-band Villar branch (SVI, MultiBazin), on the first
    `joint_sources` sources, device-resident, one warm-up and two timed steps."""
    import torch
    from lightcurve_fitting_gb300 import abi
    from lightcurve_fitting_gb300.lib import Context
    sub = batch.subset(np.arange(min(args.joint_sources, batch.n_sources)))
    keep = {k: torch.from_numpy(getattr(sub, k)).to(dev) for k in
            ["times", "flux", "flux_err", "band_obs_offsets", "source_band_offsets"]}
    ptrs = {k: v.data_ptr() for k, v in keep.items()}
    jctx = Context(dev.index)
    jctx.set_autotune(1, candidate)
    jstream = torch.cuda.ExternalStream(jctx.stream, device=dev)

    def fit():
        jctx.fit_device(ptrs, sub.n_sources, sub.n_bands, fit_all_models=False, method=abi.METHOD_SVI,
                        joint_multiband=True)

    fit()
    torch.cuda.synchronize()
    times, st = [], None
    for _ in range(2):
        flush.fill_(1.0)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(jstream)
        fit()
        e1.record(jstream)
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
        st = jctx.stats()
    jctx.close()
    ms = dist_max(float(np.mean(times)), ws, dev)
    return {"value": job_value(sub.n_sources, ws, ms), "unit": "sources/s", "ms_per_step": ms,
            "sources_per_gpu": sub.n_sources, "steps": 2, "warmup": 1,
            "config": "fit_parametric(fit_all_models=false, SVI): joint multi-band Villar swarm (200 particles, "
                      "1500 iterations, stall 60, 3 seeds), per-band SVI, refinements, MultiBazin",
            "stage_ms": {"ms_joint": st["ms_joint"], "ms_uncertainty": st["ms_uncertainty"],
                         "ms_refine": st["ms_refine"], "ms_multi_bazin": st["ms_multi_bazin"]}}


def pair_batch(batch, res, n_sources: int):
    """Every fitted (band, model) pair of the first `n_sources` sources as its
    own one-band source (the band's observations repeated per model), with
    that model's polished parameters and cost from a fit_all_models run."""
    from lightcurve_fitting_gb300 import synth
    nb = int(batch.source_band_offsets[min(n_sources, batch.n_sources)])
    have = np.isfinite(res.per_model_params[:nb, :, 0]) & (res.model[:nb, None] >= 0)
    b_idx, m_idx = np.nonzero(have)
    off = batch.band_obs_offsets
    cnt = (off[b_idx + 1] - off[b_idx]).astype(np.int64)
    new_off = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    idx = np.repeat(off[b_idx] - new_off[:-1], cnt) + np.arange(int(new_off[-1]), dtype=np.int64)
    pairs = synth.PhotometryBatch(batch.times[idx], batch.flux[idx], batch.flux_err[idx], new_off,
                                  np.arange(b_idx.size + 1, dtype=np.int32), np.zeros(b_idx.size, np.int32), "pairs")
    return pairs, m_idx.astype(np.int32), res.per_model_params[b_idx, m_idx, :], res.per_model_chi2[b_idx, m_idx]


def run_finalize(args, batch, res, flush, dev, ws, rank):
    """The reference CLI's finalisation of every (band, model) pair
    (src/bin/extract_features.rs:640-740: batched SVI of each pair seeded
    from its PSO parameters, then finalize_all_models_with_gpu_svi's
    refinements and magnitude chi2) as one lcf_finalize_batch call with SVI
    from each model's polished parameters, host buffers in and out; one
    warm-up and one timed call.  Rank 0 also times the oracle's
    restatement on the first pairs."""
    import torch
    from lightcurve_fitting_gb300 import abi
    from lightcurve_fitting_gb300.lib import Context
    pairs, model, pso, cost = pair_batch(batch, res, args.finalize_sources)
    fctx = Context(dev.index)
    fin = lambda: fctx.finalize_batch(pairs, model, pso, cost, method=abi.METHOD_SVI)
    fin()
    flush.fill_(1.0)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    fin()
    dt = dist_max(time.perf_counter() - t0, ws, dev)
    st = fctx.stats()
    fctx.close()
    out = {"value": ws * pairs.n_bands / dt, "unit": "(band, model) pairs/s", "ms_per_step": 1e3 * dt,
           "pairs_per_gpu": pairs.n_bands, "n_obs_per_gpu": pairs.n_obs, "steps": 1, "warmup": 1,
           "config": "every fitted (band, model) pair of the workload: SVI (1000 steps, 4 samples) from the "
                     "model's polished parameters, profile refinements, magnitude chi2; host buffers",
           "stage_ms": {k: st[k] for k in ["ms_total", "ms_uncertainty", "ms_refine"]},
           "h2d_bytes": int(st["h2d_bytes"]), "d2h_bytes": int(st["d2h_bytes"])}
    if rank == 0 and not args.no_cpu_baseline:
        from oracle import oracle as O
        k = min(1024, pairs.n_bands)
        sub = pairs.subset(np.arange(k))
        t0 = time.perf_counter()
        O.finalize_batch(sub, model[:k], pso[:k], cost[:k], method=abi.METHOD_SVI)
        dc = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": k / dc, "unit": "(band, model) pairs/s", "cores": O.max_threads(),
                               "kind": "port", "sample": f"first {k} pairs, oracle restatement of the "
                                                         f"finalisation, OpenMP over pairs ({dc:.1f} s wall)"}
    return out


def run_side(args, which, dev, flush, ws, rank):
    """A side leg on another of the path's workloads, device-resident, one
    warm-up and `basic_steps` / `precision_steps` timed steps, each rank its
    own copy (seed + rank):
      basic      100 sources x 3 bands x 30 points (the reference's CPU
                 benchmark case), fit_all_models, Laplace, MultiBazin;
      basic_joint  the same sources as the reference's benchmark calls them,
                 fit_parametric(.., false, Laplace): with three bands every
                 source takes the joint multi-band Villar branch;
      precision  1,000 sources x 3 bands x 2,000 points, flux range 1e5,
                 fit_all_models, Laplace, MultiBazin."""
    import torch
    from lightcurve_fitting_gb300 import abi, synth
    from lightcurve_fitting_gb300.lib import Context
    joint = which == "basic_joint"
    if which in ("basic", "basic_joint"):
        batch, steps = synth.config_basic(100, seed=1 + rank), args.basic_steps
    else:
        batch, steps = synth.config_precision(1000, seed=4 + rank), args.precision_steps
    keep = {k: torch.from_numpy(getattr(batch, k)).to(dev) for k in
            ["times", "flux", "flux_err", "band_obs_offsets", "source_band_offsets"]}
    ptrs = {k: v.data_ptr() for k, v in keep.items()}
    sctx = Context(dev.index)
    sstream = torch.cuda.ExternalStream(sctx.stream, device=dev)

    def fit():
        sctx.fit_device(ptrs, batch.n_sources, batch.n_bands, fit_all_models=not joint, method=abi.METHOD_LAPLACE,
                        joint_multiband=joint)

    fit()
    torch.cuda.synchronize()
    times = []
    for _ in range(steps):
        flush.fill_(1.0)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(sstream)
        fit()
        e1.record(sstream)
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    st = sctx.stats()
    sctx.close()
    ms = dist_max(float(np.mean(times)), ws, dev)
    return {"value": job_value(batch.n_sources, ws, ms), "unit": "sources/s", "ms_per_step": ms,
            "sources_per_gpu": batch.n_sources, "n_obs_per_gpu": batch.n_obs, "steps": steps, "warmup": 1,
            "config": batch.name + (": fit_parametric(fit_all_models=false, Laplace): the joint multi-band Villar "
                                    "branch, then per-band Laplace, refinements, MultiBazin, device-resident" if joint
                                    else ": fit_all_models=true, Laplace, MultiBazin, device-resident"),
            "stage_ms": {k: st[k] for k in ["ms_total", "ms_pso", "ms_lbfgs", "ms_uncertainty", "ms_refine",
                                            "ms_multi_bazin"] + (["ms_joint"] if joint else [])}}


def run_scale(args, dev, flush, ws, rank, candidate):
    """The full-scale workload: `scale_sources` sources x 3 bands, counts
    round(lognormal(ln 40, 0.9)) clipped to [5, 1000], the five generators,
    PSO + SVI with MultiBazin in one lcf_fit_parametric_device call (one
    graph), device-resident inputs, one warm-up and one timed step.  Each
    rank fits its own shard (seed 5 + rank)."""
    import torch
    from lightcurve_fitting_gb300 import abi, synth
    from lightcurve_fitting_gb300.lib import Context
    batch = synth.config_scale(args.scale_sources, seed=5 + rank)
    keep = {k: torch.from_numpy(getattr(batch, k)).to(dev) for k in
            ["times", "flux", "flux_err", "band_obs_offsets", "source_band_offsets"]}
    ptrs = {k: v.data_ptr() for k, v in keep.items()}
    sctx = Context(dev.index)
    sctx.set_autotune(1, candidate)
    sstream = torch.cuda.ExternalStream(sctx.stream, device=dev)

    def fit():
        sctx.fit_device(ptrs, batch.n_sources, batch.n_bands, fit_all_models=True, method=abi.METHOD_SVI)

    fit()
    torch.cuda.synchronize()
    flush.fill_(1.0)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(sstream)
    fit()
    e1.record(sstream)
    torch.cuda.synchronize()
    st = sctx.stats()
    sctx.close()
    ms = dist_max(float(e0.elapsed_time(e1)), ws, dev)
    return {"value": job_value(batch.n_sources, ws, ms), "unit": "sources/s", "ms_per_step": ms,
            "sources_per_gpu": batch.n_sources, "n_obs_per_gpu": batch.n_obs, "steps": 1, "warmup": 1,
            "config": "scale: counts round(lognormal(ln 40, 0.9)) clipped [5, 1000], five generators, "
                      "fit_all_models=true, SVI, MultiBazin, one graph",
            "stage_ms": {k: st[k] for k in ["ms_total", "ms_pso", "ms_lbfgs", "ms_t0_search", "ms_uncertainty",
                                            "ms_refine", "ms_multi_bazin"]}}


def main():
    args = parse()
    ws, rank, local = dist_setup()
    if args.impl == "reference":
        run_reference(args, ws, rank)
    else:
        run_fused(args, ws, rank, local)
    if ws > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
