"""Benchmark of the B200 beam-step path (one JSON line on rank 0).

Workload: the 4096-beam batch -- 4096 independent cantilevers, nodes U{5..21}
(order = nodes - 1, Gauss points = nodes + 2), lengths U(5, 100) m, tapered
seeded sections, tip loads A sin(2 pi f t) with A ~ U(1e3, 1e5) N and
f ~ U(0.1, 5) Hz, FP64, h = 0.01 s.  One bench step = every beam advanced one
time step (all Newton iterations to convergence or max_iter).

Metric: converged beam-steps/s (non-converged beam-steps are excluded), with
p50/p99 step latency.  `value` is measured with the loads already resident in
HBM (device-timed with CUDA events on the library's stream); `e2e` goes
through the public C ABI with host buffers: per step one pinned H2D of every
beam's loads, the step, and one D2H of every node's displacement, over the
same steps as `value` (a twin batch taken through the same warm-up steps).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from openturbine_b200 import sharding as S
from openturbine_b200 import workloads as W  # noqa: E402

L2_FLUSH_BYTES = 256 << 20


# DRAM bytes per beam-step of the step kernel from the ncu capture of
# profiles/kernel_counters.md (43.1 MB for 2048 beams: the slab read once per
# step; most of the state written stays in L2).
DRAM_BYTES_PER_BEAM_STEP = 43.1e6 / 2048


def _hbm_peak() -> float | None:
    """Measured HBM copy bandwidth of this pool's B200s, when the file is present."""
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            return float(json.load(f)["hbm_gbs"])
    except (OSError, KeyError, ValueError):
        return None


# FLOPs of the quadrature-point physics (interpolation, sections rotated,
# inertial and elastic forces and blocks) per point of an N-node beam, counted
# in the oracle's operation order by its counting build (ORC_COUNT_FLOPS;
# tests/test_flop_count.py re-derives both constants).
QP_FLOPS_FIXED = 3112.0
QP_FLOPS_PER_NODE = 55.0


def qp_flops(N: int) -> float:
    return QP_FLOPS_FIXED + QP_FLOPS_PER_NODE * N


def algorithmic_flops(N: int, Q: int, iters: int) -> float:
    """FLOPs of one clamped beam for `iters` Newton iterations (per-iteration count:
    Q*F_qp(N) + 144 N^2 Q + 200 N Q + (2/3) m^3 + 2 m^2, m = 6N - 6): the points;
    the node-pair product [N x 2Q][2Q x 36N]; its second factor and the residual;
    elimination and substitution of the free block."""
    m = 6 * N - 6
    per = Q * qp_flops(N) + 144.0 * N * N * Q + 200.0 * N * Q + (2.0 / 3.0) * m ** 3 + 2.0 * m * m
    return per * iters


def rank_draws(rank: int, beams: int, nodes: int = 0) -> list:
    """This rank's batch under weak scaling: its own `beams` beams of the
    workload (model ids rank*beams ...), every node count `nodes` if nonzero."""
    draws = W.draw_batch(beams, first_id=S.weak_shard_first_id(rank, beams))
    if nodes:
        draws = [W.BeamDraw(d.model_id, nodes, d.length, d.amp, d.freq) for d in draws]
    return draws


def job_rate(local_ms: float, local_units: float, dist=None, device=None) -> tuple:
    """Whole-job throughput of a timed region: (slowest rank's time in ms,
    units of all ranks, units / s); the time is the max over ranks."""
    t_ms = S.max_over_ranks(float(local_ms), dist, device)
    units = S.sum_over_ranks(float(local_units), dist, device)
    return t_ms, units, units / (t_ms * 1e-3)


class ClockSampler:
    """nvidia-smi sampling of SM clock and throttle reasons during a region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.lines: list[str] = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self) -> dict:
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = float(parts[2])
            except ValueError:
                continue
            for nm, val in zip(names, parts[5:9]):
                if val.lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


def measured_fp64_peak(torch, device) -> float:
    """cuBLAS FP64 GEMM (8192^3) best of 3, TFLOP/s: the FP64 roof on this GPU."""
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device=device)
    b = torch.randn(n, n, dtype=torch.float64, device=device)
    torch.matmul(a, b)
    torch.cuda.synchronize()
    best = 0.0
    for _ in range(3):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        torch.matmul(a, b)
        e.record()
        e.synchronize()
        best = max(best, 2.0 * n ** 3 / (s.elapsed_time(e) * 1e-3) / 1e12)
    del a, b
    return best


def cpu_baseline(draws, params, steps: int, threads: int) -> dict:
    """The oracle (FP64 C++ port of the reference, OpenMP over beams) on a sample."""
    from oracle.oracle_py import OracleModel, run_batch
    models = [OracleModel(W.batch_cantilever_model(d).pack()) for d in draws]
    conv, secs, iters = run_batch(models, params, steps, [d.amp for d in draws],
                                  [d.freq for d in draws], threads)
    return {"value": conv / secs, "unit": "beam-steps/s", "cores": threads, "kind": "port",
            "sample": f"{len(draws)} beams of the batch x {steps} steps ({secs:.1f} s)",
            "newton_iters": iters}


def run_reference(args) -> None:
    """--impl reference: the reference's CPU path (the oracle port: the reference
    itself needs Kokkos/KokkosKernels/a sparse solver, absent here) on all host
    cores, on the same configuration as the GPU arm: every step advances the
    whole batch (`--beams`, 4096 by default) one time step, with the same load
    schedule (time index k of the warm-up and timed steps)."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from oracle.oracle_py import OracleModel, run_batch_record
    threads = os.cpu_count() or 1
    draws = W.draw_batch(args.beams)
    if args.nodes:
        draws = [W.BeamDraw(d.model_id, args.nodes, d.length, d.amp, d.freq) for d in draws]
    models = [OracleModel(W.batch_cantilever_model(d).pack()) for d in draws]
    params = W.batch_params()
    amp = [d.amp for d in draws]
    freq = [d.freq for d in draws]
    for k in range(args.warmup):
        run_batch_record(models, params, k, 1, amp, freq, threads)
    total_conv, total_secs, lat, iters = 0, 0.0, [], 0
    for j in range(args.steps):
        st, it, secs = run_batch_record(models, params, args.warmup + j, 1, amp, freq, threads)
        total_conv += int((st == 0).sum())
        iters += int(it.sum())
        total_secs += secs
        lat.append(secs * 1e3)
    value = total_conv / total_secs
    line = {
        "impl": "reference", "metric": "converged beam-steps/s", "value": value,
        "unit": "beam-steps/s", "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": total_secs * 1e3 / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": (f"{args.beams}-beam batch of uneven cantilevers (nodes U{{5..21}}, "
                                "Gauss nodes+2, L U(5,100) m, tip A sin(2 pi f t)), every beam "
                                "one time step per bench step (CPU)"),
                   "beams_per_gpu": args.beams, "h": 0.01, "rho_inf": 0.9,
                   "max_iter": params.max_iter, "a_tol": 1e-7, "r_tol": 1e-3,
                   "precision": "plain FP64", "same_config": True},
        "latency_ms": {"p50": float(np.percentile(lat, 50)), "p99": float(np.percentile(lat, 99))},
        "converged_fraction": total_conv / (args.steps * len(models)),
        "newton_iters_per_beam_step": iters / (args.steps * len(models)),
        "cpu_baseline": {"value": value, "unit": "beam-steps/s", "cores": threads, "kind": "port",
                         "sample": f"the whole {len(models)}-beam batch x {args.steps} timed steps "
                                   f"after {args.warmup} warm-up steps"},
        "e2e": {"value": value, "unit": "beam-steps/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_single_models(args) -> None:
    """--single-models: per-step latency of the two single-model configurations
    -- the 5-node cantilever (100 steps, tip load 1e4 sin(2 pi t)) and the
    three-blade rotor with gravity (1000 steps, prescribed hub rotation) --
    through kyn_step (one model per call, results on the host after each
    call), beside the FP64 oracle on one host core.  Prints one JSON line."""
    import torch
    from oracle.oracle_py import OracleModel
    from openturbine_b200.runtime import Context
    torch.cuda.set_device(0)
    ctx = Context(0)
    out = {"metric": "step latency of single models", "unit": "ms", "higher_is_better": False,
           "n_gpus": 1, "dtype": "f64", "data": "synthetic", "configs": {}}

    def cantilever():
        m = W.cantilever_model()
        p = W.cantilever_params()

        def inputs(k, setter):
            fx = np.zeros((5, 6))
            fx[4, 2] = W.cantilever_tip_load(k)
            setter(fx)
        return m, p, 100, inputs

    def rotor():
        m, bcs = W.rotor_model(3)
        p = W.rotor_params()

        def inputs(k, setter):
            for c, u in zip(bcs, W.rotor_root_inputs(m, bcs, k)):
                setter(c, u)
        return m, p, 1000, inputs

    for name, make in (("cantilever 5 nodes, 100 steps", cantilever),
                       ("three-blade rotor 11 nodes per blade, gravity, 1000 steps", rotor)):
        m, p, steps, inputs = make()
        pm = m.pack()
        mid = ctx.create_model(pm)
        orc = OracleModel(pm)
        gpu_ms, cpu_ms, iters = [], [], 0
        for k in range(steps):
            if name.startswith("cantilever"):
                inputs(k, lambda fx: ctx.set_node_fx(mid, fx))
                inputs(k, orc.set_node_fx)
            else:
                inputs(k, lambda c, u: ctx.set_prescribed(mid, c, u))
                inputs(k, orc.set_prescribed)
            t0 = time.perf_counter()
            st, it = ctx.step([mid], p)
            gpu_ms.append((time.perf_counter() - t0) * 1e3)
            t0 = time.perf_counter()
            orc.step(p)
            cpu_ms.append((time.perf_counter() - t0) * 1e3)
            iters += int(it[0])
        g = np.array(gpu_ms[3:])
        c = np.array(cpu_ms[3:])
        out["configs"][name] = {
            "gpu_ms": {"p50": float(np.percentile(g, 50)), "p99": float(np.percentile(g, 99))},
            "oracle_1_core_ms": {"p50": float(np.percentile(c, 50)), "p99": float(np.percentile(c, 99))},
            "newton_iters_per_step": iters / steps,
            "tip_rel_err_vs_oracle": float(np.abs(ctx.state(mid, "q") - orc.state("q")).max()
                                           / max(np.abs(orc.state("q")).max(), 1e-300))}
        ctx.destroy_model(mid)
    ctx.close()
    print(json.dumps(out), flush=True)


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=30)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--beams", type=int, default=4096)
    ap.add_argument("--cpu-sample", type=int, default=1024)
    ap.add_argument("--cpu-steps", type=int, default=150)
    ap.add_argument("--oracle-sample", type=int, default=512,
                    help="beams of the EI-swept batch run on the FP64 oracle for the accuracy leg")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-fp32", action="store_true", help="skip the FP32 + refinement form")
    ap.add_argument("--no-graph", action="store_true", help="launch steps directly (no CUDA graph)")
    ap.add_argument("--no-autotune", action="store_true",
                    help="default threads per CTA instead of the autotuned choice per size class")
    ap.add_argument("--serve", type=float, default=5.0,
                    help="seconds of the serving workload per form (0: skip)")
    ap.add_argument("--serve-rate", type=float, default=2000.0, help="request arrivals per second")
    ap.add_argument("--refine", type=int, default=0,
                    help="refinement corrections of the FP32 form after convergence")
    ap.add_argument("--solver", type=int, default=1,
                    help="free-block solve of the headline legs: 1 elimination in shared memory (default), 0 "
                         "Gauss-Jordan in registers (elimination where the block does not fit)")
    ap.add_argument("--single-models", action="store_true",
                    help="time the single cantilever and rotor configurations instead")
    ap.add_argument("--bulk-sections", type=int, default=1,
                    help="1: sections staged by one bulk copy per Newton iteration, 0: per-point loads")
    ap.add_argument("--nodes", type=int, default=0,
                    help="uniform nodes per beam (0: the batch's U{5..21}); for profiling one bucket")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
        return
    if args.single_models:
        run_single_models(args)
        return

    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    dev = torch.device("cuda", local)

    from openturbine_b200.runtime import LOAD_NODE_FX, Context

    # ---- build the shard: weak scaling, each rank owns its own 4096 beams ----
    draws = rank_draws(rank, args.beams, args.nodes)
    ctx = Context(local)
    ctx.set_linear_solver(args.solver)
    ctx.set_bulk_sections(bool(args.bulk_sections))
    if not args.no_graph:
        ctx.set_cuda_graph(True)   # each step replays the captured bucket launches
    t_setup = time.perf_counter()
    ids = np.array([ctx.create_model(W.batch_cantilever_model(d).pack()) for d in draws],
                   dtype=np.int32)
    t_setup = time.perf_counter() - t_setup
    params = W.batch_params()
    nodes = np.array([d.num_nodes for d in draws])
    qps = nodes + 2
    elem_nodes = int(nodes.sum())
    tip_index = np.cumsum(nodes) - 1          # element-node row of each tip
    total_steps = args.warmup + args.steps
    # loads for every step (resident on the device for `value`, pinned host for e2e)
    loads_host = torch.zeros((total_steps, elem_nodes, 6), dtype=torch.float64).pin_memory()
    for k in range(total_steps):
        loads_host[k, tip_index, 2] = torch.from_numpy(W.tip_loads(draws, k))
    loads_dev = loads_host.to(dev)
    q_host = torch.zeros((elem_nodes, 7), dtype=torch.float64).pin_memory()
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device=dev)
    ext = torch.cuda.ExternalStream(ctx.stream_handle, device=dev)
    fp64_peak = measured_fp64_peak(torch, dev)

    tuned_solvers: dict = {}

    def tune(step_ids, step_params) -> dict:
        """Autotune threads per CTA (and in the FP64 form the free-block solver)
        per size class, timed on clones before the timed region; returns the
        threads per node count and keeps the solvers in tuned_solvers."""
        if args.no_autotune:
            return {}
        # the clones carry their sources' loads: tune on loaded steps (the
        # first step's tip loads), whose Newton iterations are the timed ones'
        ctx.set_loads_batch(step_ids, LOAD_NODE_FX, loads_dev[0].data_ptr(), True)
        ctx.autotune(step_ids, step_params)
        out, sv = {}, {}
        for i, d in enumerate(draws):
            out.setdefault(int(d.num_nodes), ctx.tuned_threads(int(step_ids[i]), step_params.precision))
            sv.setdefault(int(d.num_nodes), "gauss-jordan" if ctx.tuned_solver(
                int(step_ids[i]), step_params.precision) == 0 else
                "panel LU" if step_params.precision else "block elimination")
        tuned_solvers[step_params.precision] = dict(sorted(sv.items()))
        return dict(sorted(out.items()))

    def device_leg(step_ids, step_params, clocks_on: bool):
        """W warm-up steps, then K device-timed steps (device-resident loads, L2
        flushed before each step).  Returns per-step ms, converged counts,
        algorithmic flops, launches, clock summary and the final states."""
        def step(k):
            ctx.set_loads_batch(step_ids, LOAD_NODE_FX, loads_dev[k].data_ptr(), True)
            return ctx.step(step_ids, step_params)
        for k in range(args.warmup):
            step(k)
        torch.cuda.synchronize()
        conv, flops, ms, iters = 0, 0.0, [], 0
        ok_all = np.ones(len(step_ids), dtype=bool)   # converged at every timed step
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        l0 = ctx.kernel_launches
        sampler = ClockSampler(local) if clocks_on else None
        if sampler:
            sampler.__enter__()
        for j in range(args.steps):
            k = args.warmup + j
            with torch.cuda.stream(ext):
                flush.zero_()
                s = torch.cuda.Event(enable_timing=True)
                e = torch.cuda.Event(enable_timing=True)
                s.record(ext)
            st, it = step(k)
            with torch.cuda.stream(ext):
                e.record(ext)
            e.synchronize()
            ms.append(s.elapsed_time(e))
            conv += int((st == 0).sum())
            ok_all &= st == 0
            iters += int(it.sum())
            flops += sum(algorithmic_flops(int(nodes[i]), int(qps[i]), int(it[i]))
                         for i in range(len(step_ids)))
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        clk = None
        if sampler:
            sampler.__exit__(None, None, None)
            clk = sampler.summary()
        q = torch.zeros((elem_nodes, 7), dtype=torch.float64).pin_memory()
        ctx.get_state_batch(step_ids, "q", q.data_ptr(), False)
        return {"ms": ms, "conv": conv, "flops": flops, "iters": iters,
                "launches": ctx.kernel_launches - l0, "clocks": clk, "q": q.numpy().copy(),
                "ok_all": ok_all}

    # ---- value: plain FP64 form, device-resident inputs, device time per step --
    tuned64 = tune(ids, params)
    r64 = device_leg(ids, params, True)
    dev_ms, conv_v, flops_v, launches = r64["ms"], r64["conv"], r64["flops"], r64["launches"]
    t_value_ms, conv_all, value = job_rate(sum(dev_ms), conv_v, dist, dev)

    # ---- the FP32 forms on their own copies of the batch ------------------------
    # (a) FP32 tangent and panel LU; (b) FP32 tangent, FP32 Gauss-Jordan inverse
    # and FP64-residual refinement of every Newton correction to a 1e-10
    # backward error.  Both keep the FP64 residual, convergence test and update.
    prec = None
    if not args.no_fp32:
        tips = np.cumsum(nodes) - 1

        def tip_rel_vs(qa, qb, ok):
            a, b = qa[tips, :3], qb[tips, :3]
            rel = np.abs(b - a).max(axis=1) / np.maximum(np.abs(a).max(axis=1), 1e-300)
            return rel[ok]

        def stats(x):
            x = np.asarray(x)
            return {"beams": int(x.size), "median": float(np.median(x)),
                    "p99": float(np.percentile(x, 99)), "max": float(x.max())} if x.size else None

        def fp32_leg(solver):
            ids32 = np.array([ctx.create_model(W.batch_cantilever_model(d).pack()) for d in draws],
                             dtype=np.int32)
            p32 = W.batch_params()
            p32.precision, p32.refine_iters = 1, args.refine
            ctx.set_linear_solver(solver)
            tuned32 = tune(ids32, p32)
            ctx.reset_solve_stats()
            before = ctx.solve_stats()
            r32 = device_leg(ids32, p32, False)
            after = ctx.solve_stats()
            ctx.set_linear_solver(args.solver)
            t32, _, v32 = job_rate(sum(r32["ms"]), r32["conv"], dist, dev)
            solves = after["checked"] - before["checked"]
            out = {"value": v32, "unit": "beam-steps/s", "ratio_vs_fp64": v32 / value,
                   "threads_per_cta_by_nodes": tuned32,
                   "ms_per_step": t32 / args.steps,
                   "newton_iters_per_beam_step": r32["iters"] / (args.steps * len(ids32)),
                   "fp64_newton_iters_per_beam_step": r64["iters"] / (args.steps * len(ids)),
                   "converged_fraction": r32["conv"] / (args.steps * len(ids32)),
                   "tip_rel_err_vs_fp64_form": stats(tip_rel_vs(r64["q"], r32["q"],
                                                                r64["ok_all"] & r32["ok_all"])),
                   "latency_ms": {"p50": float(np.percentile(r32["ms"], 50)),
                                  "p99": float(np.percentile(r32["ms"], 99))}}
            if solves:
                out["refinement"] = {
                    "solves": solves,
                    "sweeps_per_solve": (after["refine_sweeps"] - before["refine_sweeps"]) / solves,
                    "solves_above_1e-10_after_8_sweeps": after["refine_short"] - before["refine_short"],
                    "largest_backward_error": after["max_backward_error"]}
            for i in ids32:
                ctx.destroy_model(int(i))
            return out

        prec = {"form": "FP32 tangent (3xTF32 integration GEMM) and FP32 panel LU (pivot chains FP32, "
                        "trailing updates on FP64 tensor cores), FP64 residual, convergence test and "
                        "rotation update"
                        + (f", {args.refine} extra Newton correction(s) after convergence"
                           if args.refine else "")}
        prec.update(fp32_leg(1))
        prec["refined"] = {"form": "FP32 tangent, FP32 Gauss-Jordan inverse of the free block in "
                                   "registers, every Newton correction refined with FP64 residuals "
                                   "of the assembled system to a 1e-10 backward error (at most 8 "
                                   "sweeps)"}
        prec["refined"].update(fp32_leg(0))

        # accuracy on the EI-swept batch (bending/torsion stiffness x 10^U(-1,2),
        # conditioned tangents ~2e7..3e9): the same steps in every form, per-beam
        # tip-displacement and root-load errors against the FP64 oracle on a
        # sample, and against the FP64 form on every beam; the FP64 Gauss-Jordan
        # leg measures the backward error of every unpivoted solve
        forms = {"fp64": (0, 1), "fp32": (1, 1), "fp32_refined": (1, 0), "fp64_gauss_jordan": (0, 0)}
        acc_ids, pa, guard = {}, {}, None
        for name, (form, solver) in forms.items():
            acc_ids[name] = np.array([ctx.create_model(W.precision_cantilever_model(d).pack())
                                      for d in draws], dtype=np.int32)
            pp = W.batch_params()
            pp.precision, pp.refine_iters = form, args.refine
            ctx.set_linear_solver(solver)
            ctx.reset_solve_stats()
            before = ctx.solve_stats()
            pa[name] = device_leg(acc_ids[name], pp, False)
            after = ctx.solve_stats()
            if name == "fp64_gauss_jordan":
                guard = {"solves": after["checked"] - before["checked"],
                         "backward_error_above_1e-10": after["guard_trips"] - before["guard_trips"],
                         "largest_backward_error": after["max_backward_error"]}
        ctx.set_linear_solver(args.solver)

        def root_err(la, lb):
            return float(np.abs(lb - la).max() / max(np.abs(la).max(), 1e-300))

        ns = min(args.oracle_sample, len(draws))
        vs_oracle = None
        if ns > 0:
            from oracle.oracle_py import OracleModel, run_batch_record
            orcs = [OracleModel(W.precision_cantilever_model(d).pack()) for d in draws[:ns]]
            ost, _, osecs = run_batch_record(orcs, W.batch_params(), 0, args.warmup + args.steps,
                                             [d.amp for d in draws[:ns]], [d.freq for d in draws[:ns]],
                                             os.cpu_count() or 1)
            oracle_ok = (ost == 0).all(axis=1)
            row0 = np.concatenate([[0], np.cumsum(nodes)[:-1]])
            vs_oracle = {}
            for name in forms:
                okf = oracle_ok & pa[name]["ok_all"][:ns]
                te, re_ = [], []
                for i in np.flatnonzero(okf):
                    oq = orcs[i].state("q")
                    gq = pa[name]["q"][row0[i]:row0[i] + nodes[i]]
                    te.append(np.abs(gq[-1, :3] - oq[-1, :3]).max() / max(np.abs(oq[-1, :3]).max(), 1e-300))
                    re_.append(root_err(orcs[i].state("lambda"),
                                        ctx.state(int(acc_ids[name][i]), "lambda")))
                vs_oracle[name] = {"tip_rel_err": stats(te), "root_load_rel_err": stats(re_)}
            vs_oracle["sample"] = (f"first {ns} beams, {args.warmup + args.steps} steps, beams "
                                   f"converged at every step in the oracle and the form "
                                   f"(oracle: {osecs:.1f} s on {os.cpu_count()} threads)")
        acc = {"workload": f"{args.beams} beams of the batch with bending/torsion stiffness x 10^U(-1,2)",
               "vs_fp64_oracle": vs_oracle, "fp64_gauss_jordan_backward_error": guard}
        for name in ("fp32", "fp32_refined"):
            both = pa["fp64"]["ok_all"] & pa[name]["ok_all"]
            rr = [root_err(ctx.state(int(acc_ids["fp64"][i]), "lambda"),
                           ctx.state(int(acc_ids[name][i]), "lambda")) for i in np.flatnonzero(both)]
            acc[name] = {"beams_converged_in_both": int(both.sum()),
                         "ratio_vs_fp64": ((pa[name]["conv"] / sum(pa[name]["ms"])) /
                                           max(pa["fp64"]["conv"] / sum(pa["fp64"]["ms"]), 1e-300)),
                         "tip_rel_err_vs_fp64_form": stats(tip_rel_vs(pa["fp64"]["q"], pa[name]["q"], both)),
                         "root_load_rel_err_vs_fp64_form": stats(rr)}
        prec["accuracy_ei_swept_batch"] = acc
        for name in forms:
            for i in acc_ids[name]:
                ctx.destroy_model(int(i))

    # ---- e2e: host buffers through the C ABI, wall time per step --------------
    # A twin of the batch, built from the same draws and taken through the same
    # W warm-up steps, is timed over the steps `value` timed (W .. W+K-1, the
    # reference arm's steps too), so both numbers cover the same work: the
    # twin's states, statuses and iteration counts are the batch's own.
    e_ids = np.array([ctx.create_model(W.batch_cantilever_model(d).pack()) for d in draws],
                     dtype=np.int32)
    for k in range(args.warmup):
        ctx.set_loads_batch(e_ids, LOAD_NODE_FX, loads_dev[k].data_ptr(), True)
        ctx.step(e_ids, params)
    e2e_ms, conv_e = [], 0
    if dist:
        dist.barrier()
    for j in range(args.steps):
        k = args.warmup + j
        with torch.cuda.stream(ext):
            flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ctx.set_loads_batch(e_ids, LOAD_NODE_FX, loads_host[k].data_ptr(), False)
        st, it = ctx.step(e_ids, params)
        ctx.get_state_batch(e_ids, "q", q_host.data_ptr(), False)
        e2e_ms.append((time.perf_counter() - t0) * 1e3)
        conv_e += int((st == 0).sum())
    e2e_same_q = bool(np.array_equal(q_host.numpy(), r64["q"], equal_nan=True))
    for i in e_ids:
        ctx.destroy_model(int(i))
    t_e2e_ms, conv_e_all, e2e = job_rate(sum(e2e_ms), conv_e, dist, dev)

    # ---- serving: Poisson request stream, continuous batching, both forms --------
    serving = None
    if args.serve > 0 and world == 1:
        from openturbine_b200.serving import StepServer, poisson_requests, request_pool
        pool_b, pool_r = request_pool(256, 32)
        serving = {"workload": f"Poisson arrivals at {args.serve_rate:g}/s for {args.serve:g} s, "
                               "90% single beams (nodes U{5..21}), 10% three-blade rotors (11 nodes "
                               "per blade, prescribed hub rotation), U{50..500} steps per request",
                   "hbm_budget_gb": 150}
        for name, form in (("fp64", 0), ("fp32", 1)):
            sctx = Context(local, 150 * 10**9)
            sctx.set_linear_solver(args.solver)
            sp = W.batch_params()
            sp.precision = form
            if not args.no_autotune:   # size classes of the request pool, tuned before serving
                pids = np.array([sctx.create_model(pm) for pm, *_ in pool_b + pool_r], dtype=np.int32)
                sctx.autotune(pids, sp)
                for i in pids:
                    sctx.destroy_model(int(i))
            srv = StepServer(sctx, sp)
            for r in poisson_requests(args.serve_rate, args.serve, pool_b, pool_r):
                srv.submit(r)
            srv.run(until_s=args.serve)
            serving[name] = srv.summary()
            sctx.close()
        if serving["fp64"]["converged_beam_steps_per_s"] > 0:
            serving["fp32_vs_fp64"] = (serving["fp32"]["converged_beam_steps_per_s"] /
                                       serving["fp64"]["converged_beam_steps_per_s"])

    if rank == 0:
        achieved = flops_v / (sum(dev_ms) * 1e-3) / 1e12
        line = {
            "metric": "converged beam-steps/s", "value": value, "unit": "beam-steps/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": t_value_ms / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": (f"{args.beams}-beam batch of cantilevers with {args.nodes} nodes"
                                    if args.nodes else
                                    f"{args.beams}-beam batch of uneven cantilevers (nodes U{{5..21}}, "
                                    "Gauss nodes+2, L U(5,100) m, tip A sin(2 pi f t))"),
                       "beams_per_gpu": args.beams, "h": 0.01, "rho_inf": 0.9,
                       "max_iter": params.max_iter, "a_tol": 1e-7, "r_tol": 1e-3,
                       "precision": "plain FP64", "l2": "flushed (256 MB write) before each step",
                       "linear_solver": ("Gauss-Jordan in registers (block elimination where the block "
                                         "exceeds the register grid)" if args.solver == 0 else
                                         "block elimination (8x8 blocks, FP64 tensor-core trailing "
                                         "updates)"),
                       "launch": "direct" if args.no_graph else "CUDA graph replay per step",
                       "threads_per_cta_by_nodes": tuned64,
                       "solver_by_nodes": tuned_solvers.get(0, {}),
                       "parallelism": f"independent beam shards x{world}"},
            "latency_ms": {"p50": float(np.percentile(dev_ms, 50)),
                           "p99": float(np.percentile(dev_ms, 99)),
                           "e2e_p50": float(np.percentile(e2e_ms, 50)),
                           "e2e_p99": float(np.percentile(e2e_ms, 99))},
            "converged_fraction": conv_v / (args.steps * len(ids)),
            "e2e": {"value": e2e, "unit": "beam-steps/s",
                    "h2d_bytes_per_step": int(elem_nodes * 6 * 8),
                    "d2h_bytes_per_step": int(elem_nodes * 7 * 8 + 2 * 4 * len(ids)),
                    "steps": f"{args.warmup}..{args.warmup + args.steps - 1} (value's steps) on a twin batch",
                    "converged_fraction": conv_e / (args.steps * len(ids)),
                    "final_q_equals_value_leg": e2e_same_q},
            "roofline": {"bound": "tensor", "achieved": achieved, "peak": fp64_peak,
                         "unit": "TFLOP/s", "frac": achieved / fp64_peak,
                         "traffic": DRAM_BYTES_PER_BEAM_STEP * len(ids),
                         "peak_source": "cuBLAS FP64 GEMM 8192^3 (FP64 tensor cores) measured in this run",
                         "traffic_source": "ncu dram bytes read+write per beam-step (2048 beams x 13 nodes, "
                                           "profiles/kernel_counters.md) x beams per step",
                         "hbm": {"achieved_gbs": DRAM_BYTES_PER_BEAM_STEP * len(ids) / (t_value_ms / args.steps * 1e-3) / 1e9,
                                 "peak_gbs": _hbm_peak(), "peak_source": "MEASURED_PEAKS.json hbm_gbs"}},
            "gpu_launches": launches,
            "setup_s": t_setup,
        }
        line["clocks"] = r64["clocks"]
        if prec is not None:
            line["precision_form"] = prec
        if serving is not None:
            line["serving"] = serving
        if not args.no_cpu and world == 1:
            line["cpu_baseline"] = cpu_baseline(draws[: args.cpu_sample], params, args.cpu_steps,
                                                os.cpu_count() or 1)
        print(json.dumps(line), flush=True)
    ctx.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
