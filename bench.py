"""Benchmark: LM iterations/s of the GB300 bundle-adjustment solver.

Workload (default): benchmark configuration 1 — one synthetic BAL problem,
250 cameras on a random walk, 60,000 points, ~296k observations, 50 LM
iterations (tolerances off so all 50 run), PCG capped at 100 iterations
(residual criterion 1e-6).  A step is one full solve.  The headline `value`
is the plain FP64 form (the reference's arithmetic) with the problem
resident in HBM (re-solved from its initial point on the device, L2 flushed
between steps); `e2e` is the same metric through the public C ABI call
(gba_solve) with host buffers: host prep, the host->device copy of the
problem, the solve and the device->host copy of the parameters inside the
timed region.  `forms.mixed` is the FP32/FP64 mixed form on the same
problem, with its accuracy against the FP64 CPU oracle.

Beside them (rank 0, one GPU): `forms.large` (configuration 2), `batched`
(configuration 3), `serving` (configuration 4), `g2o_variant` and
`local_ba` (full_slam's local-BA windows; `--local-ba-only` prints that form
alone).  The full per-kernel tables go to a detail line printed before the
headline line.

--impl reference times the CPU oracle (the C restatement of the reference's
Ceres path: LM + exact Schur complement + Cholesky of the reduced camera
matrix) on this host's cores: each step is one full 50-iteration solve of
the same problem on all cores, generated by the oracle's own generator
(the product library is never loaded on that arm); one more solve on a
single thread (Ceres' default num_threads) is reported beside it.

Multi-GPU (torchrun, N>1): replicas only — each rank solves its own copy of
the workload (weak scaling); value = all ranks' LM iterations / max time.
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

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "LM iters/s and solves/s per GB300 (mixed vs plain FP64 GPU); p50/p99 latency"
UNIT = "LM iter/s"
LM_ITERATIONS = 50


def workload_options(precision: str) -> dict:
    return dict(max_num_iterations=LM_ITERATIONS, function_tolerance=0.0, gradient_tolerance=0.0,
                parameter_tolerance=0.0, max_linear_solver_iterations=100, pcg_tolerance=1e-6, precision=precision,
                loss="trivial")


def config_dict(nc: int, np_: int, no: int) -> dict:
    return {"workload": f"config1: synthetic BAL, 250 cams random walk, 60k points, {no} obs, 50 LM iters, PCG<=100",
            "num_cameras": nc, "num_points": np_, "num_observations": no, "lm_iterations": LM_ITERATIONS,
            "pcg_cap": 100, "pcg": "residual criterion 1e-6, at most 100 iterations per LM step",
            "l2": "flushed between steps (256 MiB write on the solver stream, outside the timed events)",
            "parallelism": "replicas"}


def host_cores() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled during the timed region."""

    FIELDS = "index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown," \
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown," \
             "clocks_event_reasons.sw_power_cap"

    def __init__(self, index: int = 0):
        self.index = index
        self.proc = None
        self.lines: list[str] = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                                          "-i", str(self.index), "-lms", "200"], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

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
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def measured_peaks() -> dict:
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            return json.load(f)
    return {"hbm_gbs": 6800.0, "fallback": True}


def oracle_solve(threads: int = 0, iterations: int = LM_ITERATIONS) -> dict:
    """One solve of the configuration 1 problem by the CPU oracle (the C
    restatement of the reference's Ceres SPARSE_SCHUR path: LM, points
    eliminated, Cholesky of the reduced camera matrix in its envelope), on
    `threads` host threads (0 = all).  The problem comes from the oracle's
    own generator, bitwise the product's."""
    from oracle import oracle_py as O

    p = O.Problem.synthetic(1, seed=0)
    t0 = time.perf_counter()
    res = O.solve(p, max_num_iterations=iterations, function_tolerance=0.0, gradient_tolerance=0.0,
                  parameter_tolerance=0.0, linear_solver="dense_schur", num_threads=threads)
    res["seconds"] = time.perf_counter() - t0
    res["threads"] = threads if threads > 0 else host_cores()
    res["sizes"] = (p.num_cameras(), p.num_points(), p.num_observations())
    return res


def cpu_baseline() -> tuple[dict, dict]:
    """The oracle on all host cores, one full 50-iteration solve of the same
    problem (a few seconds of CPU work)."""
    r = oracle_solve()
    cb = {"value": r["num_iterations"] / r["seconds"], "unit": UNIT, "cores": r["threads"], "kind": "port",
          "sample": f"one full {r['num_iterations']}-iteration solve of the config1 problem (oracle LM, exact Schur "
                    f"complement, envelope Cholesky), {r['seconds']:.2f} s on {r['threads']} threads"}
    return cb, r


def accuracy_vs(oracle_res: dict, params, final_cost: float, nc: int, no: int) -> dict:
    """Final cost, RMS reprojection error and parameter RMS differences of a
    GPU result against the oracle's result on the same problem."""
    import numpy as np

    po = oracle_res["parameters"]
    pg = np.asarray(params, dtype=np.float64).reshape(-1)
    co = oracle_res["final_cost"]
    return {"final_cost": final_cost, "oracle_final_cost": co, "final_cost_rel": abs(final_cost - co) / co,
            "rms_reprojection_px": (2.0 * final_cost / no) ** 0.5, "oracle_rms_reprojection_px": (2.0 * co / no) ** 0.5,
            "camera_rms_diff": float(np.sqrt(np.mean((pg[:9 * nc] - po[:9 * nc]) ** 2))),
            "point_rms_diff": float(np.sqrt(np.mean((pg[9 * nc:] - po[9 * nc:]) ** 2)))}


def run_reference(args) -> None:
    """The CPU oracle on this host's cores, on the GPU arm's config, metric
    and unit.  Rank 0 only; the product library is not loaded."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    for _ in range(args.warmup):
        oracle_solve(iterations=1)  # thread pool, page faults
    runs = [oracle_solve() for _ in range(args.steps)]
    secs = [r["seconds"] for r in runs]
    its = runs[0]["num_iterations"]
    ms = 1e3 * statistics.median(secs)
    v = its / (ms * 1e-3)
    one = oracle_solve(threads=1)
    nc, np_, no = runs[0]["sizes"]
    line = {"metric": METRIC, "value": v, "unit": UNIT, "impl": "reference", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": config_dict(nc, np_, no),
            "reference_impl": "CPU oracle port of the reference's Ceres path (LM + exact Schur complement + "
                              "Cholesky of the reduced camera matrix); Ceres itself is not in the reference tree",
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": runs[0]["threads"], "kind": "port",
                             "sample": f"each step one full {its}-iteration solve of the config1 problem on "
                                       f"{runs[0]['threads']} threads"},
            "cpu_1thread": {"value": one["num_iterations"] / one["seconds"], "unit": UNIT, "cores": 1,
                            "seconds_per_solve": one["seconds"],
                            "sample": "one full solve on one thread (Ceres' default num_threads)"},
            "final_cost": runs[0]["final_cost"],
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def launches_per_solve(s, prof_launches: dict) -> int:
    """Kernels of one solve: setup (parameter sync, LM state, camera table,
    two evaluations of two kernels each, Jacobi scale, post-evaluation) and
    the gather = 10; per LM iteration point/Schur chunk, camera Schur, back-
    substitution, candidate cameras (with their tables), candidate cost, decide,
    evaluation (chunk + camera), post-evaluation = 9, + 1 for the formation
    of the explicit Schur complement; the PCG either as one launch per LM
    iteration (cluster or grid form) or as two kernels per PCG iteration.  prof_launches:
    launches per profile entry of a host-driven pass of the same solve."""
    per_lm = 9 + (1 if prof_launches.get("schur_form") else 0)
    pcg = prof_launches.get("pcg_cluster") or prof_launches.get("pcg_grid") or 2 * s.num_linear_solver_iterations
    return 10 + per_lm * s.num_iterations + pcg


def ncu_traffic(kernel: str, precision: str = "fp64"):
    """DRAM bytes per launch of `kernel` (a profile entry name) on this
    workload in the given form, from the committed ncu capture
    (dram__bytes_read.sum + dram__bytes_write.sum), or None."""
    p = os.path.join(ROOT, "profiles", "dram_traffic_config1.json")
    if not os.path.exists(p):
        return None
    with open(p) as f:
        d = json.load(f)
    return d.get(precision, {}).get("kernels", {}).get(kernel)


def measure_fp64_peak(torch) -> dict:
    """FP64 throughput of this GPU: a cuBLAS DGEMM (torch.matmul, float64,
    8192^3) timed with CUDA events, after warm-up."""
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, n, dtype=torch.float64, device="cuda")
    for _ in range(2):
        torch.matmul(a, b)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    reps = 3
    for _ in range(reps):
        torch.matmul(a, b)
    e1.record()
    e1.synchronize()
    s = e0.elapsed_time(e1) * 1e-3 / reps
    del a, b
    return {"tflops": 2.0 * n ** 3 / s / 1e12, "source": "cuBLAS DGEMM 8192^3 (torch.matmul float64), CUDA events"}


def fp64_rooflines(problem, prof, peak: dict) -> dict:
    """The FP64 form's kernels against the FP64 roof (the measured DGEMM
    rate), for the kernels whose FP64 work is counted: the formation of the
    explicit Schur complement (243 FMAs = 486 flops per observation pair on or
    above the diagonal: sum over points of m (m - 1) / 2 pairs for m views)."""
    import numpy as np

    out = {"peak": peak["tflops"], "unit": "TFLOP/s", "peak_source": peak["source"]}
    m = np.bincount(problem.point_index()).astype(np.int64)
    pairs = int((m * (m - 1) // 2).sum())
    for e in prof:
        if e["name"] == "schur_form":
            avg_s = e["total_ms"] / e["launches"] * 1e-3
            ach = 486.0 * pairs / avg_s / 1e12
            out["schur_form"] = {"achieved": ach, "frac": ach / peak["tflops"], "flops_per_launch": 486.0 * pairs,
                                 "avg_launch_ms": avg_s * 1e3}
    return out


def kernel_table(prof: list[dict]) -> list[dict]:
    out = []
    for e in prof:
        avg_us = 1e3 * e["total_ms"] / e["launches"]
        out.append({"name": e["name"], "launches": e["launches"], "total_ms": e["total_ms"], "avg_us": avg_us,
                    "bytes_per_launch": e["bytes"] / e["launches"],
                    "gbs": e["bytes"] / e["launches"] / (avg_us * 1e-6) / 1e9 if avg_us > 0 else None})
    return out


def run_gpu(args) -> None:
    import torch

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl")
    from slamplay_gb300 import BALProblem, Solver

    problem = BALProblem.synthetic(1, seed=0)
    nc, np_, no = problem.num_cameras(), problem.num_points(), problem.num_observations()
    stream = torch.cuda.Stream()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    def timed_form(precision: str):
        s = Solver(device=local, stream=stream.cuda_stream, **workload_options(precision))
        p0 = problem.copy()
        first = s.solve(p0)  # uploads the problem, builds the graph; p0 holds the result
        for _ in range(args.warmup):
            s.solve_resident(1)
        s.synchronize()
        times = []
        for _ in range(args.steps):
            with torch.cuda.stream(stream):
                flush.fill_(1)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            s.solve_resident(1)
            e1.record(stream)
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return s, first, p0, times

    def e2e_form(s) -> tuple[float, object]:
        # through gba_solve: host arrays in, host prep + H2D + solve + D2H
        ts = []
        su = None
        for _ in range(args.steps):
            p = problem.copy()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            su = s.solve(p)
            ts.append(time.perf_counter() - t0)
        return statistics.median(ts), su

    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    clocks = ClockSampler(local)
    clocks.start()
    t_wall0 = time.perf_counter()
    sp, first_p, res_p, times_p = timed_form("fp64")
    t_wall1 = time.perf_counter()
    clk = clocks.stop()
    torch.cuda.synchronize()
    ms_p = sum(times_p) / len(times_p)
    e2e_s, su_p = e2e_form(sp)
    sm, first_m, res_m, times_m = timed_form("mixed")
    ms_m = sum(times_m) / len(times_m)
    e2e_m, _ = e2e_form(sm)
    if dist:
        t = torch.tensor([ms_p, ms_m, e2e_s], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_p, ms_m, e2e_s = t.tolist()
    iters_p, iters_m = first_p.num_iterations, first_m.num_iterations
    value = world * iters_p / (ms_p * 1e-3)
    value_m = world * iters_m / (ms_m * 1e-3)
    h2d = 24 * no + 8 * (9 * nc + 3 * np_)
    d2h = 8 * (9 * nc + 3 * np_)
    e2e_val = world * su_p.num_iterations / e2e_s

    # per-kernel device times (host-driven pass with CUDA events per launch)
    def profile(s):
        s.set_profiling(True)
        s.solve(problem.copy())
        s.set_profiling(False)
        return [e for e in s.profile() if e["launches"] > 0]

    prof_p, prof_m = profile(sp), profile(sm)
    peaks = measured_peaks()
    peak = peaks.get("hbm_gbs", 6800.0)
    fp64_peak = measure_fp64_peak(torch) if rank == 0 else None
    top = max(prof_p, key=lambda e: e["total_ms"]) if prof_p else None
    roof = None
    if top:
        avg_ms = top["total_ms"] / top["launches"]
        bytes_per = top["bytes"] / top["launches"]
        ach = bytes_per / (avg_ms * 1e-3) / 1e9
        roof = {"kernel": top["name"], "bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s",
                "frac": ach / peak, "traffic": ncu_traffic(top["name"], "fp64"), "bytes_per_launch": bytes_per,
                "avg_launch_ms": avg_ms,
                "binding_roof": ("FP64 latency chain: exchanges between SMs and problem-wide FP64 reductions between "
                                 "the products (FP64 pipe 18% active, DRAM 0.08% of peak; "
                                 "profiles/pcg_grid_config1_fp64.md)") if top["name"] == "pcg_grid" else None,
                "timing": "CUDA events around each launch on the solver stream, host-driven pass of the same "
                          "solve (kernels inside the conditional graph cannot be bracketed one by one)",
                "peak_source": "MEASURED_PEAKS.json hbm_gbs (of measured)" if not peaks.get("fallback")
                else "fallback 6.8 TB/s (of fallback)"}
    roof_fp64 = fp64_rooflines(problem, prof_p, fp64_peak) if fp64_peak else None
    if rank == 0:
        cb, orc = cpu_baseline() if world == 1 else (None, None)
        acc_p = accuracy_vs(orc, res_p.parameters(), first_p.final_cost, nc, no) if orc else None
        acc_m = accuracy_vs(orc, res_m.parameters(), first_m.final_cost, nc, no) if orc else None
        extra_forms = {}
        if world == 1 and not args.no_extra_forms:
            serving = lambda: serving_form(n_requests=args.serving_requests,
                                           rate_mults=tuple(float(x) for x in args.serving_rates.split(",")))
            for name, form in (("large", large_form), ("batched", batched_form), ("serving", serving),
                               ("g2o_variant", g2o_variant_form), ("local_ba", local_ba_form)):
                try:
                    extra_forms[name] = form()
                except Exception as e:  # a side form never takes the headline line down
                    extra_forms[name] = {"error": repr(e)}
        forms = {
            "fp64": {"lm_iters_per_s": value, "solves_per_s": world * 1e3 / ms_p, "ms_per_solve": ms_p,
                     "lm_iterations": iters_p, "pcg_iterations": first_p.num_linear_solver_iterations,
                     "vs_oracle": acc_p},
            "mixed": {"lm_iters_per_s": value_m, "solves_per_s": world * 1e3 / ms_m, "ms_per_solve": ms_m,
                      "lm_iterations": iters_m, "pcg_iterations": first_m.num_linear_solver_iterations,
                      "e2e_lm_iters_per_s": world * iters_m / e2e_m, "vs_oracle": acc_m,
                      "final_cost_rel_vs_fp64_gpu": abs(first_m.final_cost - first_p.final_cost) / first_p.final_cost,
                      "vs_fp64": value_m / value},
        }
        detail = {"detail": "bench", "kernels_fp64": kernel_table(prof_p), "kernels_mixed": kernel_table(prof_m),
                  "forms": {**forms, **extra_forms}}
        print(json.dumps(detail), flush=True)
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_p, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic", "config": config_dict(nc, np_, no),
            "e2e": {"value": e2e_val, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "ms_per_step": 1e3 * e2e_s},
            "roofline": roof,
            "roofline_fp64": roof_fp64,
            "cpu_baseline": cb,
            "gpu_launches": args.steps * launches_per_solve(first_p, {e["name"]: e["launches"] for e in prof_p}),
            "clocks": clk,
            "forms": {**forms, **{k: compact_form(k, v) for k, v in extra_forms.items()}},
            "linear_solver": linear_solver_name(prof_p),
            "wall_s_timed": t_wall1 - t_wall0,
        }
        print(json.dumps(line), flush=True)
    sm.close()
    sp.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def linear_solver_name(prof: list[dict]) -> dict:
    names = {e["name"] for e in prof}
    pcg = "two kernels per PCG iteration"
    if "pcg_cluster" in names:
        pcg = "cluster (one launch per LM iteration)"
    elif "pcg_cluster64" in names:
        pcg = "FP64 cluster (one launch per LM iteration)"
    elif "pcg_grid" in names:
        pcg = "grid (one launch per LM iteration)"
    return {"schur": "explicit" if "schur_form" in names else "implicit", "pcg": pcg}


def compact_form(name: str, f: dict) -> dict:
    """The side forms' headline figures, for the final JSON line."""
    if "error" in f:
        return f
    try:
        if name == "large":
            return {k: {"lm_iters_per_s": f[k]["lm_iters_per_s"], "pcg_iterations": f[k]["pcg_iterations"]}
                    for k in ("mixed", "fp64")} | {"mixed_vs_fp64_final_cost_rel": f.get("mixed_vs_fp64_final_cost_rel"),
                                                   "full_solve_lm_iterations": {k: v["lm_iterations"] for k, v in
                                                                                f.get("full_solve", {}).items()}}
        if name == "batched":
            return {"mixed_solves_per_s": f["mixed"]["solves_per_s"], "fp64_solves_per_s": f["fp64"]["solves_per_s"],
                    "sequential_fp64_solves_per_s": f["sequential_fp64"]["solves_per_s"],
                    "mixed_vs_fp64_final_cost_rel": f["mixed_vs_fp64_final_cost_rel"],
                    "rms_reprojection_px_median": {k: v["median"] for k, v in f.get("rms_reprojection_px", {}).items()},
                    "mixed_vs_fp64_camera_rms_diff_median": f.get("mixed_vs_fp64_camera_rms_diff", {}).get("median")}
        if name == "serving":
            return {"sweep": [{k: x[k] for k in ("arrival_rate_per_s", "solves_per_s", "p50_ms", "p99_ms", "reforms")}
                              for x in f["sweep"]], "requests_per_rate": f.get("requests_per_rate"),
                    "sequential_fp64_solves_per_s": f["sequential_fp64_solves_per_s"]}
        if name == "g2o_variant":
            return {k: {"solves_per_s": f[k]["solves_per_s"], "final_cost": f[k]["final_cost"]}
                    for k in ("mixed", "fp64")} | {"mixed_vs_fp64_final_cost_rel": f["mixed_vs_fp64_final_cost_rel"]}
        if name == "local_ba":
            return {k: {"windows_per_s": f[k]["windows_per_s"], "e2e_windows_per_s": f[k]["e2e_windows_per_s"],
                        "final_cost_rel_vs_oracle_max": f[k]["final_cost_rel_vs_oracle_max"]}
                    for k in ("mixed", "fp64")} | {"cpu_oracle_windows_per_s": f["cpu_oracle"]["windows_per_s"]}
    except (KeyError, TypeError) as e:
        return {"error": f"summary: {e!r}"}
    return f


PCG_SMALL = dict(pcg_criterion="residual", pcg_tolerance=1e-6, max_linear_solver_iterations=100)


def batched_form(n_problems: int = 1024, repeats: int = 2, seq_sample: int = 32) -> dict:
    """Configuration 3: 1,024 local-BA windows (5-40 cameras, 200-5,000
    points, 2-8 views) solved as one batch (every LM iteration of every
    problem in one graph launch), to convergence or 50 iterations, PCG as in
    configuration 1.  Timed re-runs from the initial point on the device;
    beside it the plain FP64 solver on the same problems one at a time
    (first `seq_sample` problems)."""
    from slamplay_gb300 import BALProblem, Solver

    probs = [BALProblem.synthetic(3, index=i, seed=0) for i in range(n_problems)]
    out = {"workload": f"config3: {n_problems} problems, {sum(p.num_observations() for p in probs)} obs",
           "pcg": "residual 1e-6, <= 100"}
    solved = {}

    def timed(s, prec=None):
        work = [p.copy() for p in probs]
        sums = s.batch_solve(work)
        if prec:
            solved[prec] = work
        ts = []
        for _ in range(repeats):
            t0 = time.perf_counter()
            s.solve_resident(1)
            s.synchronize()
            ts.append(time.perf_counter() - t0)
        return sums, min(ts)

    finals = {}
    for prec in ("mixed", "fp64"):
        with Solver(precision=prec, max_num_iterations=50, **PCG_SMALL) as s:
            sums, t = timed(s, prec)
            finals[prec] = [x.final_cost for x in sums]
            tune = None
            if prec == "mixed":
                t_tune = time.perf_counter()
                tune = s.autotune(probs)
                tune_s = time.perf_counter() - t_tune
                sums_t, t_t = timed(s)
        its = sum(x.num_iterations for x in sums)
        out[prec] = {"solves_per_s": n_problems / t, "lm_iters_per_s": its / t, "s_per_batch": t,
                     "lm_iterations": its, "converged": sum(1 for x in sums if x.termination_type == "CONVERGENCE")}
        if tune:
            its_t = sum(x.num_iterations for x in sums_t)
            out[prec]["autotuned"] = {"chunk_observations": tune["chunk_observations"],
                                      "pcg_unroll": tune["pcg_unroll"], "tuning_s": tune_s,
                                      "solves_per_s": n_problems / t_t, "lm_iters_per_s": its_t / t_t,
                                      "s_per_batch": t_t}
    with Solver(precision="fp64", max_num_iterations=50, **PCG_SMALL) as s:
        t0 = time.perf_counter()
        its = sum(s.solve(p.copy()).num_iterations for p in probs[:seq_sample])
        dt = time.perf_counter() - t0
    out["sequential_fp64"] = {"solves_per_s": seq_sample / dt, "lm_iters_per_s": its / dt,
                              "sample": f"first {seq_sample} problems, one gba_solve each"}
    out["mixed_batched_vs_sequential_fp64_solves"] = out["mixed"]["solves_per_s"] / out["sequential_fp64"]["solves_per_s"]
    # accuracy of the mixed form: each problem's final cost against its FP64
    # solve (both run to their convergence test)
    rel = [abs(a - b) / b for a, b in zip(finals["mixed"], finals["fp64"]) if b > 0]
    rel.sort()
    out["mixed_vs_fp64_final_cost_rel"] = {"max": rel[-1], "median": rel[len(rel) // 2],
                                          "p99": rel[int(0.99 * (len(rel) - 1))],
                                          "within_1e-6": sum(1 for r in rel if r <= 1e-6), "problems": len(rel)}
    # RMS reprojection error of each result and the parameter RMS differences
    # of the mixed results against the FP64 ones (the FP64 GPU solve as the
    # reference of this size), as medians / p99 / max over the problems
    import numpy as np

    def dist(v):
        v = np.sort(np.asarray(v))
        return {"median": float(v[len(v) // 2]), "p99": float(v[int(0.99 * (len(v) - 1))]), "max": float(v[-1])}

    rms = {prec: [(2.0 * c / p.num_observations()) ** 0.5 for c, p in zip(finals[prec], probs)]
           for prec in ("mixed", "fp64")}
    cam_d, pt_d = [], []
    for a, b, p in zip(solved["mixed"], solved["fp64"], probs):
        n9 = 9 * p.num_cameras()
        pa, pb = a.parameters(), b.parameters()
        cam_d.append(float(np.sqrt(np.mean((pa[:n9] - pb[:n9]) ** 2))))
        pt_d.append(float(np.sqrt(np.mean((pa[n9:] - pb[n9:]) ** 2))))
    out["rms_reprojection_px"] = {prec: dist(v) for prec, v in rms.items()}
    out["mixed_vs_fp64_camera_rms_diff"] = dist(cam_d)
    out["mixed_vs_fp64_point_rms_diff"] = dist(pt_d)
    return out


def g2o_variant_form(repeats: int = 3) -> dict:
    """The g2o variant's SolveBA (test_bundle_adjustment_g2o.cpp:166-232: SO3
    left camera update, g2o's Levenberg, Huber 1.0, 40 iterations) on the
    configuration 1 problem, PCG as the headline workload; resident re-runs,
    mixed and FP64, with the FP64 oracle's final cost beside them."""
    from slamplay_gb300 import G2O_VARIANT, BALProblem, Solver

    problem = BALProblem.synthetic(1, seed=0)
    out = {"workload": "config1 problem, g2o variant (so3_left, g2o LM, Huber 1.0, 40 iterations)",
           "pcg": "residual 1e-6, <= 100"}
    for prec in ("mixed", "fp64"):
        with Solver(precision=prec, **G2O_VARIANT, **PCG_SMALL) as s:
            sm = s.solve(problem.copy())
            ts = []
            for _ in range(repeats):
                t0 = time.perf_counter()
                s.solve_resident(1)
                s.synchronize()
                ts.append(time.perf_counter() - t0)
        t = min(ts)
        out[prec] = {"lm_trials_per_s": sm.num_iterations / t, "solves_per_s": 1.0 / t, "ms_per_solve": 1e3 * t,
                     "lm_trials": sm.num_iterations, "accepted": sm.num_successful_steps,
                     "termination": sm.termination_reason, "final_cost": sm.final_cost}
    out["mixed_vs_fp64_final_cost_rel"] = abs(out["mixed"]["final_cost"] - out["fp64"]["final_cost"]) / \
        out["fp64"]["final_cost"]
    return out


def local_ba_form(n_windows: int = 256, repeats: int = 2, oracle_sample: int = 16) -> dict:
    """full_slam's local BA (Backend::Optimize, full_slam/src/backend.cpp:67-199)
    on a batch of synthetic stereo windows (7 keyframes, ~580 landmarks,
    ~5.7k edges each, 5 % gross outliers): g2o's Levenberg, 10 iterations,
    Huber 5.991, then the outlier-threshold test, all windows as one batch
    through gba_local_ba.  e2e = the whole call (host prep, copies, solve,
    chi2, outlier test); resident = device re-runs of the uploaded batch.
    The oracle solves the first `oracle_sample` windows (dense Schur) for the
    CPU rate and the parity of the final costs."""
    from oracle import oracle_py as O
    from slamplay_gb300 import LOCAL_BA, LocalBAWindow, Solver

    ws = [LocalBAWindow.synthetic(seed=1000 + i) for i in range(n_windows)]
    nobs = sum(w.num_observations for w in ws)
    out = {"workload": f"{n_windows} windows, 7 keyframes each, {nobs} edges", "options": "g2o LM, 10 iterations, "
           "Huber 5.991, exact-ish PCG (residual 1e-10, <= 500)"}
    for prec in ("mixed", "fp64"):
        with Solver(precision=prec, **LOCAL_BA) as s:
            gs = [w.copy() for w in ws]
            s.local_ba(gs)  # warm-up: graph capture, workspace
            gs = [w.copy() for w in ws]
            t0 = time.perf_counter()
            res = s.local_ba(gs)
            e2e = time.perf_counter() - t0
            ts = []
            for _ in range(repeats):
                t1 = time.perf_counter()
                s.solve_resident(1)
                s.synchronize()
                ts.append(time.perf_counter() - t1)
        t = min(ts)
        its = sum(sm.num_iterations for sm, _ in res)
        out[prec] = {"windows_per_s": n_windows / t, "lm_trials_per_s": its / t, "s_per_batch": t,
                     "e2e_windows_per_s": n_windows / e2e, "e2e_s": e2e,
                     "outliers": sum(r["num_outliers"] for _, r in res),
                     "final_costs_head": [sm.final_cost for sm, _ in res[:oracle_sample]]}
    t0 = time.perf_counter()
    orc = []
    for w in ws[:oracle_sample]:
        so = O.solve(O.window_problem(w), rig=O.rig_from_window(w), linear_solver="dense_schur", **LOCAL_BA)
        orc.append(so["final_cost"])
    dt = time.perf_counter() - t0
    import os as _os
    out["cpu_oracle"] = {"windows_per_s": oracle_sample / dt, "sample": f"first {oracle_sample} windows",
                         "cores": _os.cpu_count(), "kind": "port"}
    for prec in ("mixed", "fp64"):
        rel = [abs(a - b) / b for a, b in zip(out[prec]["final_costs_head"], orc)]
        out[prec]["final_cost_rel_vs_oracle_max"] = max(rel)
    return out


def large_form(lm_iterations: int = 10) -> dict:
    """Configuration 2: one large problem (1,800 cameras in six loops, 1.0M
    points, views per point 1 + Zipf(1.5) truncated to 2-40: ~5.8M
    observations), mixed and FP64, the first `lm_iterations` LM iterations
    (tolerances off, PCG as in configuration 1).  Reports LM iterations/s and
    each kernel's achieved bandwidth at a size where launch latency no longer
    dominates (the Jacobian alone is 0.6 GB in the mixed form); then both
    forms solved in full (Ceres' default tolerances) for their accuracy."""
    from slamplay_gb300 import BALProblem, Solver

    b = BALProblem.synthetic(2, seed=0)
    peak = measured_peaks().get("hbm_gbs", 6800.0)
    out = {"workload": f"config2: {b.num_cameras()} cameras, {b.num_points()} points, {b.num_observations()} obs, "
                       f"first {lm_iterations} LM iterations, PCG residual 1e-6 <= 100"}
    finals = {}
    for prec in ("mixed", "fp64"):
        opts = dict(max_num_iterations=lm_iterations, function_tolerance=0.0, gradient_tolerance=0.0,
                    parameter_tolerance=0.0, precision=prec, **PCG_SMALL)
        with Solver(**opts) as s:
            first = s.solve(b.copy())
            s.synchronize()
            t0 = time.perf_counter()
            s.solve_resident(1)
            s.synchronize()
            dt = time.perf_counter() - t0
            s.set_profiling(True)
            s.solve(b.copy())
            s.set_profiling(False)
            prof = [e for e in s.profile() if e["launches"] > 0]
        kern = {}
        for e in prof:
            avg = e["total_ms"] / e["launches"]
            gbs = e["bytes"] / e["launches"] / (avg * 1e-3) / 1e9 if avg > 0 else 0.0
            kern[e["name"]] = {"launches": e["launches"], "avg_us": 1e3 * avg, "gbs": gbs, "frac": gbs / peak,
                               "share": e["total_ms"] / sum(x["total_ms"] for x in prof)}
        finals[prec] = first.final_cost
        out[prec] = {"lm_iters_per_s": first.num_iterations / dt, "s_per_solve": dt,
                     "lm_iterations": first.num_iterations, "pcg_iterations": first.num_linear_solver_iterations,
                     "final_cost": first.final_cost, "kernels": kern}
    out["peak_gbs"] = peak
    out["mixed_vs_fp64_lm_iters"] = out["mixed"]["lm_iters_per_s"] / out["fp64"]["lm_iters_per_s"]
    # after the first iterations from a heavily perturbed start the two
    # forms' trajectories differ (a rounding difference grows); the accuracy
    # comparison is of full solves (Ceres' default tolerances, at most 50
    # iterations), with the FP64 GPU solve as this size's reference (the
    # dense oracle does not scale to it)
    out["first_iterations_cost_rel"] = abs(finals["mixed"] - finals["fp64"]) / finals["fp64"]
    full = {}
    for prec in ("mixed", "fp64"):
        with Solver(precision=prec, max_num_iterations=50, **PCG_SMALL) as s:
            sm = s.solve(b.copy())
        full[prec] = {"final_cost": sm.final_cost, "lm_iterations": sm.num_iterations,
                      "termination": sm.termination_reason,
                      "rms_reprojection_px": (2.0 * sm.final_cost / b.num_observations()) ** 0.5}
    out["full_solve"] = full
    out["mixed_vs_fp64_final_cost_rel"] = abs(full["mixed"]["final_cost"] - full["fp64"]["final_cost"]) / \
        full["fp64"]["final_cost"]
    return out


def _request_copy(r):
    """A request over a pool problem: its own parameter array (the solve
    writes it), the observations and indices shared."""
    from slamplay_gb300 import BALProblem

    b = BALProblem()
    b.use_quaternions = r.use_quaternions
    b.num_cameras_, b.num_points_, b.num_observations_ = r.num_cameras_, r.num_points_, r.num_observations_
    b.camera_index_, b.point_index_, b.observations_ = r.camera_index_, r.point_index_, r.observations_
    b.parameters_ = r.parameters_.copy()
    return b


def serving_form(n_requests: int = 1000, pool: int = 64, rate_mults=(2.0, 5.0, 10.0), seq_sample: int = 16) -> dict:
    """Configuration 4: requests generated as configuration 1 with 10-400
    cameras and 1k-150k points (log-uniform), solved to relative cost
    decrease < 1e-6 or 50 iterations.  `pool` distinct problems are
    generated; the `n_requests` requests of a rate cycle through them (each
    request its own parameter array).  A sequential plain FP64 loop over the
    first `seq_sample` problems sets the reference rate; the mixed-precision
    server then takes `n_requests` Poisson arrivals at each multiple of that
    rate (continuous batching over eight engine slots, requests joining
    running cohorts at LM-iteration boundaries); latency = completion seen by
    the client - submit."""
    import numpy as np

    from slamplay_gb300 import BALProblem, Solver

    problems = [BALProblem.synthetic(4, index=i, seed=0) for i in range(pool)]
    opts = dict(max_num_iterations=50, function_tolerance=1e-6, **PCG_SMALL)
    with Solver(precision="fp64", **opts) as s:
        t0 = time.perf_counter()
        for r in problems[:seq_sample]:
            s.solve(_request_copy(r))
        seq = seq_sample / (time.perf_counter() - t0)
    sweep = []
    rng = np.random.default_rng(1)
    for mult in rate_mults:
        rate = seq * mult
        gaps = rng.exponential(1.0 / rate, size=n_requests)
        sub_t, done_t = {}, {}
        with Solver(precision="mixed", **opts) as s:
            s.start_server()
            t_start = time.perf_counter()
            next_t, i, pending = t_start, 0, set()
            while i < n_requests or pending:
                now = time.perf_counter()
                while i < n_requests and now >= next_t:
                    tk = s.submit(_request_copy(problems[i % pool]))
                    sub_t[tk] = now
                    pending.add(tk)
                    next_t += gaps[i]
                    i += 1
                for tk in list(pending):
                    if s.poll(tk) is not None:
                        done_t[tk] = time.perf_counter()
                        pending.discard(tk)
                time.sleep(0.0002)
            total = time.perf_counter() - t_start
            st = s.server_stats()
            s.stop_server()
        lat = np.array([done_t[k] - sub_t[k] for k in done_t])
        sweep.append({"arrival_rate_per_s": rate, "requests": n_requests, "solves_per_s": n_requests / total,
                      "p50_ms": 1e3 * float(np.percentile(lat, 50)), "p99_ms": 1e3 * float(np.percentile(lat, 99)),
                      "peak_live": st.get("peak_live"), "batched_lm_iterations": st.get("steps"),
                      "reforms": st.get("reforms"), "host_prep_s": st.get("host_prep_s"),
                      "wall_s": total})
    best = max(sweep, key=lambda x: x["solves_per_s"])
    return {"workload": f"config4: {n_requests} Poisson requests per rate over a pool of {pool} problems, mean "
                        f"{int(np.mean([r.num_observations() for r in problems]))} obs",
            "requests_per_rate": n_requests, "sweep": sweep, "sequential_fp64_solves_per_s": seq,
            "sequential_sample": f"first {seq_sample} problems",
            "best_solves_per_s": best["solves_per_s"], "best_vs_sequential_fp64": best["solves_per_s"] / seq}


def run_profile_solve(args) -> None:
    """One solve of the workload (or of configuration 0 / 2, for a bounded
    number of LM iterations) with the host driving the loops (every kernel a
    plain stream launch, as ncu needs: it cannot profile kernels of a graph
    with conditional nodes).  No event timing: ncu times the kernels
    itself."""
    from slamplay_gb300 import BALProblem, Solver

    problem = BALProblem.synthetic(args.config, seed=0)
    opts = workload_options(args.precision)
    opts["schur"] = args.schur
    opts["persistent_pcg"] = args.persistent_pcg
    if args.lm_iterations:
        opts["max_num_iterations"] = args.lm_iterations
    with Solver(use_graphs=0, **opts) as s:
        sm = s.solve(problem.copy())
    print(json.dumps({"precision": args.precision, "schur": args.schur, "persistent_pcg": args.persistent_pcg,
                      "lm_iterations": sm.num_iterations,
                      "pcg_iterations": sm.num_linear_solver_iterations, "final_cost": sm.final_cost}), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gba", choices=["gba", "reference"])
    ap.add_argument("--profile-solve", action="store_true",
                    help="one host-driven solve with per-kernel event timing (the command profiled with ncu)")
    ap.add_argument("--precision", default="mixed", choices=["mixed", "fp64"])
    ap.add_argument("--config", type=int, default=1, choices=[0, 1, 2],
                    help="with --profile-solve: the synthetic configuration to solve")
    ap.add_argument("--schur", default="auto", choices=["auto", "implicit", "explicit"],
                    help="with --profile-solve: the Schur complement form (gba_options.schur)")
    ap.add_argument("--persistent-pcg", type=int, default=1, choices=[0, 1],
                    help="with --profile-solve: the cluster PCG (1) or two kernels per PCG iteration (0)")
    ap.add_argument("--lm-iterations", type=int, default=0,
                    help="with --profile-solve: LM iterations (0 = the workload's 50)")
    ap.add_argument("--serving-requests", type=int, default=1000,
                    help="Poisson requests per arrival rate in the serving form")
    ap.add_argument("--serving-rates", default="2,5,10",
                    help="arrival rates of the serving form, as multiples of the sequential FP64 rate")
    ap.add_argument("--no-extra-forms", action="store_true",
                    help="skip the large, batched, serving and local-BA forms")
    ap.add_argument("--local-ba-only", action="store_true",
                    help="print only the local-BA form (full_slam's windows) as one JSON line")
    args = ap.parse_args()
    if args.impl == "reference":
        # the CPU oracle alone: the product library is neither built nor loaded
        from oracle import oracle_py

        oracle_py.ensure_built()
        run_reference(args)
        return
    from slamplay_gb300 import build as B

    B.build()
    if args.local_ba_only:
        print(json.dumps({"form": "local_ba", **local_ba_form()}), flush=True)
    elif args.profile_solve:
        run_profile_solve(args)
    else:
        run_gpu(args)


if __name__ == "__main__":
    main()
