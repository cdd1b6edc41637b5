#!/usr/bin/env python
"""Benchmark of the SnuSolver numeric factorize-and-solve path on B200.

Workload (default): the 64^3 7-point convection-diffusion matrix
(n = 262,144, 1,810,432 nonzeros, cell Peclet 0.5 along (1,2,3)/sqrt(14))
with 4 right-hand sides U[-1,1] (seed 2), 8 leaves -- synthetic, generated by
snusolver_b200.generators.  One step = numeric factorization (FP32 fronts)
+ solve of the 4 right-hand sides with FP64 iterative refinement to a
relative residual of 1e-10, matrix values and right-hand sides resident in
HBM.  The plain FP64 path is timed on the same matrix for the FP32+IR vs
FP64 comparison.  Inputs (11+ GB of fronts) exceed L2 (126 MB), so no L2
flush is needed between steps.  Then a serving stream (`serve`: Poisson
arrivals at 200 requests/s of factor / refactor / solve requests on 2D and
3D Laplacians, n 1e4..5e5, 1-64 RHS, 4 slots, 120 GB budget) reports p50 /
p99 latency per request type and throughput.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

N > 1 runs one independent replica per GPU (torchrun, NCCL only for the
barrier and the max-over-ranks timing): every rank factors and solves its
own copy ("replicas only"; weak scaling).  --impl reference times the
reference SnuSolver's own CPU path (oracle/_ref, built from its sources) on
the host cores instead, on a bounded sample of the workload.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = ("factor+solve s, FP32+IR vs FP64 @1e-10 resid (64^3 7-pt); "
          "p50/p99 serve latency")
REF_BIN = os.path.join(ROOT, "oracle", "_ref", "snu_ref")


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="c2_convdiff64")
    ap.add_argument("--nleaves", type=int, default=8)
    ap.add_argument("--fp64-steps", type=int, default=3)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--serve-seconds", type=float, default=4.0,
                    help="length of the serving stream (0: skip it)")
    return ap.parse_args()


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms; start()
    returns once the first sample is in, so the timed steps that follow are
    covered even when they last a fraction of a second."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,"
              "clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.rows = []
        self.proc = None
        self.thread = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.device}",
                 f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, text=True)
        except OSError:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._read, daemon=True)
        self.thread.start()
        t0 = time.time()
        while not self.rows and time.time() - t0 < 3.0:
            time.sleep(0.01)

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        if self.thread:
            self.thread.join(timeout=2)
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown",
                 "sw_power_cap"]
        for r in self.rows:
            try:
                sm.append(float(r[1]))
                mx.append(float(r[2]))
            except (ValueError, IndexError):
                continue
            for k, name in enumerate(names):
                if len(r) > 5 + k and r[5 + k].lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


# DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum) per launch of a
# kernel family, from one ncu capture of all its launches in one
# factorization of the workload (one pass, the full-size case); the
# capture and its command are summarised in the named file
PROFILED_TRAFFIC = {
    ("c2_convdiff64", "panel_block"): {
        "bytes_per_launch": 53.80e6,
        "source": "profiles/k_panel_block_dram_c2_convdiff64.md"},
}


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return d.get("hbm_gbs", 6650.0), d.get("bf16_tflops", 1590.0), "measured"
    return 6650.0, 1590.0, "fallback"


def workload(name):
    from snusolver_b200 import generators
    rp, ci, v, B = generators.config(name)
    return rp, ci, v, np.asfortranarray(B)


def dist_setup(args):
    from snusolver_b200 import replicas
    return replicas.init()


def barrier(ws):
    from snusolver_b200 import replicas
    replicas.barrier(ws)


def max_over_ranks(ws, x):
    from snusolver_b200 import replicas
    return replicas.max_over_ranks(ws, x)


def run_ours(args):
    import torch
    import snusolver_b200 as snu
    ws, rank, local = dist_setup(args)
    rp, ci, v, B = workload(args.workload)
    n, nrhs, nnz = len(rp) - 1, B.shape[1], len(ci)
    stream = torch.cuda.Stream()
    dB = torch.from_numpy(np.ascontiguousarray(B.T)).to("cuda")  # column-major
    dX = torch.empty_like(dB)

    def make(prec):
        s = snu.Solver(nleaves=args.nleaves, precision=prec, device=local)
        s.set_stream(stream.cuda_stream)
        if prec == snu.FP32_IR:  # GEMM variants tuned at the first factorize
            s.set_autotune(True)
        s.construct(rp, ci, v)
        return s

    def step(s):
        s.factorize()
        s.solve_device(dB.data_ptr(), dX.data_ptr(), nrhs, n,
                       stream.cuda_stream)

    s32 = make(snu.FP32_IR)
    for _ in range(max(args.warmup - 1, 0)):
        step(s32)
    # one profiled warm-up step: per-family breakdown, dominant family
    s32.set_profiling(snu.KERNEL_FAMILIES).reset_profile()
    step(s32)
    torch.cuda.synchronize()
    breakdown = s32.profile()
    fam_time = {k: d["seconds"] for k, d in breakdown.items()}
    dominant = max(fam_time, key=fam_time.get)
    s32.set_profiling(()).reset_profile()  # timed steps run clean (graph)

    sampler = ClockSampler(local)
    barrier(ws)
    torch.cuda.synchronize()
    sampler.start()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        step(s32)
    e1.record(stream)
    torch.cuda.synchronize()
    barrier(ws)
    clocks = sampler.stop()
    t_step = e0.elapsed_time(e1) / 1e3 / args.steps
    t_step = max_over_ranks(ws, t_step)
    st32 = s32.stats()
    # the same steps again with CUDA events around every launch of the
    # dominant kernel family: its average launch time for the roofline
    s32.set_profiling([dominant]).reset_profile()
    for _ in range(args.steps):
        step(s32)
    torch.cuda.synchronize()
    prof = s32.profile()[dominant]
    s32.set_profiling(())
    X32 = dX.cpu().numpy().T.copy()

    # end to end through the public API: host (pinned) values and RHS in,
    # solution out, every step
    hv = torch.from_numpy(np.asarray(v, np.float64)).pin_memory().numpy()
    hB = torch.from_numpy(np.ascontiguousarray(B.T)).pin_memory().numpy().T
    hX = torch.empty((nrhs, n), dtype=torch.float64).pin_memory().numpy().T
    s32.refactor(hv)
    s32.solve(hB, allow_notconv=False)
    torch.cuda.synchronize()
    barrier(ws)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        s32.refactor(hv)
        s32.solve(hB, out=hX)
    torch.cuda.synchronize()
    t_e2e = max_over_ranks(ws, (time.perf_counter() - t0) / args.steps)

    # plain FP64 on the same matrix
    s64 = make(snu.FP64)
    step(s64)
    torch.cuda.synchronize()
    barrier(ws)
    f0 = torch.cuda.Event(enable_timing=True)
    f1 = torch.cuda.Event(enable_timing=True)
    f0.record(stream)
    for _ in range(args.fp64_steps):
        step(s64)
    f1.record(stream)
    torch.cuda.synchronize()
    t64 = max_over_ranks(ws, f0.elapsed_time(f1) / 1e3 / args.fp64_steps)
    st64 = s64.stats()
    X64 = dX.cpu().numpy().T.copy()
    fwd_err = float(np.abs(X32 - X64).max() / np.abs(X64).max())
    order, sizes = s32.ordering()
    return dict(ws=ws, rank=rank, n=n, nnz=nnz, nrhs=nrhs, t_step=t_step,
                t_e2e=t_e2e, t64=t64, st32=st32, st64=st64, clocks=clocks,
                dominant=dominant, prof=prof, breakdown=breakdown,
                fwd_err=fwd_err, s32=s32, s64=s64, x32=X32[:, 0].copy(),
                x64=X64[:, 0].copy(), order=order, sizes=sizes)


def run_reference_cpu(name, nleaves, blas_threads):
    """One complete factor+solve of the workload by the reference SnuSolver
    (oracle/_ref: its own sources, CPU dense branch), nleaves ranks.
    Returns (factsolve seconds, construct seconds, ranks x BLAS threads)."""
    rp, ci, v, B = workload(name)
    from snusolver_b200 import generators
    d = tempfile.mkdtemp(prefix="snu_ref_")
    mtx = os.path.join(d, "a.mtx")
    generators.write_mtx(mtx, rp, ci, v)
    rhs = os.path.join(d, "b.bin")
    np.asarray(B[:, 0], np.float64).tofile(rhs)
    env = dict(os.environ, SNU_MPI_NP=str(nleaves), CUDA_VISIBLE_DEVICES="",
               OPENBLAS_NUM_THREADS=str(blas_threads),
               SNU_REF_BLAS_THREADS=str(blas_threads), SNU_MPI_TIMEOUT="1800")
    summ = os.path.join(d, "summary")
    os.makedirs(summ)
    out = subprocess.run([REF_BIN, mtx, "--rhs", rhs, "--summary", summ],
                         env=env, check=True, capture_output=True, text=True,
                         timeout=1900).stdout
    line = [l for l in out.splitlines() if l.startswith("SNU_REF_RESULT")][-1]
    res = json.loads(line.split(" ", 1)[1])
    # the reference's ordering and solution, for the parity fields
    res["order"] = np.fromfile(os.path.join(summ, "r0_order.i32.bin"), np.int32)
    res["sizes"] = np.fromfile(os.path.join(summ, "r0_sizes.i32.bin"), np.int32)
    res["x"] = np.fromfile(os.path.join(summ, "r0_x.f64.bin"), np.float64)
    return res["factsolve_s"], res["construct_s"], nleaves * blas_threads, res


def run_port_cpu(name, nleaves):
    """Fallback when oracle/_ref is absent: the C restatement (oracle/),
    ranks simulated one after another in one thread."""
    import ctypes as C
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    from util import oracle_solve  # noqa: E402
    import snusolver_b200 as snu
    rp, ci, v, B = workload(name)
    h = snu.Solver(nleaves=nleaves).analyze(rp, ci)
    order, sizes = h.ordering()
    t0 = time.perf_counter()
    x, lus, blocks, lib = oracle_solve(rp, ci, v, B[:, 0], nleaves, order, sizes)
    t = time.perf_counter() - t0
    for p in blocks.values():
        lib.snu_oracle_free(C.cast(p, C.c_void_p))
    return t


def parity_vs_reference(r, res):
    """The GPU run against the reference's own run of the same system (its
    first right-hand side): ordering and separator sizes bit for bit, the
    FP64 solution and the FP32+IR solution as max-norm relative errors."""
    xr = res["x"]
    scale = float(np.abs(xr).max())
    return {"order_equal": bool(np.array_equal(r["order"], res["order"])),
            "sizes_equal": bool(np.array_equal(r["sizes"], res["sizes"])),
            "fp64_x_rel_err": float(np.abs(r["x64"] - xr).max() / scale),
            "fp32_ir_forward_error": float(np.abs(r["x32"] - xr).max() / scale),
            "fp64_x_tol": 1e-10,
            "reference": "oracle/_ref run of the cpu_baseline leg, column 0"}


def cpu_baseline(name, nleaves, r=None):
    if os.path.exists(REF_BIN):
        t, tc, cores, res = run_reference_cpu(name, nleaves, 1)
        if r is not None:
            r["parity"] = parity_vs_reference(r, res)
        return {"value": t, "unit": "s", "cores": cores, "kind": "reference",
                "sample": (f"one complete factor+solve (1 RHS) of the same "
                           f"{name} system by the reference built from its "
                           f"sources, {nleaves} ranks x 1 BLAS thread, dense "
                           f"levels on its CPU branch; construct {tc:.2f}s "
                           f"not included; max|Ax-b| "
                           f"{res['max_abs_residual']:.2e}")}
    t = run_port_cpu(name, nleaves)
    return {"value": t, "unit": "s", "cores": 1, "kind": "port",
            "sample": f"one complete factor+solve of {name} by the C "
                      f"restatement, ranks run one after another"}


def emit(d):
    print(json.dumps(d), flush=True)


def main_reference(args):
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    cores = os.cpu_count() or 8
    threads = max(1, cores // args.nleaves)
    if not os.path.exists(REF_BIN):
        t = run_port_cpu(args.workload, args.nleaves)
        kind, used = "port", 1
        sample = "C restatement, ranks one after another, 1 thread"
    else:
        # the reference holds no state between runs; every step is a full,
        # independent factor+solve (~1-2 min), so one step is timed
        t, tc, used, res = run_reference_cpu(args.workload, args.nleaves, threads)
        kind = "reference"
        sample = (f"one complete factor+solve (1 RHS; the reference takes one "
                  f"RHS per run) of {args.workload}, {args.nleaves} ranks x "
                  f"{threads} BLAS threads; construct {tc:.2f}s excluded")
    emit({"impl": "reference", "metric": METRIC, "value": t, "unit": "s",
          "n_gpus": args.gpus, "steps": 1, "warmup": 0, "ms_per_step": t * 1e3,
          "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
          "dtype": "f64", "data": "synthetic",
          "config": {"workload": args.workload, "nleaves": args.nleaves,
                     "nrhs": 1, "host_cores": cores},
          "cpu_baseline": {"value": t, "unit": "s", "cores": used,
                           "kind": kind, "sample": sample},
          "e2e": {"value": t, "unit": "s", "h2d_bytes_per_step": 0,
                  "d2h_bytes_per_step": 0}})


def main_ours(args):
    r = run_ours(args)
    if r["rank"] != 0:
        return
    hbm, bf16, src = peaks()
    prof = r["prof"]
    fam = r["dominant"]
    tensor_fams = ("gemm_schur", "gemm_trail", "gemm_panel")
    traffic = PROFILED_TRAFFIC.get((args.workload, fam))
    if fam in tensor_fams:
        # (algorithmic flops; the three-product split issues 3x that in
        # BF16 MMAs, so 1/3 of the bf16 peak is the split's own ceiling)
        ach = prof["flops"] / max(prof["seconds"], 1e-12) / 1e12
        roof = {"bound": "tensor", "achieved": ach, "peak": bf16,
                "unit": "TFLOP/s", "frac": ach / bf16,
                "traffic": traffic["bytes_per_launch"] if traffic else None,
                "kernel": fam, "launches": prof["launches"],
                "peak_source": f"{src} bf16_tflops"}
    else:
        ach = prof["bytes"] / max(prof["seconds"], 1e-12) / 1e9
        roof = {"bound": "hbm", "achieved": ach, "peak": hbm, "unit": "GB/s",
                "frac": ach / hbm,
                "traffic": traffic["bytes_per_launch"] if traffic else None,
                "kernel": fam, "launches": prof["launches"],
                "peak_source": f"{src} hbm_gbs"}
    # the same launches' algorithmic flop rate (the panel kernel is bound
    # by its tile chains, neither HBM nor the tensor pipe)
    roof["achieved_tflops"] = prof["flops"] / max(prof["seconds"], 1e-12) / 1e12
    if traffic:
        roof["traffic_source"] = traffic["source"]
        roof["algorithmic_bytes_per_launch"] = prof["bytes"] / max(prof["launches"], 1)
    # kernels per step, counted at every launch site by the library
    launches_per_step = (r["st32"]["factor_launches"]
                         + r["st32"]["solve_launches"])
    st32, st64 = r["st32"], r["st64"]
    n, nnz, nrhs = r["n"], r["nnz"], r["nrhs"]
    out = {
        "metric": METRIC, "value": r["t_step"], "unit": "s",
        "n_gpus": r["ws"], "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": r["t_step"] * 1e3, "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "f32 fronts (bf16x3/tf32x3 tensor-core GEMMs) + f64 IR",
        "data": "synthetic (seeded generator, snusolver_b200.generators)",
        "config": {"workload": args.workload, "n": n, "nnz": nnz,
                   "nrhs": nrhs, "nleaves": args.nleaves,
                   "precision": "FP32 factors + FP64 refinement to 1e-10",
                   "l2": "no flush: fronts (>5 GB) exceed L2",
                   "parallelism": f"replicas x{r['ws']}"},
        "fp64": {"value": r["t64"], "unit": "s",
                 "backward_error": st64["backward_error"],
                 "factor_s": st64["factor_s"], "solve_s": st64["solve_s"]},
        "fp32_ir_speedup_vs_fp64": r["t64"] / r["t_step"],
        "backward_error": st32["backward_error"],
        "forward_error_vs_own_fp64": r["fwd_err"],
        "ir_iters": st32["ir_iters"], "fp64_fallback": st32["fp64_fallback"],
        "factor_s": st32["factor_s"], "solve_s": st32["solve_s"],
        "factor_gflop": st32["factor_flops"] / 1e9,
        "roofline": roof,
        "breakdown_s": {k: d["seconds"] for k, d in r["breakdown"].items()},
        "gpu_launches": launches_per_step * args.steps,
        "clocks": r["clocks"],
        "e2e": {"value": r["t_e2e"], "unit": "s",
                "h2d_bytes_per_step": 8 * nnz + 8 * n * nrhs,
                "d2h_bytes_per_step": 8 * n * nrhs},
    }
    if r["ws"] == 1 and args.serve_seconds > 0:
        # serving stream: Poisson arrivals at 200/s of factor / refactor /
        # solve requests on 2D/3D Laplacians (n 1e4..5e5), 4 slots, 120 GB
        from snusolver_b200.server import run_stream
        r["s32"].close()
        r["s64"].close()
        try:
            out["serve"] = run_stream(rate=200.0, duration=args.serve_seconds,
                                      seed=5)
        except Exception as e:  # report, do not hide the GPU result
            out["serve"] = {"error": str(e)[:200]}
    if r["ws"] == 1 and not args.no_cpu_baseline:
        try:
            out["cpu_baseline"] = cpu_baseline(args.workload, args.nleaves, r)
        except Exception as e:  # report, do not hide the GPU result
            out["cpu_baseline"] = {"value": None, "error": str(e)[:200]}
        if "parity" in r:
            out["parity_vs_reference"] = r["parity"]
    emit(out)


def backward_errors(mats, row_start, x, b):
    """Per matrix of a batch: |b - A x|_inf / (|A|_inf |x|_inf + |b|_inf)."""
    out = []
    for k, (rp, ci, v) in enumerate(mats):
        sl = slice(row_start[k], row_start[k + 1])
        xk, bk = x[sl], b[sl]
        rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
        ax = np.zeros(len(rp) - 1)
        np.add.at(ax, rows, v * xk[ci])
        an = np.zeros(len(rp) - 1)
        np.add.at(an, rows, np.abs(v))
        den = an.max() * np.abs(xk).max() + np.abs(bk).max()
        out.append(float(np.abs(bk - ax).max() / den))
    return out


def main_batch(args):
    """The batched workload (256 independent 2D matrices in one handle):
    factor+solve with the FP32 GEMMs split TF32x3 and BF16x3, each with its
    per-matrix backward errors.  One JSON line; not the headline metric."""
    import torch
    import snusolver_b200 as snu
    from snusolver_b200 import generators
    mats = generators.batch_config(args.workload)
    stream = torch.cuda.Stream()
    res = {}
    for split in ("tf32", "bf16"):
        os.environ["SNU_SPLIT"] = split  # read when the engine is made
        s = snu.Solver(nleaves=args.nleaves, precision=snu.FP32_IR)
        s.set_stream(stream.cuda_stream)
        s.set_autotune(True)
        s.construct_batch(mats)
        n = s.n
        b = generators.rhs(n, 1, seed=3)[:, 0]
        dB = torch.from_numpy(b.copy()).to("cuda").reshape(1, n)
        dX = torch.empty_like(dB)

        def step():
            s.factorize()
            s.solve_device(dB.data_ptr(), dX.data_ptr(), 1, n,
                           stream.cuda_stream)
        for _ in range(args.warmup):
            step()
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            step()
        e1.record(stream)
        torch.cuda.synchronize()
        st = s.stats()
        x = dX.cpu().numpy()[0]
        be = backward_errors(mats, s.row_start, x, b)
        res[split] = {"factor_solve_s": e0.elapsed_time(e1) / 1e3 / args.steps,
                      "factor_s": st["factor_s"], "solve_s": st["solve_s"],
                      "ir_iters": st["ir_iters"],
                      "fp64_fallback": st["fp64_fallback"],
                      "backward_error_max": max(be),
                      "backward_error_median": float(np.median(be)),
                      "matrices_above_1e-10": int(sum(e > 1e-10 for e in be))}
        s.close()
    os.environ.pop("SNU_SPLIT", None)
    emit({"metric": "factor+solve s, batched FP32+IR @1e-10 (per split)",
          "value": res["tf32"]["factor_solve_s"], "unit": "s",
          "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
          "higher_is_better": False, "dtype": "f32 fronts + f64 IR",
          "data": "synthetic (seeded generator, snusolver_b200.generators)",
          "config": {"workload": args.workload, "matrices": len(mats),
                     "n": n, "nrhs": 1, "nleaves": args.nleaves},
          "splits": res})


def main():
    args = parse()
    if args.impl == "reference":
        main_reference(args)
    elif args.workload.startswith("c3_"):
        main_batch(args)
    else:
        main_ours(args)
    if args.impl == "ours":
        from snusolver_b200 import replicas
        replicas.finish(int(os.environ.get("WORLD_SIZE", "1")))


if __name__ == "__main__":
    main()
