"""Benchmark of the GB300 RHF-CCSD amplitude engine.

Metric: CCSD TFLOP/s and seconds per iteration at no=40, nv=300 (synthetic Hamiltonian,
seed 2, matched coupling), mixed precision vs plain FP64 on one GB300.

* A step is one CCSD iteration of ``solve_cc`` (residual + Jacobi update + energy + DIIS) on
  HBM-resident integrals and amplitudes, following the mixed engine's precision ladder
  (FP8 ladder + BF16 -> BF16 -> split-BF16x3) from the MP2 guess: W warm-up iterations,
  then K timed iterations.  The integral blocks (tens of GB) exceed L2 every iteration.
* TFLOP/s uses the pinned per-iteration count of the reference formulation,
  F_iter = 2 o^2 v^4 + 18 o^3 v^3 + 10 o^2 v^3 + 4 o^4 v^2 (counted once for every mode).
* ``fp64``: the plain FP64 GPU form timed over one iteration at the same size.
* ``e2e``: whole iterations through the public API (``CCwfn.iterate`` + ``diis_step``, the
  body of ``solve_cc``) with t1/t2 copied in from pinned host memory and back out every step:
  the same work per step as the CPU arm's iteration.
* ``roofline``: the <ab|ef> ladder GEMM (the dominant kernel), CUDA events on its stream;
  ``achieved`` counts its algorithmic work (2 o^2 v^4 flop per launch), ``executed_tflops``
  the tensor-core products it issues (three split-BF16 passes over the i <= j pairs).
* ``cpu_baseline``: the reference's own CCSD iteration (its unmodified ``solve_cc`` loop,
  imported from ``baseline/_ref``) on the host cores, a bounded sample at no=20, nv=180.
* ``--impl reference``: the same reference iteration, as the reference arm.

Usage: python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
from __future__ import annotations

import argparse
import gc
import json
import math
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "CCSD s/iter & TFLOP/s (no=40,nv=300): mixed vs FP64 on GB300 at 1e-6 Eh"
FP64_REF = os.path.join(ROOT, "tests", "golden", "fp64_reference.json")


# (no, nv, GEMM format) -> DRAM bytes of the ladder's GEMM launches, from a one-pass ncu
# capture of the same launches at that size
LADDER_DRAM_BYTES = {
    # no=40, nv=300, fused split-BF16x3: + part 12.43 GB read, 2.51 GB written; - part
    # 11.92 GB read, 2.58 GB written
    (40, 300, 4): 29.44e9,
}


def f_iter(o, v):
    return 2 * o**2 * v**4 + 18 * o**3 * v**3 + 10 * o**2 * v**3 + 4 * o**4 * v**2


def peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            d = json.load(f)
        return {"hbm_gbs": d["hbm_gbs"], "bf16": d["bf16_tflops"],
                "bf16_sustained": d.get("bf16_tflops_sustained", d["bf16_tflops"]),
                "source": "measured"}
    return {"hbm_gbs": 6800.0, "bf16": 1900.0, "bf16_sustained": 1700.0, "source": "fallback"}


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""
    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index=0):
        self.index = index
        self.rows = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.Q,
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.th = threading.Thread(target=self._read, daemon=True)
            self.th.start()
            time.sleep(0.3)
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, pw, reasons = [], [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in self.rows:
            try:
                sm.append(float(r[0]))
                mx.append(float(r[1]))
                pw.append(float(r[2]))
            except (ValueError, IndexError):
                continue
            for name, val in zip(names, r[3:7]):
                if val.lower() == "active":
                    reasons.add(name)
        sm.sort()
        return {"sm_mhz": sm[len(sm) // 2] if sm else None,
                "sm_max_mhz": max(mx) if mx else None,
                "power_w_max": max(pw) if pw else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def replica_time(ms, world, device):
    """The per-step time of the job: the slowest of the ``world`` replicas (each rank runs
    the whole iteration on its own GPU; no data-path collective)."""
    if world > 1:
        import torch
        import torch.distributed as dist
        t = torch.tensor([float(ms)], dtype=torch.float64, device=device)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    return ms


def job_tflops(flop_per_step, ms, world):
    """Whole-job rate: every replica does flop_per_step per step of ms milliseconds."""
    return world * flop_per_step / (ms * 1e-3) / 1e12


def dist_env():
    return (int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1")),
            int(os.environ.get("LOCAL_RANK", "0")))


REF_DIR = os.path.join(ROOT, "baseline", "_ref")
# the CPU sample's size: the largest whose reference host layout (full nmo^4 ERI and L in
# FP64, 2 x 12.8 GB at nmo=200) and iteration time (seconds) suit a bounded timing run
CPU_SAMPLE = (20, 180, 1)


def host_info():
    """CPU model, logical cores and RAM of this host (for the CPU baseline's record)."""
    model, mem_gb = None, None
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                k = line.split(":")[0].strip().lower()
                if k in ("model name", "cpu model", "hardware"):
                    model = line.split(":", 1)[1].strip()
                    break
    except OSError:
        pass
    if model is None:
        try:
            out = subprocess.run(["lscpu"], capture_output=True, text=True, timeout=10).stdout
            for line in out.splitlines():
                if line.lower().startswith(("model name", "vendor id")):
                    model = line.split(":", 1)[1].strip()
                    if line.lower().startswith("model name"):
                        break
        except (OSError, subprocess.SubprocessError):
            pass
    try:
        with open("/proc/meminfo") as f:
            for line in f:
                if line.startswith("MemTotal:"):
                    mem_gb = int(line.split()[1]) / 1024**2
                    break
    except OSError:
        pass
    return {"cpu": model, "nproc": os.cpu_count(), "ram_gb": round(mem_gb, 1) if mem_gb else None}


def blas_threads():
    for k in ("OMP_NUM_THREADS", "OPENBLAS_NUM_THREADS"):
        if os.environ.get(k):
            return int(os.environ[k])
    return os.cpu_count() or 1


def cpu_reference_iteration(steps, warmup, budget_s, sample=None):
    """The reference's own CCSD iteration (CrawfordGroup/pycc ``CCwfn.solve_cc`` loop,
    ``pycc/ccwfn.py:268-319``: residual + update + energy + DIIS), timed on the host cores.

    The reference is imported unmodified from ``baseline/_ref`` (its pip install) through
    ``oracle.reference``; when that install or its opt_einsum is missing, the numpy port of
    the same equations (``oracle/ccsd.py``) is timed instead and labelled ``port``.
    Sample: no=20, nv=180 (seed 1, matched coupling).  At no=40, nv=300 the reference keeps
    the full nmo^4 ERI and L in FP64 (214 GB of host RAM) and one iteration takes minutes
    on these cores, beyond a bounded timing run; TFLOP/s uses the same pinned flop formula
    at the sample's size.  Mean over the timed iterations (warm-up iterations excluded).
    """
    import numpy as np
    from pycc_gb300.synth import SyntheticFactors
    o_s, v_s, seed = sample or CPU_SAMPLE
    t0 = time.perf_counter()
    fac = SyntheticFactors(o_s, v_s, seed, coupling="matched")
    F, ERI, L = fac.hamiltonian()
    setup = time.perf_counter() - t0
    kind, why = "reference", None
    try:
        from oracle import reference as R
        pycc = R.import_reference(REF_DIR)
    except ImportError as e:
        kind, why = "port", "reference install unusable (%s)" % e
    if kind == "reference":
        w = R.make_ref_ccwfn(pycc, F, ERI, L, o_s, v_s)
        times, warm = R.time_solve_iterations(w, warmup, steps, budget_s=budget_s)
        del w
    else:
        from oracle import ccsd as oc
        o, v = slice(0, o_s), slice(o_s, o_s + v_s)
        t1, t2 = oc.mp2_guess(F, ERI, o_s)
        Dia, Dijab = oc.denominators(F, o_s)
        diis = oc.DIIS(t1, t2, 8)
        times, warm = [], 0
        tb = time.perf_counter()
        for k in range(warmup + steps):
            ts = time.perf_counter()
            r1, r2 = oc.residuals(o, v, F, ERI, L, t1, t2)
            t1 = t1 + r1 / Dia
            t2 = t2 + r2 / Dijab
            oc.cc_energy(o, v, F, L, t1, t2)
            diis.add_error_vector(t1, t2)
            t1, t2 = diis.extrapolate(t1, t2)
            if k < warmup:
                warm += 1
                tb = time.perf_counter()
            else:
                times.append(time.perf_counter() - ts)
                if budget_s is not None and time.perf_counter() - tb > budget_s:
                    break
    del ERI, L
    if not times:
        raise RuntimeError("CPU baseline: no timed iteration completed")
    dt = float(np.mean(times))
    threads = blas_threads()
    what = ("reference CCwfn.solve_cc iterations (baseline/_ref, unmodified, opt_einsum/numpy "
            "BLAS)" if kind == "reference" else "numpy port of the reference's iteration "
            "(oracle/ccsd.py)")
    host = host_info()
    return {"s_per_iter": dt, "tflops": f_iter(o_s, v_s) / dt / 1e12, "cores": threads,
            "kind": kind, "steps": len(times), "warmup": warm, "iter_s": [round(x, 3) for x in times],
            "integrals_s": setup, "fallback_reason": why, "host": host,
            "sample": "%s at no=%d,nv=%d (seed %d, matched coupling): mean of %d timed iterations "
                      "after %d warm-up; %d BLAS threads on %s; the no=40,nv=300 headline size is "
                      "not runnable on the host: the reference keeps the full nmo^4 ERI and L in "
                      "FP64 (214 GB; host RAM %s GB) and an iteration would take minutes"
                      % (what, o_s, v_s, seed, len(times), warm, threads, host["cpu"],
                         host["ram_gb"])}


def reference_arm(args, rank):
    """``--impl reference``: the reference's own CPU iteration, on rank 0 only, with the
    steps and warm-up that actually ran (bounded so the run ends within a few minutes)."""
    if rank != 0:
        return
    sample = tuple(args.cpu_sample) if getattr(args, "cpu_sample", None) else CPU_SAMPLE
    res = cpu_reference_iteration(args.steps, min(args.warmup, 2), args.ref_budget, sample)
    tf = res["tflops"]
    o_s, v_s, seed = sample
    line = {"metric": METRIC, "value": tf, "unit": "TFLOP/s", "n_gpus": args.gpus,
            "steps": res["steps"], "warmup": res["warmup"], "ms_per_step": res["s_per_iter"] * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "impl": "reference",
            "config": {"workload": "RHF-CCSD iteration (residual + update + energy + DIIS), "
                                   "synthetic Hamiltonian, on the host CPU",
                       "no": o_s, "nv": v_s, "seed": seed, "coupling": "matched",
                       "same_config": False,
                       "headline_config": "no=40,nv=300: not runnable on the host (the reference's "
                                          "FP64 ERI+L need 214 GB; host RAM %s GB)"
                                          % res["host"]["ram_gb"]},
            "steps_requested": args.steps, "warmup_requested": args.warmup,
            "iter_s": res["iter_s"], "host": res["host"],
            "cpu_baseline": {"value": tf, "unit": "TFLOP/s", "cores": res["cores"],
                             "kind": res["kind"], "sample": res["sample"]},
            "e2e": {"value": tf, "unit": "TFLOP/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    if res["fallback_reason"]:
        line["cpu_baseline"]["fallback_reason"] = res["fallback_reason"]
    print(json.dumps(line))


def triples_mode(args, dev):
    """(T) at no=30, nv=240 (seed 4, matched coupling): mixed CCSD, then the tensor-core (T);
    errors against the FP64 energies of tests/golden/fp64_reference.json."""
    import numpy as np
    import torch
    import pycc_gb300 as pg
    from pycc_gb300.triples_tc import t_energy_tc
    no, nv, seed = (30, 240, 4) if args.triples_size is None else tuple(args.triples_size)
    fac = pg.SyntheticFactors(no, nv, seed, coupling="matched")
    H = pg.Hamiltonian.from_factors(fac, device=dev)
    w = pg.CCwfn(H, precision="MIXED")
    t0 = time.time()
    ecc = w.solve_cc(1e-8, 1e-7, 60)
    torch.cuda.synchronize()
    t_cc = time.time() - t0
    t_energy_tc(w, batch=32)                    # warm-up (packs, kernels)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    et = t_energy_tc(w, batch=32)
    e1.record()
    torch.cuda.synchronize()
    s = e0.elapsed_time(e1) / 1e3
    flop = 2 * no**3 * nv**4 + 2 * no**4 * nv**3
    ref = json.load(open(FP64_REF)).get("%d_%d_%d" % (no, nv, seed), {})
    line = {"mode": "triples", "config": {"no": no, "nv": nv, "seed": seed, "coupling": "matched"},
            "ccsd_mixed": {"ecc": ecc, "niter": w.niter, "s": t_cc,
                           "ms_per_iter": 1e3 * float(np.mean(w.iter_times[1:]))},
            "t_s": s, "t_tflops": flop / s / 1e12, "t_flop": flop, "et": et,
            "et_fp64": ref.get("et"), "ecc_fp64": ref.get("ecc"),
            "et_err": (et - ref["et"]) if "et" in ref else None,
            "ecc_err": (ecc - ref["ecc"]) if "ecc" in ref else None,
            "t_fp64_s": ref.get("t_s")}
    print(json.dumps(line))


def term_mode(args, dev):
    """One contraction of the residual at full size, alone: synthetic FP64 operands with the
    o/v extents its labels name (i-n occupied, a-h virtual), the second operand static
    (packed once, like an integral block), the first packed on every call.  Times the pack +
    GEMM and the GEMM launch with CUDA events; the profiling target for single kernels."""
    import torch
    from pycc_gb300.tc import FMT_BF16, FMT_BF16X3, FMT_BF16X3F, Operand, TCEngine
    fmt = {"bf16": FMT_BF16, "bf16x3": FMT_BF16X3, "bf16x3f": FMT_BF16X3F}[args.term_fmt]
    lhs, rhs = args.term.split("->")
    la, lb = lhs.split(",")
    ext = lambda labs: [args.no if c in "ijklmn" else args.nv for c in labs]
    g = torch.Generator(device=dev).manual_seed(7)
    A = torch.randn(ext(la), generator=g, dtype=torch.float64, device=dev)
    B = torch.randn(ext(lb), generator=g, dtype=torch.float64, device=dev)
    out = torch.randn(ext(rhs), generator=g, dtype=torch.float64, device=dev)
    eng = TCEngine(dev)
    opa, opb = Operand.of(la, A), Operand.of(lb, B, key=("term", lb))
    times, gemm = [], []
    st = torch.cuda.current_stream()
    for it in range(args.warmup + args.steps):
        eng.timing = []
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        eng.contract(args.term, opa, opb, out, fmt=fmt)
        e1.record(st)
        torch.cuda.synchronize()
        if it >= args.warmup:
            times.append(e0.elapsed_time(e1))
            gemm.append(eng.timing[0]["start"].elapsed_time(eng.timing[0]["end"]))
    eng.check_status()
    rec = eng.timing[0]
    ms = sorted(gemm)[len(gemm) // 2]
    c_bytes = 2 * out.numel() * 8                  # read-modify-write of the FP64 output
    op_bytes = 4 * (rec["M"] + rec["N"]) * rec["Kp"]  # hi + lo BF16 pieces
    print(json.dumps({"mode": "term", "term": args.term, "fmt": args.term_fmt, "no": args.no,
                      "nv": args.nv, "M": rec["M"], "N": rec["N"], "Kp": rec["Kp"],
                      "ms_gemm": ms, "ms_pack_gemm": sorted(times)[len(times) // 2],
                      "hbm_gbs_gemm": (c_bytes + op_bytes) / (ms * 1e-3) / 1e9,
                      "c_bytes": c_bytes, "operand_bytes": op_bytes,
                      "device_gb": torch.cuda.max_memory_allocated(dev) / 1e9}))


def adjoint_mode(args, dev):
    """Adjoint at no=20, nv=180 (seed 3, matched coupling): Lambda + gradient densities,
    backward/forward cost, central finite differences along random symmetric directions;
    the tape's sweeps on the engine ``--adjoint-sweep`` names."""
    import numpy as np
    import torch
    import pycc_gb300 as pg
    from pycc_gb300.adjoint import CCSDAdjoint
    from pycc_gb300.contract import contract_f64
    no, nv, seed = 20, 180, 3
    fac = pg.SyntheticFactors(no, nv, seed, coupling="matched")
    H = pg.Hamiltonian.from_factors(fac, device=dev)
    w = pg.CCwfn(H)
    e = w.solve_cc(1e-12, 1e-12, 100, keep_tape=bool(args.keep_tape))
    fwd = float(np.mean(w.iter_times[1:]))
    torch.cuda.synchronize()
    t0 = time.time()
    adj = CCSDAdjoint(w, sweep=args.adjoint_sweep)
    t_tape = time.time() - t0
    adj.solve_lambda(1e-12, 1e-12, 200, polish=bool(args.lambda_polish))
    gF, Gam = adj.gradient()
    torch.cuda.synchronize()
    t_back = time.time() - t0
    n = no + nv
    B = torch.from_numpy(fac.B).to(dev)
    ERI = contract_f64("Qpr,Qqs->pqrs", B, B)
    F = H.F
    ident = float((gF * F).sum() + (Gam * ERI).sum()) - e
    # fourth-order central differences, every point converged (|dE| < 1e-14, rms < 1e-13)
    # from the unperturbed amplitudes: (8 (E(h) - E(-h)) - (E(2h) - E(-2h))) / 12h.  The
    # directional derivatives along random unit directions of the n^4 space are small
    # (1e-7 .. 1e-4), so h = 3e-2 keeps the rounding term (~1e-14 / h) far below 1e-6 of
    # them; the h^4 truncation term was measured below 2e-8 relative against h = 1e-2.
    h, rows = 3e-2, []
    t1c, t2c = w.t1.clone(), w.t2.clone()
    for d in range(args.fd_directions):
        g = torch.Generator(device=dev).manual_seed(100 + d)
        dF = torch.randn(n, n, dtype=torch.float64, device=dev, generator=g)
        dF = 0.5 * (dF + dF.T)
        C = torch.randn(n, n, n, n, dtype=torch.float64, device=dev, generator=g)
        C = 0.5 * (C + C.permute(1, 0, 2, 3))
        C = 0.5 * (C + C.permute(0, 1, 3, 2))
        C = 0.5 * (C + C.permute(2, 3, 0, 1))
        dE = C.permute(0, 2, 1, 3).contiguous()
        del C
        nrm = float(torch.sqrt((dF * dF).sum() + (dE * dE).sum()))
        dF /= nrm
        dE /= nrm
        an = float((gF * dF).sum() + (Gam * dE).sum())
        es = {}
        for sg in (1.0, -1.0, 2.0, -2.0):
            wp = pg.CCwfn(pg.Hamiltonian.from_full(F + sg * h * dF, ERI + sg * h * dE, no))
            wp.t1, wp.t2 = t1c, t2c
            es[sg] = wp.solve_cc(1e-14, 1e-13, 200)
            del wp
            gc.collect()            # a wave function is a reference cycle (self.contract)
        fd = (8.0 * (es[1.0] - es[-1.0]) - (es[2.0] - es[-2.0])) / (12.0 * h)
        rows.append({"fd": fd, "adjoint": an, "abs": abs(fd - an), "rel": abs(fd - an) / abs(an)})
        del dE, dF
        torch.cuda.empty_cache()
    stages = getattr(adj, "lambda_stages", [])
    st_time = {k: float(sum(t for t, s_ in zip(adj.lambda_times, stages) if s_ == k))
               for k in set(stages)}
    line = {"mode": "adjoint", "sweep": args.adjoint_sweep, "lambda_polish": bool(args.lambda_polish),
            "tape_from_last_forward_iteration": adj.tape_reused, "tape_s": t_tape,
            "lambda_stages": {k: stages.count(k) for k in set(stages)},
            "lambda_stage_s": st_time, "lambda_at_floor": getattr(adj, "lambda_at_floor", False),
            "config": {"no": no, "nv": nv, "seed": seed, "coupling": "matched"},
            "ecc": e, "forward_iter_s": fwd, "forward_niter": w.niter,
            "lambda_niter": adj.lambda_niter,
            "lambda_iter_s": float(np.mean(adj.lambda_times[1:])),
            "vjp_over_forward_iter": float(np.mean(adj.lambda_times[1:])) / fwd,
            "backward_s": t_back, "backward_over_forward_iter": t_back / fwd,
            "gradient_s": adj.timing_gradient, "energy_identity_err": ident,
            "fd_max_abs": max((r["abs"] for r in rows), default=None),
            "fd_max_rel": max((r["rel"] for r in rows), default=None),
            "fd_stencil": "4-point central, h=3e-2, points converged to |dE| < 1e-14",
            "fd": rows}
    print(json.dumps(line))


def fp64cfg2_mode(args, dev):
    """Plain FP64 RHF-CCSD on the GPU at no=20, nv=180 (seed 1, matched coupling), converged
    to 1e-10: s/iter, TFLOP/s, the fraction of the FP64 peak (cuBLAS DGEMM measured in the
    same run, and the nominal 1.25 TFLOP/s), the energy error against the reference's own
    converged energy (tests/golden/o20v180.npz), and the reference's CPU iteration on the
    host cores at the same size."""
    import numpy as np
    import torch
    import pycc_gb300 as pg
    no, nv, seed = 20, 180, 1
    fac = pg.SyntheticFactors(no, nv, seed, coupling="matched")
    H = pg.Hamiltonian.from_factors(fac, device=dev)
    w = pg.CCwfn(H)
    t0 = time.time()
    try:
        e = w.solve_cc(1e-10, 1e-10, args.fp64_maxiter)
        converged = True
    except pg.ConvergenceError:          # a short profiling run (--fp64-maxiter)
        e, converged = w.energies[-1], False
    torch.cuda.synchronize()
    solve_s = time.time() - t0
    s_iter = float(np.mean(w.iter_times[1:]))
    tf = f_iter(no, nv) / s_iter / 1e12
    # cuBLAS FP64 GEMM on the same GPU: the measured FP64 denominator
    a = torch.randn(8192, 8192, dtype=torch.float64, device=dev)
    b = torch.randn(8192, 8192, dtype=torch.float64, device=dev)
    torch.matmul(a, b)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(3):
        torch.matmul(a, b)
    e1.record()
    torch.cuda.synchronize()
    dgemm = 3 * 2 * 8192.0 ** 3 / (e0.elapsed_time(e1) * 1e-3) / 1e12
    del a, b
    ref = None
    gpath = os.path.join(ROOT, "tests", "golden", "o20v180.npz")
    if os.path.exists(gpath):
        ref = float(np.load(gpath)["ecc"])
    cpu = None
    if not args.no_cpu_baseline:
        res = cpu_reference_iteration(2, 1, 30.0, (no, nv, seed))
        cpu = {"s_per_iter": res["s_per_iter"], "tflops": res["tflops"], "kind": res["kind"],
               "cores": res["cores"], "host": res["host"], "steps": res["steps"]}
    print(json.dumps({"mode": "fp64cfg2", "config": {"no": no, "nv": nv, "seed": seed,
                                                     "coupling": "matched"},
                      "ecc": e, "converged": converged, "niter": w.niter, "solve_s": solve_s,
                      "s_per_iter": s_iter,
                      "tflops": tf, "dgemm_tflops_measured": dgemm,
                      "frac_of_measured_dgemm": tf / dgemm, "frac_of_nominal_1.25": tf / 1.25,
                      "ecc_reference": ref, "energy_error": (e - ref) if ref is not None else None,
                      "cpu_reference": cpu,
                      "speedup_vs_cpu_reference": (cpu["s_per_iter"] / s_iter) if cpu else None}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no", type=int, default=40)
    ap.add_argument("--nv", type=int, default=300)
    ap.add_argument("--seed", type=int, default=2)
    ap.add_argument("--fp64-steps", type=int, default=1)
    ap.add_argument("--e2e-steps", type=int, default=20)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--profile-terms", action="store_true")
    ap.add_argument("--force-mode", default=None, choices=[None, "bf16x3f", "bf16x3s", "bf16x3"],
                    help="run every iteration in this precision stage (profiling of that stage)")
    ap.add_argument("--converge-iters", type=int, default=60,
                    help="untimed iterations allowed after the timed ones to reach the floor")
    ap.add_argument("--fp64-maxiter", type=int, default=60,
                    help="fp64cfg2 mode: iteration limit of the FP64 solve")
    ap.add_argument("--mode", default="ccsd",
                    choices=["ccsd", "triples", "adjoint", "term", "fp64cfg2"],
                    help="ccsd: the benchmark line; triples / adjoint: the (T) and adjoint "
                         "measurements at no=30,nv=240 and no=20,nv=180; term: one residual "
                         "contraction (--term) alone at --no/--nv")
    ap.add_argument("--triples-size", type=int, nargs=3, default=None, metavar=("NO", "NV", "SEED"),
                    help="(T) mode at another size (profiling; the measurement is no=30,nv=240)")
    ap.add_argument("--adjoint-sweep", default="tc", choices=["fp64", "tc"],
                    help="adjoint mode: engine of the tape's sweeps (FP64 or tensor cores)")
    ap.add_argument("--cpu-sample", type=int, nargs=3, default=None, metavar=("NO", "NV", "SEED"),
                    help="size of the CPU sample (default no=20, nv=180, seed 1)")
    ap.add_argument("--ref-budget", type=float, default=120.0,
                    help="reference arm: seconds of timed CPU iterations at most")
    ap.add_argument("--fd-directions", type=int, default=16,
                    help="adjoint mode: random directions of the finite-difference check")
    ap.add_argument("--keep-tape", type=int, default=1, choices=[0, 1],
                    help="adjoint mode: adopt the converging forward iteration's tape")
    ap.add_argument("--lambda-polish", type=int, default=0, choices=[0, 1],
                    help="adjoint mode, tensor-core sweeps: finish Lambda on the FP64 kernels")
    ap.add_argument("--term", default="nb,mnej->mbej")
    ap.add_argument("--term-fmt", default="bf16x3f", choices=["bf16", "bf16x3", "bf16x3f"])
    args = ap.parse_args()
    rank, world, local = dist_env()
    if args.impl == "reference":
        reference_arm(args, rank)
        return
    if args.mode != "ccsd":
        import torch
        dev = torch.device("cuda:%d" % local)
        torch.cuda.set_device(dev)
        {"triples": triples_mode, "adjoint": adjoint_mode, "term": term_mode,
         "fp64cfg2": fp64cfg2_mode}[args.mode](args, dev)
        return

    import numpy as np
    import torch
    import pycc_gb300 as pg
    from pycc_gb300 import _lib
    if args.warmup < 3:
        raise SystemExit("bench.py: at least 3 warm-up steps are required")
    dev = torch.device("cuda:%d" % local)
    torch.cuda.set_device(dev)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")
    o_n, v_n = args.no, args.nv
    F_it = f_iter(o_n, v_n)
    pk = peaks()

    # ---- set-up: integral blocks built on the GPU from the 3-index factor ----------------
    t0 = time.time()
    fac = pg.SyntheticFactors(o_n, v_n, args.seed, coupling="matched")
    H = pg.Hamiltonian.from_factors(fac, device=dev)
    torch.cuda.synchronize()
    setup_s = time.time() - t0

    # ---- mixed-precision solve: W warm-up + K timed iterations ----------------------------
    w = pg.CCwfn(H, precision="MIXED")
    if args.force_mode:
        eng0 = w.mixed_engine()
        eng0.stage = eng0.stages.index(args.force_mode)
        eng0.stages = eng0.stages[:eng0.stage + 1]      # hold that stage
    diis = w.start_iterations(8)
    n = 0
    solve_s = [0.0]       # wall seconds of the solve's iterations (residual .. DIIS), summed

    def step():
        nonlocal n
        n += 1
        ts = time.perf_counter()
        w.iterate(diis, n)
        w.diis_step(diis, n)
        solve_s[0] += time.perf_counter() - ts

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()
    clk = ClockSampler(local)
    clk.start()
    l0 = _lib.launch_count()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    ev0.record()
    for _ in range(args.steps):
        step()
    ev1.record()
    torch.cuda.synchronize()
    launches = _lib.launch_count() - l0
    clocks = clk.stop()
    ms = replica_time(ev0.elapsed_time(ev1) / args.steps, world, dev)
    modes = w.mixed_engine().history[-args.steps:]
    iter_ms = [round(x * 1e3, 2) for x in w.iter_times[-args.steps:]]
    timed_energy = w.energies[-1]
    # iterate on (untimed) to the precision floor for the converged mixed energy
    e_mixed = None
    for _ in range(args.converge_iters):
        if w.mixed_engine().at_floor():
            e_mixed = float(np.mean(w.energies[-4:]))
            break
        step()
    torch.cuda.synchronize()
    hist = w.mixed_engine().history
    stages = {}
    for mode, t in zip(hist, w.iter_times):
        st_ = stages.setdefault(mode, {"iterations": 0, "ms": []})
        st_["iterations"] += 1
        st_["ms"].append(t * 1e3)
    for st_ in stages.values():
        st_["ms_per_iter"] = float(np.mean(st_["ms"][1:] or st_["ms"]))
        del st_["ms"]
    floor = {"reached": e_mixed is not None, "iterations": n if e_mixed is not None else None,
             "rms_floor": w._last_rms, "solve_s": solve_s[0],
             "energy_spread_last4": float(np.ptp(w.energies[-4:])),
             "stages": stages,
             "note": "iterations from the MP2 guess until the final stage stopped reducing the "
                     "update norm; the energy is the mean of the last four iterates"}

    # ---- dominant kernel: per-GEMM CUDA events over one iteration of the stage that ran
    # most of the timed iterations ---------------------------------------------------------
    eng = w.mixed_engine()
    dominant = max(set(modes), key=modes.count)
    saved = eng.stage
    eng.stage = eng.stages.index(dominant)
    eng.tc.timing = []
    t1s, t2s = w.t1.clone(), w.t2.clone()
    w.residuals(H.F, t1s, t2s)
    torch.cuda.synchronize()
    eng.stage = saved
    recs = []
    for r in eng.tc.timing:
        recs.append({"subs": r["subs"], "fmt": r["fmt"], "M": r["M"], "N": r["N"], "Kp": r["Kp"],
                     "ms": r["start"].elapsed_time(r["end"])})
    eng.tc.timing = None
    # the ladder's two GEMMs (symmetric and antisymmetric pair parts)
    ladder = [r for r in recs if r["subs"].startswith("ijef,abef->ijab")]
    roofline = None
    if ladder:
        fmt_l = ladder[0]["fmt"]
        npass = {0: 1, 1: 3, 2: 1, 3: 6, 4: 3, 5: 3}[fmt_l]
        ms_l = sum(r["ms"] for r in ladder)
        # algorithmic work of the launches: the reference's ladder term, 2 o^2 v^4 flop
        alg = 2.0 * o_n**2 * v_n**4
        achieved = alg / (ms_l * 1e-3) / 1e12
        # what the tensor pipe executes: every split-BF16 product pass over the pair rows,
        # columns and K of both parts (a <= b / a < b, i <= j / i < j, e <= f / e < f), and
        # the same over the padded tile grid
        P, Q = v_n * (v_n + 1) // 2, v_n * (v_n - 1) // 2
        Op, Om = o_n * (o_n + 1) // 2, o_n * (o_n - 1) // 2
        work = npass * 2.0 * (P * P * Op + Q * Q * Om)
        executed = work / (ms_l * 1e-3) / 1e12
        padded = sum(npass * 2.0 * r["M"] * r["N"] * r["Kp"] for r in ladder) / (ms_l * 1e-3) / 1e12
        # DRAM bytes of these launches (dram__bytes_read.sum + dram__bytes_write.sum) from a
        # one-pass ncu capture at this size, when one is recorded
        traffic = LADDER_DRAM_BYTES.get((o_n, v_n, fmt_l))
        roofline = {"bound": "tensor", "achieved": achieved, "peak": pk["bf16"],
                    "unit": "TFLOP/s", "frac": achieved / pk["bf16"], "traffic": traffic,
                    "traffic_unit": "bytes per ladder (ncu capture)" if traffic else None,
                    "kernel": "tc_gemm_kernel ladder ijef,abef->ijab, symmetric + antisymmetric "
                              "pair parts (2 launches)",
                    "mode": {0: "bf16", 1: "bf16x3", 2: "fp8", 3: "bf16x6", 4: "bf16x3f",
                             5: "bf16x3s"}[fmt_l],
                    "algorithmic_flop_per_launch": alg, "executed_flop_per_launch": work,
                    "passes": npass, "executed_tflops": executed,
                    "executed_frac": executed / pk["bf16"],
                    "padded_tile_tflops": padded, "ms_per_launch": ms_l,
                    "launches": [{"subs": r["subs"], "M": r["M"], "N": r["N"], "Kp": r["Kp"],
                                  "ms": r["ms"]} for r in ladder],
                    "peak_source": pk["source"] + " bf16 burst (of measured)"}
    gemm_ms = sum(r["ms"] for r in recs)

    # ---- e2e: whole iterations through the public API with host-resident amplitudes -----
    # Each step sets t1/t2 from pinned host memory, runs one solve_cc iteration (residual,
    # update, energy, DIIS) and reads the new t1/t2 back: the same work per step as the CPU
    # arm's iteration, with the host<->device copies inside the timed region.
    t1h = w.t1.detach().cpu().pin_memory()
    t2h = w.t2.detach().cpu().pin_memory()
    e2e_modes = []
    e2e_phases = []

    e2e_host = []

    def e2e_step(k):
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(5)]
        hs = [time.perf_counter()]
        ev[0].record()
        w.t1.copy_(t1h, non_blocking=True)
        w.t2.copy_(t2h, non_blocking=True)
        ev[1].record()
        hs.append(time.perf_counter())
        w.iterate(diis, k)
        ev[2].record()
        hs.append(time.perf_counter())
        w.diis_step(diis, k)
        ev[3].record()
        hs.append(time.perf_counter())
        t1h.copy_(w.t1, non_blocking=True)
        t2h.copy_(w.t2, non_blocking=True)
        ev[4].record()
        hs.append(time.perf_counter())
        torch.cuda.current_stream().synchronize()
        hs.append(time.perf_counter())
        e2e_modes.append(w.mixed_engine().mode_name())
        e2e_phases.append([ev[q].elapsed_time(ev[q + 1]) for q in range(4)])
        e2e_host.append([(hs[q + 1] - hs[q]) * 1e3 for q in range(5)])

    if args.e2e_steps > 0:
        n += 1
        e2e_step(n)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.e2e_steps):
        n += 1
        e2e_step(n)
    e1.record()
    torch.cuda.synchronize()
    e2e_ms = replica_time(e0.elapsed_time(e1) / max(args.e2e_steps, 1), world, dev)
    nb = (t1h.numel() + t2h.numel()) * 8

    # ---- plain FP64 form at the same size --------------------------------------------------
    fp64 = None
    if args.fp64_steps > 0:
        w64 = pg.CCwfn(H, precision="DP")
        d64 = w64.start_iterations(8)
        small = pg.CCwfn(pg.Hamiltonian.from_factors(pg.SyntheticFactors(5, 19, 0), device=dev))
        small.residuals(small.H.F, small.t1, small.t2)         # loads the FP64 kernels
        torch.cuda.synchronize()
        f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        f0.record()
        for k in range(args.fp64_steps):
            w64.iterate(d64, k + 1)
            w64.diis_step(d64, k + 1)
        f1.record()
        torch.cuda.synchronize()
        s64 = f0.elapsed_time(f1) / args.fp64_steps / 1e3
        fp64 = {"s_per_iter": s64, "tflops": F_it / s64 / 1e12, "steps": args.fp64_steps,
                "mixed_speedup": s64 / (ms * 1e-3)}
        if os.path.exists(FP64_REF):
            ref64 = json.load(open(FP64_REF)).get("%d_%d_%d" % (o_n, v_n, args.seed))
            if ref64:
                # FP64 converges (|dE| < 1e-9, rms < 1e-7) in ref64["niter"] iterations
                fp64["solve_iterations"] = ref64["niter"]
                fp64["time_to_solution_s"] = ref64["niter"] * s64
                if floor["reached"]:
                    fp64["mixed_time_to_solution_s"] = floor["solve_s"]
                    fp64["time_to_solution_speedup"] = ref64["niter"] * s64 / floor["solve_s"]
        del w64, d64

    # ---- FP64 oracle energy for the error of the mixed result ------------------------------
    err = None
    if os.path.exists(FP64_REF) and e_mixed is not None:
        with open(FP64_REF) as f:
            refs = json.load(f)
        key = "%d_%d_%d" % (o_n, v_n, args.seed)
        if key in refs:
            err = abs(e_mixed - refs[key]["ecc"])

    cpu = None
    if not args.no_cpu_baseline and rank == 0:
        res = cpu_reference_iteration(2, 1, budget_s=20.0)
        cpu = {"value": res["tflops"], "unit": "TFLOP/s", "cores": res["cores"],
               "kind": res["kind"], "sample": res["sample"], "host": res["host"]}

    line = {
        "metric": METRIC, "value": job_tflops(F_it, ms, world), "unit": "TFLOP/s",
        "value_vs_bf16_peak": job_tflops(F_it, ms, 1) / pk["bf16"],
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "bf16", "data": "synthetic",
        "config": {"workload": "RHF-CCSD iteration (mixed precision ladder from the MP2 guess), "
                               "synthetic Hamiltonian", "no": o_n, "nv": v_n, "seed": args.seed,
                   "coupling": "matched (lambda=%.4f)" % fac.coupling,
                   "l2": "inputs larger than L2 (integral blocks ~%.0f GB)" % (H.nbytes() / 1e9),
                   "parallelism": "replicas" if world > 1 else "single GPU"},
        "s_per_iter": ms * 1e-3, "modes_timed": modes, "iter_wall_ms": iter_ms, "energy_timed_last": timed_energy,
        "energy_mixed": e_mixed, "energy_error_vs_fp64": err, "mixed_solve": floor,
        "fp64": fp64, "roofline": roofline, "cpu_baseline": cpu,
        "e2e": {"value": job_tflops(F_it, e2e_ms, world), "unit": "TFLOP/s",
                "h2d_bytes_per_step": world * nb, "d2h_bytes_per_step": world * nb,
                "what": "one CCwfn iteration (residual, update, energy, DIIS) per step, t1/t2 "
                        "copied in from pinned host memory and back out every step",
                "modes": e2e_modes[-args.e2e_steps:],
                "phases_ms": dict(zip(("h2d", "iterate", "diis", "d2h"),
                                      np.mean(e2e_phases[-args.e2e_steps:], axis=0).round(2)
                                      .tolist())) if args.e2e_steps > 0 else None,
                "host_phases_ms": dict(zip(("h2d", "iterate", "diis", "d2h", "sync"),
                                           np.mean(e2e_host[-args.e2e_steps:], axis=0).round(2)
                                           .tolist())) if args.e2e_steps > 0 else None,
                "step_ms": [round(sum(ph), 2) for ph in e2e_phases[-args.e2e_steps:]],
                "ms_per_step": e2e_ms} if args.e2e_steps > 0 else None,
        "gpu_launches": launches, "clocks": clocks, "setup_s": setup_s,
        "gemm_ms_per_iter": gemm_ms,
    }
    if args.profile_terms:
        line["terms"] = recs
    if rank == 0:
        print(json.dumps(line))
    if world > 1:
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
