"""Benchmark: logdet(1-M) matrices per second and time-to-E for the CaPS
plane-sphere free energy at R/L=150 (Drude gold, T=300 K, ldim=1050, matrices
of dimension 2100), on the GPU through the library's C-ABI.

One step = one complete free-energy evaluation (Matsubara sum with the
reference's m cutoff 1e-9 and xi truncation 1e-6, 978 matrices), i.e. the
call caps_free_energy() a user of the library makes.  Matrices are counted over
the reference's own (xi, m) set in both arms; the CPU arm times a systematic
sample of that set.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--precision fp64|mixed]
  python bench.py --impl reference ...   # CPU restatement of the reference on host cores

Multi-GPU (torchrun, one process per GPU) runs independent replicas: every
rank evaluates the whole workload; value = all ranks' matrices / max time.
Prints one JSON line on rank 0.
"""
import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "logdetD/s and time-to-E at R/L=150: mixed+learned vs FP64 GPU, |ΔE/E|≤1e-6"
UNIT = "logdetD/s"
# workload: Drude gold, R/L=150, L=1um, T=300K, ldim=1050
R, L, T, LDIM = 150e-6, 1e-6, 300.0, 1050
OMEGAP_EV, GAMMA_EV = 9.0, 0.035
CUTOFF, EPSREL = 1e-9, 1e-6
WORKLOAD = ("Drude gold (wp=9 eV, gamma=0.035 eV), R/L=150, L=1e-6 m, T=300 K, ldim=1050 (matrix dim 2100), "
            "full Matsubara sum (cutoff 1e-9, epsrel 1e-6)")


def rank_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)), int(os.environ.get("WORLD_SIZE", 1))


class ClockSampler:
    """samples nvidia-smi clocks and throttle reasons while running"""
    FIELDS = "index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown," \
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap"

    def __init__(self, gpu_index):
        self.idx = gpu_index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.idx), "--query-gpu=" + self.FIELDS,
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for ln in self.proc.stdout:
            self.lines.append(ln.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons, power = [], [], set(), []
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
                power.append(float(f[3]))
            except ValueError:
                continue
            for k, name in enumerate(names):
                if f[5 + k].lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm), "power_w_max": max(power) if power else None}


def barrier(dist):
    if dist is not None:
        dist.barrier()


def allmax(dist, x):
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def allsum(dist, x):
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.SUM)
    return float(t.item())


def load_reference_energy():
    p = os.path.join(ROOT, "tests", "golden", "energy_drude_RbyL150_ldim1050_T300.json")
    if os.path.exists(p):
        return json.load(open(p))
    return None


def matsubara_spacing():
    return 2 * math.pi * 1.38064852e-23 * (R + L) * T / (1.0545718e-34 * 299792458.0)


def workload_pairs(ref):
    """the (xi, m) matrices of one free energy of the workload, in (n, m) order: those the
    reference's truncation visits (m cutoff 1e-9 per frequency, frequency cutoff 1e-6),
    read from the reference library's own run of the workload; with their values"""
    Ts = matsubara_spacing()
    xi, ms, vals = [], [], []
    for k, terms in enumerate(ref["terms"]):
        for m, v in enumerate(terms):
            xi.append((k + 1) * Ts)
            ms.append(m)
            vals.append(v)
    return xi, ms, vals


def cpu_sample(ref, nmat, step=0):
    """a systematic sample of nmat matrices of the workload's own (xi, m) set: every
    (N / nmat)-th matrix in (n, m) order, the offset moving with the step, so trace-rule
    matrices (the high-m end of every frequency) and full factorisations enter at their
    true shares"""
    xi, ms, _ = workload_pairs(ref)
    N = len(xi)
    nmat = min(nmat, N)
    off = (0.5 + 0.618034 * step) % 1.0
    idx = sorted(set(min(N - 1, int((i + off) * N / nmat)) for i in range(nmat)))
    return [xi[i] for i in idx], [ms[i] for i in idx], N


def cpu_baseline(ref, nmat, threads, step=0):
    """the CPU restatement of the reference (oracle port) on host threads over a sample of
    the workload: (matrices/s, seconds, matrices sampled, matrices in one free energy)"""
    from oracle import binding as ob
    xi, m, N = cpu_sample(ref, nmat, step)
    t = time.time()
    ob.logdetD_batch(R, L, LDIM, xi, m, (OMEGAP_EV, GAMMA_EV), threads=threads)
    dt = time.time() - t
    return len(xi) / dt, dt, len(xi), N


def workload_config():
    """the workload, identical in both arms"""
    return {"workload": WORKLOAD,
            "matrices": "the (xi, m) matrices of one free energy under the reference's truncation "
                        "(978 of dimension 2100, 446 of them ending at the trace rule)",
            "counted": "logdetD/s over that set: matrices a method computes beyond it are not counted",
            "l2": "no flush needed: every matrix (35 MB) and the per-chunk working set (>10 GB) exceed L2"}


def run_reference(args, dist, rank, world):
    threads = os.cpu_count() or 1
    per_step = args.cpu_sample or 2 * threads
    if rank != 0:
        return
    ref = load_reference_energy()
    for k in range(args.warmup):
        cpu_baseline(ref, per_step, threads, step=k)
    t0 = time.time()
    total, N = 0, 0
    for k in range(args.steps):
        _, _, n, N = cpu_baseline(ref, per_step, threads, step=args.warmup + k)
        total += n
    dt = time.time() - t0
    value = total / dt
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": dt / args.steps * 1e3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64", "data": "synthetic (inputs fully set by the geometry/material scalars)", "impl": "reference",
        "config": workload_config(),
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": "%d matrices per step, a systematic sample of the workload's %d, by the oracle "
                                   "port of the reference (C: adaptive Gauss-Legendre K integrals, dense LU) on %d host "
                                   "threads" % (per_step, N, threads)},
        "projected_time_to_E_s": N / value,
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def measured_hbm_peak():
    """HBM copy bandwidth of the GB300s (GB/s) from MEASURED_PEAKS.json, else the fallback"""
    p = os.path.join(os.path.dirname(os.path.abspath(__file__)), "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            v = json.load(f)["hbm_gbs"]
        return float(v), "of measured (MEASURED_PEAKS.json hbm_gbs: STREAM-style copy)"
    except (OSError, KeyError, ValueError):
        return 6800.0, "of fallback (6.8 TB/s, one earlier GB300 measurement)"


def time_energy(cg, precision, net, calls):
    """(time-to-E s, info, E, device ms per phase) of `calls` free energies after one warm-up"""
    c = cg.Caps(R, L, ldim=LDIM)
    c.set_drude(OMEGAP_EV, GAMMA_EV)
    c.set_precision(precision)
    c.free_energy(T, CUTOFF, EPSREL, mlp=net)
    cg.reset_timings()
    t = time.time()
    for _ in range(calls):
        E, info = c.free_energy(T, CUTOFF, EPSREL, mlp=net)
    t = (time.time() - t) / calls
    ph = [x / calls for x in cg.timings(cumulative=True)]
    return t, info, E, ph


def per_matrix_errors(cg, ref):
    """every matrix of the workload's set in both forms (one batch each) against the
    reference library's values: max and 99th percentile of |d logdetD| / max(1, |x|)"""
    import numpy as np
    xi, ms, want = workload_pairs(ref)
    want = np.array(want)
    got = {}
    for name, prec in (("mixed", cg.PREC_MIXED), ("fp64", cg.PREC_FP64)):
        c = cg.Caps(R, L, ldim=LDIM)
        c.set_drude(OMEGAP_EV, GAMMA_EV)
        c.set_precision(prec)
        got[name] = np.array(c.logdetD_batch(xi, ms)[0])
    scale = np.maximum(1.0, np.abs(want))

    def stats(a, b):
        e = np.abs(a - b) / scale
        return {"max": float(e.max()), "p99": float(np.percentile(e, 99)), "median": float(np.median(e))}
    return {"matrices": len(xi),
            "mixed_vs_reference": stats(got["mixed"], want),
            "fp64_vs_reference": stats(got["fp64"], want),
            "mixed_vs_fp64": stats(got["mixed"], got["fp64"]),
            "bar": "1e-10 max(1,|x|) for the FP64 form; the mixed form is judged on E (|dE/E| <= 1e-6)"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--precision", default="mixed", choices=["fp64", "mixed"])
    ap.add_argument("--cpu-sample", type=int, default=0, help="matrices in the CPU-baseline sample (0: 2 per host thread)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--plain", action="store_true",
                    help="plain truncation schedule instead of the learned proposal")
    ap.add_argument("--no-side", action="store_true",
                    help="skip the side measurements (plain forms, per-matrix errors)")
    ap.add_argument("--no-autotune", action="store_true",
                    help="keep the library's default schedule and path instead of timing the candidates (for runs under "
                         "a profiler, whose serialised launches distort the candidates' times)")
    ap.add_argument("--ncu-case", action="store_true",
                    help="profiling case: one batch of 8 matrices of the workload (n in {1,5}, m in {0,20,40,60})")
    ap.add_argument("--ncu-matrices", type=int, default=8,
                    help="matrices in the profiling case; other than 8: n = 1..4, m = 0, 4, 8, ... (all factored), "
                         "e.g. 48 for a trailing-matrix working set above L2")
    ap.add_argument("--hodlr-case", choices=["r150", "r1000"], default=None,
                    help="profiling case: --ncu-matrices matrices through the FP64 HODLR path, of this workload (r150) "
                         "or of the large-aspect one (r1000: plasma, R/L=1000, L=100 nm, ldim 6000, dimension 12000)")
    ap.add_argument("--c4", action="store_true",
                    help="the large-aspect T = 0 free energy once (plasma, R/L=1000, L=100 nm, ldim 6000, 60-point "
                         "Gauss-Laguerre rule) in the chosen precision; --path picks the FP64 determinant path")
    ap.add_argument("--path", default="auto", choices=["auto", "hodlr", "dense"])
    args = ap.parse_args()
    if args.c4:
        import caps_gb300 as cg
        caps = cg.Caps(1e-4, 1e-7, ldim=6000)
        caps.set_drude(9.0, 0.0)
        caps.set_precision(cg.PREC_MIXED if args.precision == "mixed" else cg.PREC_FP64)
        caps.set_path({"auto": cg.PATH_AUTO, "hodlr": cg.PATH_HODLR, "dense": cg.PATH_DENSE}[args.path])
        cg.counters(reset=True)
        w0 = cg.work()
        t = time.time()
        E, info = caps.free_energy_T0_gl(60)
        dt = time.time() - t
        w1 = cg.work()
        print(json.dumps({"workload": "plasma (wp=9 eV), R/L=1000, L=1e-7 m, T=0, ldim=6000 (dimension 12000), "
                                      "60-point Gauss-Laguerre rule in 2 xi L/c",
                          "precision": args.precision, "path": args.path, "E": E, "time_to_E_s": dt,
                          "matrices": info["ndet"], "matrices_beyond_cutoffs": info["nwasted"],
                          "matrices_factored": w1["nfactor"] - w0["nfactor"], "gpu_launches": cg.counters()["launches"]}))
        return
    if args.hodlr_case:
        import caps_gb300 as cg
        n = args.ncu_matrices
        if args.hodlr_case == "r150":
            caps = cg.Caps(R, L, ldim=LDIM)
            caps.set_drude(OMEGAP_EV, GAMMA_EV)
            xi, ms = [matsubara_spacing()] * n, [(10 * k) % 100 for k in range(n)]
        else:
            caps = cg.Caps(1e-4, 1e-7, ldim=6000)
            caps.set_drude(9.0, 0.0)
            xi, ms = [(250.0, 500.5, 1000.0, 2000.0)[k % 4] for k in range(n)], [(7 * k) % 200 for k in range(n)]
        caps.set_path(cg.PATH_HODLR)
        t = time.time()
        out, st = caps.logdetD_batch(xi, ms)
        print(json.dumps({"logdetD": list(out), "status": [int(s) for s in st], "seconds": time.time() - t}))
        return
    if args.ncu_case:
        import caps_gb300 as cg
        Ts = matsubara_spacing()
        caps = cg.Caps(R, L, ldim=LDIM)
        caps.set_drude(OMEGAP_EV, GAMMA_EV)
        caps.set_precision(cg.PREC_MIXED if args.precision == "mixed" else cg.PREC_FP64)
        if args.ncu_matrices == 8:
            xi = [n * Ts for n in (1, 5) for m in (0, 20, 40, 60)]
            ms = [m for n in (1, 5) for m in (0, 20, 40, 60)]
        else:  # n = 1..4, m = 0, 4, 8, ...: every matrix large enough to be factored
            per = (args.ncu_matrices + 3) // 4
            xi = [n * Ts for n in (1, 2, 3, 4) for k in range(per)][:args.ncu_matrices]
            ms = [4 * k for n in (1, 2, 3, 4) for k in range(per)][:args.ncu_matrices]
        out, st = caps.logdetD_batch(xi, ms)
        print(json.dumps({"logdetD": list(out), "status": [int(s) for s in st], "phases_ms": cg.timings()}))
        return

    rank, local_rank, world = rank_env()
    dist = None
    if world > 1:
        import torch.distributed as dist_mod
        dist_mod.init_process_group("gloo", init_method="env://")
        dist = dist_mod
    if args.impl == "reference":
        run_reference(args, dist, rank, world)
        if dist is not None:
            dist.barrier()
        return
    if world > 1 and "CUDA_VISIBLE_DEVICES" not in os.environ:
        os.environ["CUDA_VISIBLE_DEVICES"] = str(local_rank)

    import caps_gb300 as cg

    fp64_peak = cg.fp64_peak()
    prec = cg.PREC_MIXED if args.precision == "mixed" else cg.PREC_FP64
    caps = cg.Caps(R, L, ldim=LDIM)
    caps.set_drude(OMEGAP_EV, GAMMA_EV)
    caps.set_precision(prec)

    # autotuner (untimed set-up): the trailing-update schedule of the mixed form, or the FP64
    # determinant path, timed on eight matrices of the workload
    Ts = matsubara_spacing()
    t_at = time.time()
    if args.no_autotune:
        autotune = {"skipped": "library defaults: dense path at this dimension, panel images by bulk copies"}
    else:
        chosen, at_ms = caps.autotune(Ts, nprobe=8)
        autotune = {"candidates_ms_per_matrix": at_ms, "chosen": chosen, "seconds": time.time() - t_at,
                    "candidates": (["dense: panel images by bulk copies", "dense: panel staged through registers",
                                    "dense: one CTA per tile", "HODLR (float-float sampled elements, FP64 factorisation)"]
                                   if args.precision == "mixed" else ["dense Cholesky", "HODLR"])}

    net, train_info = None, None
    args.learned = not args.plain
    if args.learned:
        # trained on small geometries (R/L <= 50) and other Drude metals: the workload's
        # geometry and material are held out of the training data
        from caps_gb300 import learned
        net, train_info = learned.train(seed=0)

    E = None
    for _ in range(args.warmup):
        E, info = caps.free_energy(T, CUTOFF, EPSREL, mlp=net)

    clocks = ClockSampler(local_rank if "CUDA_VISIBLE_DEVICES" not in os.environ else os.environ["CUDA_VISIBLE_DEVICES"].split(",")[0])
    barrier(dist)
    cg.counters(reset=True)
    cg.reset_timings()
    cg.kernel_timing(True)
    clocks.start()
    t0 = time.time()
    infos = []
    for _ in range(args.steps):
        E, info = caps.free_energy(T, CUTOFF, EPSREL, mlp=net)
        infos.append(info)
    wall = time.time() - t0
    clk = clocks.stop()
    barrier(dist)
    ctr = cg.counters()
    wk = cg.work()
    ph = cg.timings(cumulative=True)   # device ms per phase, summed over the timed steps
    syrk_ms, syrk_bytes, syrk_n = cg.kernel_stats(0)
    panel_kernels = {}
    for kind, name in ((1, "k_trsm_inv (panel solve; writes the FP16 panel images)"),
                       (2, "k_potf2_w (64 x 64 diagonal block and its inverse, one CTA per matrix)")):
        ms_, by_, n_ = cg.kernel_stats(kind)
        if n_:
            panel_kernels[name] = {"launches": n_, "ms_per_step": ms_ / args.steps, "algorithmic_GBps": by_ / (ms_ * 1e-3) / 1e9,
                                   "avg_launch_us": ms_ / n_ * 1e3}
    cg.kernel_timing(False)

    ndet = sum(i["ndet"] for i in infos)
    nset = sum(i["ndet"] - i["nwasted"] for i in infos)   # matrices of the reference's set
    dev_s = ph[5] * 1e-3

    ref = load_reference_energy()
    side = {}
    if not args.no_side:
        # the same workload in the other forms (one warm-up, then timed calls), outside the
        # timed region: the plain FP64 GPU form (the metric's denominator) and, for the
        # mixed form, its plain-truncation run, which isolates what the network gains
        names = {"fp64_plain_form": (cg.PREC_FP64, None, 2)}
        if args.learned and args.precision == "mixed":
            names["mixed_plain_form"] = (cg.PREC_MIXED, None, 3)
        for name, (p, n_, calls) in names.items():
            t_, i_, E_, ph_ = time_energy(cg, p, n_, calls)
            side[name] = {"time_to_E_s": t_, "value": (i_["ndet"] - i_["nwasted"]) / (ph_[5] * 1e-3),
                          "matrices_computed": i_["ndet"], "matrices_beyond_cutoffs": i_["nwasted"], "E": E_,
                          "E_rel_err": abs(E_ - ref["E"]) / abs(ref["E"]) if ref else None,
                          "phases_ms": dict(zip(["setup_mie", "K", "I", "elements", "factor", "total"], ph_))}
        if ref is not None and "terms" in ref:
            side["per_matrix_error"] = per_matrix_errors(cg, ref)

    wall_max = allmax(dist, wall)
    dev_max = allmax(dist, dev_s)
    nset_all = allsum(dist, nset)
    if rank != 0:
        return

    value = nset_all / dev_max          # device time (CUDA events on the launching stream)
    e2e = nset_all / wall_max           # wall time of the public API call, host work and copies included
    tte = wall_max / args.steps
    fac_s = ph[4] * 1e-3
    achieved = wk["factor_flops"] / fac_s / 1e12 if fac_s > 0 else None
    hbm_peak, hbm_src = measured_hbm_peak()
    syrk_gbs = syrk_bytes / (syrk_ms * 1e-3) / 1e9 if syrk_ms > 0 else None
    err = abs(E - ref["E"]) / abs(ref["E"]) if ref else None

    cpu = None
    if not args.no_cpu_baseline and ref is not None:
        threads = os.cpu_count() or 1
        nm = args.cpu_sample or 2 * threads
        v, dt, n_, N = cpu_baseline(ref, nm, threads)
        cpu = {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
               "sample": "%d matrices, a systematic sample of the workload's %d (dim 2100), %.1f s on %d host threads, "
                         "oracle port of the reference (C: adaptive Gauss-Legendre K integrals, dense LU)" % (n_, N, dt, threads),
               "projected_time_to_E_s": N / v}

    learned_gain = None
    if train_info is not None and "mixed_plain_form" in side:
        saved = side["mixed_plain_form"]["time_to_E_s"] - tte
        cost = train_info["data_seconds"] + train_info["train_seconds"]
        learned_gain = {"time_to_E_plain_s": side["mixed_plain_form"]["time_to_E_s"], "time_to_E_learned_s": tte,
                        "saved_per_E_s": saved, "speedup": side["mixed_plain_form"]["time_to_E_s"] / tte,
                        "training_cost_s": cost,
                        "break_even_free_energies": (cost / saved) if saved > 0 else None,
                        "held_out": "the workload's geometry (R/L=150) and material (gold) are not in the training data"}

    fp64 = side.get("fp64_plain_form")
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": wall_max / args.steps * 1e3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if args.precision == "fp64" else
                 "f64 (Mie, K, log-factorials, exponents, pivot logs, correction) + float-float q-sums + f32 delta-Cholesky",
        "data": "synthetic (inputs fully set by the geometry/material scalars)",
        "config": workload_config(),
        "method": {"precision": args.precision,
                   "truncation": "learned (MLP proposal, reference rules verify)" if args.learned else "plain (extrapolating schedule)",
                   "matrices_computed_per_step": ndet / args.steps,
                   "matrices_beyond_cutoffs_per_step": (ndet - nset) / args.steps,
                   "parallelism": "replicas" if world > 1 else "single GPU"},
        "time_to_E_s": tte,
        "E": E, "E_reference": ref["E"] if ref else None, "E_rel_err": err,
        "phases_ms_per_step": {k: v / args.steps for k, v in zip(["setup_mie", "K", "I", "elements", "factor", "total"], ph)},
        "roofline": ({"bound": "fp64", "kernel": "Cholesky of the FP64 form (64-bit fixed point, digit products on the tensor cores), "
                                                      "n^3/3 flops per factored matrix against the FP64 pipe that it does without: a fraction "
                                                      "above 1 is what FP64 arithmetic could not reach",
                      "achieved": achieved, "peak": fp64_peak, "unit": "TFLOP/s",
                      "frac": achieved / fp64_peak if achieved else None,
                      "peak_source": "measured live: DFMA-chain probe kernel (caps_gpu_fp64_peak); MEASURED_PEAKS.json has no FP64 figure",
                      "traffic": None} if args.precision == "fp64" else
                     {"bound": "hbm",
                      "kernel": "tcgen05 updates of the FP32 delta-form Cholesky (512-column panels in two 256-column "
                                "halves; panel as FP16 pairs hi + lo of 2^14 x, products hi hi + hi lo + lo hi accumulated "
                                "in FP32 in TMEM; persistent and warp-specialised): k_syrk_pair for the K = 512 update of "
                                "the whole trailing matrix (row-pair items sharing the column slice) and for the middle "
                                "update of each panel (its first half onto the second half's 256 columns), k_syrk_blk for "
                                "the left-looking block updates, all fed by bulk copies of the panel images that the panel "
                                "solves write, over the items whose image blocks are not zero; algorithmic bytes = the tiles of "
                                "S that those items read + write (FP32), counted by the kernels",
                      "achieved": syrk_gbs, "peak": hbm_peak, "unit": "GB/s",
                      "frac": syrk_gbs / hbm_peak if syrk_gbs else None,
                      "traffic": None,
                      "peak_source": hbm_src,
                      "launches": syrk_n, "avg_launch_ms": syrk_ms / syrk_n if syrk_n else None,
                      "algorithmic_bytes_per_launch": syrk_bytes / syrk_n if syrk_n else None,
                      "traffic_source": "not measured at this size: ncu starts each launch with a clean L2 and ends it before "
                                        "the stores leave L2 (42 matrices of this workload: 1.05 DRAM bytes read and none "
                                        "written per byte counted here, about half of them panel images)",
                      "fp32_accurate_tflops_factorisation": achieved,
                      "panel_kernels": panel_kernels or None,
                      "panel_kernels_note": "the panel solve is bytes-bound like the update (its rate against the same peak); "
                                            "the diagonal block is latency-bound: a dependent factorisation and inverse "
                                            "per 64 x 64 block"}),
        "dominant_kernel": None if args.precision == "fp64" else {
            "kernel": "the FP32 delta-form factorisation (k_syrk_pair and k_syrk_blk, the roofline kernels above, with the panel "
                      "kernels k_trsm_inv and k_potf2_w)", "phase_share_of_step": ph[4] / ph[5] if ph[5] else None,
            "bound": "HBM for the trailing update; the panel solve streams the panel, the diagonal block is latency-bound",
            "evidence": "roofline and panel_kernels above; ncu captures of k_syrk_pair and k_syrk_blk on a 24-matrix case"},
        "assembly_kernel": None if args.precision == "fp64" else {
            "kernel": "k_rec_ff and k_elem_sweep (I table by the three-term Legendre recurrence from 4L seed q-sums; "
                      "elements from its tiles, straight into the FP32 delta matrix)",
            "phase_share_of_step": (ph[2] + ph[3]) / ph[5] if ph[5] else None,
            "bound": "issue and latency: the rows' chain of float-float sums and a barrier per row; 256 instructions per "
                     "pair of the elements at 48 % issue",
            "evidence": "ncu capture of both kernels on 40 matrices of this workload"},
        "cpu_baseline": cpu,
        "autotune": autotune,
        "learned_training": train_info,
        "learned_gain": learned_gain,
        "fp64_plain_form": fp64,
        "mixed_plain_form": side.get("mixed_plain_form"),
        "per_matrix_error": side.get("per_matrix_error"),
        "time_to_E_speedup_vs_fp64_plain": (fp64["time_to_E_s"] / tte) if fp64 else None,
        "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": ctr["h2d"] / args.steps, "d2h_bytes_per_step": ctr["d2h"] / args.steps},
        "gpu_launches": ctr["launches"],
        "clocks": clk,
    }
    print(json.dumps(line), flush=True)
    if dist is not None:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
