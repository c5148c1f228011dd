"""Headline benchmark: two-site TEBD updates per second on one GB300.

Workload (the plain-FP64 GPU configuration): Bose-Hubbard chain L=64, maxFilling=4
(d=5), J=1, U=2, mu=0, open boundaries, 2nd-order Trotter, dt=0.005, chi=128,
complex128 Gammas/Lambdas.  Initial state: unit-filling Mott product state plus a
seeded (seed 1) complex Gaussian perturbation of amplitude 1e-3 on every Gamma
entry, renormalised.  One step = one Trotter step = 95 bond updates (32 odd +
31 even + 32 odd, each sweep batched on the GPU).  Data are synthetic (the
reference has no dataset); the configuration is the one the metric is quoted on.

A bench run is the configured run itself: K Trotter steps from the initial state
(default 20, steps 1..20, about a second of timed work; --steps 200 runs the whole
configuration), after W warm-up steps (default 5) on a copy.
value: updates/s with the chain resident in HBM: CUDA events on the library's
       stream around exactly the K steps (one more event per step gives the
       per-step costs: early steps are cheap, the chain saturates chi = 128 near
       step 50 and the SVD dimension then stays near 600).  Before the timed
       pass (untimed) the autotuner sets the launch shapes on the window's own
       batches, replayed from the initial state (--no-tune-window skips it).
e2e:   the same K steps end to end through the reference-facing C ABI: the chain
       is uploaded from pinned host buffers (tebd_set_gamma/lambda), every step
       passes its gates from host memory and returns the truncation error to the
       host (tebd_trotter_step), and the chain is read back at the end
       (tebd_get_gamma/lambda): the drop-in keeps Gammas/Lambdas resident across
       steps, as a Fortran host calling it would.  Host wall clock, synchronised.
precision_form: the same K steps again with the precision form of the SVD
       (TEBD_SVD_DF), its updates/s, the ratio to the plain FP64 value and the
       largest differences of the final <n_i>, bond energies and entropies
       (the metric's "mixed vs plain FP64 at error <= 1e-8"); --no-precision skips it.
mixed_form: the same K steps in the mixed form (TEBD_SVD_RSVD + tensor-core Theta
       + the trained model), with the same comparisons.
saturated, saturated_random_start, saturated_chi512: batched sweeps over
       saturated bonds (chi = 128 prepared / from a random state, chi = 512) in
       plain FP64, the mixed form and the mixed form without the model (the A/B
       of what the network gains), each with its observable errors and the
       tensor-core products' roofline; --no-saturated / --no-chi512 skip them.
roofline: the window's dominant FP64 kernel by CUDA-event time (the QR route's
       Jacobi or the bidiagonalisation), achieved flops against the measured FP64
       peak; cpu_baseline: the oracle on one core for a bounded sample.
--impl reference: the reference's CPU algorithm (the C restatement in oracle/,
       naive FormTheta/ThetaOperation loops + LAPACK ZGESVD) on all host cores,
       one bond update per core per step.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

L, D, CHI = 64, 5, 128
J, U, MU, DT, ORDER = 1.0, 2.0, 0.0, 0.005, 2
AMP, SEED = 1e-3, 1
UPDATES_PER_STEP = (L // 2) * 2 + (L - 1) // 2  # 32 + 31 + 32 = 95
METRIC = "two-site updates/sec (Trotter steps/sec = value/95)"
SVD_MODES = {"fp64": 0, "df": 5, "rsvd": 6,  # plain FP64 / double-float / randomized (learned-rank) route
             "jacobi": 2, "bidiag": 3, "qrj": 4}  # the FP64 routes forced for every bond (route comparisons)
WORKLOAD = "bose_hubbard_L64_d5_chi128_fp64_trotter2"


def workload(H):
    carray = np.zeros((D, L), complex)
    carray[1, :] = 1.0  # one boson per site (occupation index 2, 1-based)
    gam, lam = H.perturbed_product_state(carray, CHI, AMP, SEED)
    Hb = H.bose_hubbard(L, D, J, U, MU)
    Udt = H.construct_propagators(Hb, DT, ORDER)
    return gam, lam, Udt


# ---------------------------------------------------------------------------
# clocks sampled during the timed region
# ---------------------------------------------------------------------------
REASONS = ["active", "hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]


class ClockSampler:
    def __init__(self, path):
        self.path = path
        self.proc = None

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", "--query-gpu=" + q, "--format=csv,noheader,nounits",
                                          "-lms", "200"], stdout=self.f, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            self.f.close()

    def summary(self):
        if self.proc is None or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        sm, mx, reasons = [], [], set()
        for line in open(self.path):
            p = [x.strip() for x in line.split(",")]
            if len(p) < 9 or not p[1].replace(".", "").isdigit():
                continue
            sm.append(float(p[1]))
            mx.append(float(p[2]))
            for name, v in zip(REASONS[1:], p[5:9]):
                if v.lower() in ("active", "0x1", "1"):
                    reasons.add(name)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


# ---------------------------------------------------------------------------
# CPU legs (the oracle restates the reference's algorithm; checker/baseline only)
# ---------------------------------------------------------------------------
def _cpu_update(args):
    link, gam1, gam2, l0, l1, l2, gate = args
    from oracle import oracle as O

    t0 = time.perf_counter()
    O.two_site_op(gam1, gam2, l0, l1, l2, gate)
    return time.perf_counter() - t0


def cpu_sample(gam, lam, Udt, links, workers):
    """Time bond updates of the first odd sweep; returns (updates/s, wall seconds)."""
    jobs = [(k, gam[k - 1], gam[k], lam[k - 1], lam[k], lam[k + 1], Udt[k - 1]) for k in links]
    t0 = time.perf_counter()
    if workers <= 1:
        for j in jobs:
            _cpu_update(j)
    else:
        import multiprocessing as mp

        with mp.get_context("spawn").Pool(workers) as pool:
            pool.map(_cpu_update, jobs)
    wall = time.perf_counter() - t0
    return len(jobs) / wall, wall


# ---------------------------------------------------------------------------
# replicas (bench.py --gpus N under torchrun): one independent chain per GPU;
# a gloo group serves only the barrier and the max over ranks of the timed
# region -- there is no data-path collective
# ---------------------------------------------------------------------------
def hbm_roofline(traffic_bytes, avg_launch_ms, peaks_path):
    """The dominant kernel on the HBM roofline: its measured DRAM traffic per
    launch over its average launch time, against the measured copy bandwidth of
    this GPU's kind (None when a figure is missing).  k_gebrd is bound by a serial
    chain per column and the integer pipe, so this fraction is far below one; it
    shows how far from memory-bound the kernel is."""
    if not traffic_bytes or not avg_launch_ms or not os.path.exists(peaks_path):
        return None
    try:
        peak = float(json.load(open(peaks_path))["hbm_gbs"])
    except (ValueError, KeyError, TypeError):
        return None
    achieved = traffic_bytes / (avg_launch_ms / 1e3) / 1e9
    return {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
            "traffic": traffic_bytes, "peak_source": "MEASURED_PEAKS.json hbm_gbs (measured copy bandwidth)",
            "kernel": "k_gebrd"}


def replica_env():
    """(rank, world size, local rank) from torchrun's environment; one process without it."""
    return (int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1")),
            int(os.environ.get("LOCAL_RANK", "0")))


def replica_group(world):
    """The gloo process group of N > 1 replicas, None for one process."""
    if world <= 1:
        return None
    import torch.distributed as dist

    dist.init_process_group("gloo")
    return dist


def replica_max(dist, x):
    """Largest value of x over the replicas (the job's time is its slowest rank's)."""
    if dist is None:
        return x
    import torch

    t = torch.tensor([x], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t[0])


def whole_job_rate(world, units_per_replica, ms_max):
    """Units all replicas processed per second of the slowest replica's time."""
    return world * units_per_replica / (ms_max / 1e3)


# the legs beside the headline, and what the line keeps of each
LEGS = ("precision_form", "mixed_form")
SATURATED_LEGS = ("saturated", "saturated_random_start", "saturated_chi512")


def bench_line(out, details):
    """The printed line: the headline with what it has to be judged by, and of the other
    legs their rates.  `out` holds everything (20 kB with the autotuner's tables and the legs'
    rooflines) and goes to the file `details`."""
    keep = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "cpu_baseline")
    line = {k: out[k] for k in keep}
    roof = out["roofline"]
    line["roofline"] = {k: roof[k] for k in ("kernel", "bound", "achieved", "peak", "unit", "frac", "launches",
                                             "avg_launch_ms", "share_of_timed")}
    legs = {}
    for name in LEGS:
        if out.get(name):
            legs[name] = {k: out[name][k] for k in ("value", "speedup_vs_plain_fp64", "within_error_bound")}
    for name in SATURATED_LEGS:
        if out.get(name):
            legs[name] = {form: round(leg["value"], 2) for form, leg in out[name].items()
                          if isinstance(leg, dict) and leg.get("unit") == "updates/s"}
    if legs:
        line["legs_updates_per_s"] = legs
    line["details"] = details
    return line


def run_reference(args):
    rank = replica_env()[0]
    if rank != 0:  # under torchrun rank 0 alone times the host-core reference
        return
    os.environ.setdefault("OPENBLAS_NUM_THREADS", "1")
    import __graft_entry__ as ge

    H = ge.load_package().hamiltonians
    from oracle import oracle as O

    O.build()
    gam, lam, Udt = workload(H)
    cores = os.cpu_count() or 1
    links = list(range(1, L, 2))[: max(1, min(cores, L // 2))]
    import multiprocessing as mp

    jobs = [(k, gam[k - 1], gam[k], lam[k - 1], lam[k], lam[k + 1], Udt[k - 1]) for k in links]
    # A bounded number of rounds (sized from the warm-up to ~90 s) of the first odd
    # sweep's bonds of the initial state.  ZGESVD('A','A') always runs on the full
    # 640 x 640 Theta, but its iterations converge fastest on this nearly product
    # state, so this rate overstates the reference's average over the run (the
    # default GPU run's cpu_baseline times two saturated bonds of the final state).
    with mp.get_context("spawn").Pool(len(links)) as pool:
        tw = time.perf_counter()
        for _ in range(max(1, args.warmup)):
            pool.map(_cpu_update, jobs)
        t_round = (time.perf_counter() - tw) / max(1, args.warmup)
        rounds = max(1, min(args.steps, int(90.0 / max(t_round, 1e-3))))
        t0 = time.perf_counter()
        for _ in range(rounds):
            pool.map(_cpu_update, jobs)
        wall = time.perf_counter() - t0
    value = len(links) * rounds / wall
    sample = ("%d rounds of %d concurrent bond updates (links %s of the first odd sweep, d=5, chi=128, "
              "one process per core, OpenBLAS 1 thread each) on the initial state, where ZGESVD "
              "converges fastest" % (rounds, len(links), ",".join(map(str, links[:4])) + ",..."))
    out = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "updates/s", "n_gpus": args.gpus,
        "steps": args.steps, "timed_rounds": rounds, "warmup": args.warmup, "ms_per_step": wall / rounds * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "c128 (f64)",
        "data": "synthetic", "config": {"workload": WORKLOAD, "L": L, "d": D, "chi": CHI, "dt": DT,
                                        "trotter_order": ORDER, "parallelism": "host cores",
                                        "timed_window": "bond updates of the first odd sweep of the initial "
                                                        "state, repeated; the GPU arm times Trotter steps 1..K "
                                                        "of the run, whose Thetas are the same 640 x 640 size "
                                                        "but entangle, so ZGESVD converges slower there: this "
                                                        "arm's rate overstates the reference on that window"},
        "cpu_baseline": {"value": value, "unit": "updates/s", "cores": len(links), "kind": "port",
                         "sample": sample},
        "e2e": {"value": value, "unit": "updates/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(out), flush=True)


# ---------------------------------------------------------------------------
# the mixed form's trained model and the saturated-bond legs
# ---------------------------------------------------------------------------
MODEL_PATH = os.path.join(ROOT, "opentebd-extended_gb300", "data", "rsvd_model.npz")
MODEL_TARGET = 1e-10


def load_model(pkg, device):
    """The randomized route's model trained by the package's learned.py on spectra
    of the method's own runs (the parameters committed beside it)."""
    m = pkg.Mlp(device=device)
    m.set_params(np.load(MODEL_PATH)["params"])
    return m


def measured_peak(key):
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        return float(json.load(open(path))[key]), "MEASURED_PEAKS.json " + key
    except (OSError, ValueError, KeyError, TypeError):
        return ({"hbm_gbs": 6800.0, "bf16_tflops": 1900.0, "bf16_tflops_sustained": 1700.0}[key],
                "fallback figure (no MEASURED_PEAKS.json)")


def saturated_state(Ls=L, chi=CHI, decay=16.0, d=D):
    """Every Lambda full (lambda_k ~ exp(-k/decay), normalised) and complex Gaussian
    Gammas (seed 5): each odd bond of the d=5 chain has a full (5 chi) x (5 chi)
    Theta -- at L=64, chi=128 the cost regime of the configured run after step ~50."""
    rng = np.random.default_rng(5)
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(Ls)]
    lam = []
    for _ in range(Ls + 1):
        l = np.exp(-np.arange(chi) / decay)
        lam.append(l / np.linalg.norm(l))
    return gam, lam


def saturated_legs(pkg, device, args, fp64_peak, steps=3, Ls=L, chi=CHI, decay=16.0, prepare=True,
                   tune=("fp64", "mixed", "mixed_without_model")):
    """The odd bonds of a saturated chain, updated `steps` times (one batched sweep
    each), in plain FP64 and in the mixed form, profiled: updates/s from CUDA events
    on each chain's stream, and the roofline of each form's dominant kernel from
    that leg's own launch timings (k_gebrd's 64-bit flops against the FP64 peak; the tensor-core
    product kernels against the measured bf16 peak).

    prepare: the legs start from the random state after one sweep of the same
    bonds (double-float form).  Every update of a Trotter run meets a state whose
    Schmidt rank across the bond is at most chi (the bond was truncated at its
    last update, and the gates since then act on other bonds), so that Theta's
    spectrum beyond chi comes from the one gate; the prepared state has that
    property.  Without it each Theta of the random state is full rank and the
    sweep discards a large weight -- a harder case than any step of a run.

    tune: the legs whose chain runs the autotuner (tebd_autotune) on the batch
    before it is timed; its default and tuned batch times are reported."""
    import torch

    H = pkg.hamiltonians
    gam, lam = saturated_state(Ls, chi, decay)
    gate = H.matrix_exponential(H.bose_hubbard(Ls, D, J, U, MU)[1], DT)
    links = list(range(1, Ls, 2))
    if prepare:
        with pkg.Chain(Ls, D, chi, device=device, svd_mode=SVD_MODES["df"]) as c:
            c.set_state(gam, lam)
            c.apply_bonds(links, [gate] * len(links))
            gam, lam = c.get_state()
    bf16_peak, bf16_src = measured_peak("bf16_tflops")
    bf16_sus, sus_src = measured_peak("bf16_tflops_sustained")
    n = D * chi
    out = {"workload": "saturated_bonds_L%d_d5_chi%d (%d bonds of a %d x %d Theta per step, lambda_k ~ exp(-k/%g))"
                       % (Ls, chi, len(links), n, n, decay), "steps": steps,
           "start": ("random state after one sweep of the same bonds (Schmidt rank chi across each bond, "
                     "as at every update of a run)" if prepare else
                     "random state: full-rank Theta, large discarded weight (harder than any step of a run)")}
    finals = {}
    # "mixed_without_model": the A/B leg -- the same form with the library's fixed
    # sketch (tebd_set_rsvd defaults, p = 64, q = 2) instead of the network's choice
    for name in ("fp64", "mixed", "mixed_without_model"):
        c = pkg.Chain(Ls, D, chi, device=device, svd_mode=SVD_MODES["fp64" if name == "fp64" else "rsvd"])
        model = None
        if name != "fp64":
            c.set_theta_form(107)
        if name == "mixed":
            model = load_model(pkg, device)
            c.set_rsvd_model(model, MODEL_TARGET)
        c.set_state(gam, lam)
        st_ = torch.cuda.ExternalStream(c.stream(), device=device)
        c.apply_bonds(links, [gate] * len(links))  # warm-up (workspaces, kernels)
        c.set_state(gam, lam)
        tuned = None
        if name in tune:  # untimed: the chain is left as it was
            b_ms, t_ms = c.autotune(links, [gate] * len(links))
            tuned = {"default_batch_ms": b_ms, "tuned_batch_ms": t_ms}
        c.reset_stats()
        c.set_profiling(True)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record(st_)
        for _ in range(steps):
            c.apply_bonds(links, [gate] * len(links))
        e1.record(st_)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        st = c.stats()
        num = np.diag(np.arange(D, dtype=float))
        finals[name] = ([c.two_site_rho(k) for k in links],  # device observables of the updated bonds
                        c.one_site_expval(num), c.local_energy(H.bose_hubbard(Ls, D, J, U, MU)))
        leg_ = {"ms_per_step": ms / steps, "value": len(links) * steps / (ms / 1e3), "unit": "updates/s",
                "autotune": tuned}
        if st["gebrd_ms"] > 0:
            a = st["gebrd_flops"] / (st["gebrd_ms"] / 1e3) / 1e12
            leg_["roofline_k_gebrd"] = {"bound": "fp64", "achieved": a, "peak": fp64_peak, "unit": "TFLOP/s",
                                        "frac": a / fp64_peak, "share_of_leg": st["gebrd_ms"] / ms,
                                        "algorithmic": "16 M N^2 - 16 N^3/3 per bidiagonalised matrix"}
        if st["tc_ms"] > 0:
            a = st["tc_mma_flops"] / (st["tc_ms"] / 1e3) / 1e12
            leg_["roofline_tensor_products"] = {
                "kernels": "k_tc_oz (bf16 digit-plane products)", "bound": "tensor", "achieved": a,
                "peak": bf16_peak, "unit": "TFLOP/s", "frac": a / bf16_peak, "peak_source": bf16_src,
                "frac_of_sustained": a / bf16_sus, "sustained_peak": bf16_sus, "sustained_source": sus_src,
                "launches": st["tc_launches"], "avg_launch_ms": st["tc_ms"] / max(1, st["tc_launches"]),
                "share_of_leg": st["tc_ms"] / ms,
                "algorithmic": "digit pairs x 2 x m_pad x n_pad x k_pad per product (bf16 multiply-adds issued)",
                "fp64_class_flops_per_s": st["rsvd_flops"] / (st["tc_ms"] / 1e3) / 1e12}
            leg_["rsvd"] = {"updates": st["rsvd_updates"], "fallbacks": st["rsvd_fallbacks"],
                            "skipped_by_model": st["rsvd_skipped"], "worst_residual": st["rsvd_worst_residual"],
                            "mean_oversample": st["rsvd_oversample_sum"] / max(1, st["rsvd_batches"]),
                            "mean_power_iters": st["rsvd_power_sum"] / max(1, st["rsvd_batches"]),
                            "retries": st["rsvd_retries"]}
        out[name] = leg_
        c.close()
        if model is not None:
            model.close()
    out["speedup_mixed_vs_fp64"] = out["fp64"]["ms_per_step"] / out["mixed"]["ms_per_step"]
    (r0, n0, e0), (r1, n1, e1) = finals["fp64"], finals["mixed"]
    out["max_abs_err_rho2_vs_fp64"] = float(max(np.max(np.abs(a - b)) for a, b in zip(r0, r1)))
    out["max_abs_err_vs_plain_fp64"] = {"n_i": float(np.max(np.abs(n1 - n0))),
                                        "bond_energy": float(np.max(np.abs(e1 - e0)))}
    out["within_error_bound"] = max(out["max_abs_err_vs_plain_fp64"].values()) <= 1e-8
    (r2, n2, e2) = finals["mixed_without_model"]
    out["ab_model"] = {
        "what": "the mixed form with the trained network choosing the sketch (mixed) against the same form with "
                "the fixed default sketch p = 64, q = 2 (mixed_without_model)",
        "speedup_from_model": out["mixed_without_model"]["ms_per_step"] / out["mixed"]["ms_per_step"],
        "max_abs_err_vs_plain_fp64_without_model": {"n_i": float(np.max(np.abs(n2 - n0))),
                                                    "bond_energy": float(np.max(np.abs(e2 - e0)))}}
    return out


# ---------------------------------------------------------------------------
# GPU arm
# ---------------------------------------------------------------------------
def window_autotune(pkg, chain, gam, lam, Udt, steps, every=4):
    """Autotune (tebd_autotune) the odd and the even sweep of every `every`-th
    Trotter step of the timed window, replayed from the initial state on the same
    chain: the compacted Theta grows step by step, and each tuned batch fills the
    table entries of its size; the chain is left at the replayed state and the
    timed pass uploads the initial state again.  Returns the tuned batches'
    default and tuned times."""
    odd, even = list(range(1, L, 2)), list(range(2, L, 2))
    chain.set_state(gam, lam)
    out = []
    for k in range(1, steps + 1):
        if k % every == 0 or k == steps:
            for links in (odd, even):
                b_ms, t_ms = chain.autotune(links, [Udt[i - 1] for i in links])
                out.append({"step": k, "bonds": len(links), "default_ms": b_ms, "tuned_ms": t_ms})
        chain.trotter_step(Udt, ORDER)
    return out


def run_ours(args):
    import torch

    rank, world, local = replica_env()
    dist = replica_group(world)  # independent replicas, one per GPU; gloo only for barrier/max
    torch.cuda.set_device(local)
    import __graft_entry__ as ge

    ge.build() if rank == 0 else None
    if dist is not None:
        dist.barrier()
    pkg = ge.load_package()
    H = pkg.hamiltonians
    gam, lam, Udt = workload(H)
    fp64_peak = pkg.measure_fp64_peak(local)

    chain = pkg.Chain(L, D, CHI, device=local, svd_mode=SVD_MODES[args.svd])
    chain.set_state(gam, lam)
    stream = torch.cuda.ExternalStream(chain.stream(), device=local)

    def barrier():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()

    def maxall(x):
        return replica_max(dist, x)

    # warm-up on the same chain; the timed pass then uploads the initial state
    # again, so that the timed K steps are steps 1..K of the configured run (the
    # update's cost grows with the Schmidt rank as the state entangles)
    for _ in range(args.warmup):
        chain.trotter_step(Udt, ORDER)
    tune_window = None
    if not args.no_tune_window:  # untimed: tune the launch shapes on the window's own batches
        tune_window = window_autotune(pkg, chain, gam, lam, Udt, args.steps)

    # host-side inputs of the end-to-end path: the initial chain in pinned memory
    # (Fortran order, as the reference holds it) and the gates
    pin_g = [torch.empty((CHI, D, CHI)[::-1], dtype=torch.complex128, pin_memory=True).numpy().T
             for _ in range(L)]
    pin_l = [torch.empty(CHI, dtype=torch.float64, pin_memory=True).numpy() for _ in range(L + 1)]
    for a, b in zip(pin_g, gam):
        a[...] = b
    for a, b in zip(pin_l, lam):
        a[...] = b
    gates = [np.asfortranarray(g, dtype=np.complex128) for g in Udt]
    state_bytes = sum(a.nbytes for a in pin_g) + sum(a.nbytes for a in pin_l)
    # per step: odd sweep, even sweep, odd sweep (order 2)
    gate_bytes = sum(Udt[k].nbytes for k in range(L - 1)) + sum(Udt[k].nbytes for k in range(0, L - 1, 2))

    chain.reset_stats()
    chain.set_profiling(True)
    launches0 = chain.kernel_launches()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    te_total = 0.0
    barrier()
    with ClockSampler(os.path.join(args.outdir, "clocks.csv")) as clk:
        t0 = time.perf_counter()
        for s in range(1, L + 1):
            chain.set_gamma(s, pin_g[s - 1])
        for l in range(1, L + 2):
            chain.set_lambda(l, pin_l[l - 1])
        evs[0].record(stream)
        for k in range(args.steps):
            te_total += chain.trotter_step(gates, ORDER)
            evs[k + 1].record(stream)
        for s in range(1, L + 1):
            chain.get_gamma_into(s, pin_g[s - 1])
        for l in range(1, L + 2):
            chain.get_lambda_into(l, pin_l[l - 1])
        torch.cuda.synchronize()
        e2e_wall = time.perf_counter() - t0
        barrier()
    step_ms = [evs[k].elapsed_time(evs[k + 1]) for k in range(args.steps)]
    if args.save_obs:  # final-state observables on the device, for comparing SVD modes
        num = np.diag(np.arange(D, dtype=float))
        Hb = H.bose_hubbard(L, D, J, U, MU)
        np.savez(args.save_obs, n=chain.one_site_expval(num), e=chain.local_energy(Hb),
                 lam=np.array(chain.get_state()[1]), ent=chain.chain_entropy(), step_ms=np.array(step_ms))
    ms = maxall(sum(step_ms))
    e2e_ms = maxall(e2e_wall * 1e3)
    launches = chain.kernel_launches() - launches0
    st = chain.stats()
    chain.set_profiling(False)
    state_g, state_l = pin_g, pin_l
    value = whole_job_rate(world, UPDATES_PER_STEP * args.steps, ms)
    e2e = whole_job_rate(world, UPDATES_PER_STEP * args.steps, e2e_ms)
    h2d = gate_bytes + state_bytes / args.steps
    d2h = 8 * UPDATES_PER_STEP + 16 * 3 + state_bytes / args.steps
    sat = step_ms[49:] if args.steps > 60 else []
    phases = {"ms_per_step_steps_1_20": sum(step_ms[:20]) / min(20, args.steps),
              "ms_per_step_steps_50_end": (sum(sat) / len(sat)) if sat else None,
              "ms_step_1": step_ms[0], "ms_step_last": step_ms[-1]}

    # ---- precision form beside the plain FP64 run (the metric's "mixed vs plain") --
    num = np.diag(np.arange(D, dtype=float))
    Hb = H.bose_hubbard(L, D, J, U, MU)
    ref_obs = (chain.one_site_expval(num), chain.local_energy(Hb), chain.chain_entropy())

    def leg(svd_mode, bound=0.0, mixed=False):
        """The same K steps from the initial state on a second chain: updates/s from
        CUDA events on its stream, and final-state observable errors against the
        plain FP64 run.  mixed: the mixed form (Theta in 7 digit planes on the
        tensor cores, the trained model on the randomized route), profiled."""
        pc = pkg.Chain(L, D, CHI, device=local, svd_mode=svd_mode)
        pc.set_rank_bound(bound)
        model = None
        if mixed:
            pc.set_theta_form(107)
            model = load_model(pkg, local)
            pc.set_rsvd_model(model, MODEL_TARGET)
        pc.set_state(gam, lam)
        for _ in range(args.warmup):
            pc.trotter_step(Udt, ORDER)
        if not args.no_tune_window:  # the same untimed tuning as the plain run's
            window_autotune(pkg, pc, gam, lam, Udt, args.steps)
        pc.set_state(gam, lam)
        pstream = torch.cuda.ExternalStream(pc.stream(), device=local)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        pc.reset_stats()
        barrier()
        e0.record(pstream)
        te = 0.0
        for _ in range(args.steps):
            te += pc.trotter_step(Udt, ORDER)
        e1.record(pstream)
        barrier()
        pms = maxall(e0.elapsed_time(e1))
        pst = pc.stats()
        o = (pc.one_site_expval(num), pc.local_energy(Hb), pc.chain_entropy())
        ranks = [int(np.sum(x > 0)) for x in pc.get_state()[1][1:-1]]
        pc.close()
        if model is not None:
            model.close()
        pv = whole_job_rate(world, UPDATES_PER_STEP * args.steps, pms)
        err = {"n_i": float(np.max(np.abs(o[0] - ref_obs[0]))),
               "bond_energy": float(np.max(np.abs(o[1] - ref_obs[1]))),
               "entropy": float(np.max(np.abs(o[2] - ref_obs[2])))}
        out = {"value": pv, "unit": "updates/s", "ms_per_step": pms / args.steps,
               "speedup_vs_plain_fp64": pv / value, "max_abs_err_vs_plain_fp64": err,
               "within_error_bound": max(err.values()) <= 1e-8, "error_bound": 1e-8,
               "total_truncerr": te, "final_mean_rank": float(np.mean(ranks))}
        if svd_mode == SVD_MODES["rsvd"]:
            out["rsvd"] = {"updates": pst["rsvd_updates"], "fallbacks": pst["rsvd_fallbacks"],
                           "skipped_by_model": pst["rsvd_skipped"], "worst_residual": pst["rsvd_worst_residual"]}
        return out

    prec = None
    if args.svd == "fp64" and not args.no_precision:
        prec = {"svd": "TEBD_SVD_DF: the gate and small Thetas in double-float on the FP32 pipe; the SVD as "
                       "in plain FP64"}
        prec.update(leg(SVD_MODES["df"]))
    mixed = None
    if args.svd == "fp64" and not args.no_precision:
        mixed = {"form": "TEBD_SVD_RSVD + tebd_set_theta_form(107) + trained model (target %g): Theta and the "
                         "randomized route's products on the tensor cores (bf16 digit planes, FP64 class), FP64 "
                         "Cholesky / s x s SVD, full FP64 SVD for the bonds the model or the judge sends "
                         "back" % MODEL_TARGET}
        mixed.update(leg(SVD_MODES["rsvd"], mixed=True))
    rank_form = None
    if args.svd == "fp64" and args.rank_bound:
        rank_form = []
        for b in args.rank_bound:
            for nm in ("fp64", "df"):
                r = {"rank_bound": b, "svd": nm}
                r.update(leg(SVD_MODES[nm], b))
                rank_form.append(r)

    # ---- CPU baseline: the oracle port on a bounded sample ------------------
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        os.environ.setdefault("OPENBLAS_NUM_THREADS", "1")
        links = [L // 2 - 1, L // 2 + 1, L // 2 - 3, L // 2 + 3][: args.cpu_updates]  # interior bonds
        v, wall = cpu_sample(state_g, state_l, Udt, links, 1)
        cpu = {"value": v, "unit": "updates/s", "cores": 1, "kind": "port",
               "sample": "%d bond updates (links %s of an odd sweep) of the timed chain, d=5, chi=128: "
                         "C restatement of TwoSiteOp_c (naive loops) + LAPACK ZGESVD, 1 thread, %.1f s"
                         % (len(links), ",".join(map(str, links)), wall)}

    # ---- roofline of the dominant kernel (FP64 pipe): the bidiagonalisation when
    # the window's batches take the bidiagonal route, else the QR route's Jacobi --
    def fp64_roof(kernel, t_ms, flops, launches, algorithmic):
        nl = max(1, launches)
        achieved = flops / (t_ms / 1e3) / 1e12 if t_ms > 0 else None
        return {"kernel": kernel, "bound": "fp64", "achieved": achieved, "peak": fp64_peak, "unit": "TFLOP/s",
                "frac": (achieved / fp64_peak) if achieved else None, "traffic": None,
                "peak_source": "measured FP64 FMA throughput of this GPU (tebd_measure_fp64_peak); "
                               "MEASURED_PEAKS.json carries no FP64 figure",
                "algorithmic": algorithmic, "flops_per_launch": flops / nl, "launches": launches,
                "avg_launch_ms": t_ms / nl, "share_of_timed": t_ms / ms if ms > 0 else None,
                "traffic_source": "not measured for this window: DRAM traffic comes only from an ncu capture, "
                                  "never from a run that is timed"}

    gebrd_roof = fp64_roof("k_gebrd", st["gebrd_ms"], st["gebrd_flops"], st["gebrd_launches"],
                           "16 M N^2 - 16 N^3/3 real flops per bond (complex Householder bidiagonalisation, "
                           "M >= N)")
    jacobi_roof = fp64_roof("k_jacobi_persistent<double>", st["jacobi_ms"], st["jacobi_flops"],
                            st["jacobi_launches"],
                            "counted on the device: 16 m per visited column pair (three complex dot products "
                            "over m rows) + 20 (m + n) per rotated pair (the 2 x 2 rotation of X's and V's "
                            "columns)")
    roof = dict(gebrd_roof if st["gebrd_ms"] >= st["jacobi_ms"] else jacobi_roof)
    roof["bidiag_route_share_of_timed"] = st["bidiag_ms"] / ms if ms > 0 else None
    roof["qr_route_share_of_timed"] = (st["jacobi_ms"] + st["qr_ms"]) / ms if ms > 0 else None
    roof["other"] = jacobi_roof if roof["kernel"] == "k_gebrd" else gebrd_roof
    clocks = clk.summary()
    out = {
        "metric": METRIC, "value": value, "unit": "updates/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "c128 (f64; gate and small Thetas in double-float)" if args.svd == "df" else "c128 (f64)",
        "data": "synthetic",
        "config": {"workload": WORKLOAD, "L": L, "d": D, "chi": CHI, "J": J, "U": U, "mu": MU, "dt": DT,
                   "trotter_order": ORDER, "updates_per_step": UPDATES_PER_STEP,
                   "svd": ("fp64 per bond: Householder bidiagonalisation in 64-bit fixed point + bisection + "
                           "inverse iteration (batches holding a saturated bond or one above 384 columns), else "
                           "pivoted QR + QR of R^H + one-sided Jacobi"
                           if args.svd == "fp64" else "svd_mode %s for every bond" % args.svd),
                   "timed_window": "Trotter steps 1..%d of the configured 200-step run (warm-up on a copy)" % args.steps,
                   "bidiag_updates": st["bidiag_updates"], "updates": st["updates"],
                   "mean_svd_cols": st["compact_cols"] / max(1, st["updates"]),
                   "parallelism": "replicas" if world > 1 else "single GPU",
                   "l2": "no flush: per-step working set (64 Gammas 84 MB + 32 SVD slots ~1 GB) exceeds the 129 MB L2"},
        "phases": phases,
        "steps_per_sec": value / UPDATES_PER_STEP,
        "total_truncerr_timed": te_total,
        "e2e": {"value": e2e, "unit": "updates/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                "steps": args.steps, "path": "tebd_set_gamma/lambda + tebd_trotter_step (host gates) + "
                                              "tebd_get_gamma/lambda, host wall clock"},
        "gpu_launches": launches,
        "window_autotune": tune_window,
        "roofline": roof,
        "roofline_hbm": hbm_roofline(roof["traffic"], roof["avg_launch_ms"],
                                     os.path.join(ROOT, "MEASURED_PEAKS.json")),
        "cpu_baseline": cpu,
        "precision_form": prec,
        "mixed_form": mixed,
        "saturated": (saturated_legs(pkg, local, args, fp64_peak)
                      if not args.no_precision and not args.no_saturated else None),
        "saturated_random_start": (saturated_legs(pkg, local, args, fp64_peak, prepare=False, tune=())
                                   if not args.no_precision and not args.no_saturated else None),
        "saturated_chi512": (saturated_legs(pkg, local, args, fp64_peak, steps=1, Ls=32, chi=512, decay=64.0,
                                            tune=("mixed", "mixed_without_model"))
                             if not args.no_precision and not args.no_saturated and not args.no_chi512 else None),
        "autotune_table": pkg.get_tuning(local) if not args.no_precision else None,
        **({"rank_form": {"what": "kept-rank form: per-update discarded-weight bound "
                                  "(tebd_set_rank_bound), Lambda beyond the kept rank exactly zero",
                          "legs": rank_form}} if rank_form else {}),
        "clocks": clocks,
    }
    if rank == 0:
        details = os.path.join(args.outdir, "bench_details.json")
        with open(details, "w") as f:
            json.dump(out, f, indent=1)
        print(json.dumps(bench_line(out, os.path.relpath(details, ROOT))), flush=True)
    chain.close()
    if dist is not None:
        dist.destroy_process_group()


# ---------------------------------------------------------------------------
# number-conserving workload (extra line, not the headline): Bose-Hubbard
# L=128, d=5, chi=512, U_i ~ U[1,3] (seed 3), unit-filling Mott state from
# InitialSetNC, dt=0.01, 2nd order, TrotterStepNC
# ---------------------------------------------------------------------------
NC_L, NC_D, NC_CHI, NC_N, NC_DT = 128, 5, 512, 128, 0.01


def run_nc(args):
    import torch

    import __graft_entry__ as ge

    ge.build()
    pkg = ge.load_package()
    H = pkg.hamiltonians
    gam, lam, ll, lr = H.initial_set_nc(NC_L, NC_D, NC_CHI, NC_N)
    Uvec = np.random.default_rng(3).uniform(1.0, 3.0, NC_L)
    Hb = H.bose_hubbard(NC_L, NC_D, 1.0, Uvec)
    Udt = H.construct_propagators(Hb, NC_DT, 2)
    num = np.diag(np.arange(NC_D, dtype=float))
    per_step = NC_L - 1 + (NC_L // 2)  # 64 + 63 + 64

    def run(svd_mode, theta_form=0):
        chain = pkg.Chain(NC_L, NC_D, NC_CHI, mode=pkg.MODE_NC, tot_num=NC_N, svd_mode=svd_mode)
        chain.set_theta_form(theta_form)
        chain.set_state(gam, lam, ll, lr)
        stream = torch.cuda.ExternalStream(chain.stream())
        for _ in range(args.warmup):
            chain.trotter_step(Udt, 2)
        chain.set_state(gam, lam, ll, lr)
        chain.reset_stats()
        chain.set_profiling(True)
        evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
        torch.cuda.synchronize()
        evs[0].record(stream)
        for k in range(args.steps):
            chain.trotter_step(Udt, 2)
            evs[k + 1].record(stream)
        torch.cuda.synchronize()
        step_ms = [evs[k].elapsed_time(evs[k + 1]) for k in range(args.steps)]
        st = chain.stats()
        lam_end = chain.get_state()[1]
        obs = (chain.one_site_expval(num), chain.local_energy(Hb), chain.chain_entropy())
        chain.close()
        return step_ms, st, lam_end, obs

    step_ms, st, lam_end, ref_obs = run(SVD_MODES[args.svd], args.theta_form)
    ms = sum(step_ms)
    value = per_step * args.steps / (ms / 1e3)
    out = {"metric": "two-site updates/sec, number-conserving (TwoSiteOpNC)", "value": value,
           "unit": "updates/s", "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps,
           "svd": args.svd, "theta_form": args.theta_form,
           "config": {"workload": "nc_bose_hubbard_L128_d5_chi512", "L": NC_L, "d": NC_D, "chi": NC_CHI,
                      "tot_num": NC_N, "dt": NC_DT, "U": "uniform[1,3] seed 3", "trotter_order": 2,
                      "timed_window": "steps 1..%d from the Mott state" % args.steps,
                      "blocks": "charge blocks with both sides >= 16 bidiagonalised, the rest grouped Jacobi"},
           "jacobi_ms": st["jacobi_ms"], "gebrd_ms": st["gebrd_ms"], "gebrd_launches": st["gebrd_launches"],
           "gpu_launches": st["kernel_launches"],
           "phases": {"ms_step_1": step_ms[0], "ms_step_last": step_ms[-1],
                      "ms_per_step_last_10": sum(step_ms[-10:]) / min(10, args.steps)},
           "final_rank": {"max": int(max(np.sum(x > 0) for x in lam_end)),
                          "mean": float(np.mean([np.sum(x > 0) for x in lam_end[1:-1]]))}}
    if args.svd == "fp64" and not args.no_precision:
        p_ms, _, _, p_obs = run(SVD_MODES["df"])
        pv = per_step * args.steps / (sum(p_ms) / 1e3)
        err = {"n_i": float(np.max(np.abs(p_obs[0] - ref_obs[0]))),
               "bond_energy": float(np.max(np.abs(p_obs[1] - ref_obs[1]))),
               "entropy": float(np.max(np.abs(p_obs[2] - ref_obs[2])))}
        out["precision_form"] = {"svd": "TEBD_SVD_DF (double-float bidiagonalisation of the large blocks)",
                                 "value": pv, "unit": "updates/s", "speedup_vs_plain_fp64": pv / value,
                                 "max_abs_err_vs_plain_fp64": err, "error_bound": 1e-8,
                                 "within_error_bound": max(err.values()) <= 1e-8}
        m_ms, m_st, _, m_obs = run(SVD_MODES["df"], 107)
        mv = per_step * args.steps / (sum(m_ms) / 1e3)
        err = {"n_i": float(np.max(np.abs(m_obs[0] - ref_obs[0]))),
               "bond_energy": float(np.max(np.abs(m_obs[1] - ref_obs[1]))),
               "entropy": float(np.max(np.abs(m_obs[2] - ref_obs[2])))}
        out["mixed_form"] = {"form": "TEBD_SVD_DF + tebd_set_theta_form(107): the charge blocks' class sums as "
                                     "grouped digit-plane products on the tensor cores, the gate applied in "
                                     "place, double-float bidiagonalisation of the large blocks",
                             "value": mv, "unit": "updates/s", "speedup_vs_plain_fp64": mv / value,
                             "ms_per_step_last_10": sum(m_ms[-10:]) / min(10, args.steps),
                             "theta_products_ms": m_st["tc_ms"], "theta_products_launches": m_st["tc_launches"],
                             "theta_products_share": m_st["tc_ms"] / sum(m_ms),
                             "max_abs_err_vs_plain_fp64": err, "error_bound": 1e-8,
                             "within_error_bound": max(err.values()) <= 1e-8}
    print(json.dumps(out), flush=True)


# ---------------------------------------------------------------------------
# Fermi-Hubbard precision-form configuration (extra line, not the headline):
# spin-1/2 Hubbard chain L=64, d=4, t=1, U=4, mu=0 (half filling), a seeded random
# MPS at chi=256 (complex Gaussian Gammas, seed 2, flat Lambdas) made canonical
# with CanonicalFormAll on the device, then Forest-Ruth steps at dt=0.01.  Every
# bond is a saturated 1024 x 1024 Theta from the first step.  The same K steps run
# in plain FP64 and in the double-float form from the same canonical state;
# observables after K steps are compared.
# ---------------------------------------------------------------------------
FH_L, FH_D, FH_CHI, FH_T, FH_U, FH_DT = 64, 4, 256, 1.0, 4.0, 0.01


def run_fermi(args):
    import torch

    import __graft_entry__ as ge

    ge.build()
    pkg = ge.load_package()
    H = pkg.hamiltonians
    rng = np.random.default_rng(2)
    gam = [np.asfortranarray(rng.standard_normal((FH_CHI, FH_D, FH_CHI)) + 1j * rng.standard_normal((FH_CHI, FH_D, FH_CHI)))
           for _ in range(FH_L)]
    lam = [np.full(FH_CHI, 1.0 / np.sqrt(FH_CHI)) for _ in range(FH_L + 1)]
    lam[0] = np.eye(FH_CHI)[0]
    lam[FH_L] = np.eye(FH_CHI)[0]
    Hb = H.fermi_hubbard(FH_L, FH_T, FH_U)
    Udt = H.construct_propagators(Hb, FH_DT, 5)
    with pkg.Chain(FH_L, FH_D, FH_CHI) as c:
        c.set_state(gam, lam)
        c.canonical_form_all()
        gam, lam = c.get_state()
    _, _, _, nop, _, _ = H.fermi_ops()
    per_step = 4 * (FH_L // 2) + 3 * ((FH_L - 1) // 2)  # 4 odd + 3 even sweeps
    legs = {}
    for nm in ("fp64", "df"):
        chain = pkg.Chain(FH_L, FH_D, FH_CHI, svd_mode=SVD_MODES[nm])
        chain.set_state(gam, lam)
        stream = torch.cuda.ExternalStream(chain.stream())
        chain.trotter_step(Udt, 5)  # warm-up (kernels, workspaces) on the same chain ...
        chain.set_state(gam, lam)   # ... then the timed steps from the canonical state
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record(stream)
        te = 0.0
        for _ in range(args.steps):
            te += chain.trotter_step(Udt, 5)
        e1.record(stream)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        legs[nm] = {"ms": ms, "te": te, "obs": (chain.one_site_expval(nop), chain.local_energy(Hb),
                                                chain.chain_entropy()),
                    "bidiag_updates": chain.stats()["bidiag_updates"]}
        chain.close()
    v = per_step * args.steps / (legs["fp64"]["ms"] / 1e3)
    pv = per_step * args.steps / (legs["df"]["ms"] / 1e3)
    ref, o = legs["fp64"]["obs"], legs["df"]["obs"]
    err = {"n_i": float(np.max(np.abs(o[0] - ref[0]))), "bond_energy": float(np.max(np.abs(o[1] - ref[1]))),
           "entropy": float(np.max(np.abs(o[2] - ref[2])))}
    out = {"metric": "two-site updates/sec, Fermi-Hubbard chi=256 (Forest-Ruth)", "value": v, "unit": "updates/s",
           "steps": args.steps, "ms_per_step": legs["fp64"]["ms"] / args.steps, "svd": "fp64",
           "config": {"workload": "fermi_hubbard_L64_d4_chi256_forest_ruth", "L": FH_L, "d": FH_D, "chi": FH_CHI,
                      "t": FH_T, "U": FH_U, "mu": 0.0, "dt": FH_DT, "trotter_order": 5,
                      "updates_per_step": per_step,
                      "initial": "random MPS chi=256 (seed 2) made canonical with CanonicalFormAll",
                      "timed_window": "Forest-Ruth steps 1..%d" % args.steps},
           "bidiag_updates": legs["fp64"]["bidiag_updates"], "total_truncerr": legs["fp64"]["te"],
           "precision_form": {"svd": "TEBD_SVD_DF", "value": pv, "unit": "updates/s",
                              "speedup_vs_plain_fp64": pv / v, "max_abs_err_vs_plain_fp64": err,
                              "error_bound": 1e-8, "within_error_bound": max(err.values()) <= 1e-8}}
    print(json.dumps(out), flush=True)


# ---------------------------------------------------------------------------
# saturated-bond batch (extra line, not the headline): the cost regime that
# dominates the configured run after step ~50.  The chain (default L=64, d=5,
# chi=128; --sat-L, --sat-d, --sat-chi, --sat-decay) with every Lambda full
# (lambda_k ~ exp(-k/decay), normalised) and complex Gaussian Gammas (seed 5),
# after one sweep of the odd bonds in the double-float form (--random-start
# skips it): each odd bond has a full (d chi) x (d chi) Theta.  One step = one
# batched TwoSiteOp sweep over the odd bonds with the Bose-Hubbard bond gate
# exp(-i dt h) (dt = 0.005).  --svd rsvd loads the trained model as the mixed
# form does.
# ---------------------------------------------------------------------------
def run_saturated(args):
    import torch

    import __graft_entry__ as ge

    ge.build()
    pkg = ge.load_package()
    H = pkg.hamiltonians
    Ls, chi, d = args.sat_L, args.sat_chi, args.sat_d
    gam, lam = saturated_state(Ls, chi, args.sat_decay, d)
    gate = H.matrix_exponential(H.bose_hubbard(Ls, d, J, U, MU)[1], DT)
    links = list(range(1, Ls, 2))
    if not args.random_start:
        with pkg.Chain(Ls, d, chi, svd_mode=SVD_MODES["df"]) as c:
            c.set_state(gam, lam)
            c.apply_bonds(links, [gate] * len(links))
            gam, lam = c.get_state()
    chain = pkg.Chain(Ls, d, chi, svd_mode=SVD_MODES[args.svd])
    chain.set_theta_form(args.theta_form)
    model = None
    if args.svd == "rsvd":  # the mixed form's model sizes the sketches, as in the headline run's legs
        model = load_model(pkg, 0)
        chain.set_rsvd_model(model, MODEL_TARGET)
    chain.set_state(gam, lam)
    stream = torch.cuda.ExternalStream(chain.stream())
    for _ in range(args.warmup):
        chain.apply_bonds(links, [gate] * len(links))
    chain.set_state(gam, lam)
    chain.reset_stats()
    chain.set_profiling(True)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    ev0.record(stream)
    for _ in range(args.steps):
        chain.apply_bonds(links, [gate] * len(links))
    ev1.record(stream)
    torch.cuda.synchronize()
    ms = ev0.elapsed_time(ev1)
    st = chain.stats()
    n = d * chi
    out = {"metric": "two-site updates/sec, saturated bonds (%d x %d Theta)" % (n, n),
           "value": len(links) * args.steps / (ms / 1e3), "unit": "updates/s", "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": ms / args.steps,
           "config": {"workload": "saturated_bonds_L%d_d%d_chi%d" % (Ls, d, chi), "bonds_per_step": len(links),
                      "theta_form": args.theta_form, "decay": args.sat_decay,
                      "start": "random" if args.random_start else "random + one double-float sweep"},
           "gebrd_tflops": st["gebrd_flops"] / (st["gebrd_ms"] / 1e3) / 1e12 if st["gebrd_ms"] > 0 else None,
           "gebrd_share": st["gebrd_ms"] / ms, "bidiag_share": st["bidiag_ms"] / ms,
           "tc_share": st["tc_ms"] / ms, "gpu_launches": st["kernel_launches"],
           "rsvd": {"updates": st["rsvd_updates"], "fallbacks": st["rsvd_fallbacks"],
                    "worst_residual": st["rsvd_worst_residual"], "tc_flops": st["rsvd_flops"],
                    "mean_oversample": st["rsvd_oversample_sum"] / max(1, st["rsvd_batches"]),
                    "mean_power_iters": st["rsvd_power_sum"] / max(1, st["rsvd_batches"])}}
    print(json.dumps(out), flush=True)
    chain.close()
    if model is not None:
        model.close()


# ---------------------------------------------------------------------------
# learned-rank configuration (extra line, not the headline): spin-1 Heisenberg
# chain L=128, J=1, Delta=1, single-ion anisotropy D_i ~ U[-0.5, 0.5] (seed 4),
# from a seeded random MPS at chi=64 (complex Gaussian Gammas, seed 4, made
# canonical on the device) growing to chi_max=1024; 2nd order, dt=0.01; kept
# rank: discarded weight <= 1e-10 per update (tebd_set_rank_bound).  The same
# steps run in plain FP64 and in the learned-rank form (randomized route sized
# by the trained model, Theta on the tensor cores, the full SVD as fallback and
# judge); per-step times and the final observables are compared.  Under the
# 1e-10 bound the first steps keep ~190 values per bond (Thetas up to 576 x 576),
# so the randomized route, which takes saturated bonds only, waits for the
# entanglement to grow; --spin1-steps (default 3) bounds the run (a saturated
# plain-FP64 step of 3072 x 3072 Thetas would take minutes).
# ---------------------------------------------------------------------------
S1_L, S1_D, S1_CHI0, S1_CHI, S1_DT, S1_BOUND = 128, 3, 64, 1024, 0.01, 1e-10


def spin1_state(pkg):
    rng = np.random.default_rng(4)
    g = [np.asfortranarray(rng.standard_normal((S1_CHI0, S1_D, S1_CHI0)) +
                           1j * rng.standard_normal((S1_CHI0, S1_D, S1_CHI0))) for _ in range(S1_L)]
    lm = [np.full(S1_CHI0, 1.0 / np.sqrt(S1_CHI0)) for _ in range(S1_L + 1)]
    lm[0] = np.eye(S1_CHI0)[0]
    lm[S1_L] = np.eye(S1_CHI0)[0]
    with pkg.Chain(S1_L, S1_D, S1_CHI0) as c:
        c.set_state(g, lm)
        c.canonical_form_all()
        g, lm = c.get_state()
    gam, lam = [], []
    for x in g:  # embedded in chi_max storage: the rest exactly zero
        y = np.zeros((S1_CHI, S1_D, S1_CHI), complex, order="F")
        y[:S1_CHI0, :, :S1_CHI0] = x
        gam.append(y)
    for x in lm:
        y = np.zeros(S1_CHI)
        y[:S1_CHI0] = x
        lam.append(y)
    return gam, lam


def run_spin1(args):
    import torch

    import __graft_entry__ as ge

    ge.build()
    pkg = ge.load_package()
    H = pkg.hamiltonians
    Di = np.random.default_rng(4).uniform(-0.5, 0.5, S1_L)
    Hb = H.spin1_xxz_anisotropy(S1_L, 1.0, 1.0, Di)
    Udt = H.construct_propagators(Hb, S1_DT, 2)
    gam, lam = spin1_state(pkg)
    sz = H.spin_ops(1.0)[2]
    per_step = (S1_L // 2) * 2 + (S1_L - 1) // 2
    legs = {}
    for name in ("fp64", "learned"):
        c = pkg.Chain(S1_L, S1_D, S1_CHI, svd_mode=SVD_MODES["fp64" if name == "fp64" else "rsvd"])
        c.set_rank_bound(S1_BOUND)
        model = None
        if name == "learned":
            c.set_theta_form(107)
            model = load_model(pkg, 0)
            c.set_rsvd_model(model, MODEL_TARGET)
        c.set_state(gam, lam)
        c.reset_stats()
        c.set_profiling(True)
        stream = torch.cuda.ExternalStream(c.stream())
        evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.spin1_steps + 1)]
        torch.cuda.synchronize()
        evs[0].record(stream)
        ranks = []
        for k in range(args.spin1_steps):
            c.trotter_step(Udt, 2)
            evs[k + 1].record(stream)
            ranks.append(int(max(np.sum(c.get_lambda(l) > 0) for l in range(2, S1_L + 1))))
        torch.cuda.synchronize()
        step_ms = [evs[k].elapsed_time(evs[k + 1]) for k in range(args.spin1_steps)]
        st = c.stats()
        legs[name] = {"step_ms": step_ms, "max_rank_after_step": ranks,
                      "obs": (c.one_site_expval(sz), c.local_energy(Hb), c.chain_entropy()),
                      "rsvd": {"updates": st["rsvd_updates"], "fallbacks": st["rsvd_fallbacks"],
                               "skipped_by_model": st["rsvd_skipped"],
                               "worst_residual": st["rsvd_worst_residual"]},
                      "tc_share": st["tc_ms"] / max(sum(step_ms), 1e-9)}
        c.close()
        if model is not None:
            model.close()
    f, m = legs["fp64"], legs["learned"]
    v = per_step * args.spin1_steps / (sum(f["step_ms"]) / 1e3)
    mv = per_step * args.spin1_steps / (sum(m["step_ms"]) / 1e3)
    err = {"sz_i": float(np.max(np.abs(m["obs"][0] - f["obs"][0]))),
           "bond_energy": float(np.max(np.abs(m["obs"][1] - f["obs"][1]))),
           "entropy": float(np.max(np.abs(m["obs"][2] - f["obs"][2])))}
    out = {"metric": "two-site updates/sec, spin-1 chi 64 -> 1024 (learned-rank form vs plain FP64)",
           "value": mv, "unit": "updates/s", "steps": args.spin1_steps,
           "config": {"workload": "spin1_anisotropy_L128_d3_chi64_to_1024", "L": S1_L, "d": S1_D,
                      "chi0": S1_CHI0, "chi_max": S1_CHI, "dt": S1_DT, "trotter_order": 2, "J": 1.0, "Delta": 1.0,
                      "D_i": "uniform[-0.5,0.5] seed 4", "rank_bound": S1_BOUND,
                      "initial": "random MPS chi=64 (seed 4) made canonical with CanonicalFormAll"},
           "plain_fp64": {"value": v, "unit": "updates/s", "step_ms": f["step_ms"],
                          "max_rank_after_step": f["max_rank_after_step"]},
           "learned": {"value": mv, "unit": "updates/s", "step_ms": m["step_ms"],
                       "max_rank_after_step": m["max_rank_after_step"], "rsvd": m["rsvd"],
                       "tensor_product_share": m["tc_share"]},
           "speedup_vs_plain_fp64": mv / v, "max_abs_err_vs_plain_fp64": err, "error_bound": 1e-8,
           "within_error_bound": max(err.values()) <= 1e-8}
    print(json.dumps(out), flush=True)


# ---------------------------------------------------------------------------
# tensor-core product micro-benchmark (extra line): one batched complex product
# C_p = A_p B_p through the C ABI (tebd_zgemm_tc) at the randomized route's
# shapes, operands from a seeded normal generator on the device, checked against
# torch's complex128 product; --zgemm-shape NBxMxNxK, --zgemm-form 107 (7 bf16
# digit planes), 3 (3xTF32) or 1 (1xTF32).
# ---------------------------------------------------------------------------
def run_zgemm(args):
    import torch

    import __graft_entry__ as ge

    ge.build()
    pkg = ge.load_package()
    lib = pkg.load_library()
    nb, m, n, k = (int(x) for x in args.zgemm_shape.split("x"))
    g = torch.Generator(device="cuda").manual_seed(0)
    A = torch.randn((nb, k, m), dtype=torch.complex128, device="cuda", generator=g)
    B = torch.randn((nb, n, k), dtype=torch.complex128, device="cuda", generator=g)
    C = torch.zeros((nb, n, m), dtype=torch.complex128, device="cuda")

    def call():
        rc = lib.tebd_zgemm_tc(nb, m, n, k, A.data_ptr(), k * m, m, B.data_ptr(), n * k, k, C.data_ptr(), n * m, m,
                               args.zgemm_form, None)
        if rc:
            raise RuntimeError("tebd_zgemm_tc failed: %d" % rc)

    for _ in range(max(1, args.warmup)):
        call()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    for _ in range(args.steps):
        call()
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / args.steps
    ref = torch.einsum("bkm,bnk->bnm", A, B)
    err = ((C - ref).abs().max() / ref.abs().max()).item()
    f = args.zgemm_form
    mp, np_ = -(-m // 128) * 128, -(-2 * n // 128) * 128
    kp = -(-2 * k // 32) * 32
    pairs = (f - 100) * (f - 99) // 2 if f > 100 else 3 if f == 3 else 1
    mma = pairs * 2.0 * mp * np_ * kp * nb
    print(json.dumps({"metric": "batched complex product through tebd_zgemm_tc (operand packing included)",
                      "shape": args.zgemm_shape, "form": f, "ms_per_call": ms, "calls": args.steps,
                      "fp64_class_tflops": 8.0 * nb * m * n * k / ms / 1e9,
                      "tensor_tflops_issued": mma / ms / 1e9, "rel_err_vs_complex128": err}), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="headline",
                    choices=["headline", "nc", "saturated", "fermi_hubbard", "spin1", "zgemm"])
    ap.add_argument("--zgemm-shape", default="2x2560x640x2560", help="--workload zgemm: NBxMxNxK")
    ap.add_argument("--zgemm-form", type=int, default=107, help="--workload zgemm: 107, 3 or 1")
    ap.add_argument("--spin1-steps", type=int, default=3, help="--workload spin1: Trotter steps per leg")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-tune-window", action="store_true",
                    help="skip autotuning the plain run's launch shapes on the window's batches before timing")
    ap.add_argument("--svd", default="fp64", choices=sorted(SVD_MODES))
    ap.add_argument("--save-obs", default=None, help="write final <n_i>, bond energies, Lambdas (npz)")
    ap.add_argument("--no-precision", action="store_true", help="skip the precision, mixed and saturated legs")
    ap.add_argument("--no-chi512", action="store_true", help="skip the chi=512 saturated leg")
    ap.add_argument("--no-saturated", action="store_true",
                    help="skip the saturated legs (e.g. for the whole 200-step run: --steps 200)")
    ap.add_argument("--rank-bound", type=float, nargs="*", default=None,
                    help="extra legs of the kept-rank form at these discarded-weight bounds (FP64 and "
                         "double-float), with speedup and observable errors against the plain run")
    ap.add_argument("--cpu-updates", type=int, default=2)
    ap.add_argument("--sat-L", type=int, default=L, help="--workload saturated: chain length")
    ap.add_argument("--sat-chi", type=int, default=CHI, help="--workload saturated: chi")
    ap.add_argument("--sat-d", type=int, default=D, help="--workload saturated: local dimension (Bose-Hubbard, max filling d-1)")
    ap.add_argument("--sat-decay", type=float, default=16.0, help="--workload saturated: lambda_k ~ exp(-k/decay)")
    ap.add_argument("--random-start", action="store_true", help="--workload saturated: no preparing sweep")
    ap.add_argument("--theta-form", type=int, default=0,
                    help="Theta formation: 0 CUDA cores, 3 = 3xTF32, 100+S = S bf16 digit planes (tensor cores)")
    ap.add_argument("--outdir", default=os.path.join(ROOT, "bench_out"),
                    help="where the clock samples of the timed region are written")
    args = ap.parse_args()
    os.makedirs(args.outdir, exist_ok=True)
    if args.impl == "reference":
        run_reference(args)
    elif args.workload == "nc":
        run_nc(args)
    elif args.workload == "saturated":
        run_saturated(args)
    elif args.workload == "fermi_hubbard":
        run_fermi(args)
    elif args.workload == "spin1":
        run_spin1(args)
    elif args.workload == "zgemm":
        run_zgemm(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
