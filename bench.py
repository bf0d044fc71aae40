"""Benchmark: time to E_CCSD for the L=6, A=28 lattice nucleus on one B200.

Workload: periodic cubic lattice L=6 (864 states), A=28 closed shell (site
(0,0,0) and its six neighbours, four spin-isospin states each; 836 particle
states), kinetic hopping + on-site SU(4) contact C2=-3 + three-body contact
C3=+1 in units of hbar^2/(M a^2) (the reference's unit is half of that, so
vT1=vS1=-6, w3=+2).  The Hamiltonian is built in-process; nothing is read
from disk.

A *step* is one complete CCSD solve from the MP2 start:

* ``mixed`` (the headline): T2 in FP32 with FP64 T1 / energy / DIIS
  (subspace 8), energy test 1e-8, then the FP64 refinement sweep: FP64 steps
  until the FP64 energy test passes at the same 1e-8 (``--no-refine`` drops
  the sweep);
* ``mixed_tight``: the same with the FP64 steps run to 1e-10;
* ``mixed32``: the FP32 phase alone;
* ``fp64``: the plain FP64 path with the reference's NumPy algorithm
  (Jacobi + mixing 0.5, no DIIS, energy test 1e-8);
* ``fp64_diis``: FP64 with the torch solver's pulsed DIIS (subspace 8).

``value`` is the mixed time-to-solution (device time, CUDA events, inputs
resident); its energy must lie within 1e-6 relative of the FP64 fixed point
(a tight FP64 solve, eps=1e-12, run once untimed).  L2 (126 MB) is flushed
by a 256 MiB write before every timed solve.

``--impl reference`` times the CPU oracle (a numpy restatement of the
reference's CCSD, evaluating every diagram as the reference does) on the host
cores: one Jacobi iteration at L=4, A=28 per step, one each at L=3 and L=5
for the size dependence, and the L=6 time to solution projected from them
(the power-law exponent fitted to the measured sizes) with the FP64
iteration count at L=6; the output names the sizes it ran.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "time-to-E_CCSD (<=1e-6 rel vs FP64 oracle) and s/iter, mixed vs FP64, 1 B200"
L_BENCH, A_BENCH, C2, C3 = 6, 28, -3.0, 1.0
L_SAMPLE = 4                 # CPU sample size (same A=28 closed shell)
# FP64 Jacobi iteration count at L=6, A=28 (eps=1e-8), measured by the FP64
# GPU path; the reference arm runs on the host alone and uses this value.
FP64_ITERS_L6_MEASURED = 70


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-refine", action="store_true",
                    help="headline without the final FP64 refinement sweep of the mixed solve")
    ap.add_argument("--profile", action="store_true", help="one short mixed solve, no JSON (for ncu)")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU-baseline sample")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-adjoint", action="store_true", help="skip the dE/dC2, dE/dC3 leg")
    ap.add_argument("--no-batch", action="store_true", help="skip the 64-instance batched scan")
    ap.add_argument("--profile-lambda", action="store_true", help="one short Lambda solve at L=6, A=28 (for ncu)")
    ap.add_argument("--profile-gemm", action="store_true",
                    help="the general engine's tensor-core contraction (3xTF32) against the FP64 GEMM path")
    ap.add_argument("--pw-case", action="append", default=None, metavar="L,A",
                    help="with --profile-planewave: only this (L, A) (repeatable)")
    ap.add_argument("--profile-planewave", action="store_true",
                    help="momentum-block solves of closed-shell plane waves (L=6 A=4, L=6 A=28, L=8 A=28), "
                         "and 20 timed steps of each; no JSON")
    return ap.parse_args()


def dist_setup():
    import torch
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    elif torch.cuda.is_available():
        torch.cuda.set_device(0)
    return rank, ws, local


def build_problem(L, A, dense=False):
    from nulattice_b200 import hamiltonian as ham
    v2, w3 = ham.contact_couplings(C2, C3)
    e_ref, fock, two = ham.normal_ordered_hamiltonian(L, ham.closed_shell_holes(L, A), v2, v2, w3, dense=dense)
    return e_ref, fock, two


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self, index):
        import tempfile
        self.index = index
        self.proc = None
        self.path = os.path.join(tempfile.mkdtemp(prefix="nlb_clocks_"), "clocks.csv")

    def __enter__(self):
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index),
                 "--query-gpu=clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
                 "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                 "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap",
                 "--format=csv,noheader,nounits", "-lms", "100"], stdout=self.f, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            time.sleep(0.25)
            self.proc.terminate()
            self.proc.wait(timeout=10)
            self.f.close()

    def summary(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 8:
                continue
            try:
                sm.append(float(parts[0]))
                smax = float(parts[1])
            except ValueError:
                continue
            for n, v in zip(names, parts[4:8]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": smax,
                "samples": len(sm), "reasons": sorted(reasons)}


def cpu_model():
    try:
        for line in open("/proc/cpuinfo"):
            if line.startswith("model name"):
                return line.split(":", 1)[1].strip()
    except OSError:
        pass
    import platform
    return platform.processor() or "unknown"


def oracle_iteration(L, A=A_BENCH):
    """Seconds of one Jacobi iteration of the CPU port of the reference CCSD
    at (L, A): every diagram evaluated as the reference evaluates it, zero
    blocks included.  Returns (seconds, p)."""
    import numpy as np
    from oracle import ccsd_oracle as O
    O.SKIP_ZERO_BLOCKS = False
    e_ref, fock, two = build_problem(L, A, dense=True)
    H = O.Hamiltonian(fock, two)
    t1, t2 = O.t1_init(H), O.t2_init(H)
    t0 = time.perf_counter()
    r = O.ppph_intermediates(H.ppph_idx, H.ppph_val, t1, t2)
    n1 = O.t1_step(H, t1, t2, r)
    n2 = O.t2_step(H, t1, t2, r)
    dt = time.perf_counter() - t0
    assert np.isfinite(n1).all() and np.isfinite(n2).all()
    return dt, H.p


def oracle_tts(L, A=4, eps=1e-8):
    """Time to solution of the CPU port of the reference CCSD (every diagram,
    FP64 Jacobi + mixing 0.5, the NumPy solver's energy test) from the MP2
    start at (L, A).  Returns (seconds, iterations, E_corr)."""
    from oracle import ccsd_oracle as O
    O.SKIP_ZERO_BLOCKS = False
    e_ref, fock, two = build_problem(L, A, dense=True)
    t0 = time.perf_counter()
    e, _, _, iters, status = O.solve(fock, two, eps=eps, maxSteps=4000, max_diis=0, criterion="numpy")
    return time.perf_counter() - t0, iters, e


def configs_leg(dev):
    """The A=4 configurations (L=3, 4, 5; the bench's couplings) through the
    public ccsd_solver on host numpy inputs, wall clock of a second (warm)
    call: FP64 with the reference's NumPy algorithm (Jacobi + mixing 0.5,
    energy test 1e-8) at every L; at L=5 also FP64 with pulsed DIIS 8 and the
    mixed recipe (FP32 T2 phase with DIIS 8, then FP64 steps to the same
    test)."""
    import torch
    from nulattice_b200 import ccsd_solver
    out = {}
    for L in (3, 4, 5):
        e_ref, fock, two = build_problem(L, 4)
        modes = [("fp64_jacobi", dict(max_diis=0, criterion="numpy"))]
        if L == 5:
            modes += [("fp64_diis8", dict(max_diis=8)),
                      ("mixed", dict(max_diis=8, precision="mixed", mixed_eps=1e-8))]
        res = {}
        for name, kw in modes:
            for _ in range(2):
                info = {}
                torch.cuda.synchronize(dev)
                t0 = time.perf_counter()
                e, _, _ = ccsd_solver(fock, two, eps=1e-8, maxSteps=4000, device=dev, info=info, **kw)
                torch.cuda.synchronize(dev)
                t = time.perf_counter() - t0
            res[name] = {"s": t, "iterations": info["iterations"], "e_corr": e}
        out[f"A4_L{L}"] = res
    return out


def project(samples, p_target, iters):
    """Time to solution at p_target from measured (p, s/iter) samples: the
    power law s = c p^x through the two largest samples, times the FP64
    iteration count.  Returns (seconds, x)."""
    import math
    (p1, s1), (p2, s2) = sorted(samples)[-2:]
    x = math.log(s2 / s1) / math.log(p2 / p1)
    return s2 * (p_target / p2) ** x * iters, x


def run_reference(args):
    """The reference arm: the reference's CPU algorithm (the numpy port in
    oracle/, every diagram) on the host cores.  Each step is one measured
    Jacobi iteration at L=4, A=28; one iteration at L=3 and one at L=5 (16 GB)
    are measured once for the size dependence; the L=6 time to solution is
    projected from them with the fitted exponent and the FP64 iteration count
    of the L=6 solve."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    threads = os.cpu_count() or 1
    p6 = 4 * L_BENCH ** 3 - A_BENCH
    times = []
    for k in range(args.warmup + args.steps):
        dt, p4 = oracle_iteration(L_SAMPLE)
        if k >= args.warmup:
            times.append(dt)
    s_iter = statistics.median(times)
    samples = {4: (p4, s_iter)}
    for L in (3, 5):
        try:
            dt, pL = oracle_iteration(L)
            samples[L] = (pL, dt)
        except MemoryError:
            pass
    val, x = project(list(samples.values()), p6, FP64_ITERS_L6_MEASURED)
    configs = {}
    for L in (3, 4):
        dt, iters, e = oracle_tts(L)
        configs[f"A4_L{L}"] = {"s": dt, "iterations": iters, "e_corr": e}
    sample = (f"measured one Jacobi iteration of the numpy port of the reference CCSD (every diagram) at A={A_BENCH}: "
              + ", ".join(f"L={L} (p={pp}) {ss:.2f} s" for L, (pp, ss) in sorted(samples.items()))
              + f" (L={L_SAMPLE}: median of {args.steps}); L=6 (p={p6}) projected as s/iter ~ p^{x:.2f} "
              f"(exponent fitted to the two largest samples) x {FP64_ITERS_L6_MEASURED} FP64 iterations")
    out = {"metric": METRIC, "value": val, "unit": "s", "n_gpus": args.gpus, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": s_iter * 1e3, "higher_is_better": False,
           "scaling": "weak", "vs_baseline": None, "dtype": "f64", "impl": "reference",
           "data": "synthetic lattice Hamiltonian built in-process",
           "config": {"workload": "ccsd_L6_A28 time to solution, projected from measured iterations",
                      "L_measured": sorted(samples), "A": A_BENCH, "C2": C2, "C3": C3,
                      "step": f"one Jacobi iteration at L={L_SAMPLE}, A={A_BENCH}",
                      "path": "the reference's CPU algorithm (FP64 Jacobi + mixing, every diagram)"},
           "measured_s_per_iter": {f"L{L}": ss for L, (pp, ss) in sorted(samples.items())},
           "projection": {"target_L": L_BENCH, "exponent": x, "fp64_iterations": FP64_ITERS_L6_MEASURED},
           "configs_time_to_solution": {"measured": configs,
                                        "path": "FP64 Jacobi + mixing 0.5 from the MP2 start, energy test 1e-8, "
                                                "A=4, C2=-3, C3=+1"},
           "cpu_baseline": {"value": val, "unit": "s", "cores": threads, "cpu": cpu_model(), "kind": "port",
                            "sample": sample},
           "e2e": {"value": val, "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out), flush=True)


def profile_gemm(dev, reps=10):
    """The general engine's GEMM-shaped contraction on the tensor cores
    (tcgen05, 3xTF32, nlb_contract_gemm_tf32x3) and on the FP64 library GEMM
    path (nlb_contract_gemm_f64), CUDA events, median of `reps`: a square
    4096^3 product and a ring-diagram shape (bkcj,acik->abij at p=400, h=8).
    TFLOP/s count the useful 2MNK; the tensor pipe runs three TF32 products."""
    import torch
    from nulattice_b200 import dense as D
    out = {}
    cases = {"square_4096": ("mk,kn->mn", (4096, 4096), (4096, 4096), (4096, 4096), 2 * 4096 ** 3),
             "ring_p400_h8": ("bkcj,acik->abij", (400, 8, 400, 8), (400, 400, 8, 8), (400, 400, 8, 8),
                              2 * (400 * 8) ** 3)}
    g = torch.Generator().manual_seed(0)
    for name, (spec, sa, sb, sc, flops) in cases.items():
        A = torch.randn(sa, generator=g, dtype=torch.float64).to(dev)
        B = torch.randn(sb, generator=g, dtype=torch.float64).to(dev)
        res = {}
        outs = {}
        for path in ("tensor_cores", "fp64"):
            C = torch.zeros(sc, dtype=torch.float64, device=dev)
            E = D.GpuEinsum(torch.cuda.current_stream(dev).cuda_stream)
            E.tensor_cores = path == "tensor_cores"
            E.pair(spec, A, B, C)
            ts = []
            for _ in range(reps):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                E.pair(spec, A, B, C)
                b.record()
                torch.cuda.synchronize()
                ts.append(a.elapsed_time(b) / 1e3)
            t = statistics.median(ts)
            res[path] = {"ms": t * 1e3, "tflops": flops / t / 1e12}
            outs[path] = C
        res["max_rel_err"] = float((outs["tensor_cores"] - outs["fp64"]).abs().max() / outs["fp64"].abs().max())
        out[name] = res
    # open-shell 3He (three nucleons on one site: ring and quadratic diagrams
    # are real contractions), ccsd_solver to 1e-10 through the general engine,
    # mixed (tensor-core phase to the default 1e-6, then FP64) against FP64;
    # wall clock of a second, warm call
    from nulattice_b200 import ccsd_solver, hamiltonian as ham
    he3 = [(0, 0, 0, 0, 0), (0, 0, 0, 1, 0), (0, 0, 0, 0, 1)]
    for L in (4, 6):
        e_ref, fock, two = ham.normal_ordered_hamiltonian(L, he3, -8.0, -8.0, 5.5)
        res = {}
        for prec in ("mixed", "fp64"):
            for _ in range(2):
                info = {}
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                e, _, _ = ccsd_solver(fock, two, eps=1e-10, maxSteps=3000, max_diis=8, device=dev,
                                      precision=prec, info=info)
                torch.cuda.synchronize()
                t = time.perf_counter() - t0
            res[prec] = {"s": t, "s_per_iter": t / max(1, info.get("iterations") or 1),
                         "iterations": info.get("iterations"), "mixed_iters": info.get("mixed_iters"),
                         "tc_gemms": info.get("tc_gemms"), "gemms": info.get("gemms"), "e_corr": e,
                         "status": info.get("status")}
        res["speedup"] = res["fp64"]["s"] / res["mixed"]["s"]
        res["e_diff"] = abs(res["mixed"]["e_corr"] - res["fp64"]["e_corr"])
        out[f"he3_L{L}_solve"] = res
    print(json.dumps({"profile_gemm": out}), flush=True)


def profile_planewave(dev, cases=None):
    """Momentum-block path on closed-shell plane waves (couplings vT1 = vS1 =
    -4, w3 = 1): solves to 1e-10 (pulsed DIIS 8) on a warm engine in FP64 and
    mixed precision (FP32 phase to 1e-8, then FP64), wall clock of the second
    of two; then 20 steps of each precision timed with CUDA events."""
    import torch
    from nulattice_b200 import momentum as MB
    from nulattice_b200 import planewave as PW
    for (L, A) in (cases or ((6, 4), (6, 28), (8, 28))):
        plan = MB.MomentumPlan(L, PW.momentum_holes(L, A))
        V = MB.contact_tensor(L, plan.n_k, -4.0, -4.0, 1.0)
        fpp, fhh, e_ref = MB.fock_blocks(L, plan.n_k, plan.hmom, plan.pmom, -4.0, -4.0, 1.0)
        eng = MB.MomentumEngine(plan, V, fpp, fhh, dev)
        for prec in ("fp64", "mixed"):
            for _ in range(2):
                info = {}
                torch.cuda.synchronize(dev)
                t0 = time.perf_counter()
                e, t2 = MB.solve(plan, V, fpp, fhh, eps=1e-10, maxSteps=1000, max_diis=8, engine=eng, info=info,
                                 precision=prec, mixed_eps=1e-8)
                torch.cuda.synchronize(dev)
                t = time.perf_counter() - t0
            print(f"L={L} A={A} n_t2={plan.n_t2} {prec} E_corr={e:.12f} {info['status']} "
                  f"iterations={info['iterations']} (fp32 {info.get('mixed_iters', 0)}) solve_s={t:.4f}",
                  flush=True)
        for e_ in (eng, getattr(eng, "_f32_twin", None)):
            if e_ is None:
                continue
            x, y = e_.zeros(), e_.zeros()
            e_.init(x)
            e_.energy(x)
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            for _ in range(3):
                e_.step(x, y)
            ev[0].record()
            for _ in range(20):
                e_.step(x, y)
            ev[1].record()
            torch.cuda.synchronize(dev)
            print(f"   {'fp32' if e_.f32 else 'fp64'} step_us={ev[0].elapsed_time(ev[1]) / 20 * 1e3:.1f}", flush=True)


def main():
    args = parse()
    if args.impl == "reference":
        run_reference(args)
        return
    import numpy as np
    import torch
    from nulattice_b200 import _lib
    from nulattice_b200 import ccsd as C
    from nulattice_b200 import hamiltonian as ham
    from nulattice_b200 import structure as S

    if args.profile_planewave:
        cases = [tuple(int(x) for x in c.split(",")) for c in args.pw_case] if args.pw_case else None
        profile_planewave(torch.device("cuda", 0), cases)
        return
    if args.profile_gemm:
        profile_gemm(torch.device("cuda", 0))
        return
    rank, ws, local = dist_setup()
    dev = torch.device("cuda", local)
    e_ref, fock, two = build_problem(L_BENCH, A_BENCH)
    plan, why = S.detect(fock, two)
    assert plan is not None, why
    eng = C.StructuredEngine(plan, fock, dev)
    # launch shapes of the lattice kernels (timed per variant, cached per GPU and shape)
    from nulattice_b200 import tune as T
    tune_info = {}
    T.tune(eng, info=tune_info)

    refine = not args.no_refine
    # the solve modes: "mixed" is the headline (FP32 T2 with FP64 T1/energy/
    # DIIS to |dE|/|E| < 1e-8, then the FP64 refinement sweep: FP64 steps
    # until the FP64 energy test passes at the same 1e-8 as the FP64 paths;
    # --no-refine drops the sweep); "mixed_tight" sweeps to 1e-10; "mixed32"
    # stops after the FP32 phase; "fp64" is the reference's NumPy algorithm
    # (FP64 Jacobi + mixing, no DIIS); "fp64_diis" the torch solver's (FP64,
    # pulsed DIIS 8)
    def solve(mode, t2_events=None, **kw):
        info = {}
        if mode in ("mixed", "mixed_tight", "mixed32"):
            ref = (refine and mode == "mixed") or mode == "mixed_tight"
            e, t1, t2 = C.solve_structured(eng, eps=1e-10 if mode == "mixed_tight" else 1e-8, maxSteps=4000,
                                           max_diis=8, precision="mixed", mixed_eps=1e-8, t2_format="compact",
                                           info=info, t2_events=t2_events, refine=ref, **kw)
            if not ref:
                info["refine_iters"] = 0
        elif mode == "fp64":
            e, t1, t2 = C.solve_structured(eng, eps=1e-8, maxSteps=4000, max_diis=0, precision="fp64",
                                           criterion="numpy", t2_format="compact", info=info,
                                           t2_events=t2_events, **kw)
        else:
            e, t1, t2 = C.solve_structured(eng, eps=1e-8, maxSteps=4000, max_diis=8, precision="fp64",
                                           criterion="soa", t2_format="compact", info=info,
                                           t2_events=t2_events, **kw)
        return e, info

    if args.profile:
        # stage by stage (t2_events): kernels inside the device-loop graph are
        # not seen by a kernel profiler
        C.solve_structured(eng, eps=0.0, maxSteps=12, max_diis=8, precision="mixed", mixed_eps=0.0,
                           t2_format="compact", t2_events=[])
        torch.cuda.synchronize()
        print("profile run done", flush=True)
        return
    if args.profile_lambda:
        # converged amplitudes, then 12 FP32 Lambda steps (lattice kernels)
        from nulattice_b200 import adjoint as A
        prob = A.lattice_problem(L_BENCH, ham.closed_shell_holes(L_BENCH, A_BENCH))
        e, t1, t2c = C.solve_structured(eng, eps=1e-10, maxSteps=500, max_diis=8, precision="mixed",
                                        mixed_eps=1e-8, t2_format="compact")
        try:
            A.lambda_gradient(eng, t1, t2c, [prob.dv, prob.dw], tol=0.0, tol_fp32=0.0, max_steps=12, max_diis=8,
                              precision="mixed")
        except RuntimeError:
            pass   # 12 steps, not converged: only the kernels are wanted
        torch.cuda.synchronize()
        print("profile run done", flush=True)
        return

    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    # FP64 fixed point used as the accuracy reference (untimed)
    e_tight, _, _ = C.solve_structured(eng, eps=1e-12, maxSteps=6000, max_diis=8, precision="fp64",
                                       t2_format="compact")
    modes = ("mixed", "mixed_tight", "mixed32", "fp64", "fp64_diis")
    for _ in range(args.warmup):
        for mode in modes:
            solve(mode)
    torch.cuda.synchronize()

    def timed(precision):
        """K solves through the production path (steps captured in CUDA graphs),
        then one more solve launched stage by stage with CUDA events around
        every T2 update (the roofline's kernel time; not part of the value)."""
        evs, t2ev, infos, energies = [], [], [], []
        eng.launches = 0
        if ws > 1:
            torch.distributed.barrier()
        torch.cuda.synchronize()
        for _ in range(args.steps):
            flush.fill_(1.0)
            a = torch.cuda.Event(enable_timing=True)
            b = torch.cuda.Event(enable_timing=True)
            a.record()
            e, info = solve(precision)
            b.record()
            evs.append((a, b))
            infos.append(info)
            energies.append(e)
        torch.cuda.synchronize()
        launches = eng.launches
        if ws > 1:
            torch.distributed.barrier()
        flush.fill_(1.0)
        solve(precision, t2_events=t2ev)
        torch.cuda.synchronize()
        step_ms = [a.elapsed_time(b) for a, b in evs]
        k_ms = [a.elapsed_time(b) for a, b in t2ev]
        return step_ms, k_ms, infos, energies, launches

    dev_index = torch.cuda.current_device()
    with Clocks(dev_index) as clk:
        m_ms, m_k, m_info, m_e, m_launch = timed("mixed")
    clocks = clk.summary()
    others = {mode: timed(mode) for mode in modes[1:]}

    from nulattice_b200 import batch as B

    def gmax(x):
        return B.max_over_ranks(x, dev)

    def rel_err(e):
        return abs((e + e_ref) - (e_tight + e_ref)) / abs(e_tight + e_ref)

    tts_mixed = gmax(statistics.mean(m_ms)) / 1e3
    it_mixed = m_info[-1]["iterations"]
    e_corr = m_e[-1]
    rel = rel_err(e_corr)
    paths = {}
    for mode, (ms, _, infos, es, _) in others.items():
        t = gmax(statistics.mean(ms)) / 1e3
        paths[mode] = {"time_to_solution_s": t, "iterations": infos[-1]["iterations"],
                       "s_per_iter": t / infos[-1]["iterations"], "e_ccsd_rel_err": rel_err(es[-1])}
    paths["mixed32"]["algorithm"] = "FP32 T2 (FP64 T1, energy, DIIS 8) to |dE|/|E| < 1e-8, no FP64 sweep"
    paths["mixed_tight"]["algorithm"] = "the FP32 phase, then FP64 steps to |dE|/|E| < 1e-10"
    paths["fp64"]["algorithm"] = "FP64 Jacobi + mixing 0.5, no DIIS (the reference's NumPy algorithm), eps 1e-8"
    paths["fp64_diis"]["algorithm"] = "FP64 with pulsed DIIS 8 (the reference's torch algorithm), eps 1e-8"
    tts_fp64 = paths["fp64"]["time_to_solution_s"]
    it_fp64 = paths["fp64"]["iterations"]

    # roofline of the T2 update kernel (mixed, FP32 storage, DIIS ring write)
    # of the problem that runs: one channel when the labels are alike
    n_t2 = plan.n_t2
    work = eng.reduced() or eng
    # two-launch steps: T2 read, written, error written (no Ga table); the
    # events then span the row and the pair kernel
    paired = _lib.lib().nlb_struct_step_launches(work.prob, _lib.NLB_F32) == 2
    alg_bytes = (3 * work.plan.n_t2 + (0 if paired else work.n_g)) * 4
    k_ms = statistics.mean(m_k)
    achieved = alg_bytes / (k_ms * 1e-3) / 1e9
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
        peak, peak_src = float(peaks["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        peak, peak_src = 6650.0, "fallback"
    kernel = "k_sym_row + k_sym_update" if paired else T.t2_kernel_fp32(int(eng.prob.tune))
    traffic = None
    tfile = os.path.join(ROOT, "profiles", "t2_update_traffic.json")
    if os.path.exists(tfile):
        rec = json.load(open(tfile))
        traffic = rec.get("bytes_per_launch") if rec.get("kernel") == kernel else None
    roofline = {"kernel": kernel, "bound": "hbm", "achieved": achieved, "peak": peak,
                "peak_source": peak_src, "unit": "GB/s", "frac": achieved / peak, "traffic": traffic,
                "alg_bytes_per_launch": alg_bytes, "avg_launch_us": k_ms * 1e3, "launches": len(m_k)}

    out = {"metric": METRIC, "value": tts_mixed, "unit": "s", "n_gpus": ws, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": tts_mixed * 1e3, "higher_is_better": False,
           "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
           "data": "synthetic: lattice Hamiltonian built in-process (no dataset)",
           "config": {"workload": "ccsd_L6_A28_mixed", "L": L_BENCH, "A": A_BENCH, "p": plan.p, "h": plan.h,
                      "C2": C2, "C3": C3, "units": "hbar^2/(M a^2)", "n_t2_compact": n_t2, "n_t2_stored": work.plan.n_t2,
                      "tune": {"word": int(eng.prob.tune), "choice": T.describe(int(eng.prob.tune)),
                               "cached": tune_info.get("cached")},
                      "max_diis": 8, "mixed_eps": 1e-8, "refine": refine,
                      "l2": "256 MiB flush write before every timed solve (excluded from step time)",
                      "parallelism": "replicas" if ws > 1 else "single"},
           "s_per_iter": tts_mixed / it_mixed, "iterations": it_mixed,
           "mixed_iters": m_info[-1].get("mixed_iters"), "refine_iters": m_info[-1].get("refine_iters", 0),
           "headline": ("FP32 T2 phase to |dE|/|E| < 1e-8, then the FP64 refinement sweep: FP64 steps until the "
                        "FP64 energy test passes at 1e-8, the test of the FP64 paths" if refine
                        else "FP32 T2 phase to |dE|/|E| < 1e-8 (no FP64 sweep)"),
           "fp64": paths["fp64"], "fp64_diis": paths["fp64_diis"], "mixed32": paths["mixed32"],
           "mixed_tight": paths["mixed_tight"],
           "speedup_mixed_vs_fp64": tts_fp64 / tts_mixed,
           "speedup_mixed_vs_fp64_diis": paths["fp64_diis"]["time_to_solution_s"] / tts_mixed,
           "e_ccsd": (e_corr + e_ref), "e_ccsd_fp64_fixed_point": e_tight + e_ref,
           "e_ccsd_rel_err": rel,
           "accuracy_reference": "FP64 engine at eps 1e-12 (the reference cannot run at L=6: ~50 GB RSS, ~13 "
                                 "min/iteration); the engine is pinned to the reference's tight fixed points at "
                                 "A=4, L=3-5 and A=28, L=4 by the GPU tests",
           "roofline": roofline, "gpu_launches": m_launch, "clocks": clocks,
           "tune_us": tune_info.get("us")}

    if not args.no_e2e:
        out["e2e"] = e2e_leg(args, fock, two, dev)
    if not args.no_adjoint:
        out["adjoint"] = adjoint_leg(dev)
    if rank == 0:
        out["configs"] = configs_leg(dev)
    batch = batch_leg(dev, peak, rank, ws) if not args.no_batch else None
    if not args.no_cpu and rank == 0:
        # one iteration each at L=3 and L=4 (about 10-15 s of CPU work), the
        # L=6 time to solution projected with the exponent they give
        samples = [oracle_iteration(L)[::-1] for L in (3, L_SAMPLE)]
        val, x = project(samples, plan.p, it_fp64)
        c1 = oracle_tts(3)
        out["cpu_baseline"] = {"value": val, "unit": "s", "cores": os.cpu_count(), "cpu": cpu_model(),
                               "kind": "port", "projected": True,
                               "measured_time_to_solution_A4_L3": {"s": c1[0], "iterations": c1[1],
                                                                   "e_corr": c1[2]},
                               "measured_s_per_iter": {f"L{L}": ss for L, (pp, ss) in zip((3, L_SAMPLE), samples)},
                               "sample": "measured one Jacobi iteration of the numpy port of the reference CCSD "
                                         f"(every diagram) at A={A_BENCH}, L=3 (p={samples[0][0]}) "
                                         f"{samples[0][1]:.2f} s and L={L_SAMPLE} (p={samples[1][0]}) "
                                         f"{samples[1][1]:.2f} s; L=6 (p={plan.p}) projected as s/iter ~ "
                                         f"p^{x:.2f} x {it_fp64} FP64 iterations"}
    if batch is not None:
        out["batch"] = batch
    # the contract keys and the short summaries first, the long detail blocks
    # (per-path results, configurations, tuner timings, batch) last
    first = ["metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
             "vs_baseline", "dtype", "data", "config", "roofline", "gpu_launches", "clocks", "e2e", "cpu_baseline",
             "adjoint", "s_per_iter", "iterations", "mixed_iters", "refine_iters", "e_ccsd_rel_err",
             "speedup_mixed_vs_fp64", "speedup_mixed_vs_fp64_diis"]
    last = ["fp64", "fp64_diis", "mixed32", "mixed_tight", "configs", "tune_us", "batch"]
    out = {**{k: out[k] for k in first if k in out},
           **{k: v for k, v in out.items() if k not in first and k not in last},
           **{k: out[k] for k in last if k in out}}
    if rank == 0:
        print(json.dumps(out), flush=True)
    if ws > 1:
        torch.distributed.destroy_process_group()


def batch_leg(dev, peak_gbs, rank=0, ws=1):
    """Batched scan: 64 (A, L, C2, C3) instances from numpy's default_rng(0),
    energies and dE/dC2, dE/dC3 in one graph launch (mixed precision with
    FP64 finishes), against the same instances solved one at a time in FP64
    (Jacobi + mixing, forward and Lambda) and one at a time with the batch's
    own algorithm.  With N ranks each GPU solves its share of the 64 instances
    (cost-balanced, no communication); times are the max over ranks."""
    import math
    import torch
    from nulattice_b200 import adjoint as A
    from nulattice_b200 import batch as B
    from nulattice_b200.ccsd import solve_structured
    inst_all = B.draw_instances(64, 0)
    inst = B.shard(inst_all, rank, ws)
    t0 = time.perf_counter()
    scan = B.BatchScan(inst, device=dev)
    t_setup = time.perf_counter() - t0
    times = []
    for _ in range(3):
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize(dev)
        ev[0].record()
        scan.launch()
        ev[1].record()
        torch.cuda.synchronize(dev)
        times.append(ev[0].elapsed_time(ev[1]) / 1e3)
    t_batch = statistics.median(times)

    def gmax(x):
        return B.max_over_ranks(x, dev)
    t_batch = gmax(t_batch)
    res = scan.results()
    ok = [r for r in res if r["status"] == "converged" and r["lambda_status"] == "converged"]
    # algorithmic bytes of the steps that ran: 3 passes over the stored T2
    # (read, write, DIIS error) per forward or Lambda step, FP32 or FP64
    alg = 0.0
    for r in res:
        n2 = r["n_t2_stored"]
        alg += 3 * n2 * (4 * r["mixed_iterations"] + 8 * (r["iterations"] - r["mixed_iterations"]))
        alg += 3 * n2 * 6 * r["lambda_iterations"]   # FP32 and FP64 Lambda steps, ~6 bytes on average
    # one at a time: the batch's algorithm and plain FP64 Jacobi, on the same engines
    seq = {"mixed": [], "fp64": []}
    diffs = []
    for x, r in zip(scan.instances, res):
        for mode in ("mixed", "fp64"):
            kw = (dict(precision="mixed", max_diis=8, mixed_eps=1e-8) if mode == "mixed"
                  else dict(precision="fp64", max_diis=0))
            torch.cuda.synchronize(dev)
            t1 = time.perf_counter()
            info = {}
            e, t1v, t2c = solve_structured(x.eng, eps=1e-10, maxSteps=500, t2_format="compact", info=info,
                                           loop="eager", **kw)
            g = None
            if info["status"] == "converged":
                try:
                    g = A.lambda_gradient(x.eng, t1v, t2c, [x.prob.dv, x.prob.dw], tol=1e-8, max_steps=500,
                                          max_diis=kw["max_diis"], precision=kw["precision"])
                except RuntimeError:
                    g = None
            torch.cuda.synchronize(dev)
            seq[mode].append(time.perf_counter() - t1)
            if mode == "fp64" and g is not None and r in ok:
                diffs.append((abs(e - r["E_corr"]) / abs(r["E_corr"]), abs(2 * g[0] - r["dE_dC2"]) / abs(r["dE_dC2"]),
                              abs(2 * g[1] - r["dE_dC3"]) / abs(r["dE_dC3"])))
        if r not in ok:
            # the reason: the reference's own algorithms on the same instance in
            # FP64, ten times the batch's step limit (NumPy solver: Jacobi with
            # mixing 0.5; torch solver: pulsed DIIS 8)
            out = {}
            for name, kw in (("fp64_jacobi_5000", dict(max_diis=0, criterion="numpy")),
                             ("fp64_diis8_5000", dict(max_diis=8))):
                info = {}
                e, _, _ = solve_structured(x.eng, eps=1e-10, maxSteps=5000, t2_format="compact", info=info,
                                           loop="eager", precision="fp64", **kw)
                out[name] = {"status": info["status"], "iterations": info["iterations"], "E_corr": round(e, 4)}
            r["reference_algorithms"] = out
    scan.close()
    # one compact record per failure: the instance, the batch's statuses and
    # E_corr, and [status, steps, E_corr] of the reference's two algorithms
    failed = [{"inst": [r["A"], r["L"], round(r["C2"], 4), round(r["C3"], 4)],
               "batch": [r["status"], r["lambda_status"], round(r["E_corr"], 3)],
               **{k: [v["status"], v["iterations"], round(v["E_corr"], 3)]
                  for k, v in r["reference_algorithms"].items()}} for r in res if r not in ok]
    if ws > 1:
        gathered = B.gather_results([(res, failed, diffs, alg)])
        res = [r for g in gathered for r in g[0]]
        failed = [f for g in gathered for f in g[1]]
        diffs = [d for g in gathered for d in g[2]]
        alg = sum(g[3] for g in gathered)
        ok = [r for r in res if r["status"] == "converged" and r["lambda_status"] == "converged"]
    n = len(inst_all)
    t_f64, t_mix = gmax(sum(seq["fp64"])), gmax(sum(seq["mixed"]))
    classes = {}
    for a_, l_, _, _ in inst_all:
        classes[f"A{a_}_L{l_}"] = classes.get(f"A{a_}_L{l_}", 0) + 1
    achieved = alg / t_batch / 1e9
    return {"instances": n, "converged": len(ok), "failures": failed, "classes": classes, "seed": 0,
            "t_batch_s": t_batch, "instances_per_s": n / t_batch,
            "t_one_at_a_time_fp64_s": t_f64, "instances_per_s_fp64_sequential": n / t_f64,
            "t_one_at_a_time_mixed_s": t_mix, "instances_per_s_mixed_sequential": n / t_mix,
            "speedup_vs_fp64_sequential": t_f64 / t_batch, "speedup_vs_mixed_sequential": t_mix / t_batch,
            "max_rel_diff_vs_fp64_sequential": {"E_corr": max(d[0] for d in diffs) if diffs else None,
                                                "dE_dC2": max(d[1] for d in diffs) if diffs else None,
                                                "dE_dC3": max(d[2] for d in diffs) if diffs else None},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak_gbs * ws, "unit": "GB/s",
                         "frac": achieved / (peak_gbs * ws), "alg_bytes": alg},
            "ranks": ws, "t_setup_s": t_setup}


def adjoint_leg(dev):
    """dE_CCSD/dC2 and dE_CCSD/dC3 at the headline configuration through the
    Lambda kernels, timed against the forward solve, and checked against
    central differences (step 1e-4) of tight FP64 solves."""
    import torch
    from nulattice_b200 import adjoint as A
    from nulattice_b200 import hamiltonian as ham
    from nulattice_b200 import structure as S
    from nulattice_b200.ccsd import StructuredEngine, solve_structured
    holes = ham.closed_shell_holes(L_BENCH, A_BENCH)
    info = {}
    E, g2, g3 = A.ccsd_energy_and_gradient(L_BENCH, holes, C2, C3, device=dev, precision="mixed", eps=1e-10,
                                           mixed_eps=1e-8, lambda_tol=1e-8, info=info)
    from nulattice_b200 import tune as T
    T.tune(info["engine"])
    # timed on the warm engine (buffers allocated, step graphs captured with
    # the tuned shapes by one more untimed call): forward and Lambda solves
    # measured the same way, median of three
    A.ccsd_energy_and_gradient(L_BENCH, holes, C2, C3, device=dev, precision="mixed", eps=1e-10, mixed_eps=1e-8,
                               lambda_tol=1e-8, info={}, engine=info["engine"])
    runs = []
    for _ in range(3):
        info2 = {}
        E, g2, g3 = A.ccsd_energy_and_gradient(L_BENCH, holes, C2, C3, device=dev, precision="mixed", eps=1e-10,
                                               mixed_eps=1e-8, lambda_tol=1e-8, info=info2,
                                               engine=info["engine"])
        runs.append(info2)
    runs.sort(key=lambda r: r["t_forward"] + r["t_lambda"])
    info2 = runs[1]

    def etot(c2, c3):
        v, w = ham.contact_couplings(c2, c3)
        e_ref, fock, two = ham.normal_ordered_hamiltonian(L_BENCH, holes, v, v, w, dense=False)
        plan, _ = S.detect(fock, two)
        eng = StructuredEngine(plan, fock, dev)
        e, _, _ = solve_structured(eng, eps=1e-14, maxSteps=6000, max_diis=8, t2_format="compact")
        return e + e_ref

    h = 1e-4
    fd2 = (etot(C2 + h, C3) - etot(C2 - h, C3)) / (2 * h)
    fd3 = (etot(C2, C3 + h) - etot(C2, C3 - h)) / (2 * h)
    return {"dE_dC2": g2, "dE_dC3": g3, "fd_dE_dC2": fd2, "fd_dE_dC3": fd3,
            "rel_err_vs_fd": [abs(g2 - fd2) / abs(fd2), abs(g3 - fd3) / abs(fd3)],
            "t_forward_s": info2["t_forward"], "t_lambda_s": info2["t_lambda"],
            "lambda_over_forward": info2["t_lambda"] / info2["t_forward"],
            "lambda_iters": info2["lambda_iters"], "forward_iters": info2["iterations"],
            "lambda_iters_fp32": info2.get("lambda_iters_fp32"), "lambda_path": info2.get("lambda_path"),
            "t_lambda_fp32_phase_s": info2.get("t_lambda_fp32"), "t_lambda_fp64_phase_s": info2.get("t_lambda_fp64")}


def e2e_leg(args, fock, two, dev):
    """The public ccsd_solver on host (numpy) inputs: H2D of the Hamiltonian,
    plan build, mixed solve, D2H of E, t1 and the compact t2."""
    import numpy as np
    import torch
    from nulattice_b200 import ccsd_solver
    h2d = sum(np.asarray(f).nbytes for f in fock) + sum(
        (b.indices.nbytes + b.values.nbytes) if hasattr(b, "indices") else np.asarray(b).nbytes for b in two)
    times, phases = [], {}
    for k in range(args.warmup + args.steps):
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        info = {}
        e, t1, t2 = ccsd_solver(fock, two, eps=1e-8, maxSteps=4000, max_diis=8, device=dev, precision="mixed",
                                mixed_eps=1e-8, t2_format="compact", info=info)
        b.record()
        torch.cuda.synchronize()
        if k >= args.warmup:
            times.append(a.elapsed_time(b) / 1e3)
            for name in ("t_detect", "t_engine", "t_solve", "t_output"):
                phases.setdefault(name, []).append(info.get(name, 0.0))
    d2h = 8 + t1.nbytes + t2.nbytes
    return {"value": statistics.mean(times), "unit": "s", "h2d_bytes_per_step": int(h2d),
            "d2h_bytes_per_step": int(d2h), "iterations": info.get("iterations"),
            "phases_ms": {k: round(statistics.mean(v) * 1e3, 3) for k, v in phases.items()},
            "path": "ccsd_solver(numpy inputs): structure detection, engine build, eager mixed solve, "
                    "E/t1/compact-t2 to host (page-locked)"}


if __name__ == "__main__":
    main()
