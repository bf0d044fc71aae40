"""The work that a user of this framework has it do, as cases that can be timed and compared.

Every case is one call path a program takes through the public entry points:

* ``solver``    ``ccsd_solver`` on host arrays, results back on the host;
* ``engine``    ``solve_structured`` on an engine the program keeps (a fixed number of steps);
* ``lambda``    the Lambda iteration at converged amplitudes (``LambdaSolver.run``, a fixed number of steps);
* ``gradient``  ``ccsd_energy_and_gradient``: energy and coupling derivatives, everything included;
* ``batch``     one launch of a ``BatchScan`` over instances of uneven size;
* ``momentum``  ``momentum.solve`` on a plane-wave engine the program keeps;
* ``general``   ``ccsd_solver`` on open-shell inputs (the general engine).

Sizes: lattices L = 3 .. 6, nuclei of closed sites (A = 4 ``sites``; 1 and 7 are the configurations of the
benchmark, the others generic) and closed momentum shells (A = 4, 28), FP64 and mixed precision.  A fixed number
of steps makes a pass the same work whatever the rounding of a kernel; the calls that iterate to a tolerance use
one that FP32 rounding does not blur.  The extrapolation of a DIIS pulse multiplies rounding by 1e3 to 1e10 (its
error vectors are nearly parallel, most of all in plane waves), so the passes of fixed steps are the nine before
the first pulse of the default subspace of ten, error vectors stored; the pulses run in the FP64 passes of the
lattice engine and in the whole solves.
"""
import math

import numpy as np
import torch

import nulattice_b200 as nlb
from nulattice_b200 import _lib, adjoint, batch, ccsd, hamiltonian, momentum, planewave, structure, tune

SEVEN = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the smallest configuration, through the drop-in entry point: ⁴He on 3^3 sites, the NumPy algorithm
        # (Jacobi, no DIIS) to 1e-10; launches and host work count
        dict(name="solver_A4_L3_fp64", kind="solver", L=3, sites=1, precision="fp64"),
        # ⁴He on 5^3 sites on an engine in hand: small kernels, one graph launch
        dict(name="engine_A4_L5_fp64", kind="engine", L=5, sites=1, precision="fp64", steps=20, diis=8),
        # an ordinary size of the scans: 28 nucleons on 4^3 sites, FP32 amplitudes
        dict(name="engine_A28_L4_fp32", kind="engine", L=4, sites=7, precision="fp32", steps=9, diis=10),
        # the headline size, 28 nucleons on 6^3 sites: the FP32 phase of the mixed solve ...
        dict(name="engine_A28_L6_fp32", kind="engine", L=6, sites=7, precision="fp32", steps=9, diis=10),
        # ... and the plain FP64 solve
        dict(name="engine_A28_L6_fp64", kind="engine", L=6, sites=7, precision="fp64", steps=20, diis=8),
        # the headline size end to end: host arrays in, mixed solve (FP32, then FP64), compact amplitudes out
        dict(name="solver_A28_L6_mixed", kind="solver", L=6, sites=7, precision="mixed"),
        # the backward direction: Lambda multipliers at the headline size, FP32 phase
        dict(name="lambda_A28_L6_fp32", kind="lambda", L=6, sites=7, precision="fp32", steps=9, diis=10),
        # energy and both coupling derivatives in one call, the default precision of the torch function
        dict(name="gradient_A28_L4_fp64", kind="gradient", L=4, sites=7, precision="fp64"),
        # a scan over nuclei, lattices and couplings in one graph launch
        dict(name="batch_6", kind="batch", count=6, L=5),
        # plane waves, closed shells of 28 nucleons, FP64 (the default) ...
        dict(name="momentum_A28_L6_fp64", kind="momentum", L=6, A=28, precision="fp64", steps=9, diis=10),
        # ... and the FP32 phase of a mixed plane-wave solve of a small nucleus
        dict(name="momentum_A4_L5_fp32", kind="momentum", L=5, A=4, precision="fp32", steps=9, diis=10),
        # open-shell ³He through the general engine, tensor-core phase of the mixed solve
        dict(name="general_he3_L4_mixed", kind="general", L=4, nucleus="he3", precision="mixed", steps=9, diis=10),
    ]


def draw(rng):
    kind = rng.choice(["engine", "engine", "engine", "lambda", "lambda", "momentum", "momentum", "solver", "gradient",
                       "batch", "general"])
    before = dict(steps=rng.randint(4, 9), diis=10)      # no pulse
    pulsed = dict(steps=rng.randint(4, 20), diis=8)
    if kind == "engine":
        precision = rng.choice(["fp32", "fp64"])
        return dict(kind=kind, L=rng.choice([3, 4, 5, 5, 6]), sites=rng.choice([1, 2, 3, 5, 7, 7, 7, 7]),
                    precision=precision, **(pulsed if precision == "fp64" else before))
    if kind == "lambda":
        sites = rng.choice([1, 3, 7, 7, 7])
        precision = rng.choice(["fp32", "fp64"]) if sites == 7 else "fp64"
        return dict(kind=kind, L=rng.choice([3, 4, 5, 6] if sites == 7 else [3, 4, 5]), sites=sites,
                    precision=precision, **before)
    if kind == "momentum":
        return dict(kind=kind, L=rng.randint(3, 6), A=rng.choice([4, 28]), precision=rng.choice(["fp32", "fp64"]),
                    **before)
    if kind == "solver":
        return dict(kind=kind, L=rng.randint(3, 5), sites=rng.choice([1, 2, 7]),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "gradient":
        return dict(kind=kind, L=rng.choice([3, 4, 5]), sites=rng.choice([1, 7]), precision=rng.choice(["fp64", "mixed"]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 6), L=rng.choice([4, 5]))
    return dict(kind=kind, L=rng.choice([3, 4]), nucleus=rng.choice(["he3", "li6"]),
                precision=rng.choice(["fp64", "mixed"]), **before)


def _couplings(seed, k=0):
    """(C2, C3) in hbar^2/(M a^2): around the benchmark's (-3, 1), inside the range where CCSD converges quickly."""
    rng = np.random.default_rng([int(seed), k])
    return float(rng.uniform(-3.4, -2.8)), float(rng.uniform(0.5, 1.1))


def _holes(L, sites):
    return [[x % L, y % L, z % L, t, s] for (x, y, z) in SEVEN[:sites] for t in (0, 1) for s in (0, 1)]


def _open_holes(nucleus):
    if nucleus == "he3":
        return [[0, 0, 0, 0, 0], [0, 0, 0, 0, 1], [0, 0, 0, 1, 0]]
    return [[0, 0, 0, t, s] for t in (0, 1) for s in (0, 1)] + [[1, 0, 0, 0, 0], [1, 0, 0, 1, 1]]


def _instances(case, seed):
    """(A, L, C2, C3) of a scan: sizes from a fixed cycle, couplings from the seed."""
    size = [(28, case["L"]), (4, case["L"]), (28, 4), (4, 6), (28, 4), (4, 4)]
    return [size[k] + _couplings(seed, k) for k in range(case["count"])]


# ----------------------------------------------------------------- inputs --
def _engine(case, seed):
    C2, C3 = _couplings(seed)
    _, fock, two = nlb.normal_ordered_hamiltonian(case["L"], _holes(case["L"], case["sites"]), 2 * C2, 2 * C2, 2 * C3,
                                                  dense=False)
    plan, why = structure.detect(fock, two)
    if plan is None:
        raise ValueError(why)
    eng = ccsd.StructuredEngine(plan, fock, torch.device("cuda", torch.cuda.current_device()))
    eng.prob.tune = tune.known_word(eng)
    return eng


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    C2, C3 = _couplings(seed)
    if kind == "solver":
        _, state["fock"], state["two"] = nlb.normal_ordered_hamiltonian(
            case["L"], _holes(case["L"], case["sites"]), 2 * C2, 2 * C2, 2 * C3, dense=False)
    elif kind == "engine":
        state["eng"] = _engine(case, seed)
    elif kind == "lambda":
        eng = state["eng"] = _engine(case, seed)
        _, t1, t2 = ccsd.solve_structured(eng, eps=1e-12, max_diis=8, t2_format="compact", loop="eager")
        solver = state["solver"] = adjoint.LambdaSolver(eng)
        b = state["buffers"] = solver.buffers(_lib.NLB_F32 if case["precision"] == "fp32" else _lib.NLB_F64, case["diis"])
        b["t1"].copy_(t1.reshape(-1))
        b["t2"].copy_(t2)
        eng._bufs.clear()      # the forward buffers are not needed any more
    elif kind == "gradient":
        state["holes"] = _holes(case["L"], case["sites"])
        state["C"] = (C2, C3)
    elif kind == "batch":
        state["scan"] = batch.BatchScan(_instances(case, seed), device="cuda", mixed_eps=1e-6,
                                        autotune=False)
    elif kind == "momentum":
        plan = momentum.MomentumPlan(case["L"], planewave.momentum_holes(case["L"], case["A"]))
        V = momentum.contact_tensor(case["L"], plan.n_k, 2 * C2, 2 * C2, 2 * C3)
        fpp, fhh, _ = momentum.fock_blocks(case["L"], plan.n_k, plan.hmom, plan.pmom, 2 * C2, 2 * C2, 2 * C3)
        state["args"] = (plan, V, fpp, fhh)
        state["eng"] = momentum.MomentumEngine(*state["args"], device="cuda")
    else:
        _, state["fock"], state["two"] = nlb.normal_ordered_hamiltonian(
            case["L"], _open_holes(case["nucleus"]), 2 * C2, 1.8 * C2, 2 * C3, dense=True)
    return state


# -------------------------------------------------------------------- run --
def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "solver":
        small = case["sites"] == 1
        return nlb.ccsd_solver(state["fock"], state["two"], eps=1e-10 if case["precision"] == "fp64" else 1e-11,
                               maxSteps=100, max_diis=8, criterion="numpy" if small else "soa",
                               precision=case["precision"], mixed_eps=1e-6, t2_format="dense" if small else "compact")
    if kind == "engine":
        fp32 = case["precision"] == "fp32"
        return ccsd.solve_structured(state["eng"], eps=0.0, mixed_eps=0.0, maxSteps=case["steps"], max_diis=case["diis"],
                                     precision="mixed" if fp32 else "fp64", refine=False, t2_format="compact")
    if kind == "lambda":
        b = state["buffers"]
        c = state["solver"].run(b, 0.0, 0.5, case["steps"], case["diis"], False)
        return b["lam1"][c.parity], b["lam2"][c.parity]
    if kind == "gradient":
        return np.array(adjoint.ccsd_energy_and_gradient(case["L"], state["holes"], *state["C"], device="cuda",
                                                         precision=case["precision"], eps=1e-11, lambda_tol=1e-9))
    if kind == "batch":
        state["scan"].launch()
        res = state["scan"].results()
        return [np.array([r[k] for r in res]) for k in ("E_corr", "E", "dE_dC2", "dE_dC3")]
    if kind == "momentum":
        fp32 = case["precision"] == "fp32"
        return momentum.solve(*state["args"], engine=state["eng"], eps=0.0, mixed_eps=0.0, maxSteps=case["steps"],
                              max_diis=case["diis"], precision="mixed" if fp32 else "fp64")
    return nlb.ccsd_solver(state["fock"], state["two"], eps=0.0, mixed_eps=0.0, maxSteps=case["steps"], max_diis=case["diis"],
                           precision=case["precision"])


# ------------------------------------------------------------------- work --
def _n_t2(L, sites):
    return 6 * (L ** 3 - sites) ** 2 * sites ** 2


def _struct_work(L, sites, s, steps):
    """Per step: read t2, write t2, write its error vector and read it once for the extrapolation; per amplitude
    the f_pp stencils (7 + 7), the hole mixing (h + h) and the rank-h parts (h + h)."""
    n = _n_t2(L, sites)
    return steps * 4 * n * s, steps * n * 2 * (14 + 4 * sites)


def _momentum_size(L, A):
    """Amplitudes of the momentum blocks and multiply-adds per step."""
    h = A // 4
    n = 256 * h * h * (L ** 3 - 2 * h)
    return n, n * 2 * (16 + 16 + 2 * 16 + 8.0 * h)


def work(case):
    kind = case["kind"]
    if kind == "solver":
        s = 8 if case["precision"] == "fp64" else 4
        b, f = _struct_work(case["L"], case["sites"], s, 60 if case["sites"] == 1 else 14)
        if case["precision"] == "mixed":
            b2, f2 = _struct_work(case["L"], case["sites"], 8, 18)
            b, f = b + b2, f + f2
        return dict(bytes=b, flops=f)
    if kind == "engine":
        b, f = _struct_work(case["L"], case["sites"], 4 if case["precision"] == "fp32" else 8, case["steps"])
        return dict(bytes=b, flops=f)
    if kind == "lambda":
        # the amplitudes are read beside the multipliers
        b, f = _struct_work(case["L"], case["sites"], 4 if case["precision"] == "fp32" else 8, case["steps"])
        return dict(bytes=b * 5 / 4, flops=f * 1.6)
    if kind == "gradient":
        b, f = _struct_work(case["L"], case["sites"], 8, 24)
        return dict(bytes=b * 9 / 4, flops=f * 2.6)
    if kind == "batch":
        b = f = 0.0
        for A, L, _, _ in _instances(case, 0):
            for s, n in ((4, 16), (8, 8)):
                x, y = _struct_work(L, A // 4, s, n)
                b, f = b + 9 / 4 * x, f + 2.6 * y
        return dict(bytes=b, flops=f)
    if kind == "momentum":
        n, f = _momentum_size(case["L"], case["A"])
        return dict(bytes=case["steps"] * 4 * n * (4 if case["precision"] == "fp32" else 8), flops=case["steps"] * f)
    h = len(_open_holes(case["nucleus"]))
    p = 4 * case["L"] ** 3 - h
    # t2 read and written, its error vector written and read; four (ph)^3 products
    return dict(bytes=case["steps"] * 4 * 8.0 * p * p * h * h, flops=case["steps"] * 4 * 2.0 * (p * h) ** 3)


def tolerance(case):
    """About four times the largest difference from ``exact`` over the declared ranges."""
    kind, precision = case["kind"], case.get("precision")
    if kind == "solver":
        if precision == "mixed":          # where the energy test at 1e-11 leaves the amplitudes
            return {"rel": 1e-7, "max": 3e-6}
        # Jacobi steps alone, or with extrapolations (which multiply the rounding)
        return {"rel": 1e-13, "max": 1e-11} if case["sites"] == 1 else {"rel": 1e-8, "max": 1e-6}
    if kind == "engine":
        if precision == "fp32":
            return {"rel": 4e-7, "max": 1e-6}
        return {"rel": 2e-14, "max": 1e-12} if case["steps"] < case["diis"] else {"rel": 1e-7, "max": 2e-6}
    if kind == "lambda":                  # in FP64 the convergence of the amplitudes that it starts from
        return {"rel": 2.5e-7, "max": 1e-6} if precision == "fp32" else {"rel": 1e-8, "max": 1e-7}
    if kind == "gradient":
        return {"rel": 1e-9, "max": 1e-9}
    if kind == "batch":                   # the energy test at 1e-10 can pass by chance between two extrapolations
        return {"rel": 1e-6, "max": 1e-6}
    if kind == "momentum":
        return {"rel": 6e-7, "max": 1.5e-6} if precision == "fp32" else {"rel": 1e-14, "max": 1e-13}
    # three TF32 products with FP32 sums in the mixed phase
    return {"rel": 3e-5, "max": 1e-4} if precision == "mixed" else {"rel": 2e-11, "max": 1e-10}


# ------------------------------------------- the same results in plain torch --
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=_dev())


def _diis(errs, hist, weights):
    """Pulsed DIIS: the extrapolated amplitudes of the stored steps, or None where the system is singular.
    ``errs``, ``hist``: lists of tuples of tensors; ``weights``: how often each tensor counts in the Gram matrix."""
    m = len(errs)
    B = torch.tensor([[float(sum(w * torch.dot(x.reshape(-1), y.reshape(-1)) for w, x, y in zip(weights, a, b)))
                       for b in errs] for a in errs], dtype=torch.float64)
    A = -torch.ones(m + 1, m + 1, dtype=torch.float64)
    A[:m, :m] = B / (B.abs().max() + 1e-16)
    A[m, m] = 0.0
    rhs = torch.zeros(m + 1, dtype=torch.float64)
    rhs[m] = -1.0
    try:
        c = torch.linalg.solve(A, rhs)[:m]
    except RuntimeError:
        return None
    return tuple(sum(float(c[k]) * hist[k][q] for k in range(m)) for q in range(len(hist[0])))


class _Lattice:
    """A closed-site nucleus on the periodic lattice.  The contact treats the four spin-isospin labels alike, so
    every label has the same t1[a, i] and every pair of labels the same t2[a, b, i, j] (sites a, b; hole sites i, j)."""

    def __init__(self, L, sites, C2, C3):
        v, w = 2 * C2, 2 * C3
        hole = [((x % L) * L + y % L) * L + z % L for x, y, z in SEVEN[:sites]]
        part = [s for s in range(L ** 3) if s not in hole]
        F = np.zeros((L ** 3, L ** 3))
        for s in range(L ** 3):
            c = (s // (L * L), (s // L) % L, s % L)
            F[s, s] += 6.0
            for d in range(3):
                for e in (1, -1):
                    q = list(c)
                    q[d] = (q[d] + e) % L
                    F[s, (q[0] * L + q[1]) * L + q[2]] -= 1.0
        self.n, self.nh, self.v, self.w = len(part), sites, v, w
        self.f_pp, self.f_ph = _t(F[np.ix_(part, part)]), _t(F[np.ix_(part, hole)])
        # three other nucleons on a hole site, three pairs of them
        self.f_hh = _t(F[np.ix_(hole, hole)] + (3 * v + 3 * w) * np.eye(sites))
        self.vpp, self.vhh = v * torch.eye(self.n, **_kw()), (v + 2 * w) * torch.eye(sites, **_kw())
        self.e_ref = sites * (24 + 6 * v + 4 * w)

    def start(self):
        den = torch.diagonal(self.f_hh)[None, :] - torch.diagonal(self.f_pp)[:, None]
        return self.f_ph / den, torch.zeros(self.n, self.n, self.nh, self.nh, **_kw())

    def energy(self, t):
        return 4.0 * float((self.f_ph * t).sum())

    def dressed(self, t, x):
        """X_pp and X_hh with the factor x (1/2 in the T1 equation, 1 in the T2 equation)."""
        return self.f_pp - x * t @ self.f_ph.T, -self.f_hh - x * self.f_ph.T @ t

    def r1(self, t, B):
        xp, xh = self.dressed(t, 0.5)
        return self.f_ph + 3.0 * torch.einsum("ck,acik->ai", self.f_ph, B) + xp @ t + t @ xh

    def r2(self, ta, tb, B):
        n, nh = self.n, self.nh
        (pa, ha), (pb, hb) = self.dressed(ta, 1.0), self.dressed(tb, 1.0)
        along_a = (pa @ B.reshape(n, -1)).reshape(B.shape)
        along_b = (pb @ B.reshape(n, n, nh * nh))
        mix = torch.einsum("ki,abkj->abij", ha, B) + torch.einsum("kj,abik->abij", hb, B)
        tau = B + ta[:, None, :, None] * tb[None, :, None, :]
        return along_a + along_b.reshape(B.shape) + mix + (self.vpp[:, :, None, None] + self.vhh) * tau

    def denominators(self, t):
        (p1, h1), (p2, h2) = self.dressed(t, 0.5), self.dressed(t, 1.0)
        dg = torch.diagonal
        d1 = -(dg(p1)[:, None] + dg(h1)[None, :])
        dp, dh = dg(p2), dg(h2)
        d2 = -(dp[:, None, None, None] + dp[None, :, None, None] + dh[:, None] + dh[None, :])
        return d1, d2

    def solve(self, t, B, e, eps, steps, diis, criterion="soa"):
        """Jacobi steps with mixing 1/2; returns (E, t, B, steps)."""
        errs, hist = [], []
        for it in range(1, steps + 1):
            d1, d2 = self.denominators(t)
            nt, nB = t + 0.5 * self.r1(t, B) / d1, B + 0.5 * self.r2(t, t, B) / d2
            prev, e = e, self.energy(nt)
            errs.append((nt - t, nB - B))
            hist.append((nt, nB))
            t, B = nt, nB
            if abs(e - prev) / (max(1.0, abs(e)) if criterion == "soa" else abs(e)) < eps:
                break
            if not diis or criterion != "soa":
                errs, hist = [], []
            elif len(errs) == diis:
                got = _diis(errs, hist, (4.0, 24.0))
                t, B = got if got is not None else (t, B)
                errs, hist = [], []
        return e, t, B, it

    def converged(self):
        t, B = self.start()
        return self.solve(t, B, self.energy(t), 1e-13, 200, 8)

    def multipliers(self, t, B, steps, tol=0.0, diis=8):
        """The Lambda equations at (t, B) from zero: Jacobi steps with the forward denominators, DIIS."""
        d1, d2 = self.denominators(t)
        l1, l2 = torch.zeros_like(t), torch.zeros_like(B)
        errs, hist = [], []
        for _ in range(steps):
            z1, z2 = self.adjoint(t, B, l1, l2)
            n1, n2 = l1 + 0.5 * z1 / d1, l2 + 0.5 * z2 / d2
            errs.append((n1 - l1, n2 - l2))
            hist.append((n1, n2))
            l1, l2 = n1, n2
            norm = lambda x, y: math.sqrt(4 * float((x * x).sum()) + 24 * float((y * y).sum()))  # noqa: E731
            if norm(*errs[-1]) < tol * max(1.0, norm(l1, l2)):
                break
            if len(errs) == diis:
                got = _diis(errs, hist, (4.0, 24.0))
                l1, l2 = got if got is not None else (l1, l2)
                errs, hist = [], []
        return l1, l2

    def adjoint(self, t, B, l1, l2):
        """Z1 and Z2: the derivatives of E + <lam1, R1> + <Lam, R2> by one label's t1 and one label pair's t2."""
        with torch.enable_grad():
            x, y, z = (u.detach().clone().requires_grad_(True) for u in (t, B, t))
            # of the three pairs that hold a label, each gives <Lam, R2> by that label's t1
            s1 = (self.f_ph * x).sum() + (l1 * self.r1(x, y.detach())).sum() \
                + 3.0 * (l2 * self.r2(x, z.detach(), y.detach())).sum()
            z1, = torch.autograd.grad(s1, x)
            s2 = (l2 * self.r2(t, t, y)).sum()
            z2, = torch.autograd.grad(s2, y)
        f = self.f_ph
        return z1, z2 + l1[:, None, :, None] * f[None, :, None, :] + f[:, None, :, None] * l1[None, :, None, :]

    def coupling_derivatives(self, t, B, l1, l2):
        """dE/dC2 and dE/dC3: the residuals depend on v and w through f_hh and the two ladders."""
        eye = torch.eye(self.nh, **_kw())
        tau = B + t[:, None, :, None] * t[None, :, None, :]
        mix = torch.einsum("ki,abkj->abij", eye, B) + torch.einsum("kj,abik->abij", eye, B)
        out = []
        for dfh, dhh, dpp, dref in ((3.0, 1.0, 1.0, 6.0), (3.0, 2.0, 0.0, 4.0)):
            r1 = -dfh * t
            lad = dhh * eye + (dpp * torch.eye(self.n, **_kw()))[:, :, None, None]
            r2 = -dfh * mix + lad * tau
            out.append(2.0 * (self.nh * dref + 4.0 * float((l1 * r1).sum()) + 6.0 * float((l2 * r2).sum())))
        return out

    def full_t1(self, t):
        out = torch.zeros(self.n, 4, self.nh, 4, **_kw())
        for g in range(4):
            out[:, g, :, g] = t
        return out.reshape(4 * self.n, 4 * self.nh)

    def full_t2(self, B):
        out = torch.zeros(self.n, 4, self.n, 4, self.nh, 4, self.nh, 4, **_kw())
        for g in range(4):
            for k in range(4):
                if g != k:
                    out[:, g, :, k, :, g, :, k] = B
                    out[:, g, :, k, :, k, :, g] = -B.transpose(2, 3)
        return out.reshape(4 * self.n, 4 * self.n, 4 * self.nh, 4 * self.nh)


def _kw():
    return dict(dtype=torch.float64, device=_dev())


def _contact(vT1, vS1):
    """On-site antisymmetric matrix elements <pq||rs> of the spin-isospin states 2 tz + sz."""
    V = np.zeros((4, 4, 4, 4))
    for p in range(4):
        for q in range(4):
            if p == q:
                continue
            same_t, same_s = p // 2 == q // 2, p % 2 == q % 2
            direct = vT1 if same_t else vS1 if same_s else 0.5 * (vS1 + vT1)
            V[p, q, p, q] += direct
            V[p, q, q, p] -= direct
            if not same_t and not same_s:
                # (tz, sz) pairs (00, 11) and (01, 10) mix
                r, s = p ^ 1, q ^ 1
                x = 0.5 * (vS1 - vT1)
                x = x if (p < q) == (r < s) else -x
                V[p, q, r, s] += x
                V[p, q, s, r] -= x
    return V


class _PlaneWaves:
    """Closed momentum shells: t2[i, j, a; s_i, s_j, s_a, s_b] over hole momenta i, j and a particle momentum a (the
    other one, b = i + j - a, follows; entries whose a or b is a hole are zero)."""

    def __init__(self, L, A, C2, C3):
        h = A // 4
        v, w = 2 * C2, 2 * C3
        n3 = self.n3 = L ** 3
        xyz = np.stack([np.arange(n3) // (L * L), (np.arange(n3) // L) % L, np.arange(n3) % L], 1)
        index = lambda c: ((c[..., 0] % L) * L + c[..., 1] % L) * L + c[..., 2] % L  # noqa: E731
        hole = self.hole = np.sort(np.array([index(np.array(s)) for s in SEVEN[:h]]))
        V = _contact(v, v) / n3
        kin = (2.0 - 2.0 * np.cos(2.0 * np.pi * xyz / L)).sum(1)
        trace = h * np.einsum("asbs->ab", V)
        f3 = 0.5 * (3 * h) * (2 * h) * w / L ** 6
        V = self.V = V + _contact(2.0 * h * w / n3, 2.0 * h * w / n3) / n3
        f = kin[:, None, None] * np.eye(4) + trace + f3 * np.eye(4)
        self.fpp, self.fhh = _t(f), _t(f[hole])
        i, j = np.meshgrid(np.arange(h), np.arange(h), indexing="ij")
        K = self.K = index(xyz[hole][:, None] + xyz[hole][None, :])           # [i, j]
        b = index(xyz[K][:, :, None] - xyz[None, None])                       # [i, j, a]
        is_hole = np.isin(np.arange(n3), hole)
        self.live = ~is_hole[None, None, :] & ~is_hole[b]
        dev = _dev()
        self.b = torch.as_tensor(b, device=dev)
        self.mask = torch.as_tensor(self.live, device=dev)[..., None, None, None, None]
        self.ij = [torch.as_tensor(x, device=dev)[:, :, None].expand(h, h, n3) for x in (i, j)]
        Ks = self.Ks = np.unique(K)
        self.group = torch.as_tensor(np.searchsorted(Ks, K).reshape(-1), device=dev)
        self.h, self.V = h, _t(V)

    def swap_ab(self, x):
        """x[i, j, a; si, sj, sa, sb] -> x[i, j, b; si, sj, sb, sa]."""
        return x[self.ij[0], self.ij[1], self.b].transpose(-1, -2)

    def swap_ij(self, x):
        return x.transpose(0, 1).transpose(3, 4)

    def start(self):
        ep, eh = torch.diagonal(self.fpp, dim1=1, dim2=2), torch.diagonal(self.fhh, dim1=1, dim2=2)
        den = self.sums(-ep, eh)
        vijab = self.V.permute(2, 3, 0, 1)
        return torch.where(self.mask, vijab / torch.where(self.mask, den, 1.0), 0.0)

    def sums(self, dp, dh):
        """dp[a, sa] + dp[b, sb] + dh[i, si] + dh[j, sj]."""
        return dp[None, None, :, None, None, :, None] + dp[self.b][:, :, :, None, None, None, :] \
            + dh[:, None, None, :, None, None, None] + dh[None, :, None, None, :, None, None]

    def energy(self, T):
        return 0.25 * float(torch.einsum("abij,klmijab->", self.V, T))

    def step(self, T):
        V, h, b = self.V, self.h, self.b
        M = T.sum(2)                                                          # [i, j; si, sj, sc, sd]
        N = torch.zeros(len(self.Ks), *T.shape[2:], **_kw())
        N.index_add_(0, self.group, T.reshape(h * h, *T.shape[2:]))           # [K, a; sk, sl, sa, sb]
        N = N[self.group].reshape(T.shape)
        H = V.permute(2, 3, 0, 1)[None, None, None] + 0.5 * torch.einsum("abcd,xyijcd->xyijab", V, M)[:, :, None]
        W = 0.5 * V[None, None] + 0.25 * torch.einsum("cdkl,xyijcd->xyklij", V, M)
        H = H + torch.einsum("xyklij,xyzklab->xyzijab", W, N)
        R = T.sum(1)                                                          # [i, a; si, sk, sa, sc]
        xpp = self.fpp - 0.5 * torch.einsum("cdkl,xyzklbd->zbc", V, T)
        xhh = -self.fhh - 0.5 * torch.einsum("cdkl,xyjlcd->xkj", V, M)
        xb = xpp[b]
        H = H + torch.einsum("xyzbc,xyzijac->xyzijab", xb, T) + torch.einsum("zac,xyzijcb->xyzijab", xpp, T)
        H = H + torch.einsum("ykj,xyzikab->xyzijab", xhh, T) + torch.einsum("xki,xyzkjab->xyzijab", xhh, T)
        ring = -torch.einsum("bkcj,xzikac->xzijab", V, R)[:, None].expand(T.shape)
        U = torch.einsum("cdkl,xzikac->xziald", V, R)                         # [i, a; si, sa, sl, sd]
        Rb = R[self.ij[1], b]                                                 # [i, j, a; sj, sl, sb, sd]
        ring = ring + 0.5 * torch.einsum("xziald,xyzjlbd->xyzijab", U, Rb)
        ring = ring - self.swap_ab(ring)
        H = H + ring - self.swap_ij(ring)
        H = H - self.swap_ab(H)
        H = 0.25 * (H - self.swap_ij(H))
        dg = lambda x: torch.diagonal(x, dim1=1, dim2=2)  # noqa: E731
        D = -self.sums(dg(xpp), dg(xhh))
        return torch.where(self.mask, T + 0.5 * H / D, 0.0)

    def solve(self, steps, diis):
        T = self.start()
        errs, hist, e = [], [], self.energy(T)
        for _ in range(steps):
            n = self.step(T)
            errs.append((n - T,))
            hist.append((n,))
            T, e = n, self.energy(n)
            if len(errs) == diis:
                got = _diis(errs, hist, (1.0,))
                T = got[0] if got is not None else T
                errs, hist = [], []
        return e, T

    def blocks(self, T):
        """The blocked order: total momenta ascending; rows (a, sa, sb), columns (i, si, sj)."""
        out = []
        for K in self.Ks:
            i, j = np.nonzero(self.K == K)
            x = T[torch.as_tensor(i), torch.as_tensor(j)][:, torch.as_tensor(self.live[i[0], j[0]])]
            out.append(x.permute(1, 4, 5, 0, 2, 3).reshape(-1))
        return torch.cat(out)


# T1 and T2 diagrams of the full equations: (factor, einsum, operands, antisymmetriser of abij)
_H1 = [(1, "ck,acik->ai", "f T", ""), (-1, "akci,ck->ai", "phph t", ""), (-.5, "cikl,cakl->ai", "phhh T", ""),
       (1, "cdkl,ck,dali->ai", "pphh t T", "")]
_XH1 = [(-.5, "ck,ci->ki", "f t"), (-1, "bijk,bj->ki", "phhh t"), (-.5, "cdlk,cdli->ki", "pphh T"),
        (-.5, "cdlk,cl,di->ki", "pphh t t")]
_XP1 = [(-.5, "ck,ak->ac", "f t"), (-.5, "dckl,dakl->ac", "pphh T"), (.5, "cdkl,dk,al->ac", "pphh t t")]
_XH2 = [(-1, "ck,cj->kj", "f t"), (-.5, "cdkl,cdjl->kj", "pphh T"), (-1, "cdlk,cl,dj->kj", "pphh t t")]
_XP2 = [(-1, "ck,bk->bc", "f t"), (-.5, "cdkl,bdkl->bc", "pphh T"), (-1, "cdlk,dk,bl->bc", "pphh t t")]
_H2 = [(.5, "klij,abkl->abij", "hhhh T", ""), (.5, "klij,ak,bl->abij", "hhhh t t", "ab"),
       (-1, "bkcj,acik->abij", "phph T", "abij"), (-1, "bkci,ak,cj->abij", "phph t t", "abij"),
       (1, "bkij,ak->abij", "phhh t", "ab"), (-1, "cikl,ck,ablj->abij", "phhh t T", "ij"),
       (-1, "cikl,al,bcjk->abij", "phhh t T", "abij"), (.5, "cjkl,ci,abkl->abij", "phhh t T", "ij"),
       (.5, "cjkl,ci,ak,bl->abij", "phhh t t t", "abij"), (.5, "cdkl,acik,dblj->abij", "pphh T T", "abij"),
       (.25, "cdkl,cdij,abkl->abij", "pphh T T", ""), (.25, "cdkl,ci,dj,abkl->abij", "pphh t t T", "ij"),
       (.25, "cdkl,ak,bl,cdij->abij", "pphh t t T", "ab"), (1, "cdkl,ci,bl,adkj->abij", "pphh t t T", "abij"),
       (.25, "cdkl,ci,ak,dj,bl->abij", "pphh t t t t", "abij"), (-1, "da,dbij->abij", "r3 T", "ab"),
       (1, "acik,bcjk->abij", "r4 T", "abij"), (.5, "bijk,ak->abij", "r5 t", "ab"),
       (.5, "bijk,ak->abij", "r6 t", "abij"), (.5, "abcd,cdij->abij", "pppp T", ""), (1, "abij->abij", "r2", "ij"),
       (.5, "abcd,ci,dj->abij", "pppp t t", "ij"), (1, "bc,acij->abij", "xp T", "ab"),
       (1, "kj,abik->abij", "xh T", "ij")]


def _antisym(x, which):
    if "ab" in which:
        x = x - x.transpose(0, 1)
    if "ij" in which:
        x = x - x.transpose(2, 3)
    return x


class _General:
    """Open-shell inputs: the whole factorised equation set on dense tensors; v_pppp and v_ppph as row lists."""

    def __init__(self, fock, two):
        self.f_pp, self.f_ph, self.f_hh = (_t(x) for x in fock)
        self.p, self.h = self.f_ph.shape
        self.ops = dict(zip(("pphh", "phph", "phhh", "hhhh"), (_t(x) for x in two[2:])), f=self.f_ph)
        self.rows = [(torch.as_tensor(np.asarray(x)[:, :4].astype(np.int64), device=_dev()), _t(np.asarray(x)[:, 4]))
                     for x in two[:2]]

    def term(self, spec, names, ops):
        if names.startswith("pppp"):
            idx, val = self.rows[0]
            a, b, c, d = idx.T
            x = ops["T"][c, d] if names == "pppp T" else ops["t"][c][:, :, None] * ops["t"][d][:, None, :]
            out = torch.zeros(self.p * self.p, self.h, self.h, **_kw())
            out.index_add_(0, a * self.p + b, val[:, None, None] * x)
            return out.reshape(self.p, self.p, self.h, self.h)
        args = [ops[n] for n in names.split()]
        return args[0] if len(args) == 1 else torch.einsum(spec, *args)

    def ppph(self, t, T):
        """The intermediates of v_ppph[c, d, a, k]."""
        p, h = self.p, self.h
        idx, v = self.rows[1]
        c, d, a, k = idx.T
        z = lambda *s: torch.zeros(*s, **_kw())  # noqa: E731
        add = lambda n, where, x, *s: z(n, *s).index_add_(0, where, x)  # noqa: E731
        r0 = add(p, a, -0.5 * v[:, None] * T[c, d, k], h)
        r1 = add(p * p, a * p + d, -v * t[c, k]).reshape(p, p)
        r3 = add(p * p, d * p + a, v * t[c, k]).reshape(p, p)
        r2 = add(p * p * h, (c * p + d) * h + k, v[:, None] * t[a], h).reshape(p, p, h, h).transpose(2, 3)
        r4 = add(p * p * h, (a * p + d) * h + k, v[:, None] * t[c], h).reshape(p, p, h, h).transpose(2, 3)
        r5 = add(p * h, a * h + k, v[:, None, None] * T[c, d], h, h).reshape(p, h, h, h).permute(0, 2, 3, 1)
        r6 = add(p * h, a * h + k, v[:, None, None] * t[c][:, :, None] * t[d][:, None, :], h, h)
        return r0, r1, r2, r3, r4, r5, r6.reshape(p, h, h, h).permute(0, 2, 3, 1)

    def step(self, t, T):
        r = self.ppph(t, T)
        ops = dict(self.ops, t=t, T=T, r2=r[2], r3=r[3], r4=r[4], r5=r[5], r6=r[6])
        total = lambda start, terms: start + sum(x[0] * self.term(x[1], x[2], ops) for x in terms)  # noqa: E731
        h1, xh1, xp1 = total(self.f_ph + r[0], _H1), total(-self.f_hh, _XH1), total(self.f_pp + r[1], _XP1)
        ops["xh"], ops["xp"] = total(-self.f_hh, _XH2), total(self.f_pp, _XP2)
        h1 = h1 + xp1 @ t + t @ xh1
        h2 = self.ops["pphh"].clone()
        for x in _H2:
            h2 += x[0] * _antisym(self.term(x[1], x[2], ops), x[3])
        dg = torch.diagonal
        d1 = -(dg(xp1)[:, None] + dg(xh1)[None, :])
        dp, dh = dg(ops["xp"]), dg(ops["xh"])
        d2 = -(dp[:, None, None, None] + dp[None, :, None, None] + dh[:, None] + dh[None, :])
        return t + 0.5 * h1 / d1, T + 0.5 * h2 / d2

    def energy(self, t, T):
        v = self.ops["pphh"]
        return float((self.f_ph * t).sum() + 0.25 * (v * T).sum() + 0.5 * torch.einsum("abij,ai,bj->", v, t, t))

    def solve(self, steps, diis):
        ep, eh = torch.diagonal(self.f_pp), torch.diagonal(self.f_hh)
        t = self.f_ph / (eh[None, :] - ep[:, None])
        T = self.ops["pphh"] / (eh[:, None] + eh[None, :] - ep[:, None, None, None] - ep[None, :, None, None])
        errs, hist, e = [], [], 0.0
        for _ in range(steps):
            n, N = self.step(t, T)
            errs.append((n - t, N - T))
            hist.append((n, N))
            t, T = n, N
            e = self.energy(t, T)
            if len(errs) == diis:
                got = _diis(errs, hist, (1.0, 1.0))
                t, T = got if got is not None else (t, T)
                errs, hist = [], []
        return e, t, T


def exact(case, seed):
    with torch.no_grad():
        return _exact(case, seed)


def _exact(case, seed):
    kind = case["kind"]
    C2, C3 = _couplings(seed)
    if kind == "momentum":
        pw = _PlaneWaves(case["L"], case["A"], C2, C3)
        e, T = pw.solve(case["steps"], case["diis"])
        return e, pw.blocks(T)
    if kind == "general":
        s = prepare(case, seed)
        return _General(s["fock"], s["two"]).solve(case["steps"], case["diis"])
    if kind == "batch":
        out = [[], [], [], []]
        for A, L, c2, c3 in _instances(case, seed):
            lat = _Lattice(L, A // 4, c2, c3)
            e, t, B, _ = lat.converged()
            g = lat.coupling_derivatives(t, B, *lat.multipliers(t, B, 200, 1e-12))
            for x, y in zip(out, (e, e + lat.e_ref, *g)):
                x.append(y)
        return [np.array(x) for x in out]
    lat = _Lattice(case["L"], case["sites"], C2, C3)
    six = lambda B: B.reshape(1, -1).expand(6, -1).reshape(-1)  # noqa: E731
    if kind == "solver":
        small = case["sites"] == 1
        crit = "numpy" if small else "soa"
        t, B = lat.start()
        if case["precision"] == "fp64":
            e, t, B, _ = lat.solve(t, B, lat.energy(t), 1e-10, 100, 8, crit)
        else:
            e, t, B, _ = lat.converged()
        return e, lat.full_t1(t), lat.full_t2(B) if small else six(B)
    if kind == "engine":
        t, B = lat.start()
        e, t, B, _ = lat.solve(t, B, lat.energy(t), 0.0, case["steps"], case["diis"])
        return e, lat.full_t1(t), six(B)
    e, t, B, _ = lat.converged()
    if kind == "lambda":
        l1, l2 = lat.multipliers(t, B, case["steps"], diis=case["diis"])
        return lat.full_t1(l1).reshape(-1), six(l2)
    g = lat.coupling_derivatives(t, B, *lat.multipliers(t, B, 200, 1e-12))
    return np.array([e + lat.e_ref, g[0], g[1]])
