"""Label-symmetric problems: one label and one channel stand for all of them.

On the CPU the conditions under which the labels count as alike; on the GPU
every path that then runs on one label (solves, Lambda steps, gradients)
against the same path with every label stored."""
import numpy as np
import pytest
import torch

from nulattice_b200 import _lib
from nulattice_b200 import adjoint as A
from nulattice_b200 import hamiltonian as ham
from nulattice_b200 import structure as S
from nulattice_b200 import tune
from nulattice_b200.ccsd import StructuredEngine, solve_structured

SEVEN = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]


def _inputs(L, sites, C2=-3.1, C3=0.9):
    holes = [[x % L, y % L, z % L, t, s] for (x, y, z) in SEVEN[:sites] for t in (0, 1) for s in (0, 1)]
    v, w = ham.contact_couplings(C2, C3)
    _, fock, two = ham.normal_ordered_hamiltonian(L, holes, v, v, w, dense=False)
    return holes, [f.copy() for f in fock], two


@pytest.mark.parametrize("L,sites", [(3, 1), (3, 2), (4, 7)])
def test_lattice_labels_are_alike(L, sites):
    _, fock, two = _inputs(L, sites)
    plan, _ = S.detect(fock, two)
    one, m = S.alike_labels(plan, fock[2])
    assert m == 4 and one.n_labels == 1 and len(one.channels) == 1
    assert (one.p, one.h, one.n_t2) == (plan.p // 4, plan.h // 4, plan.n_t2 // 6)


@pytest.mark.parametrize("what", ["f_pp", "f_ph", "f_hh", "pp", "hh", "exchange"])
def test_labels_that_differ_are_not_alike(what):
    _, fock, two = _inputs(3, 2)
    plan, _ = S.detect(fock, two)
    P, H = plan.p_of[1], plan.h_of[1]
    if what == "f_pp":
        fock[0][P[3], P[3]] += 1e-9
    elif what == "f_ph":
        i, j = np.argwhere(fock[1][np.ix_(P, H)])[0]
        fock[1][P[i], H[j]] *= 1.5
    elif what == "f_hh":
        fock[2][H[0], H[0]] += 0.25
    plan, _ = S.detect(fock, two)
    if what == "pp":
        plan.pp_val[2] = plan.pp_val[2] * 2
    elif what == "hh":
        plan.hh_val[5] = plan.hh_val[5] + 1
    elif what == "exchange":   # the same in every channel, but not under exchange of the labels
        for n in range(6):
            plan.pp_ptr[n] = np.concatenate([[0, 0], np.ones(plan.channels[n].np1 ** 2 - 1, np.int64)])
            plan.pp_col[n], plan.pp_val[n] = np.array([1]), np.array([1.0])   # pair (0, 1) only
    assert S.alike_labels(plan, fock[2]) is None


def test_a_new_engine_has_its_tables():
    """The device problem of an engine exists before anything asks for it: a
    program may first use it inside a stream capture."""
    _, fock, two = _inputs(3, 1)
    plan, _ = S.detect(fock, two)
    eng = StructuredEngine(plan, fock, torch.device("cpu"))
    built = eng._prob
    assert built is not None and built.p == plan.p and eng.prob is built


def _engine(L, sites, full=False):
    holes, fock, two = _inputs(L, sites)
    plan, _ = S.detect(fock, two)
    eng = StructuredEngine(plan, fock, torch.device("cuda:0"))
    if full:
        eng.cache["reduced"] = None
    assert (eng.reduced() is None) == full
    return holes, eng


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites", [(3, 1), (3, 2), (4, 3), (3, 7), (4, 7), (5, 7)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 4e-7)])
def test_solve_on_one_label(L, sites, precision, tol):
    """Six steps before a DIIS pulse (rounding only), both layouts of t2, then
    a pulsed FP64 solve to convergence."""
    out = {}
    for full in (False, True):
        _, eng = _engine(L, sites, full)
        for fmt in ("compact", "dense") if L == 3 else ("compact",):
            for loop in ("graph", "eager"):
                info = {}
                e, t1, t2 = solve_structured(eng, eps=0.0, mixed_eps=0.0, maxSteps=6, max_diis=8, refine=False,
                                             precision=precision, t2_format=fmt, loop=loop, info=info)
                out[full, fmt, loop] = e, t1.cpu().numpy(), t2.double().cpu().numpy()
                assert info["n_t2_stored"] == (eng.plan.n_t2 if full else eng.plan.n_t2 // 6)
        info = {}
        e, t1, t2 = solve_structured(eng, eps=1e-12, maxSteps=400, max_diis=8, t2_format="compact", info=info)
        assert info["status"] == "converged"
        out[full, "converged"] = e, t1.cpu().numpy(), t2.cpu().numpy()
    for key in out:
        if key[0]:
            continue
        lim = 1e-7 if key[1] == "converged" else tol
        for got, want in zip(out[key], out[(True,) + key[1:]]):
            assert np.abs(np.asarray(got) - want).max() <= lim * np.abs(want).max(), key


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites", [(2, 1), (3, 4), (3, 5), (3, 6), (4, 6), (5, 1), (7, 1)])
@pytest.mark.parametrize("precision,eps", [("fp64", 2.0 ** -53), ("mixed", 2.0 ** -24)])
def test_step_kernels_over_hole_counts_and_row_lengths(L, sites, precision, eps):
    """Three steps on one label (row and pair kernels) against every label stored
    (general kernels): rows shorter than a warp up to longer than a block, every
    hole count.  A step's sum has at most 14 + 4 h + 2 roundings of terms no
    larger than the result's norm; eight for their ratio to the largest element."""
    out = {}
    for full in (False, True):
        _, eng = _engine(L, sites, full)
        e, t1, t2 = solve_structured(eng, eps=0.0, mixed_eps=0.0, maxSteps=3, max_diis=0, refine=False,
                                     precision=precision, t2_format="compact")
        out[full] = e, t1.cpu().numpy(), t2.double().cpu().numpy()
    for got, want in zip(out[False], out[True]):
        assert np.abs(np.asarray(got) - want).max() <= 3 * 8 * (16 + 4 * sites) * eps * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites,C2,C3,steps", [(3, 2, -3.1, 0.9, (18, 28)), (3, 7, -2.9, 0.6, (15, 29)),
                                                 (4, 7, -3.1, 0.9, (12, 30)), (4, 7, -3.3, 0.7, (12, 27)),
                                                 (4, 2, -3.0, 1.0, (15, 33)), (6, 7, -3.1, 0.9, (12, 30))])
@pytest.mark.parametrize("loop", ["eager", "graph"])
def test_mixed_solves_to_fp64_keep_every_label(L, sites, C2, C3, steps, loop):
    """Where the energy test stops such a solve hangs on the roundings of its FP32
    pulses: it runs on every label, bit for bit what the kernels for every label
    give, and its (FP32, all) step counts on a B200 are those it had before labels
    were reduced."""
    _, fock, two = _inputs(L, sites, C2, C3)
    plan, _ = S.detect(fock, two)
    out = []
    for full in (False, True):
        eng = StructuredEngine(plan, fock, torch.device("cuda:0"))
        eng.prob.tune = tune.word(fwd32=6, chunks=2)   # the roundings are those of one launch shape
        if full:
            eng.cache["reduced"] = None
        info = {}
        out.append(solve_structured(eng, eps=1e-11, mixed_eps=1e-6, maxSteps=100, max_diis=8, precision="mixed",
                                    t2_format="compact", loop=loop, info=info))
        assert info["n_t2_stored"] == eng.plan.n_t2
        assert (info["mixed_iters"], info["iterations"]) == steps
    assert out[0][0] == out[1][0] and torch.equal(out[0][1], out[1][1]) and torch.equal(out[0][2], out[1][2])
    # an answer of the FP32 phase alone, and a phase too short for a pulse, run on one label
    for kw in (dict(eps=1e-6), dict(eps=1e-11, refine=False), dict(eps=1e-11, maxSteps=7)):
        eng = StructuredEngine(plan, fock, torch.device("cuda:0"))
        solve_structured(eng, mixed_eps=1e-6, max_diis=8, precision="mixed", t2_format="compact", loop="eager",
                         info=info, **kw)
        assert info["n_t2_stored"] == plan.n_t2 // 6


@pytest.mark.gpu
def test_a_start_that_treats_labels_differently_runs_on_all():
    _, eng = _engine(3, 7)
    t1 = np.zeros((eng.plan.p, eng.plan.h))
    P, H = eng.plan.p_of[2], eng.plan.h_of[2]
    t1[P[0], H[0]] = 1e-3
    out = []
    for full in (False, True):
        _, eng = _engine(3, 7, full)
        info = {}
        out.append(solve_structured(eng, t1initial=t1, eps=0.0, maxSteps=4, max_diis=8, t2_format="compact", info=info))
        assert info["n_t2_stored"] == eng.plan.n_t2
    assert out[0][0] == out[1][0] and torch.equal(out[0][2], out[1][2])


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites,code,tol", [(3, 1, _lib.NLB_F64, 1e-12), (3, 3, _lib.NLB_F64, 1e-12),
                                              (4, 7, _lib.NLB_F64, 1e-12), (4, 7, _lib.NLB_F32, 2e-6)])
def test_lambda_steps_on_one_label(L, sites, code, tol):
    """Lambda steps (from zero, then kept), U and T included; amplitudes that
    treat one pair of labels differently run with every label stored."""
    got = {}
    for full in (False, True):
        _, eng = _engine(L, sites, full)
        _, t1, t2 = solve_structured(eng, eps=1e-13, max_diis=8, maxSteps=2000, t2_format="compact")
        if not full:
            start = t1, t2
        solver = A.LambdaSolver(eng)
        solver.label_from = 1    # small labels, too
        b = solver.buffers(code, 0)
        b["t1"].copy_(start[0].reshape(-1))
        b["t2"].copy_(start[1])
        c = solver.run(b, 0.0, 0.5, 3, 0, False)
        ph, hh = eng.plan.p * eng.plan.h, eng.plan.h ** 2
        b["lam1"][0].copy_(b["lam1"][c.parity].clone())
        b["lam2"][0].copy_(b["lam2"][c.parity].clone())
        c = solver.run(b, 0.0, 0.5, 3, 0, True)
        assert (solver._label is None) == full
        got[full] = [x.double().cpu().numpy() for x in (b["lam1"][c.parity], b["lam2"][c.parity],
                                                        b["acc"][ph:ph + 2 * hh])]
        if not full:
            b["t2"][-1] += 0.5
            assert solver._alike(b, False) is None
    for x, y in zip(got[False], got[True]):
        assert np.abs(x - y).max() <= tol * np.abs(y).max()


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites,precision", [(3, 1, "fp64"), (3, 7, "mixed")])
def test_gradient_on_one_label(L, sites, precision):
    grads = []
    for full in (False, True):
        holes, eng = _engine(L, sites, full)
        prob = A.lattice_problem(L, holes)
        _, t1, t2 = solve_structured(eng, eps=1e-13, max_diis=8, maxSteps=2000, t2_format="compact")
        grads.append(A.lambda_gradient(eng, t1, t2, [prob.dv, prob.dw], tol=1e-10, precision=precision))
    np.testing.assert_allclose(grads[0], grads[1], rtol=1e-8)


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites,code,eps", [(3, 2, _lib.NLB_F64, 2.0 ** -53), (3, 7, _lib.NLB_F64, 2.0 ** -53),
                                              (4, 7, _lib.NLB_F32, 2.0 ** -24)])
def test_lambda_pulse_extrapolates_every_entry(L, sites, code, eps):
    """A pulse of the Lambda iteration on one label, from multipliers without
    exchange symmetry: every entry is the same combination of its own last value
    and its own stored errors.  The weights come from the pulse's t1 part, as those
    that fit it best; FP32: the result is rounded once."""
    _, eng = _engine(L, sites)
    red = eng.reduced()
    solver = A.LambdaSolver(red)
    b = solver.buffers(code, 2)
    gen = torch.Generator(device="cuda").manual_seed(5)
    for x in (b["t1"], b["t2"], b["lam1"][0], b["lam2"][0]):
        x.copy_(torch.randn(x.shape, generator=gen, device="cuda", dtype=torch.float64) * 0.1)
    lib, sp = _lib.lib(), torch.cuda.current_stream().cuda_stream
    _lib.check(lib.nlb_lambda_init(red.prob, b["state"], 0.0, 0.5, 100, 2, _lib.NLB_LAMBDA_KEEP, sp), "init")
    for _ in range(2):
        _lib.check(lib.nlb_lambda_step(red.prob, b["state"], sp), "step")
    before = b["lam1"][0].cpu().numpy(), b["lam2"][0].double().cpu().numpy()   # two steps: parity 0 again
    e1, e2 = b["diis_t1"].view(2, -1).cpu().numpy(), b["diis_t2"].view(2, -1).double().cpu().numpy()
    _lib.check(lib.nlb_lambda_diis(red.prob, b["state"], 2, sp), "diis")
    after = b["lam1"][0].cpu().numpy(), b["lam2"][0].double().cpu().numpy()
    w = np.linalg.lstsq(np.stack([before[0], *e1], 1), after[0], rcond=None)[0]
    assert np.abs(w[1:]).max() > 1e-3      # the pulse did something
    want = np.tensordot(w, np.stack([before[1], *e2]), 1)
    assert np.abs(after[1] - want).max() <= (eps + 1e-11) * max(1.0, np.abs(want).max())


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites", [(4, 3), (4, 7)])
def test_derivative_that_treats_labels_differently(L, sites):
    """Alike amplitudes and a derivative Hamiltonian with one pair of labels apart:
    the multipliers may run on one label, the coupling sums take all of them."""
    grads = []
    for full in (False, True):
        holes, eng = _engine(L, sites, full)
        prob = A.lattice_problem(L, holes)
        de, dfock, dtwo = prob.dv
        idx, val = (np.asarray(x) for x in S._coo(dtwo[0]))
        one = np.isin(eng.plan.p_label[idx[:, :2]], (0, 1)).all(1)    # v_pppp of labels 0 and 1 only, doubled
        dtwo = [(idx, np.where(one, 2.0, 1.0) * val)] + list(dtwo[1:])
        _, t1, t2 = solve_structured(eng, eps=1e-13, max_diis=8, maxSteps=2000, t2_format="compact")
        if not full:
            start = t1, t2
            assert A._label_coefficients(eng.reduced(), dfock, dtwo) is None
        grads.append(A.lambda_gradient(eng, *start, [(de, dfock, dtwo), prob.dw], tol=1e-11, precision="fp64"))
    np.testing.assert_allclose(grads[0], grads[1], rtol=1e-9)


def _labels(plan, fock, two, keep):
    """The inputs of some of a plan's labels: Fock blocks and ladders of their states."""
    P, H = (np.flatnonzero(np.isin(x, keep)) for x in (plan.p_label, plan.h_label))
    ladders = []
    for block, states in ((two[0], P), (two[5], H)):
        idx, val = S._coo(block)
        m = np.isin(idx, states).all(1)
        ladders.append((np.searchsorted(states, idx[m]), val[m]))
    return [fock[0][np.ix_(P, P)], fock[1][np.ix_(P, H)], fock[2][np.ix_(H, H)]], \
        [ladders[0]] + list(two[1:5]) + [ladders[1]]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,step", [(torch.float64, 1e-12), (torch.float32, 1e-6)])
def test_amplitudes_count_as_alike_bit_for_bit(dtype, step):
    """Labels that differ, an exchange that does not hold to the last bit, and a NaN
    are each seen, also where two labels leave one block and no copy to compare."""
    holes, fock, two = _inputs(3, 3)
    for keep in ([0, 1, 2, 3], [0, 1]):
        f, t = _labels(S.detect(fock, two)[0], fock, two, keep)
        plan, why = S.detect(f, t)
        eng = StructuredEngine(plan, f, torch.device("cuda:0"))
        red = eng.reduced()
        assert red.labels == len(keep)
        _, t1, t2 = solve_structured(eng, eps=1e-12, max_diis=8, t2_format="compact")
        t2 = t2.to(dtype)
        np.testing.assert_array_equal(red.compress(t1, t2).cpu().numpy(),
                                      t1.cpu().numpy()[np.ix_(plan.p_of[0], plan.h_of[0])].ravel())
        n = red.plan.n_t2
        for value in (1.0 + step, float("nan")):
            x = t2.clone()
            k = red.plan.h ** 2                   # a = 0, b = 1, i = j = 0
            assert x[k] != 0
            x.view(-1, n)[:, k] *= value          # the same in every pair of labels
            assert red.compress(t1, x) is None
        x, y = t2.clone(), t1.clone()
        x[-1] += 1.0
        y[plan.p_of[1][0], plan.h_of[1][0]] += 1e-15
        assert len(keep) == 2 or red.compress(t1, x) is None
        assert red.compress(y, t2) is None
        y = t1.clone()
        y[plan.p_of[0][1], plan.h_of[0][0]] = float("nan")
        assert red.compress(y, t2) is None


def _one_step(red, t1, t2, code):
    """One step on one label from (t1, t2): the next (t1, t2)."""
    lib, sp = _lib.lib(), torch.cuda.current_stream().cuda_stream
    assert lib.nlb_struct_step_launches(red.prob, code) == 2
    b = red.buffers(code, 0)
    b["t1"][0].copy_(torch.as_tensor(t1.ravel()))
    b["t2"][0].copy_(torch.as_tensor(t2.ravel()))
    _lib.check(lib.nlb_struct_ctrl_init(b["ctrl"].data_ptr(), 0.0, 0.5, 10, _lib.NLB_CRIT_SOA, 0, 0, 0.0, sp), "init")
    _lib.check(lib.nlb_struct_step(red.prob, b["state"], sp), "step")
    return b["t1"][1].cpu().numpy().reshape(t1.shape), b["t2"][1].double().cpu().numpy().reshape(t2.shape)


@pytest.mark.gpu
@pytest.mark.parametrize("code", [_lib.NLB_F32, _lib.NLB_F64])
def test_t1_adds_the_holes_of_its_t2_term_in_fp64(code):
    """Holes whose terms 1, 2^-26 and -1 leave 2^-26: lost where they are added in
    FP32.  t1 = 0, so a step is t1 = (1 - m) (f_ph + 3 F2) / -(f_aa - f_ii)."""
    _, eng = _engine(3, 3)
    red = eng.reduced()
    n, h = red.plan.p, red.plan.h
    t2 = np.zeros((n, n, h, h))
    ptr, col, val = (np.asarray(x) for x in (red.plan.fph_ptr, red.plan.fph_col, red.plan.fph_val))
    # a particle next to each hole alone
    near = [next(int(c) for c in col[ptr[k]:ptr[k + 1]] if np.sum(col == c) == 1) for k in range(h)]
    a = next(x for x in range(n) if x not in near)
    for k, x in enumerate((1.0, 2.0 ** -26, -1.0)):
        f = float(val[ptr[k]:ptr[k + 1]][col[ptr[k]:ptr[k + 1]] == near[k]][0])
        t2[a, near[k], :, k] = x / f
    t2 += t2.transpose(1, 0, 3, 2)                        # exchange-symmetric
    t1, _ = _one_step(red, np.zeros((n, h)), t2, code)
    want = 0.5 * (red.f_ph_np[a] + 3 * 2.0 ** -26) / (np.diag(red.f_hh_np) - red.f_pp_np[a, a])
    np.testing.assert_allclose(t1[a], want, rtol=0, atol=1e-14)


@pytest.mark.gpu
@pytest.mark.parametrize("code,eps", [(_lib.NLB_F32, 2.0 ** -24), (_lib.NLB_F64, 2.0 ** -53)])
def test_denominators_round_once(code, eps):
    """Diagonals of 1e6 in f_pp and f_hh whose sums leave a few units.  t2 = 0, so a
    step is t2 = (1 - m) R / D with R the ladders on t1 t1; its error is that of R
    (two products and a sum), of D (one rounding), of the quotient (2 ulp) and of
    the update, D's FP64 terms and the FP64 sums over f_ph t1 aside."""
    _, eng = _engine(4, 3)
    f = [eng.f_pp_np + 1e6 * np.eye(eng.plan.p), eng.f_ph_np, eng.f_hh_np + 1e6 * np.eye(eng.plan.h)]
    _, _, two = _inputs(4, 3)
    plan, _ = S.detect(f, two)
    red = StructuredEngine(plan, f, torch.device("cuda:0")).reduced()
    n, h = red.plan.p, red.plan.h
    t1 = 0.01 * np.random.default_rng(1).standard_normal((n, h))
    _, t2 = _one_step(red, t1, np.zeros((n, n, h, h)), code)
    pp, hh = np.zeros(n * n), np.zeros(h * h)
    pp[np.diff(red.plan.pp_ptr[0]) > 0], hh[np.diff(red.plan.hh_ptr[0]) > 0] = red.plan.pp_val[0], red.plan.hh_val[0]
    R = (pp.reshape(n, n)[:, :, None, None] + hh.reshape(h, h)) * t1[:, None, :, None] * t1[None, :, None, :]
    dp = np.diag(red.f_pp_np) - (red.f_ph_np * t1).sum(1)
    dh = -np.diag(red.f_hh_np) - (red.f_ph_np * t1).sum(0)
    D = -((dp[:, None, None, None] + dp[None, :, None, None]) + (dh[:, None] + dh[None, :]))
    want = 0.5 * R / D
    assert np.abs(D).max() < 100 and np.abs(want).max() > 0
    # 4e6 * 2^-53 from the FP64 additions of the diagonals, against the smallest |D|
    lim = 10 * eps + 4 * 4e6 * 2.0 ** -53 / np.abs(D).min()
    assert np.all(np.abs(t2 - want) <= lim * np.abs(want))


@pytest.mark.gpu
def test_a_new_engine_steps_inside_a_capture():
    """Steps of a fresh engine's problem with the caller's buffers, captured: no
    allocation in between, and the replay is the step."""
    _, eng = _engine(3, 2)
    lib = _lib.lib()
    b = StructuredEngine(eng.plan, [eng.f_pp_np, eng.f_ph_np, eng.f_hh_np], eng.dev).buffers(_lib.NLB_F64, 0)
    fresh = StructuredEngine(eng.plan, [eng.f_pp_np, eng.f_ph_np, eng.f_hh_np], eng.dev)
    t1 = torch.as_tensor(eng.f_ph_np * 0.01).cuda()
    out = []
    for capture in (False, True):
        b["t1"][0].copy_(t1.reshape(-1))
        b["t2"][0].zero_()
        sp = torch.cuda.current_stream().cuda_stream
        _lib.check(lib.nlb_struct_ctrl_init(b["ctrl"].data_ptr(), 0.0, 0.5, 10, _lib.NLB_CRIT_SOA, 0, 0, 0.0, sp), "init")
        if capture:
            before = torch.cuda.memory_allocated()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                _lib.check(lib.nlb_struct_step(fresh.prob, b["state"], torch.cuda.current_stream().cuda_stream), "step")
                assert torch.cuda.memory_allocated() == before
            g.replay()
        else:
            _lib.check(lib.nlb_struct_step(eng.prob, b["state"], sp), "step")
        out.append((b["t1"][1].cpu(), b["t2"][1].cpu()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.gpu
def test_launches_ask_for_attributes_once_per_kernel():
    """After steps of seventy problem sizes a step is its two launches and nothing
    else: no table of launch attributes is full."""
    from torch.profiler import ProfilerActivity, profile
    lib, sp = _lib.lib(), torch.cuda.current_stream().cuda_stream
    for L in (2, 3, 4, 5, 6):
        for sites in range(1, 8):
            _, fock, two = _inputs(L, sites)
            plan, _ = S.detect(fock, two)
            red = StructuredEngine(plan, fock, torch.device("cuda:0")).reduced()
            for code in (_lib.NLB_F32, _lib.NLB_F64):
                _one_step(red, np.zeros((red.plan.p, red.plan.h)), np.zeros(red.plan.n_t2), code)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        for _ in range(3):
            _lib.check(lib.nlb_struct_step(red.prob, red.buffers(_lib.NLB_F64, 0)["state"], sp), "step")
        torch.cuda.synchronize()
    calls = [e.name for e in prof.events()]
    assert sum(x == "cudaLaunchKernel" for x in calls) == 6
    assert not [x for x in calls if "Attribute" in x or "Occupancy" in x]


NINE = SEVEN + [(1, 1, 0), (1, -1, 0)]


def _exchange_hops(plan, strength):
    """v_pppp that moves a pair (x, y) of any two labels to (y, x), for some x, y."""
    rows = []
    for g in range(plan.n_labels):
        for k in range(plan.n_labels):
            for x, y in ((0, 1), (1, 0), (2, 5), (5, 2)):
                if g != k:
                    a, b, c, d = plan.p_of[g][x], plan.p_of[k][y], plan.p_of[g][y], plan.p_of[k][x]
                    rows += [(a, b, c, d, strength), (b, a, c, d, -strength)]
    return np.array(rows)


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites,keep,hops", [(3, 3, (0, 1), 0), (3, 3, (0, 2, 3), 0), (4, 7, (1, 2), 0),
                                               (4, 7, (0, 1, 3), 0), (4, 9, (0, 1, 2, 3), 0), (3, 8, (0, 1, 2), 0),
                                               (3, 2, (0, 1, 2, 3), 0.3), (4, 7, (0, 1), 0.3), (4, 9, (0, 1, 2), 0.3)])
def test_other_alike_problems(L, sites, keep, hops):
    """Two and three labels, more than seven holes, ladders that are not diagonal:
    steps, a converged solve and (diagonal ladders) gradients on one label against
    every label stored."""
    holes = [[x % L, y % L, z % L, t, s] for (x, y, z) in NINE[:sites] for t in (0, 1) for s in (0, 1)]
    v, w = ham.contact_couplings(-3.1, 0.9)
    _, fock, two = ham.normal_ordered_hamiltonian(L, holes, v, v, w, dense=False)
    plan, _ = S.detect(fock, two)
    prob = A.lattice_problem(L, holes)
    derivs = [(de, *_labels(plan, df, dt, keep)) for de, df, dt in (prob.dv, prob.dw)]
    fock, two = _labels(plan, fock, two, keep)
    if hops:
        part, _ = S.detect(fock, two)
        idx, val = two[0]
        extra = _exchange_hops(part, hops)
        two[0] = np.concatenate([idx, extra[:, :4]]).astype(np.int64), np.concatenate([val, extra[:, 4]])
    plan, why = S.detect(fock, two)
    assert plan is not None, why
    out, start = {}, None
    for full in (False, True):
        eng = StructuredEngine(plan, fock, torch.device("cuda:0"))
        assert bool(eng.prob.diag_ladders) == (not hops)
        if full:
            eng.cache["reduced"] = None
        else:
            assert eng.reduced().labels == len(keep)
        for precision, fmt in (("fp64", "dense"), ("fp64", "compact"), ("mixed", "compact")):
            e, t1, t2 = solve_structured(eng, eps=0.0, mixed_eps=0.0, maxSteps=4, max_diis=0, refine=False,
                                         precision=precision, t2_format=fmt)
            out[full, precision, fmt] = e, t1.cpu().numpy(), t2.double().cpu().numpy()
        info = {}
        e, t1, t2 = solve_structured(eng, eps=1e-13, maxSteps=2000, max_diis=8, t2_format="compact", info=info)
        assert info["status"] == "converged"
        out[full, "converged"] = e, t1.cpu().numpy(), t2.cpu().numpy()
        start = (t1, t2) if start is None else start
        if not hops:
            out[full, "gradient"] = A.lambda_gradient(eng, *start, derivs, tol=1e-11, precision="fp64")
    for key, got in out.items():
        if key[0]:
            continue
        lim = {"converged": 1e-7, "gradient": 1e-9, "fp64": 1e-13, "mixed": 4e-6}[key[1]]
        for x, y in zip(got, out[(True,) + key[1:]]):
            assert np.abs(np.asarray(x) - y).max() <= lim * np.abs(y).max(), key


@pytest.mark.gpu
def test_amplitudes_from_the_host_and_of_a_wrong_size():
    """A gradient takes amplitudes from wherever they are, and refuses those that are
    not the engine's; a start of another shape is refused, too."""
    holes, fock, two = _inputs(3, 3)
    plan, _ = S.detect(fock, two)
    prob = A.lattice_problem(3, holes)
    kw = dict(tol=1e-10, precision="fp64")
    want = None
    for device in ("cuda", "cuda:0"):
        eng = StructuredEngine(plan, fock, torch.device(device))
        _, t1, t2 = solve_structured(eng, eps=1e-13, max_diis=8, maxSteps=2000, t2_format="compact")
        got = A.lambda_gradient(eng, t1, t2, [prob.dv], **kw)
        want = want or got
        assert got == want
    for x, y in ((t1.cpu(), t2.cpu()), (t1.reshape(-1), t2.reshape(6, -1)), (t1.t().contiguous().t(), t2.cpu())):
        assert A.lambda_gradient(eng, x, y, [prob.dv], **kw) == want
    for x, y in ((t1, t2[:-1]), (t1, t2[:t2.numel() // 6]), (t1[:-1], t2), (t1, torch.cat([t2, t2]))):
        with pytest.raises((ValueError, RuntimeError)):
            A.lambda_gradient(eng, x, y, [prob.dv], **kw)
    for shape in ((eng.plan.p + 1, eng.plan.h), (eng.plan.p, eng.plan.h + 2), (1, eng.plan.h)):
        with pytest.raises(ValueError):
            solve_structured(eng, t1initial=np.zeros(shape), eps=0.0, maxSteps=2)


@pytest.mark.gpu
@pytest.mark.parametrize("L,sites,one", [(3, 1, False), (3, 7, False), (4, 7, True)])
def test_short_lambda_runs_of_small_labels_keep_every_label(L, sites, one):
    """The check and the copies of a run on one label cost more than four steps of
    some twenty particles gain."""
    _, eng = _engine(L, sites)
    _, t1, t2 = solve_structured(eng, eps=1e-12, max_diis=8, t2_format="compact")
    solver = A.LambdaSolver(eng)
    b = solver.buffers(_lib.NLB_F64, 0)
    b["t1"].copy_(t1.reshape(-1))
    b["t2"].copy_(t2)
    solver.run(b, 0.0, 0.5, 4, 0, False)
    assert (solver._label is not None) == one


@pytest.mark.gpu
@pytest.mark.parametrize("precision,one", [("mixed", False), ("fp64", True)])
def test_gradients_build_the_engine_they_run_on(precision, one):
    """A mixed gradient runs on every label from start to end; nothing of the
    problem of one label is made for it."""
    holes = [[0, 0, 0, t, s] for t in (0, 1) for s in (0, 1)]
    info = {}
    A.ccsd_energy_and_gradient(3, holes, -3.1, 0.9, precision=precision, eps=1e-11, lambda_tol=1e-9, info=info)
    assert ("reduced" in info["engine"].cache) == one
