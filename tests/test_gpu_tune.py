"""Every launch shape the autotuner can pick computes the same steps."""
import numpy as np
import pytest
import torch

from nulattice_b200 import adjoint as A
from nulattice_b200 import hamiltonian as ham
from nulattice_b200 import structure as S
from nulattice_b200 import tune as T
from nulattice_b200.ccsd import StructuredEngine, solve_structured

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _engine(L=4, A_=28):
    v2, w3 = ham.contact_couplings(-3.0, 1.0)
    e_ref, fock, two = ham.normal_ordered_hamiltonian(L, ham.closed_shell_holes(L, A_), v2, v2, w3, dense=False)
    plan, _ = S.detect(fock, two)
    return StructuredEngine(plan, fock, torch.device(DEV))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-5)])
def test_forward_launch_shapes_agree(precision, tol):
    out = []
    words = [T.word(fwd32=v) for v in T.FWD_F32] if precision == "mixed" else [T.word(fwd64=v) for v in T.FWD_F64]
    for w in words:
        eng = _engine()
        eng.cache["reduced"] = None   # every label stored: one label has kernels of its own
        assert all(T._lib.lib().nlb_struct_step_launches(eng.prob, c) == 4 for c in (T._lib.NLB_F32, T._lib.NLB_F64))
        eng.prob.tune = w
        e, t1, t2 = solve_structured(eng, eps=0.0, maxSteps=9, max_diis=4, precision=precision, mixed_eps=0.0,
                                     refine=False, t2_format="compact")
        out.append((e, t1.cpu().numpy(), t2.double().cpu().numpy()))
    for e, t1, t2 in out[1:]:
        assert e == pytest.approx(out[0][0], rel=tol)
        np.testing.assert_allclose(t2, out[0][2], atol=tol * np.abs(out[0][2]).max())


def test_lambda_launch_shapes_agree():
    eng = _engine()
    e, t1, t2c = solve_structured(eng, eps=1e-12, maxSteps=2000, max_diis=8, t2_format="compact")
    prob = A.lattice_problem(4, ham.closed_shell_holes(4, 28))
    ref = None
    for k, w in enumerate(2 * [T.word(), T.word(lam32=1), T.word(chunks=2), T.word(lam32=1, chunks=4)]):
        if k == 4:
            eng.cache["reduced"] = None   # one label, then every label stored
        eng.prob.tune = w
        g = A.lambda_gradient(eng, t1, t2c, [prob.dv, prob.dw], tol=1e-10, precision="mixed")
        if ref is None:
            ref = g
        np.testing.assert_allclose(g, ref, rtol=1e-8)


def test_tuner_picks_a_valid_word(tmp_path, monkeypatch):
    monkeypatch.setenv("NLB_TUNE_CACHE", str(tmp_path / "tune.json"))
    eng = _engine()
    info = {}
    w = T.tune(eng, info=info)
    d = T.describe(w)
    assert d["t2_fp32"] in T.FWD_F32.values() and d["t2_fp64"] in T.FWD_F64.values()
    assert d["lambda_fp32"] in T.LAM_F32.values() and not info["cached"]
    eng2 = _engine()
    info2 = {}
    assert T.tune(eng2, info=info2) == w and info2["cached"]


def test_tuner_times_the_shapes_it_names(tmp_path, monkeypatch):
    """Every forward shape is timed on the problem whose kernels read it (every
    label stored: four launches a step), the Lambda shapes on both problems, from
    amplitudes of whole steps."""
    monkeypatch.setenv("NLB_TUNE_CACHE", str(tmp_path / "tune.json"))
    lib, stages, inits = T._lib.lib(), [], []

    class Spy:
        def __getattr__(self, name):
            return getattr(lib, name)

        def nlb_struct_stage(self, prob, st, stage, sp):
            assert stage == T._lib.NLB_STAGE_T2 and lib.nlb_struct_step_launches(prob, st.dtype) == 4
            stages.append((st.dtype, int(prob.tune)))
            return lib.nlb_struct_stage(prob, st, stage, sp)

        def nlb_lambda_init(self, prob, *a):
            inits.append((int(prob.tune) >> 24, int(prob.tune) & 0xffff0))
            return lib.nlb_lambda_init(prob, *a)

    monkeypatch.setattr(T._lib, "lib", Spy)
    eng = _engine()
    seen = []
    buffers = A.LambdaSolver.buffers
    monkeypatch.setattr(A.LambdaSolver, "buffers", lambda s, *a: seen.append(buffers(s, *a)) or seen[-1])
    w = T.tune(eng)
    assert {x for x in stages if x[0] == T._lib.NLB_F32} == {(T._lib.NLB_F32, v) for v in T.FWD_F32}
    assert {x for x in stages if x[0] == T._lib.NLB_F64} == {(T._lib.NLB_F64, v << 16) for v in T.FWD_F64}
    for labels in (0, 4):
        assert {x[1] for x in inits if x[0] == labels} >= {T.word(lam32=v, chunks=c) & 0xffff0 for v in T.LAM_F32
                                                           for c in (0, 2, 4, 8)}
    _, t1, t2 = solve_structured(_engine(), eps=0.0, mixed_eps=0.0, maxSteps=3, max_diis=0, precision="mixed",
                                 refine=False, t2_format="compact")
    one, every = seen
    assert one["t2"].numel() * 6 == every["t2"].numel() == t2.numel()
    for b in (one["t2"], every["t2"]):
        np.testing.assert_allclose(b.cpu().numpy(), t2[:b.numel()].cpu().numpy(), atol=1e-5 * float(t2.abs().max()))
    assert eng.tune == w and eng.reduced().tune == T.label_word(w)


@pytest.mark.parametrize("label", [(0, 0), (1, 0), (0, 2), (1, 8)])
def test_word_keeps_the_shapes_of_one_label(label):
    w = T.word(fwd32=6, lam32=1, chunks=4, fwd64=1, label=label)
    assert T.label_word(w) == T.word(fwd32=6, lam32=label[0], chunks=label[1], fwd64=1) & 0xfffff
    assert T.describe(w)["label_chunks"] == (label[1] or "auto") and T.describe(w)["lambda_chunks"] == 4
    # one choice for both, unless told apart
    assert T.label_word(T.word(lam32=1, chunks=4)) == T.word(lam32=1, chunks=4) & 0xfffff


def test_untuned_word_leaves_the_chunks_of_one_label_to_the_kernel(tmp_path, monkeypatch):
    """Two row chunks are the choice for six channels; one has a sixth of the blocks."""
    monkeypatch.setenv("NLB_TUNE_CACHE", str(tmp_path / "none.json"))
    eng = _engine()
    eng.prob.tune = T.known_word(eng)
    assert (eng.prob.tune >> 8) & 255 == 2 and (eng.reduced().prob.tune >> 8) & 255 == 0
