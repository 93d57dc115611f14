"""The strong-form GTS step is the one that runs: Godunov flux solvers of elastic and anelastic media
are found to be of rank 3 (free surface, outflow, layered and jittered inner faces), other flux solvers
send the context to the weak-form kernels, and both agree with the oracle."""
import dataclasses

import numpy as np
import pytest

from edge_b200._lib import lib
from edge_b200.solver import Solver
from helpers import OracleRun, random_dofs, rel_l2, small_problem

pytestmark = pytest.mark.gpu

# (order, runs, mechanisms, precision): every order, run count and both kinds of rows, odd group tails
FORMS = [(2, 1, 0, 32), (2, 1, 0, 64), (3, 4, 0, 32), (4, 8, 0, 32), (5, 16, 0, 32), (5, 1, 0, 64), (6, 4, 0, 32),
         (6, 1, 0, 64), (3, 16, 3, 32), (4, 8, 3, 32), (4, 1, 3, 64), (5, 4, 3, 32)]


@pytest.mark.parametrize("order,runs,rm,prec", FORMS)
def test_strong_form_runs_and_matches(order, runs, rm, prec):
    prob = small_problem(n=(3, 2, 3), order=order, runs=runs, rm=rm, jitter=0.15, n_steps=6, source="random",
                         layers=[3000.0, 6000.0], lognormal_sigma=0.2)
    e0, a0 = random_dofs(prob, seed=4)
    s = Solver(prob, precision=prec)
    assert lib().edge_b200_step_form(s._h) == 1
    s.upload_dofs(e0, a0)
    for k in (1, 4):
        s.step(k)
    orc = OracleRun(prob, e0, a0)
    orc.step(5)
    e, a = s.download_dofs()
    tol = 1e-12 if prec == 64 else 1e-4
    assert rel_l2(e, orc.state["dofsE"]) < tol
    if rm:
        assert rel_l2(a, orc.state["dofsA"]) < tol
    rb, _, rc = s.receivers()
    k = int(rc[0])
    assert k > 0 and rel_l2(rb[:, :k], orc.recv["buf"][:, :k]) < tol
    s.close()


def test_anelastic_order_6_keeps_the_weak_form():
    prob = small_problem(n=2, order=6, runs=4, rm=3, n_steps=1, source=None, n_receivers=0)
    s = Solver(prob, precision=32)
    assert lib().edge_b200_step_form(s._h) == 0
    s.close()


@pytest.mark.parametrize("order,runs,rm,prec", [(4, 1, 0, 64), (5, 16, 0, 32), (4, 8, 3, 32)])
def test_full_rank_flux_solvers_take_the_weak_form(order, runs, rm, prec):
    """A penalty on the jump makes one inner face's flux solvers full rank: weak form, same results as
    the oracle with those solvers; the next element data decide anew."""
    prob = small_problem(n=2, order=order, runs=runs, rm=rm, jitter=0.1, n_steps=3, source=None, n_receivers=0)
    good = prob.fsE.copy()
    e, f = map(int, np.argwhere(prob.mesh.el_fa_type == 0)[5])
    pen = 0.05 * np.abs(prob.fsE[0, e, f].reshape(9, 9)).max(axis=1).min() * np.eye(9)
    prob.fsE[0, e, f] -= pen.ravel()
    prob.fsE[1, e, f] += pen.ravel()
    e0, a0 = random_dofs(prob, seed=8)
    s = Solver(prob, precision=prec)
    assert lib().edge_b200_step_form(s._h) == 0
    s.upload_dofs(e0, a0)
    s.step(3)
    orc = OracleRun(prob, e0, a0)
    orc.step(3)
    got, _ = s.download_dofs()
    assert rel_l2(got, orc.state["dofsE"]) < (1e-12 if prec == 64 else 1e-4)
    prob.fsE[:] = good
    arr = [None if v is None else np.ascontiguousarray(v, np.float64)
           for v in (prob.starE, prob.fsE, prob.starA, prob.srcA, prob.fsA, prob.omega)]
    ptrs = [None if v is None else v.ctypes.data for v in arr]
    assert lib().edge_b200_upload_element_data(s._h, *ptrs) == 0
    assert lib().edge_b200_step_form(s._h) == 1
    s.close()


@pytest.mark.parametrize("order,runs,prec", [(5, 16, 32), (3, 8, 32), (4, 1, 64)])
def test_lts_in_strong_form_matches(order, runs, prec):
    """Rate-2 LTS through the strong-form kernels (two-step sums, half-step rows, three groups)."""
    import oracle
    from test_lts import _grouped, _lts_state
    prob, gf, flags, rel = _grouped(order=order, n=4, runs=runs, n_receivers=4, source="random", n_steps=30)
    e0, _ = random_dofs(prob, seed=9, scale=1e-2)
    ref = OracleRun(prob, e0.copy())
    st = _lts_state(prob, e0.copy())
    oracle.lts_cycles(ref.d, st, gf, 0.0, prob.dt, 2, flags, rel, ref.recv, ref.src)
    s = Solver(prob, precision=prec)
    assert lib().edge_b200_step_form(s._h) == 1
    s.upload_dofs(e0.astype(s.dtype))
    s.set_time_groups(gf)
    s.step_lts(1)
    s.step_lts(1)
    e, _ = s.download_dofs()
    assert rel_l2(e, st["dofsE"]) < (1e-12 if prec == 64 else 1e-4)
    s.close()


def _penalised(prob, share=0.05, faces=slice(5, 6)):
    """A copy of the problem whose flux solvers penalise the jump at some inner faces: full rank there."""
    p = dataclasses.replace(prob, fsE=prob.fsE.copy())
    for e, f in np.argwhere(p.mesh.el_fa_type == 0)[faces]:
        pen = share * np.abs(p.fsE[0, e, f].reshape(9, 9)).max(axis=1).min() * np.eye(9)
        p.fsE[0, e, f] -= pen.ravel()
        p.fsE[1, e, f] += pen.ravel()
    return p


def _upload_data(s, p):
    arr = [None if v is None else np.ascontiguousarray(v, np.float64)
           for v in (p.starE, p.fsE, p.starA, p.srcA, p.fsA, p.omega)]
    assert lib().edge_b200_upload_element_data(s._h, *[None if v is None else v.ctypes.data for v in arr]) == 0


@pytest.mark.parametrize("order,runs,rm,prec", [(5, 16, 0, 32), (4, 1, 0, 64), (5, 1, 0, 64), (4, 8, 3, 32)])
def test_batch_takes_over_new_element_data(order, runs, rm, prec):
    """Element data set between two calls of a batch: strong to strong with another material, strong to
    weak, weak to weak, weak to strong and back; each call's result is the oracle's with the data of the
    time."""
    from edge_b200.batch import Batch
    kw = dict(n=2, order=order, runs=runs, rm=rm, jitter=0.1, n_steps=3, source="random", n_receivers=0)
    prob, layered = small_problem(**kw), small_problem(layers=[3000.0, 5000.0], **kw)
    other = small_problem(n=2, order=3, runs=1, n_steps=3, source=None, n_receivers=0)
    e0, a0 = random_dofs(prob, seed=2)
    s, mate = Solver(prob, precision=prec), Solver(other, precision=64)
    s.upload_dofs(e0, a0)
    b = Batch([s, mate])
    orc = OracleRun(prob, e0, a0)
    for p, form in ((prob, 1), (layered, 1), (_penalised(prob), 0), (_penalised(layered), 0), (prob, 1),
                    (_penalised(prob), 0)):
        _upload_data(s, p)
        assert lib().edge_b200_step_form(s._h) == form
        b.run(4)
        orc.d = p.oracle_dict()
        orc.step(4)
        got, _ = s.download_dofs()
        assert rel_l2(got, orc.state["dofsE"]) < (1e-12 if prec == 64 else 1e-4)
    b.close()
    s.close()
    mate.close()


def test_batch_takes_over_new_sources():
    """A longer source list set between two calls of a batch (its arrays move)."""
    from edge_b200.batch import Batch
    prob = small_problem(n=2, order=4, runs=8, jitter=0.1, n_steps=12, source="random", n_receivers=0)
    one = small_problem(n=2, order=4, runs=8, jitter=0.1, n_steps=12, source=None, n_receivers=0)
    e0, _ = random_dofs(prob, seed=2, scale=1e-3)
    s, ref = Solver(one, precision=32), Solver(one, precision=32)
    src = prob.sources
    from edge_b200._lib import ptr
    b = Batch([s])
    for x in (s, ref):
        x.upload_dofs(e0)
    b.run(3)
    ref.step(3)
    for x in (s, ref):
        x._chk(lib().edge_b200_set_sources(x._h, src["n"], ptr(src["el"]), ptr(src["run"]), ptr(src["scal"]),
                                           ptr(src["bEval"]), ptr(src["t0"]), ptr(src["dt"]), ptr(src["tsOff"]),
                                           ptr(src["nPts"]), len(src["ts"]), ptr(src["ts"])), "set_sources")
    b.run(6)
    ref.step(6)
    got, want = s.download_dofs()[0], ref.download_dofs()[0]
    assert rel_l2(want, e0) > 1e-6 and rel_l2(got, want) < 1e-6
    b.close()
    s.close()
    ref.close()


@pytest.mark.parametrize("order,runs,rm,prec", [(5, 16, 0, 32), (4, 1, 0, 64), (5, 1, 0, 64), (4, 8, 3, 32), (6, 4, 3, 32)])
def test_borrowers_follow_new_element_data(order, runs, rm, prec):
    """A context that borrows element data steps (and samples its receivers) with what its lender
    uploads later, in the form that those data allow, on its own and in a batch."""
    from edge_b200.batch import Batch
    kw = dict(n=2, order=order, runs=runs, rm=rm, jitter=0.1, n_steps=12, source=None)
    prob, layered = small_problem(**kw), small_problem(layers=[3000.0, 5000.0], **kw)
    e0, a0 = random_dofs(prob, seed=6)
    lender = Solver(prob, precision=prec)
    s = Solver(prob, precision=prec, share_from=lender)
    quiet = Solver(dataclasses.replace(prob, receivers=None), precision=prec, share_from=s)  # borrows through s
    b = Batch([quiet])
    s.upload_dofs(e0, a0)
    quiet.upload_dofs(e0, a0)
    orc = OracleRun(prob, e0, a0)
    tol = 1e-12 if prec == 64 else 1e-4
    strong = lib().edge_b200_step_form(lender._h)
    for p, form in ((prob, strong), (layered, strong), (_penalised(layered), 0), (prob, strong)):
        for x in (s, quiet):
            x.sync()
        _upload_data(lender, p)
        s.step(3)
        b.run(3)
        assert lib().edge_b200_step_form(s._h) == form
        orc.d = p.oracle_dict()
        orc.step(3)
        for x in (s, quiet):
            assert rel_l2(x.download_dofs()[0], orc.state["dofsE"]) < tol
    rb, _, rc = s.receivers()
    k = int(rc[0])
    assert k > 0 and rel_l2(rb[:, :k], orc.recv["buf"][:, :k]) < tol
    b.close()
    for x in (lender, quiet, s):  # the lender first: the data live as long as a borrower
        x.close()


@pytest.mark.parametrize("order,rm", [(4, 0), (5, 0), (4, 3)])
@pytest.mark.parametrize("share", [3e-9, 1e-10, 3e-12])
def test_small_full_rank_parts_are_kept_in_fp64(order, rm, share):
    """Flux solvers a little off rank 3 at every inner face: what they add to the result (seen against
    the oracle with and without it) is not dropped."""
    prob = small_problem(n=2, order=order, runs=1, rm=rm, jitter=0.1, n_steps=3, source=None, n_receivers=0)
    off = _penalised(prob, share, slice(None))
    e0, a0 = random_dofs(prob, seed=8)
    e0[:, 6:] *= 1e-7  # velocities of the stresses' energy: both rows of a solver count
    s = Solver(off, precision=64)
    s.upload_dofs(e0, a0)
    s.step(4)
    orc, plain = (OracleRun(p, e0.copy(), None if a0 is None else a0.copy()) for p in (off, prob))
    orc.step(4)
    plain.step(4)
    got, _ = s.download_dofs()
    for q in (slice(0, 6), slice(6, 9)):
        added = rel_l2(plain.state["dofsE"][:, q], orc.state["dofsE"][:, q])
        assert rel_l2(got[:, q], orc.state["dofsE"][:, q]) < 0.1 * added + 1e-14
    s.close()


@pytest.mark.parametrize("order,rm", [(4, 0), (4, 3)])
def test_godunov_solvers_of_strong_contrasts_take_the_strong_form(order, rm):
    prob = small_problem(n=4, order=order, runs=1, rm=rm, jitter=0.2, n_steps=3, layers=[300.0, 9000.0],
                         lognormal_sigma=1.0, n_receivers=0)
    e0, a0 = random_dofs(prob, seed=8)
    s = Solver(prob, precision=64)
    assert lib().edge_b200_step_form(s._h) == 1
    s.upload_dofs(e0, a0)
    s.step(4)
    orc = OracleRun(prob, e0, a0)
    orc.step(4)
    assert rel_l2(s.download_dofs()[0], orc.state["dofsE"]) < 1e-12
    s.close()


@pytest.mark.parametrize("order,runs,rm,prec,full_rank,fuses", [
    (5, 16, 0, 32, True, True), (4, 8, 0, 32, True, True), (3, 1, 0, 32, True, True), (3, 4, 0, 32, True, True),
    (6, 16, 0, 32, True, False), (4, 1, 0, 64, True, False), (5, 1, 0, 64, True, False), (5, 4, 0, 32, True, False), (4, 8, 3, 32, True, False),
    (5, 16, 0, 32, False, True), (5, 1, 0, 64, False, True), (4, 8, 3, 32, False, True)])
def test_steps_fuse_in_both_forms(order, runs, rm, prec, full_rank, fuses):
    """Multi-step calls fold each step's surface integrals into the next step's kernel in the strong form,
    and the neighbour steps of weak-form contexts at orders 3 to 5 in FP32 with pre-mixed projections: one
    closing launch a call instead of one a step, the same DOFs and receiver samples as without."""
    prob = small_problem(n=3, order=order, runs=runs, rm=rm, jitter=0.15, n_steps=6, source="random",
                         layers=[3000.0, 6000.0], lognormal_sigma=0.2)
    if full_rank:
        prob = _penalised(prob)
    e0, a0 = random_dofs(prob, seed=3)
    a, b = Solver(prob, precision=prec), Solver(prob, precision=prec)
    assert lib().edge_b200_set_fused(b._h, 0) == 0
    for x in (a, b):
        assert lib().edge_b200_step_form(x._h) == (0 if full_rank else 1)
        x.upload_dofs(e0, a0)
    for k in (1, 3, 2):  # calls of one and of several steps
        a.step(k)
        b.step(k)
        assert b.launches() - a.launches() == (k - 1 if fuses else 0)
    for x, y in zip(a.download_dofs(), b.download_dofs()):
        np.testing.assert_array_equal(x, y)
    ra, rb = a.receivers(), b.receivers()
    k = int(ra[2][0])
    assert k > 0
    np.testing.assert_array_equal(ra[2], rb[2])
    np.testing.assert_array_equal(ra[0][:, :k], rb[0][:, :k])
    orc = OracleRun(prob, e0, a0)
    orc.step(6)
    assert rel_l2(a.download_dofs()[0], orc.state["dofsE"]) < (1e-12 if prec == 64 else 1e-4)
    a.close()
    b.close()


# (order, runs, precision), then for the strong and the weak form: CTAs per SM of the local and the
# neighbour kernel, fused steps
SHAPES = [((3, 1, 64), (2, 2, 1), (1, 1, 0)), ((4, 1, 64), (1, 2, 1), (1, 1, 0)), ((5, 16, 32), (2, 3, 1), (2, 2, 1)),
          ((6, 16, 32), (1, 2, 1), (1, 2, 0))]


@pytest.mark.parametrize("cfg,strong,weak", SHAPES)
def test_kernel_config_and_autotuner_know_the_kernels_that_run(cfg, strong, weak):
    import torch
    from edge_b200._lib import ptr
    order, runs, prec = cfg
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    prob = small_problem(n=3, order=order, runs=runs, jitter=0.1, n_steps=1, source=None, n_receivers=0)
    for p, (local, neigh, fused), form in ((prob, strong, 2), (_penalised(prob), weak, 1)):
        s = Solver(p, precision=prec)
        info, caps = np.zeros(6, np.int32), np.zeros(2, np.int32)
        assert lib().edge_b200_kernel_config(s._h, ptr(info)) == 0
        assert (info[1], info[3], info[4], info[5]) == (form, local * sms, neigh * sms, fused)
        s.step(3)
        assert s.launches() == (4 if fused else 6)
        assert lib().edge_b200_autotune(s._h, prob.dt, ptr(caps)) == 0
        groups = -(-p.n_el * runs // 32)
        for cap, grid in zip(caps, info[3:5]):
            assert cap in (0, grid // 2) or cap == groups > grid
        s.close()


@pytest.mark.parametrize("order,runs,prec", [(5, 16, 32), (3, 8, 32), (4, 1, 64)])
def test_lts_in_weak_form_matches(order, runs, prec):
    """Elastic rate-2 LTS with flux solvers of full rank at one face: the weak-form LTS kernels."""
    import oracle
    from test_lts import _grouped, _lts_state
    prob, gf, flags, rel = _grouped(order=order, n=4, runs=runs, n_receivers=4, source="random", n_steps=30, jitter=0.1)
    prob = _penalised(prob)
    e0, _ = random_dofs(prob, seed=9, scale=1e-2)
    ref = OracleRun(prob, e0.copy())
    st = _lts_state(prob, e0.copy())
    oracle.lts_cycles(ref.d, st, gf, 0.0, prob.dt, 2, flags, rel, ref.recv, ref.src)
    s = Solver(prob, precision=prec)
    assert lib().edge_b200_step_form(s._h) == 0
    s.upload_dofs(e0.astype(s.dtype))
    s.step(2)  # (fused where weak steps fuse: the LTS steps after it use one face buffer)
    s.upload_dofs(e0.astype(s.dtype))
    s._chk(lib().edge_b200_rewind_receivers(s._h, prob.receivers["t_first"]), "rewind_receivers")
    s.set_time_groups(gf)
    s.t = 0.0
    s.step_lts(1)
    s.step_lts(1)
    tol = 1e-12 if prec == 64 else 1e-4
    assert rel_l2(s.download_dofs()[0], st["dofsE"]) < tol
    rb, _, rc = s.receivers()
    assert np.array_equal(rc, ref.recv["count"])
    for i, k in enumerate(rc):
        assert rel_l2(rb[i, :k], ref.recv["buf"][i, :k]) < tol
    s.close()


@pytest.mark.parametrize("prec", [32, 64])
def test_source_integrals_of_several_blocks_of_steps(prec):
    """So many sources that a call's series integrals are computed in blocks of four steps."""
    prob = small_problem(n=2, order=4, runs=8 if prec == 32 else 1, jitter=0.1, n_steps=12, source="random",
                         n_receivers=0)
    src, k = prob.sources, -(-30000 // prob.sources["n"])
    for key in ("el", "run", "scal", "bEval", "t0", "dt", "tsOff", "nPts"):
        src[key] = np.repeat(src[key], k, axis=0)
    src["scal"] = src["scal"] / k
    src["n"] *= k
    assert 4 <= 131072 // src["n"] < 5
    e0, _ = prob.zero_dofs()
    s = Solver(prob, precision=prec)
    s.upload_dofs(e0)
    for n in (11, 2, 3):
        s.step(n)
    orc = OracleRun(prob, e0.copy())
    orc.step(16)
    assert np.abs(orc.state["dofsE"]).max() > 0
    # a DOF takes k sums a step, each rounded by half a unit: at most 16 * 30,000 * 2^-53, 16 * 3,750 * 2^-24
    assert rel_l2(s.download_dofs()[0], orc.state["dofsE"]) < 16 * k * 2.0 ** (-53 if prec == 64 else -24)
    s.close()
