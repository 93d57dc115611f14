"""Halo exchange on the device: the parts of a partition as separate contexts on one GPU, their
face rows moved by pack / device copy / unpack between the two halves of every step, against the
one-domain run (the device half of the multi-GPU form; the transport between GPUs is NCCL). Every
other step runs the overlapped order: the send elements' local step, the pack, then the inner
elements' local step before the exchanged rows are unpacked."""
import numpy as np
import pytest

from edge_b200 import host, shard
from edge_b200.solver import Solver
from helpers import random_dofs, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_parts,precision,order,runs", [(2, 64, 4, 1), (3, 64, 3, 1), (2, 32, 5, 16)])
def test_parts_match_one_domain(n_parts, precision, order, runs):
    prob = host.build_problem(4, order, runs, jitter=0.15, seed=12, n_receivers=0, source=None)
    e0, _ = random_dofs(prob, seed=5, scale=1e-2)
    dtype = np.float64 if precision == 64 else np.float32
    ref = Solver(prob, precision=precision)
    try:
        ref.upload_dofs(e0.astype(dtype))
        ref.step(6)
        want, _ = ref.download_dofs()
    finally:
        ref.close()
    parts = [shard.PartSolver(prob, p, precision=precision) for p in shard.plan(prob.mesh, n_parts)]
    try:
        for ps in parts:
            ps.upload_owned(e0.astype(dtype))
        t = 0.0
        for step in range(6):
            # odd steps: the send elements' local step, the pack, then the inner elements' local
            # step (the overlapped order); even steps: the whole local step first
            for ps in parts:
                if step % 2:
                    ps.phase_send(t, prob.dt)
                else:
                    ps.phase0(t, prob.dt)
            sent = {ps.part.rank: ps.pack() for ps in parts}
            if step % 2:
                for ps in parts:
                    ps.phase_inner(t, prob.dt)
            for ps in parts:
                for q, buf in ps.recv_buf.items():
                    buf.copy_(sent[q][ps.part.rank])
                ps.unpack()
            for ps in parts:
                ps.phase1(t, prob.dt)
            t += prob.dt
        got = np.concatenate([ps.download_owned()[0] for ps in parts])
    finally:
        for ps in parts:
            ps.close()
    assert np.array_equal(got, want) or rel_l2(got, want) < 1e-14


def test_send_then_inner_equals_whole_local_step():
    """Phases 2 + 3 (send elements, then the rest with the sources) equal phase 0 bit for bit, with
    sources and receivers on."""
    prob = host.build_problem(3, 4, 1, jitter=0.1, seed=4, n_receivers=3, source="explosive", n_steps=8)
    e0, _ = random_dofs(prob, seed=2, scale=1e-2)
    out = []
    for split in (False, True):
        s = Solver(prob, precision=64)
        try:
            from edge_b200._lib import lib
            s._chk(lib().edge_b200_set_owned(s._h, prob.n_el), "set_owned")
            s._chk(lib().edge_b200_set_send_count(s._h, prob.n_el // 3), "set_send_count")
            s.upload_dofs(e0)
            t = 0.0
            for _ in range(4):
                if split:
                    s._chk(lib().edge_b200_step_phase(s._h, t, prob.dt, 2), "phase 2")
                    s._chk(lib().edge_b200_step_phase(s._h, t, prob.dt, 3), "phase 3")
                else:
                    s._chk(lib().edge_b200_step_phase(s._h, t, prob.dt, 0), "phase 0")
                s._chk(lib().edge_b200_step_phase(s._h, t, prob.dt, 1), "phase 1")
                t += prob.dt
            e, _ = s.download_dofs()
            rb, rt, rc = s.receivers()
            out.append((e, rb, rc))
        finally:
            s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][2], out[1][2]) and int(out[0][2][0]) > 0
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n_parts,precision,order,runs,rm", [(2, 64, 4, 1, 0), (2, 64, 5, 1, 0), (3, 32, 5, 16, 0),
                                                             (2, 32, 6, 4, 0), (2, 32, 4, 8, 3), (2, 64, 4, 1, 3)])
def test_parts_of_different_forms(n_parts, precision, order, runs, rm):
    """One part's flux solvers are full rank at one face, so it takes the weak form and the others the
    strong one (pre-mixed rows or projections against characteristics): the parts still equal the
    oracle's one domain; with Godunov solvers again in every part, they do in one form."""
    from edge_b200._lib import lib, ptr
    from helpers import OracleRun
    prob = host.build_problem(4, order, runs, rm=rm, jitter=0.15, seed=12, n_receivers=0, source=None,
                              layers=[3000.0, 5000.0])
    good = prob.fsE.copy()
    plan = shard.plan(prob.mesh, n_parts)
    p = plan[n_parts // 2]
    far = p.owned[p.n_send:]  # no other part knows these elements
    e, f = next((e, f) for e in far for f in range(4)
                if prob.mesh.el_fa_type[e, f] == host.FACE_INNER and prob.mesh.el_fa_el[e, f] in far)
    pen = 0.05 * np.abs(prob.fsE[0, e, f].reshape(9, 9)).max(axis=1).min() * np.eye(9)
    prob.fsE[0, e, f] -= pen.ravel()
    prob.fsE[1, e, f] += pen.ravel()
    e0, a0 = random_dofs(prob, seed=5, scale=1e-2)
    orc = OracleRun(prob, e0.copy(), None if a0 is None else a0.copy())
    parts = [shard.PartSolver(prob, q, precision=precision) for q in plan]
    tol = 1e-12 if precision == 64 else 1e-4

    def steps(n, t):
        for _ in range(n):
            for ps in parts:
                ps.phase0(t, prob.dt)
            sent = {ps.part.rank: ps.pack() for ps in parts}
            for ps in parts:
                for q, buf in ps.recv_buf.items():
                    buf.copy_(sent[q][ps.part.rank])
                ps.unpack()
            for ps in parts:
                ps.phase1(t, prob.dt)
            t += prob.dt
        for k in range(2 if rm else 1):
            got = np.concatenate([ps.download_owned()[k] for ps in parts])
            assert rel_l2(got, orc.state["dofsA" if k else "dofsE"]) < tol
        return t

    try:
        for ps in parts:
            ids = ps.part.global_ids()
            ps.solver.upload_dofs(e0[ids], None if a0 is None else a0[ids])
        forms = [lib().edge_b200_step_form(ps.solver._h) for ps in parts]
        assert forms == [0 if q is p else 1 for q in plan]
        orc.step(5)
        t = steps(5, 0.0)
        prob.fsE[:] = good
        for ps in parts:
            loc = ps.prob
            loc.fsE[:] = good[:, ps.part.global_ids()]
            d = [loc.starE, loc.fsE, loc.starA, loc.srcA, loc.fsA, loc.omega]
            assert lib().edge_b200_upload_element_data(ps.solver._h, *[ptr(x) for x in d]) == 0
            assert lib().edge_b200_step_form(ps.solver._h) == 1
        orc.d = prob.oracle_dict()
        orc.step(3)
        steps(3, t)
    finally:
        for ps in parts:
            ps.close()
