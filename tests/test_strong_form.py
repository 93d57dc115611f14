"""The strong-form step with characteristic exchange, restated in numpy, equals the oracle's weak-form
step: the volume integral as the Taylor update, own and neighbour flux of a face through three incoming
characteristics (free surface, outflow, layered and jittered inner faces), and the anelastic update
unrolled over the levels of the recursion."""
import numpy as np
import pytest

from edge_b200 import dgmat
from helpers import OracleRun, random_dofs, rel_l2, small_problem

STAR = ([0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 4, 4, 5, 5, 6, 6, 6, 7, 7, 7, 8, 8, 8],
        [6, 7, 8, 6, 7, 8, 6, 7, 8, 6, 7, 7, 8, 6, 8, 0, 3, 5, 1, 3, 4, 2, 4, 5])
STAR_A = ([0, 1, 2, 3, 3, 4, 4, 5, 5], [6, 7, 8, 6, 7, 7, 8, 6, 8])
SRC = ([0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 4, 5], [0, 1, 2, 0, 1, 2, 0, 1, 2, 3, 4, 5])
NORMALS = np.array([(0, 0, -1), (0, -1, 0), (-1, 0, 0), (1, 1, 1)], float)


def _scale(m):
    """Scales of the stress and velocity rows and columns (rows r, columns c)."""
    r, c = np.ones(9), np.ones(9)
    for g in (slice(0, 6), slice(6, 9)):
        r[g] = np.abs(m[g]).max() or 1.0
    for g in (slice(0, 6), slice(6, 9)):
        c[g] = np.abs(m / r[:, None])[:, g].max() or 1.0
    return r, c


def _basis(s):
    rest, q = s.copy(), np.zeros((3, 9))
    for k in range(3):
        v = rest[np.argmax((rest * rest).sum(1))].copy()
        for _ in range(2):
            v -= q[:k].T @ (q[:k] @ v)
        q[k] = v / np.linalg.norm(v)
        rest -= np.outer(rest @ q[k], q[k])
    return q, (rest * rest).sum(1).max()


def _coefficients(p):
    """U [nEl][4][9 or 15][3], V0, V1 [nEl][4][9][3] of every face (V1: what its neighbour forms)."""
    ne, nq = p.n_el, 15 if p.rm else 9
    st = np.zeros((ne, 3, nq, 9))
    st[:, :, STAR[0], STAR[1]] = p.starE
    fs = np.zeros((2, ne, 4, nq, 9))
    fs[:, :, :, :9] = p.fsE.reshape(2, ne, 4, 9, 9)
    if p.rm:
        st[:, :, 9 + np.array(STAR_A[0]), STAR_A[1]] = p.starA
        fs[:, :, :, 9:] = p.fsA.reshape(2, ne, 4, 6, 9)
    u, v0, v1 = np.zeros((ne, 4, nq, 3)), np.zeros((ne, 4, 9, 3)), np.zeros((ne, 4, 9, 3))
    for e in range(ne):
        for f in range(4):
            ty = p.mesh.el_fa_type[e, f]
            own = fs[0, e, f] + np.einsum("d,dij->ij", NORMALS[f], st[e])
            if ty == 1:
                own = own + fs[1, e, f]
            m = fs[1, e, f] if ty == 0 else own
            r, c = _scale(fs[1 if ty == 0 else 0, e, f][:9])
            q, res = _basis(m[:9] / r[:, None] / c)
            assert res < 1e-20
            u[e, f] = (m / c) @ q.T
            v1[e, f] = (q * c).T
            x = np.linalg.lstsq(u[e, f, :9] / r[:, None], own[:9] / r[:, None], rcond=None)[0]
            v0[e, f] = x.T
            top = np.where(np.arange(9) < 6, c[0], c[8])
            assert np.abs(own[:9] / r[:, None] - (u[e, f, :9] / r[:, None]) @ x).max(0).max() < 1e-12 * top.max()
            if p.rm:
                scale = np.abs(fs[0, e, f, 9:]).max()
                assert np.abs(own[9:] - u[e, f, 9:] @ x).max() < 1e-11 * scale
    return st, u, v0, v1


@pytest.mark.parametrize("order,rm", [(2, 0), (3, 0), (5, 0), (3, 3), (4, 3)])
def test_strong_form_equals_the_oracle(order, rm):
    p = small_problem(n=2, order=order, runs=1, rm=rm, jitter=0.15, layers=[3000.0, 6000.0], lognormal_sigma=0.2,
                      source=None, n_receivers=0)
    m = dgmat.matrices(order)
    e0, a0 = random_dofs(p, seed=1)
    orc = OracleRun(p, e0.copy(), None if a0 is None else a0.copy())
    orc.step(2)
    st, u, v0, v1 = _coefficients(p)
    src = np.zeros((p.n_el, max(rm, 1), 6, 6))
    if rm:
        src[:, :, SRC[0], SRC[1]] = p.srcA
    dt, c = p.dt, [p.dt]
    for d in range(1, order + 1):
        c.append(c[-1] * dt / (d + 1))
    q = e0[..., 0].copy()
    a = a0[..., 0].copy() if rm else None
    for _ in range(2):
        der, der_a = q, a
        new, ti, psi = q.copy(), c[0] * q, []
        for d in range(order if rm else order - 1):
            nxt = sum(np.einsum("eij,ejk->eik", st[:, k], der) @ -m["stiffT"][k] for k in range(3))
            psi.append(nxt[:, 9:])
            nxt = nxt[:, :9]
            if rm:
                nxt[:, :6] += np.einsum("emij,emjk->eik", src, der_a)
                der_a = p.omega[None, :, None, None] * (psi[-1][:, None] + der_a)
            der = nxt
            new += c[d] * der
            if d + 1 < order:
                ti += c[d + 1] * der
        if rm:
            upd = np.zeros_like(a)
            for k in range(rm):
                w, tail = p.omega[k], 0.0
                lam = np.zeros(order)
                for d in range(order - 1, -1, -1):
                    lam[d] = w * (c[d] - tail)
                    tail = w * (c[d] + tail)
                upd[:, k] = (1 - tail) * a[:, k] + sum(lam[d] * psi[d] for d in range(order))
            a = upd
        for f in range(4):
            w = np.einsum("eik,ein->ekn", v0[:, f], ti @ m["fluxL"][f])
            for e in np.flatnonzero(p.mesh.el_fa_type[:, f] == 0):
                n, v, fo = p.mesh.el_fa_el[e, f], p.mesh.vid[e, f], p.mesh.fid[e, f]
                w[e] += v1[e, f].T @ (ti[n] @ m["fluxN"][4 * v + fo])
            up = np.einsum("eik,ekn->ein", u[:, f], w) @ m["fluxT"][f]
            new += up[:, :9]
            if rm:
                a += p.omega[None, :, None, None] * up[:, None, 9:]
        q = new
    assert rel_l2(q, orc.state["dofsE"][..., 0]) < 1e-13
    if rm:
        assert rel_l2(a, orc.state["dofsA"][..., 0]) < 1e-13
