"""Performance cases of the tet4 ADER-DG element update: what a user's program asks of it.

A program builds a mesh with its element data (``edge_b200.host``), keeps them in a ``Solver`` and
steps it in calls of several time steps; the DOFs stay on the device (``Solver.device_ptrs``) or
travel with every call. The cases cover the smallest calls (launch latency), ordinary and large
meshes, every order, one and several fused runs, FP64 and FP32, elastic and viscoelastic physics,
homogeneous and heterogeneous materials, jittered meshes, local time stepping, the server's chunk
(receivers read back) and batches of uneven simulations.

``exact`` restates the update in 64-bit torch from its published form (weak-form ADER-DG: Taylor
expansion of the predictor, volume integral, fluxes of both sides), with DG matrices it integrates
itself; it shares with ``prepare`` only the inputs.
"""
import ctypes

import numpy as np
import torch

from edge_b200 import host
from edge_b200._lib import lib
from edge_b200.batch import Batch
from edge_b200.solver import Solver

EXT = 1e4                  # edge length of the box [m]
LAYERS = [4000.0, 5500.0, 6500.0]   # vp of the layered materials, from the top [m/s]


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def _case(name, kind="gts", order=4, runs=1, rm=0, precision=32, nx=8, ny=8, nz=8, steps=4, jitter=0.0,
          layered=False, sources=True, receivers=0, groups=0, sims=0):
    c = dict(kind=kind, order=order, runs=runs, rm=rm, precision=precision, nx=nx, ny=ny, nz=nz, steps=steps,
             jitter=jitter, layered=layered, sources=sources, receivers=receivers, groups=groups, sims=sims)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a test-sized mesh stepped one step at a time: launch latency
        _case("one_step_o3_fp64", order=3, precision=64, nx=3, ny=3, nz=3, steps=1, jitter=0.1),
        # the plain method: one forward run in FP64 on the 12^3 box, its receivers sampled
        _case("plain_o4_fp64", order=4, precision=64, nx=12, ny=12, nz=12, steps=20, receivers=8),
        # the same method at a production mesh and order
        _case("plain_o5_fp64", order=5, precision=64, nx=24, ny=25, nz=23, steps=4, jitter=0.1, layered=True),
        # sixteen fused forward runs, order 5: a source study or the columns of an inversion
        _case("fused_o5_r16_fp32", order=5, runs=16, nx=28, ny=28, nz=28, steps=4),
        # eight fused runs over a heterogeneous jittered mesh of odd size
        _case("fused_o4_r8_fp32", order=4, runs=8, nx=21, ny=17, nz=23, steps=6, jitter=0.2, layered=True),
        # the highest order
        _case("fused_o6_r16_fp32", order=6, runs=16, nx=14, ny=13, nz=15, steps=3, jitter=0.1),
        # one forward run in FP32 (a server's pool with a single request)
        _case("single_o5_fp32", order=5, runs=1, nx=23, ny=24, nz=22, steps=4, jitter=0.1, layered=True),
        # a server's chunk: four slots on a small mesh, receivers rewound, stepped and read back
        _case("serve_o3_r4_fp32", kind="serve", order=3, runs=4, nx=12, ny=12, nz=12, steps=20, receivers=12),
        # viscoelastic, three mechanisms, eight fused runs on the jittered layered box
        _case("visco_o4_r8_fp32", order=4, runs=8, rm=3, nx=20, ny=20, nz=20, steps=3, jitter=0.2, layered=True),
        # viscoelastic in plain FP64
        _case("visco_o4_fp64", order=4, rm=3, precision=64, nx=12, ny=11, nz=13, steps=5, jitter=0.1, layered=True),
        # rate-2 local time stepping over three groups of the layered box
        _case("lts_o5_r16_fp32", kind="lts", order=5, runs=16, nx=16, ny=16, nz=16, steps=1, layered=True,
              sources=False, groups=3),
        # uneven simulations stepped together through one captured batch
        _case("batch_mixed_fp32", kind="batch", order=4, runs=8, nx=10, ny=10, nz=10, steps=10, sims=4),
    ]


def draw(rng):
    """One more case of the same ranges; the largest of its kind costs about as much as the listed."""
    kind = rng.choice(["gts"] * 7 + ["serve", "lts", "batch"])
    log = lambda lo, hi: int(round(lo * (hi / lo) ** rng.random()))  # noqa: E731
    layered, jitter = rng.random() < 0.5, rng.choice([0.0, 0.1, 0.2])
    if kind == "lts":
        order, n = rng.choice([3, 4, 5]), log(6, 15)
        return _case(None, "lts", order, rng.choice([8, 16]), 0, 32, n, n, n, rng.choice([1, 2]), 0.0, True, False,
                     0, rng.choice([2, 3]))
    if kind == "batch":
        n = log(4, 10)
        return _case(None, "batch", rng.choice([4, 5]), rng.choice([4, 8]), 0, 32, n, n, n, rng.choice([5, 10]), 0.0,
                     False, True, 0, 0, rng.choice([2, 3, 4]))
    rm = 3 if kind == "gts" and rng.random() < 0.3 else 0
    precision = 64 if kind == "gts" and rng.random() < 0.35 else 32
    if precision == 64:
        order, runs = (rng.choice([3, 4]) if rm else rng.choice([2, 3, 4, 5, 6])), 1
    else:
        order, runs = rng.choice([3, 4, 5, 6]), rng.choice([1, 4, 8, 16])
    # the largest mesh of a configuration keeps its DOFs at or below the largest listed case's
    words = 9 * host.n_modes(order) * runs * (precision // 32) * (3 if rm else 1)
    top = min(24.0, (131712 * 5040 / words / 6 / 1.5) ** (1 / 3))
    n = log(3, max(4, top))
    n = [max(2, n + rng.choice([-1, 0, 0, 1])) for _ in range(3)]
    steps = rng.choice([1, 2, 3, 5, 8]) if max(n) < 14 else rng.choice([1, 2, 3])
    if kind == "serve":
        return _case(None, "serve", order, runs, 0, 32, *n, rng.choice([5, 10]), jitter, layered, True,
                     rng.choice([4, 8, 16]))
    return _case(None, "gts", order, runs, rm, precision, *n, steps, jitter, layered, rng.random() < 0.8,
                 rng.choice([0, 0, 4]))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _problem(c, seed, mesh=None):
    kw = {}
    if c["layered"]:
        kw.update(layers=LAYERS if c["kind"] != "lts" else [1500.0, 3000.0, 6000.0], lognormal_sigma=0.0 if
                  c["kind"] == "lts" else 0.1)
    if c["rm"]:
        kw.update(q_range=(50.0, 200.0), freq_cen=1.0, freq_rat=100.0)
    return host.build_problem((c["nx"], c["ny"], c["nz"]), c["order"], c["runs"], rm=c["rm"], ext=EXT,
                              jitter=c["jitter"], seed=seed, source="random" if c["sources"] else None,
                              n_receivers=c["receivers"], n_steps=400, f0_window=0.5, mesh=mesh, **kw)


def _inputs(c, seed):
    """[(problem, group_first, seed of its DOFs)] of a case: one entry, one per simulation of a batch."""
    if c["kind"] == "batch":
        out = []
        for k in range(c["sims"]):
            # meshes of different sizes; alternately the case's order and runs, and one order less
            d = dict(c, nx=max(2, c["nx"] - k), ny=max(2, c["ny"] - 2 * k), nz=max(2, c["nz"] - k),
                     order=c["order"] - (k % 2), runs=c["runs"] if k % 2 == 0 else 4)
            out.append((_problem(d, seed + 100 * k), None, seed + 100 * k))
        return out
    prob, gf = _problem(c, seed), None
    if c["kind"] == "lts":
        tg = host.time_groups(prob.mesh, host.dt_cfl_el(prob.mesh, c["order"], prob.rho, prob.lam, prob.mu), c["groups"])
        mesh, _, gf = host.sort_by_groups(prob.mesh, tg)
        prob = _problem(c, seed, mesh)
    return [(prob, gf, seed)]


def _degrees(order):
    return [d for d in range(order) for _ in range((d + 1) * (d + 2) // 2)]


def _start_rows(prob, precision, seed, device):
    """Wave-like initial DOFs as device rows [nEl][9][R][B] (and [nEl][rm*6][R][B]): stresses of
    1e6 Pa, velocities to match the impedance, coefficients falling with the mode's degree."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    dt = torch.float64 if precision == 64 else torch.float32
    amp = torch.tensor([2.0 ** -(2 * d) for d in _degrees(prob.order)], dtype=dt, device=device)
    q = torch.tensor([1e6] * 6 + [0.06] * 3, dtype=dt, device=device)
    e = torch.randn((prob.n_el, 9, prob.runs, prob.B), generator=g, dtype=dt, device=device)
    e.mul_(amp).mul_(q[None, :, None, None])
    a = None
    if prob.rm:
        a = torch.randn((prob.n_el, prob.rm * 6, prob.runs, prob.B), generator=g, dtype=dt, device=device)
        a.mul_(amp).mul_(1e-4)
    return e, a


class _Device:
    """A device array of a solver as seen by torch (no copy); a tensor over it keeps the solver alive."""

    def __init__(self, solver, ptr, shape, precision):
        self.solver = solver
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8" if precision == 64 else "<f4",
                                             data=(ptr, False), version=2, strides=None)


def _rows(solver):
    """The resident DOFs (Solver.device_ptrs): stresses, velocities, anelastic rows, without the padding."""
    p = solver.prob
    w = 16 // (solver.precision // 8)
    gb = -(-p.B // w) * w
    pe, pa, _ = solver.device_ptrs()
    e = torch.as_tensor(_Device(solver, pe, (p.n_el, 9, p.runs, gb), solver.precision), device="cuda")[..., :p.B]
    out = [e[:, :6], e[:, 6:]]
    if p.rm:
        out.append(torch.as_tensor(_Device(solver, pa, (p.n_el, p.rm * 6, p.runs, gb), solver.precision),
                                   device="cuda")[..., :p.B])
    return out


def prepare(case, seed):
    c = case
    solvers, rows = [], []
    for prob, gf, s in _inputs(c, seed):
        solver = Solver(prob, precision=c["precision"], stream=torch.cuda.current_stream().cuda_stream)
        e, a = _start_rows(prob, c["precision"], s, "cuda")
        view = _rows(solver)
        view[0].copy_(e[:, :6])
        view[1].copy_(e[:, 6:])
        if a is not None:
            view[2].copy_(a)
        if gf is not None:
            solver.set_time_groups(gf)
        solvers.append(solver)
        rows.append(view)
    torch.cuda.synchronize()
    return dict(case=c, solvers=solvers, rows=rows, batch=Batch(solvers) if c["kind"] == "batch" else None)


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    c, s = state["case"], state["solvers"][0]
    if c["kind"] == "batch":
        state["batch"].run(c["steps"])
        return state["rows"]
    if c["kind"] == "lts":
        s.step_lts(c["steps"])
        return state["rows"]
    if c["receivers"]:
        # samples of this call only, as the server reads them chunk by chunk
        s._chk(lib().edge_b200_rewind_receivers(s._h, ctypes.c_double(s.t)), "rewind_receivers")
    s.step(c["steps"])
    if c["receivers"]:
        return state["rows"] + [[s.receivers()[0]]]
    return state["rows"]


_COUNT = {}


def _element_steps(c):
    """[(order, runs, element updates per run)] of one pass."""
    if c["kind"] == "batch":
        return [(c["order"] - (k % 2), c["runs"] if k % 2 == 0 else 4,
                 6 * max(2, c["nx"] - k) * max(2, c["ny"] - 2 * k) * max(2, c["nz"] - k) * c["steps"])
                for k in range(c["sims"])]
    n = 6 * c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "lts":
        key = (c["order"], c["nx"], c["ny"], c["nz"], c["groups"])
        if key not in _COUNT:
            (_, gf, _), = _inputs(dict(c, runs=1, sources=False), 0)
            g = len(gf) - 1
            _COUNT[key] = sum(int(gf[i + 1] - gf[i]) << (g - 1 - i) for i in range(g))
        return [(c["order"], c["runs"], _COUNT[key] * c["steps"])]
    return [(c["order"], c["runs"], n * c["steps"])]


def work(case):
    """Bytes: per element update the DOFs read and written and the element's star matrices, flux
    solvers of both sides (FP64, as the caller gives them) and connectivity read once. Flops: the
    reference algorithm's dense products (recursion, volume, both surface integrals)."""
    c, byts, flops = case, 0.0, 0.0
    p, rm = c["precision"] // 8, c["rm"]
    nm, nf = host.n_modes, host.n_face_modes
    for order, runs, upd in _element_steps(c):
        b, f = nm(order), nf(order)
        nq = 9 + 6 * rm
        const = (72 + 648 + (27 + 12 * rm + 432 if rm else 0)) * 8 + 28
        byts += upd * (2 * nq * b * runs * p + const)
        mq = 9 + (6 if rm else 0)
        ck = sum(3 * (9 * nm(order - (1 if rm else d) + 1) * nm(order - (1 if rm else d)) +
                      mq * 3 * nm(order - (1 if rm else d))) for d in range(1, order))
        vol = 3 * (9 * nm(order - 1) * b + mq * 3 * b)
        src = rm * 12 * b * (order + 1)
        face = 2 * 4 * (9 * b * f + mq * 9 * f + mq * f * b)
        flops += upd * runs * 2.0 * (ck + vol + src + face)
    return dict(bytes=byts, flops=flops)


def tolerance(case):
    """FP32 rounding of a few steps, FP64 rounding likewise: about four times the largest distance
    from ``exact`` seen over the listed cases and draws of every kind (stresses and velocities each
    on their own): 6.2e-7 and 1.2e-5 in FP32, 6.8e-15 and 1.5e-13 in FP64."""
    if case["precision"] == 64:
        return {"rel": 4e-14, "max": 1e-12}
    return {"rel": 2.5e-6, "max": 6e-5}


# ------------------------------------------------------------------------------------------------
# 64-bit restatement
# ------------------------------------------------------------------------------------------------
_DG = {}
# non-zeros (row, column) of the 9x9 elastic star matrix, the 6x3 anelastic star (velocities) and
# the 6x6 anelastic source, in the order the setup lists them
_STAR = list(zip([0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 4, 4, 5, 5, 6, 6, 6, 7, 7, 7, 8, 8, 8],
                 [6, 7, 8, 6, 7, 8, 6, 7, 8, 6, 7, 7, 8, 6, 8, 0, 3, 5, 1, 3, 4, 2, 4, 5]))
_STAR_A = list(zip([0, 1, 2, 3, 3, 4, 4, 5, 5], [0, 1, 2, 0, 1, 1, 2, 0, 2]))
_SRC = list(zip([0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 4, 5], [0, 1, 2, 0, 1, 2, 0, 1, 2, 3, 4, 5]))


def _jacobi(n, a, x, w):
    """w^n P_n^(a,0)(2 x / w - 1) (values)."""
    from math import comb
    return sum(comb(n + a, n - s) * comb(n, s) * (x - w) ** s * x ** (n - s) for s in range(n + 1))


def _tet_basis(order, p):
    x, y, z = p.T
    out = []
    for d in range(order):
        for i in range(d + 1):
            for j in range(d + 1 - i):
                k = d - i - j
                out.append(_jacobi(i, 0, x, 1 - y - z) * _jacobi(j, 2 * i + 1, y, 1 - z) *
                           _jacobi(k, 2 * i + 2 * j + 2, z, np.ones_like(z)))
    return np.stack(out, 1)


def _tri_basis(order, p):
    x, y = p.T
    return np.stack([_jacobi(i, 0, x, 1 - y) * _jacobi(d - i, 2 * i + 1, y, np.ones_like(y))
                     for d in range(order) for i in range(d + 1)], 1)


def _matrices(order):
    """Stiffness (both sides), face projection, neighbour projection [4 v + f] and lift matrices by
    collapsed Gauss quadrature of the hierarchical orthogonal basis."""
    if order in _DG:
        return _DG[order]
    x, w = np.polynomial.legendre.leggauss(order + 3)
    x, w = (x + 1) / 2, w / 2
    c, b, a = np.meshgrid(x, x, x, indexing="ij")
    wc, wb, wa = np.meshgrid(w, w, w, indexing="ij")
    pt = np.stack([(a * (1 - b) * (1 - c)).ravel(), (b * (1 - c)).ravel(), c.ravel()], 1)
    wt = (wa * wb * wc * (1 - b) * (1 - c) ** 2).ravel()
    V = _tet_basis(order, pt)
    # derivatives of the polynomials by a complex step (no cancellation)
    D = [_tet_basis(order, pt + 1e-30j * np.eye(3)[dim]).imag / 1e-30 for dim in range(3)]
    mass = np.einsum("p,pi,pi->i", wt, V, V)
    stiff = [np.einsum("p,pi,pj->ij", wt, V, d) for d in D]
    b2, a2 = np.meshgrid(x, x, indexing="ij")
    wb2, wa2 = np.meshgrid(w, w, indexing="ij")
    pf = np.stack([(a2 * (1 - b2)).ravel(), b2.ravel()], 1)
    wf = (wa2 * wb2 * (1 - b2)).ravel()
    T = _tri_basis(order, pf)
    mf = np.einsum("p,pi,pi->i", wf, T, T)
    s, t, z = pf[:, 0], pf[:, 1], np.zeros(len(pf))
    face = [np.stack(v, 1) for v in ((t, s, z), (s, z, t), (z, t, s), (1 - s - t, s, t))]
    turn = [np.stack(v, 1) for v in ((t, s), (1 - s - t, t), (s, 1 - s - t))]
    proj = [np.einsum("p,pi,pj->ij", wf, _tet_basis(order, f), T) for f in face]
    ori = [np.einsum("p,pi,pj->ij", wf, _tri_basis(order, v), T) for v in turn]
    m = dict(ckT=[-(k.T / mass) for k in stiff], vol=[k / mass for k in stiff], proj=proj,
             nproj=[proj[f] @ (ori[v] / mf[:, None]) for v in range(3) for f in range(4)],
             lift=[(p / mf).T / mass for p in proj])
    clean = lambda v: [np.where(np.abs(x) < 1e-12 * np.abs(x).max(), 0.0, x) for x in v]  # noqa: E731
    _DG[order] = {k: clean(v) for k, v in m.items()}
    return _DG[order]


def _dense(v, pattern, rows, cols, dev):
    out = torch.zeros(v.shape[:-1] + (rows, cols), dtype=torch.float64, device=dev)
    t = torch.as_tensor(np.asarray(v, np.float64), device=dev)
    for i, (r, k) in enumerate(pattern):
        out[..., r, k] = t[..., i]
    return out


def _mix(m, x):
    """m [e][a][b] applied to the rows of x [e][b][R][B]."""
    return torch.bmm(m, x.flatten(2)).view(x.shape[0], m.shape[1], *x.shape[2:])


class _Exact:
    """The update of one problem in 64 bits on rows [nEl][9][R][B]."""

    def __init__(self, prob, e, a, dev):
        self.p, self.dev = prob, dev
        to = lambda v: [torch.as_tensor(x, device=dev) for x in v]  # noqa: E731
        self.m = {k: to(v) for k, v in _matrices(prob.order).items()}
        self.q = e.to(torch.float64)
        self.a = None if a is None else a.to(torch.float64).view(prob.n_el, prob.rm, 6, prob.runs, prob.B)
        self.ti = torch.zeros_like(self.q)
        self.t = 0.0
        self.fs = torch.as_tensor(prob.fsE, device=dev).view(2, -1, 4, 9, 9)
        self.fsa = torch.as_tensor(prob.fsA, device=dev).view(2, -1, 4, 6, 9) if prob.rm else None
        self.om = torch.as_tensor(prob.omega, device=dev) if prob.rm else None
        ty = np.asarray(prob.mesh.el_fa_type)
        self.free = [torch.as_tensor(np.flatnonzero(ty[:, f] == host.FACE_FREE_SURFACE), device=dev) for f in range(4)]
        self.nbr = {}
        for f in range(4):
            for k in range(12):
                on = (ty[:, f] == host.FACE_INNER) & (4 * prob.mesh.vid[:, f].astype(int) + prob.mesh.fid[:, f] == k)
                i = np.flatnonzero(on)
                if len(i):
                    self.nbr[f, k] = (torch.as_tensor(i, device=dev),
                                      torch.as_tensor(prob.mesh.el_fa_el[i, f].astype(np.int64), device=dev))

    def chunks(self, lo=0, hi=None):
        hi = self.p.n_el if hi is None else hi
        n = max(1, int(2.0e7 / (9 * self.p.runs * self.p.B)))
        for s in range(lo, hi, n):
            yield torch.arange(s, min(s + n, hi), device=self.dev)

    def star(self, i):
        k = i.cpu().numpy()
        p = self.p
        st = _dense(p.starE[k], _STAR, 9, 9, self.dev)
        if not p.rm:
            return st, None, None
        return st, _dense(p.starA[k], _STAR_A, 6, 3, self.dev), _dense(p.srcA[k], _SRC, 6, 6, self.dev)

    def taylor(self, i, st, sa, sr):
        """Time derivatives of the rows (and anelastic rows) of elements i."""
        p, d = self.p, [self.q[i]]
        da = [self.a[i]] if p.rm else None
        for _ in range(1, p.order):
            x = d[-1]
            y = sum(_mix(st[:, k], x) @ self.m["ckT"][k] for k in range(3))
            if p.rm:
                v = sum(_mix(sa[:, k], x[:, 6:]) @ self.m["ckT"][k] for k in range(3))
                for m in range(p.rm):
                    y[:, :6] += _mix(sr[:, m], da[-1][:, m])
                da.append(self.om[None, :, None, None, None] * (v[:, None] + da[-1]))
            d.append(y)
        return d, da

    def integral(self, d, dt):
        s, out = dt, dt * d[0]
        for k in range(1, len(d)):
            s = s * dt / (k + 1)
            out = out + s * d[k]
        return out

    def local(self, lo, hi, dt, half=None):
        """Predictor, volume and own flux of the elements [lo, hi); half: rows for the integral over
        the first half of the step."""
        p, m = self.p, self.m
        for i in self.chunks(lo, hi):
            st, sa, sr = self.star(i)
            d, da = self.taylor(i, st, sa, sr)
            ti = self.integral(d, dt)
            self.ti[i] = ti
            if half is not None:
                half[i] = self.integral(d, dt / 2)
            up = sum(_mix(st[:, k], ti) @ m["vol"][k] for k in range(3))
            upa = None
            if p.rm:
                tia = self.integral(da, dt)
                upa = sum(_mix(sa[:, k], ti[:, 6:]) @ m["vol"][k] for k in range(3))[:, None] - tia
                for k in range(p.rm):
                    up[:, :6] += _mix(sr[:, k], tia[:, k])
            for f in range(4):
                x = ti @ m["proj"][f]
                up += _mix(self.fs[0, i, f], x) @ m["lift"][f]
                if p.rm:
                    upa += (_mix(self.fsa[0, i, f], x) @ m["lift"][f])[:, None]
            self.q[i] += up
            if p.rm:
                self.a[i] += self.om[None, :, None, None, None] * upa

    def add_flux(self, i, f, x):
        self.q.index_add_(0, i, _mix(self.fs[1, i, f], x) @ self.m["lift"][f])
        if self.p.rm:
            up = _mix(self.fsa[1, i, f], x) @ self.m["lift"][f]
            self.a.index_add_(0, i, self.om[None, :, None, None, None] * up[:, None])

    def neigh(self, lo, hi, pick):
        """Flux from the face neighbours of the elements [lo, hi); pick(i, j): the rows that the
        elements i read of their neighbours j."""
        for f in range(4):
            i = self.free[f]
            i = i[(i >= lo) & (i < hi)]
            for i in i.split(8192):
                if len(i):
                    self.add_flux(i, f, self.ti[i] @ self.m["proj"][f])
            for k in range(12):
                if (f, k) not in self.nbr:
                    continue
                i, j = self.nbr[f, k]
                on = (i >= lo) & (i < hi)
                for i, j in zip(i[on].split(8192), j[on].split(8192)):
                    self.add_flux(i, f, pick(i, j) @ self.m["nproj"][k])

    def sources(self, t, dt):
        s = self.p.sources
        for n in range(s["n"] if s else 0):
            o, k = int(s["tsOff"][n]), int(s["nPts"][n])
            v, h, x0 = s["ts"][o:o + k], float(s["dt"][n]), float(s["t0"][n])
            area = np.concatenate([[0.0], np.cumsum(0.5 * h * (v[1:] + v[:-1]))])

            def upto(x):
                y = min(max((x - x0) / h, 0.0), k - 1.0)
                c = min(int(y), k - 2)
                r = y - c
                return area[c] + h * (r * v[c] + 0.5 * r * r * (v[c + 1] - v[c]))
            add = np.outer(s["scal"][n], s["bEval"][n]) * (upto(t + dt) - upto(t))
            self.q[int(s["el"][n]), :, int(s["run"][n])] += torch.as_tensor(add, device=self.dev)

    def sample(self, t, dt, clock, buf):
        """Receiver samples of the step [t, t + dt); clock: the next sample's time and slot."""
        r = self.p.receivers
        if not r or not r.get("n", 0):
            return
        times = []
        while t - 1e-9 < clock[0] < t + dt - 1e-9:
            times.append((clock[0] - t, clock[1]))
            clock[0] += r["period"]
            clock[1] += 1
        if not times:
            return
        i = torch.as_tensor(r["el"], device=self.dev)
        d, _ = self.taylor(i, *self.star(i))
        basis = torch.as_tensor(r["basis"], device=self.dev)
        for tau, slot in times:
            v, s = torch.zeros_like(d[0]), 1.0
            for k in range(len(d)):
                s = s * tau / k if k else 1.0
                n = host.n_modes(self.p.order - k)
                v[..., :n] += s * d[k][..., :n]
            buf[:, slot] = torch.einsum("eqrb,eb->eqr", v, basis).cpu().numpy()

    def steps(self, n):
        """n steps of the whole mesh; the receivers' buffer."""
        r, dt, buf = self.p.receivers, self.p.dt, None
        clock = [self.t, 0]
        if r and r.get("n", 0):
            buf = np.zeros((r["n"], r["maxbuf"], 9, self.p.runs))
        for _ in range(n):
            self.sample(self.t, dt, clock, buf)
            self.local(0, self.p.n_el, dt)
            self.sources(self.t, dt)
            self.neigh(0, self.p.n_el, lambda i, j: self.ti[j])
            self.t += dt
        return buf

    def cycles(self, gf, n):
        """n cycles of rate-2 local time stepping over the groups [gf[g], gf[g+1])."""
        g_n = len(gf) - 1
        grp = torch.zeros(self.p.n_el, dtype=torch.long, device=self.dev)
        for g in range(g_n):
            grp[int(gf[g]):int(gf[g + 1])] = g
        two, half = torch.zeros_like(self.q), torch.zeros_like(self.q)
        for k in range(n << (g_n - 1)):
            for g in range(g_n):
                if k % (1 << g) == 0:
                    lo, hi = int(gf[g]), int(gf[g + 1])
                    self.local(lo, hi, self.p.dt * (1 << g), half)
                    two[lo:hi] = self.ti[lo:hi] + (two[lo:hi] if (k >> g) & 1 else 0)
            for g in range(g_n):
                if (k + 1) % (1 << g) == 0:
                    second = bool(((k + 1 - (1 << g)) >> g) & 1)

                    def pick(i, j, g=g, second=second):
                        x = self.ti[j].clone()
                        small, large = grp[j] < g, grp[j] > g
                        x[small] = two[j[small]]
                        h = half[j[large]]
                        x[large] = x[large] - h if second else h
                        return x
                    self.neigh(int(gf[g]), int(gf[g + 1]), pick)


def exact(case, seed, device="cuda"):
    out, buf = [], None
    for prob, gf, s in _inputs(case, seed):
        e, a = _start_rows(prob, case["precision"], s, device)
        x = _Exact(prob, e, a, device)
        del e, a
        if case["kind"] == "lts":
            x.cycles(gf, case["steps"])
        else:
            buf = x.steps(case["steps"])
        view = [x.q[:, :6], x.q[:, 6:]]
        if prob.rm:
            view.append(x.a.reshape(prob.n_el, prob.rm * 6, prob.runs, prob.B))
        out.append(view)
    rows = out if case["kind"] == "batch" else out[0]
    if case["kind"] != "lts" and case["kind"] != "batch" and case["receivers"]:
        return rows + [[buf]]
    return rows
