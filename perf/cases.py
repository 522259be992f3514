"""Performance cases of the explicit RDS solver: what a program that uses it has it do.

A case is a dict of plain values. `kind` says which calls one pass makes:

  steps    the reference examples' own loop, driven by the host: assemble_lhs_and_rhs, solve,
           compute_residual_norm, one call after the other (small meshes; latency counts)
  iterate  set_solution, the device loop over `sweeps` sweeps, solution
  rk3      set_solution, `sweeps` third-order Runge-Kutta steps, solution
  blend    every step: the nodal LF_Blend coefficient from the current state, installed, then
           assemble_lhs_and_rhs and solve (shock capturing, as the Burgers example does)
  drop     set_solution, the device loop until the residual has dropped by 1e-10, solution: what
           the mixed form is for (its single-precision sweeps leave the converged state alone)
  batch    many independent problems of uneven size in one context: set_solutions, the device
           loop over all of them, solutions; with `drop`, each to its own 1e-10

The meshes are jittered unit squares of triangles (scalar physics), the bump channel of triangles
and quadrilaterals (euler2d) and the bump box of tetrahedra (euler3d), with the quadrature rules
of the benchmark configurations. A mesh belongs to its case; the initial state comes from the
seed. Every pass starts from that state again, so all passes on a state are alike.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pdekit_b200 import meshgen, workloads
from pdekit_b200 import reference_element as ref
from pdekit_b200.batch import BatchedRDS
from pdekit_b200.rds import PGRDMethodExplicit
from pdekit_b200.stabilisation import RDBlendingCoeff

DROP, MOST_SWEEPS = 1e-10, 200000
MACH = {"euler2d": 0.5, "euler3d": 0.6}
GAS_R = 287.046


def listed():
    return [
        # a first run on a coarse mesh, each step called by the host and its norm looked at
        dict(name="steps burgers p2 16x16", kind="steps", physics="burgers", scheme="b", order=2,
             n=16, cfl=0.5, sweeps=24, precision="fp64"),
        # steady advection on the small benchmark mesh, about half of its way to convergence
        dict(name="advection p1 64x64", kind="iterate", physics="advconst", scheme="lda", order=1,
             n=64, cfl=0.9, sweeps=240, precision="fp64"),
        # the headline configuration: Burgers with a shock, P2, 524,288 cells
        dict(name="burgers p2 512x512", kind="iterate", physics="burgers", scheme="b", order=2,
             n=512, cfl=0.5, sweeps=64, precision="fp64"),
        # cubic elements, an odd mesh
        dict(name="burgers p3 181x181", kind="iterate", physics="burgers", scheme="n", order=3,
             n=181, cfl=0.45, sweeps=64, precision="fp64"),
        # the mixed form to convergence, on a mesh between the small and the headline one
        dict(name="burgers p2 320x320 mixed", kind="drop", physics="burgers", scheme="n", order=2,
             n=320, cfl=0.5, precision="mixed"),
        # a parameter study: uneven advection and Burgers problems of all orders at once
        dict(name="batch of 24", kind="batch", nprob=24, max_cells=40000, mesh_seed=5, sweeps=128,
             precision="fp64"),
        # a study of smaller ones, each to its own convergence, in the mixed form
        dict(name="batch of 20 mixed", kind="batch", nprob=20, max_cells=4000, mesh_seed=11,
             sweeps=0, precision="mixed"),
        # subsonic channel flow on a hybrid P3 mesh of triangles and quadrilaterals
        dict(name="euler2d p3 hybrid", kind="iterate", physics="euler2d", scheme="b", order=3,
             nx_tri=125, nx_quad=250, ny=125, cfl=0.5, sweeps=24, precision="fp64"),
        # a coarser channel of P2 triangles only, time-accurate stepping
        dict(name="euler2d p2 rk3", kind="rk3", physics="euler2d", scheme="n", order=2, nx_tri=150,
             nx_quad=0, ny=61, cfl=0.5, sweeps=12, precision="fp64"),
        # the bump box, P2 tetrahedra
        dict(name="euler3d p2 lda", kind="iterate", physics="euler3d", scheme="lda", order=2,
             nx=64, ny=16, nz=16, cfl=0.5, sweeps=24, precision="fp64"),
        # a coarse channel converged in the mixed form
        dict(name="euler2d p1 mixed", kind="drop", physics="euler2d", scheme="n", order=1,
             nx_tri=24, nx_quad=0, ny=8, cfl=0.5, precision="mixed"),
        # shock capturing with the blending coefficient recomputed every step
        dict(name="burgers p2 blend 160x160", kind="blend", physics="burgers", scheme="b", order=2,
             n=160, cfl=0.5, sweeps=16, precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "iterate", "iterate", "iterate", "iterate", "rk3", "drop",
                       "blend", "batch", "batch"])
    if kind == "batch":
        if rng.random() < 0.5:
            return dict(kind=kind, nprob=rng.randint(6, 30), mesh_seed=rng.randint(0, 10**6),
                        max_cells=_log_int(rng, 3000, 40000), sweeps=rng.randint(40, 128),
                        precision="fp64")
        return dict(kind=kind, nprob=rng.randint(6, 20), mesh_seed=rng.randint(0, 10**6),
                    max_cells=_log_int(rng, 2000, 4500), sweeps=0, precision="mixed")
    if kind == "blend":
        return dict(kind=kind, physics=rng.choice(["advconst", "burgers"]), scheme="b",
                    order=rng.randint(1, 3), n=_log_int(rng, 20, 250), cfl=0.5,
                    sweeps=rng.randint(4, 16), precision="fp64")
    if kind == "drop":
        # the combinations that converge: advection with LDA or N, Burgers and Euler with N
        physics = rng.choice(["advconst", "burgers", "burgers", "euler2d"])
        c = dict(kind=kind, physics=physics, scheme="n", cfl=round(rng.uniform(0.4, 0.55), 3))
        if physics == "euler2d":
            ny = rng.randint(4, 8)
            return dict(c, order=1, nx_tri=3 * ny + rng.randint(0, 2), nx_quad=0, ny=ny,
                        precision="mixed")
        return dict(c, scheme=rng.choice(["lda", "n"]) if physics == "advconst" else "n",
                    order=rng.randint(1, 3), n=_log_int(rng, 12, 160), precision="mixed")
    physics = rng.choice(["advconst", "burgers", "euler2d", "euler3d"])
    c = dict(kind=kind, physics=physics, scheme=rng.choice(["lda", "n", "b"]))
    small = kind == "steps"
    if physics in ("advconst", "burgers"):
        c.update(order=rng.randint(1, 3), n=_log_int(rng, 8, 40 if small else 300),
                 cfl=round(rng.uniform(0.3, 0.6), 3), sweeps=rng.randint(8, 48))
    elif physics == "euler2d":
        ny = _log_int(rng, 6, 20 if small else 110)
        tri, quad = rng.choice([(1, 2), (1, 2), (3, 0), (0, 3)])
        c.update(order=rng.randint(1, 3), nx_tri=ny * tri + (rng.randint(0, 3) if tri else 0),
                 nx_quad=ny * quad + (rng.randint(0, 3) if quad else 0), ny=ny, cfl=0.5,
                 sweeps=rng.randint(6, 20))
    else:
        ny = _log_int(rng, 3, 5 if small else 14)
        c.update(order=rng.choice([1, 2, 2]), nx=ny * 4 + rng.randint(0, 2), ny=ny,
                 nz=ny + rng.randint(0, 2), cfl=0.5, sweeps=rng.randint(6, 20))
    return dict(c, precision="fp64")


# ---- meshes and states ---------------------------------------------------------------------


@functools.lru_cache(maxsize=2)
def _problem(key):
    """The host description of a case's problem, or a list of them and their CFLs (batch)."""
    c = dict(key)
    if c["kind"] == "batch":
        return workloads.config5(c["nprob"], c["mesh_seed"], 1000, c["max_cells"])[:3:2]
    p, rules = c["order"], {1: 4, 2: 5, 3: 8}
    tri = ref.triag_tables(p, rules[p])
    if c["physics"] in ("advconst", "burgers"):
        bcs = workloads.ADV_BCS if c["physics"] == "advconst" else workloads.BURGERS_BCS
        return workloads.tri_problem(c["physics"], c["scheme"], p, c["n"], 0.15, 7, bcs, tri)
    if c["physics"] == "euler2d":
        # cells' dual volumes by the rule of their own order, as the quadrilaterals' tables do
        if p == 3:
            rule = ref.triag_gauss(p)
            tri = dict(tri, wv=rule[1], dVgeo_v=ref.lagrange_triag(1, rule[0])[1])
        quad = ref.quad_tables(p, {1: 4, 2: 5, 3: 8}[p], tensor=True)
        mesh = meshgen.channel_2d(c["nx_tri"], c["nx_quad"], c["ny"], jitter=0.1, seed=3)
        tables = {"triag": tri, "quad": quad}
        return workloads.mesh_problem(mesh, "euler2d", c["scheme"], p, tables,
                                      workloads.euler_bcs(2))
    mesh = meshgen.box_tet(c["nx"], c["ny"], c["nz"], jitter=0.1, seed=4)
    tables = {"tetra": ref.tet_tables(p, {1: 2, 2: 5}[p])}
    return workloads.mesh_problem(mesh, "euler3d", c["scheme"], p, tables, workloads.euler_bcs(3))


def _key(case):
    drop = ("name", "sweeps", "cfl", "precision")
    return tuple(sorted((k, v) for k, v in case.items() if k not in drop))


def _state(prob, rng):
    """An initial state [nodes, equations]: the configurations' own, changed by the seed."""
    xy = prob.sol_coords
    if prob.neq > 1:
        # freestream of the bump cases, density and pressure perturbed by up to 1% per node
        mach = MACH[prob.physics]
        f = 1.0 + 0.2 * mach * mach
        T, p0 = workloads.T_TOT / f, workloads.P_TOT / f**3.5
        rho = p0 / (GAS_R * T) * (1.0 + rng.uniform(-0.01, 0.01, len(xy)))
        p = p0 * (1.0 + rng.uniform(-0.01, 0.01, len(xy)))
        ux = mach * math.sqrt(1.4 * GAS_R * T)
        u = np.zeros((len(xy), prob.neq))
        u[:, 0], u[:, 1] = rho, rho * ux
        u[:, -1] = p / 0.4 + 0.5 * rho * ux * ux
        return u
    x, y = xy[:, 0], xy[:, 1]
    a, b, phase = rng.uniform(2.0, 8.0), rng.uniform(2.0, 8.0), rng.uniform(0.0, 6.0)
    wave = 0.1 * np.sin(a * x + b * y + phase)
    u = 1.5 - 2.0 * x + wave * y if prob.physics == "burgers" else wave
    return u.reshape(-1, 1)


def _states(case, seed):
    rng = np.random.default_rng(seed)
    got = _problem(_key(case))
    if case["kind"] == "batch":
        return got[0], got[1], [_state(p, rng) for p in got[0]]
    return got, case["cfl"], _state(got, rng)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    prob, cfl, u0 = _states(case, seed)
    if case["kind"] == "batch":
        solver = BatchedRDS(prob, cfl, precision=case["precision"])
        return dict(case=case, solver=solver, u0=u0)
    solver = PGRDMethodExplicit(prob.physics, prob.scheme, case["precision"])
    solver.configure_mesh_data(prob)
    solver.initialize_work_data()
    start, out = _pinned(u0.shape), _pinned(u0.shape)
    start[:] = u0
    s = dict(case=case, solver=solver, cfl=cfl, u0=start, out=out)
    if case["kind"] == "blend":
        s["blend"] = RDBlendingCoeff().setup(solver, "LF_Blend")
    return s


def run(s):
    case, solver = s["case"], s["solver"]
    kind, sweeps = case["kind"], case.get("sweeps", 0)
    if kind == "batch":
        solver.set_solutions(s["u0"])
        if sweeps == 0:
            solver.iterate(MOST_SWEEPS, drop=DROP)
            return dict(u=np.concatenate(solver.solutions()))
        iters, drop = solver.iterate(sweeps, drop=0.0)
        return dict(u=np.concatenate(solver.solutions()), iters=iters, drop=drop)
    solver.set_solution(s["u0"])
    got = {}
    if kind == "drop":
        solver.iterate(s["cfl"], MOST_SWEEPS, DROP)
    elif kind == "iterate":
        got["norms"] = solver.iterate(s["cfl"], sweeps)[1]
    elif kind == "steps":
        norms = []
        for _ in range(sweeps):
            solver.assemble_lhs_and_rhs(s["cfl"])
            solver.solve()
            norms.append(solver.compute_residual_norm())
        got["norms"] = np.stack(norms)
    elif kind == "rk3":
        solver.advance_rk3tvd(s["cfl"], sweeps)
    else:
        for _ in range(sweeps):
            got["theta"] = s["blend"].calculate(install=True)
            solver.assemble_lhs_and_rhs(s["cfl"])
            solver.solve()
    got["u"] = solver.solution(s["out"])
    return got


def _typical_sweeps(case, prob, cfl):
    """Sweeps of one pass; of one that goes to its drop about as many as it takes (measured:
    waves crossing the mesh some times for the scalar physics, far more in a channel)."""
    if case.get("sweeps", 0) > 0:
        return case["sweeps"] * (3 if case["kind"] == "rk3" else 1)
    if prob.neq > 1:
        return 600.0 * case["ny"] / cfl
    across = math.sqrt(prob.ncells / 2.0) * prob.groups[0].order
    return (16.0 if prob.physics == "burgers" else 7.0) * across / cfl


def work(case):
    """Per sweep: the connectivity, the geometry and the state read once, the state written
    once; the operations of the scheme with every quantity formed once per point and node."""
    got = _problem(_key(case))
    probs = zip(*got) if case["kind"] == "batch" else [(got, case["cfl"])]
    nbytes = flops = 0.0
    for p, cfl in probs:
        sweeps = _typical_sweeps(case, p, cfl)
        nbytes += sweeps * (8.0 * p.geo_coords.size + 16.0 * p.nnodes * p.neq)
        d, e = p.dim, p.neq
        for g in p.groups:
            nbytes += sweeps * 4.0 * (g.sol_conn.size + g.geo_conn.size)
            dofs = 1 if p.scheme == "lda" else 2  # LDA part, N part
            if e == 1:
                per_q = 4 * g.nfl + (2 * g.ndof if p.physics == "burgers" else 0) + 8
                per_qn = 5 + 2 + 5 * (dofs - 1)
                per_f = 2 * g.ndof + 8
            else:
                sums = 2 * e * g.nfl * d + 2 * e * g.ndof + 2 * e**3 // 3 + 4 * e * e
                per_q = sums + (0 if g.shape != "quad" else 2 * e * d * d)
                # gradient, |gradient|, three eigenvalues, two rank-one terms summed and applied
                per_qn = 2 * d * d + 20 + (d + 1) * (d + 2) + dofs * 4 * (e + d)
                per_f = 2 * e * g.ndof + 6 * e * d
            flops += sweeps * g.ncells * float(g.nq * per_q + g.nq * g.ndof * per_qn + g.nfl * per_f)
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits, plain torch ------------------------------------------------------


class _Cells:
    """One cell group on the device: geometry at the points, gradients of the basis."""

    def __init__(self, p, g, dev):
        def t(a):
            return torch.as_tensor(np.ascontiguousarray(a), device=dev)

        self.conn, self.w, self.V, self.Vsf = t(g.sol_conn).long(), t(g.w), t(g.V), t(g.Vsf)
        self.dV, self.dVf, self.dVgeo = t(g.dV), t(g.dVf), t(g.dVgeo)
        self.X = t(p.geo_coords)[t(g.geo_conn).long()]
        rule = (g.w, g.dVgeo) if g.wv is None else (g.wv, g.dVgeo_v)
        jac = torch.einsum("dqg,cgx->cqdx", t(rule[1]), self.X)
        self.vol = torch.linalg.det(jac) @ t(rule[0])
        # per point: w det J, the flux basis' and the solution basis' gradients [c, node, x]
        self.points = []
        for q in range(len(g.w)):
            jac = torch.einsum("dg,cgx->cdx", self.dVgeo[:, q], self.X)
            inv = torch.linalg.inv(jac)  # [c, x, xi]
            self.points.append((self.w[q] * torch.linalg.det(jac),
                                torch.einsum("cxd,df->cfx", inv, self.dVf[:, q]),
                                torch.einsum("cxd,dn->cnx", inv, self.dV[:, q])))


class _Exact:
    """Residual-distribution sweeps of a problem, vectorised over its cells."""

    def __init__(self, p):
        self.p = p
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.cells = [_Cells(p, g, self.dev) for g in p.groups]
        self.X = torch.as_tensor(p.geo_coords, device=self.dev)
        self.blend = None
        self.vol = torch.zeros(p.nnodes, dtype=torch.float64, device=self.dev)
        for k in self.cells:
            self._add(self.vol, k.conn, k.vol[:, None].expand(k.conn.shape))

    @staticmethod
    def _add(to, conn, values):
        to.index_add_(0, conn.reshape(-1), values.reshape(conn.numel(), *to.shape[1:]))

    # physics
    def _props(self, u):
        d = self.p.dim
        V = u[..., 1:1 + d] / u[..., :1]
        P = (self.p.gamma - 1.0) * (u[..., -1] - 0.5 * (u[..., 1:1 + d] * V).sum(-1))
        return V, P, torch.sqrt(self.p.gamma * P / u[..., 0])

    def _flux(self, u):
        """F [..., equation, direction]"""
        p, d = self.p, self.p.dim
        if p.physics == "burgers":
            return torch.stack([0.5 * u * u, u], -1)
        if p.physics == "advconst":
            return torch.stack([p.adv[0] * u, p.adv[1] * u], -1)
        V, P, _ = self._props(u)
        F = u[..., :, None] * V[..., None, :]
        for k in range(d):
            F[..., 1 + k, k] += P
        F[..., d + 1, :] += P[..., None] * V
        return F

    def _split(self, u, g, sign):
        """K with its eigenvalues clipped (max(0, .) for sign 1, min(0, .) for -1), direction g;
        and the largest |eigenvalue|. u [..., neq], g [..., dim]."""
        p, d = self.p, self.p.dim

        def clip(x):
            return torch.clamp(x, min=0.0) if sign > 0 else torch.clamp(x, max=0.0)

        if p.neq == 1:
            if p.physics == "burgers":
                k = u[..., 0] * g[..., 0] + g[..., 1]
            else:
                k = p.adv[0] * g[..., 0] + p.adv[1] * g[..., 1]
            return clip(k)[..., None, None], k.abs()
        V, P, a = self._props(u)
        rho, gm1 = u[..., 0], p.gamma - 1.0
        H = (u[..., -1] + P) / rho
        norm = torch.linalg.vector_norm(g, dim=-1)
        n = g / torch.where(norm > 0, norm, torch.ones_like(norm))[..., None]
        vn, ke = (V * n).sum(-1), 0.5 * (V * V).sum(-1)
        lc, lp, lm = norm * vn, norm * (vn + a), norm * (vn - a)
        K = torch.diag_embed(clip(lc)[..., None].expand(lc.shape + (p.neq,)))
        one = torch.ones_like(vn)
        # the differential of pressure and of the normal momentum, as row vectors
        dp = gm1 * torch.cat([ke[..., None], -V, one[..., None]], -1)
        dm = torch.cat([-vn[..., None], n, torch.zeros_like(vn)[..., None]], -1)
        for lam, s in ((lp, 1.0), (lm, -1.0)):
            c = s * a
            r = torch.cat([one[..., None], V + c[..., None] * n, (H + c * vn)[..., None]], -1)
            row = 0.5 * (dp / (a * a)[..., None] + dm / c[..., None])
            K = K + (clip(lam) - clip(lc))[..., None, None] * r[..., :, None] * row[..., None, :]
        return K, torch.maximum(lc.abs(), torch.maximum(lp.abs(), lm.abs()))

    # cells
    def cells_residual(self, u):
        """Cell residuals summed at the nodes, and the nodes' wave speeds."""
        p = self.p
        res, ws = torch.zeros_like(u), torch.zeros_like(self.vol)
        for k in self.cells:
            lda, dis, phi, wave, vol = self._points(k, u[k.conn])
            if p.scheme != "b":
                r = lda + dis  # dis is zero for LDA
            elif self.blend is None:
                r = lda + self._theta(lda, dis, phi)[:, None, None] * dis
            else:
                t = self.blend[k.conn]
                t = torch.where(t.amax(1, keepdim=True) < 1e-6, torch.zeros_like(t), t)
                r = lda + t[..., None] * dis
            self._add(res, k.conn, r)
            self._add(ws, k.conn, (vol * wave)[:, None].expand(k.conn.shape))
        return res, ws

    @staticmethod
    def _theta(lda, dis, phi):
        return phi[:, 0].abs() / ((lda + dis)[..., 0].abs().sum(1) + 1e-6)

    def _points(self, k, un):
        """LDA part, N part, Phi, largest eigenvalue and volume of the cells of states un."""
        p = self.p
        F = self._flux(torch.einsum("fn,cne->cfe", k.Vsf, un))
        lda, dis, phi, wave, vol = torch.zeros_like(un), torch.zeros_like(un), 0.0, None, 0.0
        for q in range(len(k.w)):
            wq, fgrad, grad = k.points[q]
            r = torch.einsum("cfx,cfex->ce", fgrad, F)
            uq = torch.einsum("n,cne->ce", k.V[q], un)
            K, lam = self._split(uq[:, None].expand(un.shape), grad, 1)
            lam = lam.clamp(min=1e-6).amax(1)
            wave = lam if wave is None else torch.maximum(wave, lam)
            S = K.sum(1)
            rhs = [r]
            if p.scheme != "lda":
                d0 = un - un[:, :1]  # the N part acts on differences of the states
                rhs.append((K @ d0[..., None])[..., 0].sum(1))
            rhs = torch.stack(rhs, -1)
            x = torch.linalg.solve(S, rhs) if p.neq > 1 else rhs / S
            lda += wq[:, None, None] * (K @ x[:, None, :, :1])[..., 0]
            if p.scheme != "lda":
                dis += wq[:, None, None] * (K @ (d0 - x[:, None, :, 1])[..., None])[..., 0]
            phi, vol = phi + wq[:, None] * r, vol + wq
        return lda, dis, phi, wave, vol

    # boundary facets
    def facets_residual(self, u, res, ws):
        p, dev = self.p, self.dev
        for b in p.bcs:
            conn = torch.as_tensor(b.sol_conn, device=dev).long()
            X = self.X[torch.as_tensor(b.geo_conn, device=dev).long()]
            fV, dV = torch.as_tensor(b.fV, device=dev), torch.as_tensor(b.fdVgeo, device=dev)
            gq = torch.as_tensor(np.ascontiguousarray(b.gq), device=dev)
            un = u[conn]
            out, total = torch.zeros_like(un), 0.0
            coeff = torch.full_like(un[:, 0, 0], 1e-9)
            for q in range(len(b.fw)):
                t = torch.einsum("dg,fgx->fdx", dV[:, q], X)
                if p.dim == 2:
                    n = torch.stack([t[:, 0, 1], -t[:, 0, 0]], -1)
                else:
                    n = torch.linalg.cross(t[:, 0], t[:, 1])
                jd = torch.linalg.vector_norm(n, dim=-1)
                n = n / jd[:, None]
                uq = torch.einsum("n,fne->fe", fV[q], un)
                K, lam = self._split(uq, n, -1)
                coeff = torch.maximum(coeff, lam)
                if b.kind == "WeakWall":
                    flux = self._through(self._slip(uq, n), n) - self._through(uq, n)
                else:
                    ghost = gq[:, q] if b.kind == "WeakDirichlet" else self._ghost(b, uq)
                    flux = (K @ (ghost - uq)[..., None])[..., 0]
                wq = (jd * float(b.fw[q]))[:, None]
                total = total + wq * flux
                relax = 1.0 / (3.0 * b.order) if b.kind == "WeakWall" and b.order > 1 else 1.0
                out += relax * fV[q][None, :, None] * (wq * flux)[:, None]
            both = out.sum(1)
            scale = torch.where(both.abs() > 1e-14, total / both, torch.ones_like(both))
            self._add(res, conn, out * scale[:, None])
            self._add(ws, conn, self.vol[conn] * coeff[:, None])

    def _through(self, u, n):
        return (self._flux(u) * n[:, None, :]).sum(-1)

    def _slip(self, u, n):
        V, _, _ = self._props(u)
        W = V - (V * n).sum(-1, keepdim=True) * n
        E = u[:, -1] + 0.5 * u[:, 0] * ((W * W).sum(-1) - (V * V).sum(-1))
        return torch.cat([u[:, :1], u[:, :1] * W, E[:, None]], -1)

    def _ghost(self, b, u):
        gamma, d = self.p.gamma, self.p.dim
        g = torch.zeros_like(u)
        if b.kind == "WeakSubInlet":
            V, _, a = self._props(u)
            mach = torch.linalg.vector_norm(V, dim=-1) / a
            f = 1.0 + 0.5 * (gamma - 1.0) * mach * mach
            T, P = b.params[0] / f, b.params[1] / f ** (gamma / (gamma - 1.0))
            g[:, 0] = P / (GAS_R * T)
            g[:, 1] = mach * torch.sqrt(gamma * GAS_R * T) * g[:, 0]
            g[:, -1] = P / (gamma - 1.0) + 0.5 * (g[:, 1:1 + d] ** 2).sum(-1) / g[:, 0]
            return g
        if b.kind == "WeakSubOutlet":
            g[:] = u
            g[:, -1] = b.params[0] / (gamma - 1.0) + 0.5 * (u[:, 1:1 + d] ** 2).sum(-1) / u[:, 0]
            return g
        raise ValueError(b.kind)

    # sweeps
    def assemble(self, u, cfl):
        """Residual (divided by the dual volumes) and time steps."""
        res, ws = self.cells_residual(u)
        self.facets_residual(u, res, ws)
        return res / self.vol[:, None], (cfl * self.vol / ws)[:, None]

    def iterate(self, u, cfl, sweeps):
        norms = []
        for _ in range(sweeps):
            res, dt = self.assemble(u, cfl)
            norms.append(torch.sqrt(((res * dt) ** 2).mean(0)))
            u = u - dt * res
        return u, torch.stack(norms)

    def rk3(self, u, cfl, steps):
        for _ in range(steps):
            r, dt = self.assemble(u, cfl)
            v = u - dt * r
            r = self.assemble(v, cfl)[0]
            w = 0.75 * u + 0.25 * v - 0.25 * dt * r
            r = self.assemble(w, cfl)[0]
            u = u / 3.0 + 2.0 / 3.0 * w - 2.0 / 3.0 * dt * r
        return u

    def lf_blend(self, u):
        """Nodal LF_Blend coefficient of the first equation (one group of triangles)."""
        k, p, g = self.cells[0], self.p, self.p.groups[0]
        uc = u[:, 0][k.conn]
        avg = uc.mean(1, keepdim=True)
        ksi = ((uc - avg).abs() / (uc.abs() + avg.abs() + 1e-12)).amax(1)
        most = torch.zeros_like(self.vol)
        flat = k.conn.reshape(-1)
        most.scatter_reduce_(0, flat, ksi[:, None].expand(k.conn.shape).reshape(-1), "amax")
        theta = 1.0 - most[k.conn].amax(1)
        verts = k.conn[:, :3]
        node = torch.zeros_like(self.vol)
        node.scatter_reduce_(0, verts.reshape(-1), theta[:, None].expand(-1, 3).reshape(-1),
                             "amax")
        # every other node: the linear interpolant of its cell's vertices
        X = p.sol_coords[g.sol_conn[0]]
        lam = np.linalg.solve(np.vstack([X[:3].T, np.ones(3)]), np.vstack([X.T, np.ones(len(X))]))
        interp = torch.as_tensor(np.ascontiguousarray(lam.T), device=self.dev)
        values = node[verts] @ interp.T
        for n in range(3, k.conn.shape[1]):
            node[k.conn[:, n]] = values[:, n]
        return node


def exact(case, seed):
    prob, cfl, u0 = _states(case, seed)
    kind, sweeps = case["kind"], case.get("sweeps", 0)
    if sweeps == 0:
        return None  # thousands of sweeps
    if kind == "batch":
        us, drops = [], []
        for p, c, u in zip(prob, cfl, u0):
            e = _Exact(p)
            u, norms = e.iterate(torch.as_tensor(u, device=e.dev), float(c), sweeps)
            us.append(u.reshape(-1))
            drops.append(norms[-1, 0] / norms[0, 0])
        return dict(u=torch.cat(us).cpu().numpy(), iters=None,
                    drop=torch.stack(drops).cpu().numpy())
    e = _Exact(prob)
    u = torch.as_tensor(u0, device=e.dev)
    got = {}
    if kind == "rk3":
        u = e.rk3(u, cfl, sweeps)
    elif kind == "blend":
        for _ in range(sweeps):
            e.blend = e.lf_blend(u)
            res, dt = e.assemble(u, cfl)
            u = u - dt * res
        got["theta"] = e.blend.cpu().numpy()
    else:
        u, norms = e.iterate(u, cfl, sweeps)
        got["norms"] = norms.cpu().numpy()
    got["u"] = u.cpu().numpy()
    return got
