"""Rounding errors of the scalar cells' residual, against the same sums in 80-bit arithmetic: they
grow by a tenth when the larger of two products is rounded before a fused operation adds them."""

import numpy as np
import pytest

from pdekit_b200 import reference_element as ref
from pdekit_b200 import workloads

LONG = np.longdouble


def _residual(p, u):
    """LDA residual over the dual volume of the nodes off the boundary, Burgers on triangles."""
    g = p.groups[0]
    X, un = p.geo_coords.astype(LONG)[g.geo_conn], u[:, 0].astype(LONG)[g.sol_conn]
    jac = np.einsum("dg,cgx->cdx", g.dVgeo[:, 0].astype(LONG), X)
    det = jac[:, 0, 0] * jac[:, 1, 1] - jac[:, 0, 1] * jac[:, 1, 0]
    inv = np.stack([jac[:, 1, 1], -jac[:, 0, 1], -jac[:, 1, 0], jac[:, 0, 0]], 1) / det[:, None]
    inv = inv.reshape(-1, 2, 2)  # [cell, x, xi]
    s = un @ g.Vsf.astype(LONG).T
    lda, vol = np.zeros_like(un), np.zeros_like(det)
    for q in range(len(g.w)):
        fgrad = np.einsum("cxd,df->cfx", inv, g.dVf[:, q].astype(LONG))
        grad = np.einsum("cxd,dn->cnx", inv, g.dV[:, q].astype(LONG))
        r = (fgrad[..., 0] * s * s / 2 + fgrad[..., 1] * s).sum(1)
        kp = np.maximum((un @ g.V[q].astype(LONG))[:, None] * grad[..., 0] + grad[..., 1], 0)
        wj = LONG(g.w[q]) * det
        lda += (wj * r / kp.sum(1))[:, None] * kp
        vol += wj
    res, V = np.zeros(p.nnodes, LONG), np.zeros(p.nnodes, LONG)
    np.add.at(res, g.sol_conn, lda)
    np.add.at(V, g.sol_conn, np.broadcast_to(vol[:, None], un.shape))
    return res / V


@pytest.mark.gpu
def test_burgers_p1_lda_rounding():
    """Mean over six states of the root mean square error, in units of the largest residual:
    6.1e-16 with the smaller product rounded, 6.7e-16 with the larger one."""
    from pdekit_b200.rds import PGRDMethodExplicit

    errors = []
    for seed in range(6):
        p = workloads.tri_problem("burgers", "lda", 1, 40, 0.15, 7 + seed, workloads.BURGERS_BCS,
                                  ref.triag_tables(1, 4))
        rng = np.random.default_rng(seed)
        x, y = p.sol_coords[:, 0], p.sol_coords[:, 1]
        a, b, c = rng.uniform(2, 8), rng.uniform(2, 8), rng.uniform(0, 6)
        u = (1.5 - 2.0 * x + 0.1 * np.sin(a * x + b * y + c) * y).reshape(-1, 1)
        s = PGRDMethodExplicit(p.physics, p.scheme)
        s.configure_mesh_data(p)
        s.initialize_work_data()
        s.set_solution(u)
        s.assemble_lhs_and_rhs(0.3)
        got = s.fields()[0][:, 0]
        s.close()
        inner = np.ones(p.nnodes, bool)
        for bc in p.bcs:
            inner[bc.sol_conn] = False
        want = _residual(p, u)[inner]
        errors.append(float(np.sqrt(np.mean((got[inner] - want) ** 2)) / np.abs(want).max()))
    assert np.mean(errors) <= 6.4e-16
