"""The Euler cells and conditions in supersonic flow, where the branches of the upwind matrices are
others than at the Mach numbers of the bump cases (lambda_- positive in some directions, negative in
others), with the conditions such a flow has: supersonic inlet, farfield, symmetry.

Tolerance 1e-12 of the largest magnitude of a field, as for the subsonic states: a residual is a sum
of some tens of terms of the size of the flux, each rounded to 1.1e-16."""

import numpy as np
import pytest

from oracle.rds_oracle import Oracle
from pdekit_b200 import meshgen, workloads
from pdekit_b200 import reference_element as ref

RULES = {1: 4, 2: 5, 3: 8}


def _problem(shape, order, scheme, mach):
    dim = 3 if shape == "tetra" else 2
    if dim == 3:
        mesh = meshgen.box_tet(4, 3, 2, jitter=0.1, seed=2)
        tables = {"tetra": ref.tet_tables(order, {1: 2, 2: 5}[order])}
        walls = ("bottom_wall", "side_walls", "top_wall")
    else:
        mesh = meshgen.channel_2d(7 if shape == "triag" else 0, 7 if shape == "quad" else 0, 3,
                                  jitter=0.1, seed=2)
        tables = {"triag": ref.triag_tables(order, RULES[order]),
                  "quad": ref.quad_tables(order, RULES[order], tensor=True)}
        walls = ("bottom_wall", "top_wall")
    free = np.zeros(dim + 2)
    free[0], free[1] = 1.2, 1.2 * mach * np.sqrt(1.4 * 1e5 / 1.2)
    free[-1] = 1e5 / 0.4 + 0.5 * free[1] ** 2 / free[0]
    bcs = [("WeakSymmetry", f"{w}_bc", w) for w in walls]
    bcs += [("WeakSuperInlet", "inlet_bc", "inlet"), ("WeakFarfield", "outlet_bc", "outlet", free)]
    p = workloads.mesh_problem(mesh, f"euler{dim}d", scheme, order, tables, bcs)
    return p, workloads.bump_state(p.sol_coords, dim, mach)


@pytest.mark.gpu
@pytest.mark.parametrize("mach", [1.2, 3.0])
@pytest.mark.parametrize("scheme", ["lda", "n", "b"])
@pytest.mark.parametrize("shape,order", [("triag", 1), ("triag", 2), ("triag", 3), ("quad", 1),
                                         ("quad", 2), ("quad", 3), ("tetra", 1), ("tetra", 2)])
def test_first_residual(shape, order, scheme, mach):
    from pdekit_b200.rds import PGRDMethodExplicit

    p, u0 = _problem(shape, order, scheme, mach)
    want = Oracle(p).assemble(u0, 0.3)
    s = PGRDMethodExplicit(p.physics, scheme)
    s.configure_mesh_data(p)
    s.initialize_work_data()
    s.set_solution(u0)
    s.assemble_lhs_and_rhs(0.3)
    res, dt, ws, _ = s.fields()
    s.close()
    for e in ((0,), tuple(range(1, p.dim + 1)), (p.dim + 1,)):
        assert np.abs(res - want[0])[:, e].max() <= 1e-12 * np.abs(want[0][:, e]).max()
    for got, w in ((ws, want[1]), (dt, want[2])):
        assert np.abs(got - w).max() <= 1e-12 * np.abs(w).max()
