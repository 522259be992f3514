"""The Euler cell kernels where their work split can go wrong: warps that walk units of 4 or 8 cells
(fewer cells than one unit, a ragged last unit, more units than the grid has warps), rounds of the
lanes over points and nodes with idle lanes, every element type, scheme and Jacobian form; and the
branch-free reciprocals they use.

Tolerance 1e-12 of the largest magnitude of a field: a residual is a sum of some tens of terms of
the size of the flux, a hundred times that of the residual of a state perturbed by a per cent, each
rounded to 1.1e-16."""

import os
import subprocess

import numpy as np
import pytest

from oracle.rds_oracle import Oracle
from pdekit_b200 import meshgen, workloads
from pdekit_b200 import reference_element as ref

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RULES = {1: 4, 2: 5, 3: 8}


def _problem(shape, order, scheme, size, jitter):
    if shape == "tetra":
        nx, ny, nz = size
        mesh = meshgen.box_tet(nx, ny, nz, jitter=jitter, seed=2)
        tables = {"tetra": ref.tet_tables(order, {1: 2, 2: 5}[order])}
        dim = 3
    else:
        nx, ny = size
        tri, quad = (nx, 0) if shape == "triag" else (0, nx)
        bump = 0.0 if jitter == 0.0 else 0.1  # without: a channel of equal parallelograms
        mesh = meshgen.channel_2d(tri, quad, ny, jitter=jitter, seed=2, bump_h=bump)
        tables = {"triag": ref.triag_tables(order, RULES[order]),
                  "quad": ref.quad_tables(order, RULES[order], tensor=True)}
        dim = 2
    p = workloads.mesh_problem(mesh, f"euler{dim}d", scheme, order, tables,
                               workloads.euler_bcs(dim))
    return p, workloads.bump_state(p.sol_coords, dim, 0.5)


CASES = [(shape, order, scheme, size, jitter)
         for scheme in ("lda", "n", "b")
         for shape, order, size, jitter in (
             ("triag", 1, (3, 1), 0.1),     # 6 cells of a unit's 8
             ("triag", 1, (160, 61), 0.1),  # 19,520 cells: 2,440 units, 2,368 warps
             ("triag", 2, (3, 3), 0.1),     # 18 cells: a last unit of 2
             ("triag", 3, (5, 1), 0.1),
             ("quad", 1, (3, 3), 0.1),
             ("quad", 2, (5, 3), 0.1),
             ("quad", 3, (3, 3), 0.1),      # units of 4
             ("quad", 3, (3, 3), 0.0),      # constant Jacobian
             ("quad", 2, (4, 2), 0.0),
             ("tetra", 1, (3, 1, 1), 0.1),
             ("tetra", 2, (3, 2, 1), 0.1))]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,order,scheme,size,jitter", CASES)
def test_first_residual(shape, order, scheme, size, jitter):
    from pdekit_b200.rds import PGRDMethodExplicit

    p, u0 = _problem(shape, order, scheme, size, jitter)
    want = Oracle(p).assemble(u0, 0.5)
    s = PGRDMethodExplicit(p.physics, scheme)
    s.configure_mesh_data(p)
    s.initialize_work_data()
    s.set_solution(u0)
    s.assemble_lhs_and_rhs(0.5)
    res, dt, ws, _ = s.fields()
    s.close()
    # mass, momentum (one scale for its components, which share the pressure) and energy
    for e in ((0,), tuple(range(1, p.dim + 1)), (p.dim + 1,)):
        assert np.abs(res - want[0])[:, e].max() <= 1e-12 * np.abs(want[0][:, e]).max()
    for got, w in ((ws, want[1]), (dt, want[2])):
        assert np.abs(got - w).max() <= 1e-12 * np.abs(w).max()


@pytest.mark.gpu
def test_reciprocals(tmp_path):
    """At most 1 unit in the last place from the correctly rounded 1 / x (one rounding of the last
    operation, the others act on the correction), 2 from the library's rsqrt (off by one itself)."""
    exe = tmp_path / "math_test"
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-I" + os.path.join(ROOT, "pdekit_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "math_test.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    a, b, c = map(int, out.split())
    assert a <= 1 and b <= 1 and c <= 2
