"""The device loop's stop flag with one chunk of nodes a block, one block for several chunks and
several equations: the launches after the one that sets it do nothing, and the next call starts
from a clean count."""

import numpy as np
import pytest

from pdekit_b200 import meshgen, workloads
from pdekit_b200 import reference_element as ref


def _scalar(n):
    p = workloads.tri_problem("burgers", "n", 2, n, 0.1, 7, workloads.BURGERS_BCS,
                              ref.triag_tables(2, 5))
    x, y = p.sol_coords[:, 0], p.sol_coords[:, 1]
    return p, (1.5 - 2.0 * x + 0.1 * np.sin(5.0 * x + 3.0 * y)).reshape(-1, 1)


def _euler():
    mesh = meshgen.channel_2d(9, 6, 3, jitter=0.1, seed=2)
    tables = {"triag": ref.triag_tables(1, 4), "quad": ref.quad_tables(1, 4, tensor=True)}
    p = workloads.mesh_problem(mesh, "euler2d", "n", 1, tables, workloads.euler_bcs(2))
    return p, workloads.bump_state(p.sol_coords, 2, 0.5)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda: _scalar(7),    # 225 nodes: one chunk
                                  lambda: _scalar(400),  # 2,507 chunks on 1,184 resident blocks
                                  _euler], ids=["one", "several", "euler"])
def test_loops_stop_and_start_again(make):
    """7 sweeps in one call, then 5: the states and the histories of 12 in one (bit for bit), and
    the norm of the last sweep's residual is the last of the history."""
    from pdekit_b200.rds import PGRDMethodExplicit

    p, u0 = make()
    s = PGRDMethodExplicit(p.physics, p.scheme)
    s.configure_mesh_data(p)
    s.initialize_work_data()
    s.set_solution(u0)
    it, want = s.iterate(0.3, 12)
    u = s.solution().copy()
    assert it == 12
    s.set_solution(u0)
    parts = []
    for sweeps in (7, 5):
        it, hist = s.iterate(0.3, sweeps)
        assert it == sweeps
        parts.append(np.array(hist))
        assert np.array_equal(s.compute_residual_norm(), parts[-1][-1])
    assert np.array_equal(np.concatenate(parts), want)
    assert np.array_equal(s.solution(), u)
    s.close()
