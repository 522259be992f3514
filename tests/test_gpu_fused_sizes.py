"""The fused correction sweeps at sizes where their work split changes: one item or several a
thread, more nodes than threads (P2 and P3), cluster and grid form, each rule of the P3 triangles."""

import numpy as np
import pytest

from pdekit_b200 import reference_element as ref
from pdekit_b200 import workloads

CASES = [(physics, scheme, order, rule, n)
         for physics, scheme in (("advconst", "n"), ("advconst", "b"), ("burgers", "lda"),
                                 ("burgers", "b"))
         for order, rule, n in ((1, 4, 33),    # cluster, two items a thread
                                (1, 4, 100),   # grid, one item a thread
                                (2, 5, 61),    # grid, fewer threads than nodes
                                (3, 6, 41), (3, 8, 41),
                                (3, 8, 150))]  # grid, as many items as threads


@pytest.mark.gpu
@pytest.mark.parametrize("physics,scheme,order,rule,n", CASES)
def test_fused_equal_separate_launches(physics, scheme, order, rule, n):
    """Bit for bit: the arithmetic is the same."""
    from pdekit_b200.rds import PGRDMethodExplicit

    bcs = workloads.ADV_BCS if physics == "advconst" else workloads.BURGERS_BCS
    p = workloads.tri_problem(physics, scheme, order, n, 0.15, 7, bcs,
                              ref.triag_tables(order, rule))
    x, y = p.sol_coords[:, 0], p.sol_coords[:, 1]
    u0 = (1.5 - 2.0 * x + 0.1 * np.sin(5.0 * x + 3.0 * y)).reshape(-1, 1)
    out = []
    for fuse in (0, 1 << 16):
        s = PGRDMethodExplicit(physics, scheme, "mixed")
        s.configure_mesh_data(p)
        s.initialize_work_data()
        s.set_option("mixed_refresh", 6)
        s.set_option("mixed_fuse_cells", fuse)
        s.set_solution(u0)
        it, hist = s.iterate(0.3, 19)
        assert it == 19
        out.append((s.solution(), hist))
        s.close()
    assert np.isfinite(out[0][0]).all()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
