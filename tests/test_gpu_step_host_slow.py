"""Pipelined host-buffer steps whose downloads fall behind: other streams keep the copies to the host
busy, so that steps are computed while the results of earlier ones still wait for their download."""

import numpy as np
import pytest

from pdekit_b200 import reference_element as ref
from pdekit_b200 import workloads


@pytest.mark.gpu
def test_late_downloads_keep_every_step():
    """State and norm of every step, bit for bit those of the same steps one after the other."""
    import torch
    from pdekit_b200.rds import PGRDMethodExplicit

    steps, cfl = 24, 0.3
    p = workloads.tri_problem("burgers", "b", 2, 100, 0.15, 7, workloads.BURGERS_BCS,
                              ref.triag_tables(2, 5))
    x, y = p.sol_coords[:, 0], p.sol_coords[:, 1]

    def pinned(*shape):
        return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()

    ins, outs, norms = pinned(steps, p.nnodes, 1), pinned(steps, p.nnodes, 1), pinned(steps, 1)
    for i in range(steps):
        ins[i, :, 0] = 1.5 - 2.0 * x + (0.05 + 0.01 * i) * np.sin(5.0 * x + 3.0 * y)
    s = PGRDMethodExplicit(p.physics, p.scheme).configure_mesh_data(p)
    s.initialize_work_data()
    want = []
    for i in range(steps):
        s.set_solution(ins[i])
        s.assemble_lhs_and_rhs(cfl)
        s.solve()
        want.append((s.solution().copy(), np.array(s.compute_residual_norm())))
    s.step_host(ins[0], outs[0], cfl, norms[0])  # buffers and streams are there
    s.step_sync()
    busy = [(torch.empty(1 << 24, device="cuda"), torch.empty(1 << 24, pin_memory=True),
             torch.cuda.Stream()) for _ in range(4)]
    torch.cuda.synchronize()
    for _ in range(3):
        for src, dst, stream in busy:
            with torch.cuda.stream(stream):
                dst.copy_(src, non_blocking=True)
    for i in range(steps):
        s.step_host(ins[i], outs[i], cfl, norms[i])
    s.step_sync()
    torch.cuda.synchronize()
    s.close()
    for i, (u, n) in enumerate(want):
        assert np.array_equal(outs[i], u), i
        assert np.array_equal(norms[i], n), i
