"""Weak conditions that do not fit one launch (more than eight of one facet type), conditions of a
single facet and of a ragged last block, and more parallel branches than there are side streams."""

import dataclasses

import numpy as np
import pytest

from oracle.rds_oracle import Oracle
from pdekit_b200 import meshgen, workloads
from pdekit_b200 import reference_element as ref

RULES = {1: 4, 2: 5, 3: 8}


def _split(p, pieces):
    """The problem with its condition of most facets cut into `pieces` consecutive ones: 1, 2, 3, ...
    facets, the rest in the last. Every node sums the same facets in the same order."""
    k = max(range(len(p.bcs)), key=lambda i: p.bcs[i].nfacets)
    b, parts, at = p.bcs[k], [], 0
    for i in range(pieces):
        n = i + 1 if i + 1 < pieces else b.nfacets - at
        assert n > 0
        s = slice(at, at + n)
        gq = b.gq[s] if b.kind == "WeakDirichlet" else b.gq
        parts.append(dataclasses.replace(b, name=f"{b.name}_{i:02d}", sol_conn=b.sol_conn[s],
                                         geo_conn=b.geo_conn[s], gq=gq))
        at += n
    return dataclasses.replace(p, bcs=p.bcs[:k] + parts + p.bcs[k + 1:])


def _problem(physics):
    if physics == "euler2d":
        mesh = meshgen.channel_2d(60, 0, 7, jitter=0.1, seed=2)
        p = workloads.mesh_problem(mesh, physics, "n", 2, {"triag": ref.triag_tables(2, 5)},
                                   workloads.euler_bcs(2))
        return p, workloads.bump_state(p.sol_coords, 2, 0.5)
    if physics == "euler3d":
        mesh = meshgen.box_tet(12, 3, 3, jitter=0.1, seed=2)
        p = workloads.mesh_problem(mesh, physics, "lda", 1, {"tetra": ref.tet_tables(1, 2)},
                                   workloads.euler_bcs(3))
        return p, workloads.bump_state(p.sol_coords, 3, 0.5)
    return _scalar(physics, "b", 2, 60, 7)


def _scalar(physics, scheme, order, n, seed):
    bcs = workloads.ADV_BCS if physics == "advconst" else workloads.BURGERS_BCS
    p = workloads.tri_problem(physics, scheme, order, n, 0.15, seed, bcs,
                              ref.triag_tables(order, RULES[order]))
    x, y = p.sol_coords[:, 0], p.sol_coords[:, 1]
    return p, (1.5 - 2.0 * x + 0.1 * np.sin(5.0 * x + 3.0 * y)).reshape(-1, 1)


def _run(p, u0, sweeps):
    from pdekit_b200.rds import PGRDMethodExplicit

    s = PGRDMethodExplicit(p.physics, p.scheme)
    s.configure_mesh_data(p)
    s.initialize_work_data()
    s.set_solution(u0)
    s.assemble_lhs_and_rhs(0.3)
    fields = [f.copy() for f in s.fields()]
    s.set_solution(u0)
    s.iterate(0.3, sweeps)
    u = s.solution().copy()
    s.close()
    return fields, u


@pytest.mark.gpu
@pytest.mark.parametrize("pieces", [8, 9, 10])
@pytest.mark.parametrize("physics", ["advconst", "burgers", "euler2d", "euler3d"])
def test_many_conditions_of_one_facet_type(physics, pieces):
    """Bit for bit the unsplit problem, and the oracle's residual to 1e-12 of its size."""
    p, u0 = _problem(physics)
    q = _split(p, pieces)
    assert len(q.bcs) == len(p.bcs) + pieces - 1
    (f0, v0), (f1, v1) = _run(p, u0, 9), _run(q, u0, 9)
    for a, b in zip(f0, f1):
        assert np.array_equal(a, b)
    assert np.array_equal(v0, v1)
    res, ws, dt = Oracle(q).assemble(u0, 0.3)[:3]
    momentum = tuple(range(1, p.neq - 1))  # one scale for its components, which share the pressure
    for e in ((0,), momentum, (p.neq - 1,)) if p.neq > 1 else ((0,),):
        assert np.abs(f1[0] - res)[:, e].max() <= 1e-12 * np.abs(res[:, e]).max()
    for got, w in ((f1[1], dt), (f1[2], ws)):
        assert np.abs(got - w).max() <= 1e-12 * np.abs(w).max()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_more_branches_than_side_streams(precision):
    """A batch of 18 cell groups and 6 facet types (23 branches, 12 side streams), some conditions
    in two launches: bit for bit the separate problems."""
    from pdekit_b200.batch import BatchedRDS
    from pdekit_b200.rds import PGRDMethodExplicit

    probs, states = [], []
    for physics in ("advconst", "burgers"):
        for scheme in ("lda", "n", "b"):
            for order in (1, 2, 3):
                p, u0 = _scalar(physics, scheme, order, 24 + 3 * order, 7 + len(probs))
                probs.append(_split(p, 6) if scheme == "n" else p)
                states.append(u0)
    cfls = [0.3] * len(probs)
    b = BatchedRDS(probs, cfls, precision)
    assert len(b.merged.groups) == 18
    b.set_solutions(states)
    b.iterate(49, drop=0.0)
    got = b.solutions()
    b.close()
    for p, u0, u in zip(probs, states, got):
        s = PGRDMethodExplicit(p.physics, p.scheme, precision).configure_mesh_data(p)
        s.initialize_work_data()
        s.set_solution(u0)
        s.iterate(0.3, 49)
        assert np.array_equal(s.solution(), u)
        s.close()
