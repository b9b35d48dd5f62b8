"""The line factorization of short lines, one warp a line: lines of one cell,
of every length up to a dozen, a longest line on both sides of the rule, zero
pivots, and the reciprocals bit for bit.  Against the oracle; tolerance: that
of TBS_ALGO_FP64."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from test_reciprocal_gpu import divisors, first_update, system
from triblocksolve_b200 import ALGO_FP64, ALGO_MIXED, Jacobian, Mesh, Solver, TbsError

pytestmark = pytest.mark.gpu

MESHES = {
    "one cell": lambda: Mesh.structured(1, 1),
    "cells": lambda: Mesh.structured(700, 1),
    "2x3": lambda: Mesh.structured(2, 3),
    "40x6": lambda: Mesh.structured(40, 6),
    "40x7": lambda: Mesh.structured(40, 7),
    "2500x8": lambda: Mesh.structured(2500, 8),
    "ragged": lambda: ragged_mesh([1 + (5 * k) % 12 for k in range(1600)], seed=2),
    "30 among 3": lambda: ragged_mesh([30] + [3] * 4000, seed=4),
    "90 among 3": lambda: ragged_mesh([90] + [3] * 4000, seed=5),
}


@pytest.mark.parametrize("name", list(MESHES))
def test_equals_the_oracle(name):
    mesh = MESHES[name]()
    jac = Jacobian.generate(mesh, 9.0, 4)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    h = s.sweep(4)
    U = s.solution()
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, 4, threads=4)
    assert np.all(np.abs(h - r["hist"]) <= 1e-12 * r["hist"][0])
    assert np.linalg.norm(U - r["U"]) <= 1e-12 * np.linalg.norm(r["U"])
    s.factor(ALGO_MIXED)
    n, h = s.solve(1e-10, 60)
    assert h[-1] <= 1e-10 * h[0]
    s.close()


def test_reciprocals():
    mesh = Mesh.structured(900, 5)
    rng = np.random.default_rng(1)
    d = divisors(9 * mesh.nelem, -1020, 1020, [-1001, -1000, -999, 999, 1000, 1001], rng)
    rhs = rng.choice([-1.0, 1.0], d.size)
    got = first_update(mesh, system(mesh, d, rhs), ALGO_FP64)
    np.testing.assert_array_equal(got, -rhs * (1.0 / d))


@pytest.mark.parametrize("cell", [0, 2, 4])
def test_zero_pivot_is_refused(cell):
    mesh = Mesh.structured(30, 5)
    jac = Jacobian.generate(mesh, 9.0, 4)
    # the twist cell's pivot is its own block less the chains' parts: all of it is cleared
    e = int(mesh.lines[mesh.linepoint[7] + cell])
    jac.jacD.reshape(-1, 81)[e] = 0.0
    jac.jacO1[:] = 0.0
    jac.jacO2[:] = 0.0
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    with pytest.raises(TbsError):
        s.factor(ALGO_FP64)
    s.close()
