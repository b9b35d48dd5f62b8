"""Solves whose sweeps run as one cooperative launch (few lines) against the
same solves with a launch per kernel (profiling), bit for bit: iterates,
history, checks.  At the edges: one tile, lines of one cell, as many lines as
there are CTAs, uneven lines, more tiles than two a CTA, a sweep limit, a
failed check that sends the loop round again, and the oracle."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu

MESHES = {
    "tile": lambda: Mesh.structured(2, 3),
    "cells": lambda: Mesh.structured(40, 1),
    "ragged": lambda: ragged_mesh([5, 1, 7, 3, 3, 8, 13, 2, 9, 40, 17, 33], seed=4),
    "60x64": lambda: Mesh.structured(60, 64),
    "296x9": lambda: Mesh.structured(296, 9),
    "297x9": lambda: Mesh.structured(297, 9),
    "130x150": lambda: Mesh.structured(130, 150),
    "long": lambda: Mesh.structured(3, 700),
}


def setup(mesh, jac):
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    return s


def both(s, tol, limit):
    n, h = s.solve(tol, limit)
    a = n, h, s.solution(), s.update(), s.solve_check()
    s.profile(True)
    n, h = s.solve(tol, limit)
    s.profile(False)
    b = n, h, s.solution(), s.update(), s.solve_check()
    return a, b


@pytest.mark.parametrize("name", list(MESHES))
def test_equals_a_launch_per_kernel(name):
    mesh = MESHES[name]()
    jac = Jacobian.generate(mesh, 9.0, 2)
    s = setup(mesh, jac)
    for tol, limit in ((1e-10, 100), (1e-30, 4), (1e-10, 1), (1e-3, 100)):
        a, b = both(s, tol, limit)
        assert a[0] == b[0]
        for x, y in zip(a[1:4], b[1:4]):
            np.testing.assert_array_equal(x, y)
        assert a[4] == b[4]
    n, h = s.solve(1e-10, 100)
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, n, threads=4)
    assert np.all(np.abs(h - r["hist"]) <= 1e-12 * r["hist"][0])
    assert np.linalg.norm(s.solution() - r["U"]) <= 1e-12 * np.linalg.norm(r["U"])
    s.close()


def test_failed_check_goes_on():
    """New block values on an old factorization: the recursive residual passes,
    the true one does not, and the sweeps go on from it."""
    mesh = Mesh.structured(50, 40)
    jac = Jacobian.generate(mesh, 9.0, 5)
    s = setup(mesh, jac)
    rng = np.random.default_rng(1)
    s.update_values(*[a * (1.0 + 1e-3 * rng.uniform(-1, 1, a.size)) for a in (jac.jacD, jac.jacO1, jac.jacO2)])
    a, b = both(s, 1e-9, 200)
    assert a[4][2] >= 1  # the loop went round again
    assert a[0] == b[0]
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[2], b[2])
    assert a[4] == b[4]
    s.close()


def test_several_systems_and_right_hand_sides():
    """Contexts that take turns, each with its own meeting words, and a new
    right-hand side between solves."""
    solvers = []
    for k, m in enumerate((Mesh.structured(20, 30), Mesh.structured(60, 16))):
        j = Jacobian.generate(m, 9.0, 7 + k)
        solvers.append((setup(m, j), m, j))
    rng = np.random.default_rng(2)
    for _ in range(3):
        for s, m, j in solvers:
            rhs = rng.uniform(-1, 1, j.rhs.size)
            s.set_rhs(rhs)
            n, h = s.solve(1e-9, 50)
            r = oracle.lij(m, j.jacD, j.jacO1, j.jacO2, rhs, n)
            assert np.all(np.abs(h - r["hist"]) <= 1e-12 * r["hist"][0])
            assert np.linalg.norm(s.solution() - r["U"]) <= 1e-12 * np.linalg.norm(r["U"])
    for s, _, _ in solvers:
        s.close()
