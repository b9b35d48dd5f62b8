"""The reference order at block size 9 with more lines than the two-warp
kernels are for: the one-warp kernels, and shapes on both sides of the rule.
Bit for bit against the oracle, zero numerators and a scaled system among
them."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_REFERENCE, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu

MESHES = {
    "cells": lambda: Mesh.structured(1500, 1),
    "590x3": lambda: Mesh.structured(590, 3),
    "700x3": lambda: Mesh.structured(700, 3),
    "1300x8": lambda: Mesh.structured(1300, 8),
    "2500x16": lambda: Mesh.structured(2500, 16),
    "ragged": lambda: ragged_mesh([1 + (5 * k) % 11 for k in range(1900)], seed=2),
    "one long": lambda: ragged_mesh([300] + [2] * 1400, seed=3),
}


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -420])
def test_equals_the_oracle(name, scale):
    mesh = MESHES[name]()
    jac = Jacobian.generate(mesh, 9.0, 6)
    rhs = jac.rhs.reshape(-1, 9)
    rhs[np.random.default_rng(0).random(rhs.shape) < 0.2] = 0.0
    for a in (jac.jacD, jac.jacO1, jac.jacO2):
        a *= scale
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_REFERENCE)
    s.sweep(2)
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, 2, threads=4)
    np.testing.assert_array_equal(s.solution(), r["U"])
    np.testing.assert_array_equal(s.residual(), r["R"])
    np.testing.assert_array_equal(s.update(), r["dU"])
    s.close()
