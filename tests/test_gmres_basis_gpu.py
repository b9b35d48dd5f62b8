"""GMRES with a basis of many vectors: the fused orthogonalization over one
and several chunks of eight vectors and at the largest restart, against the
oracle.  Tolerance as for GMRES elsewhere: the same steps, every history
entry within 1e-9 ||rhs||, the solution within 1e-9."""
import numpy as np
import pytest

import oracle
from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart,iters", [(1, 6), (8, 16), (9, 18), (17, 17), (64, 24)])
@pytest.mark.parametrize("L,K", [(9, 14), (40, 33)])
def test_basis_sizes(restart, iters, L, K):
    mesh = Mesh.structured(L, K)
    jac = Jacobian.generate(mesh, 3.0, 3)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    n, h = s.gmres(1e-10, restart, 1, iters)
    U = s.solution()
    s.close()
    r = oracle.gmres(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, restart, 1, 1e-10, iters)
    assert n == r["iters"]
    r0 = r["hist"][0]
    assert np.all(np.abs(h - np.asarray(r["hist"])[: n + 1]) <= 1e-9 * r0)
    assert np.linalg.norm(U - r["U"]) <= 1e-9 * np.linalg.norm(r["U"])
