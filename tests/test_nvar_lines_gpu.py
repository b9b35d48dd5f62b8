"""The line solve at block sizes other than 9, in each of its launch forms
(copy warp with the line in shared memory, copy warp alone, one warp), at the
edges of its chunks: lines of every length around multiples of the chunk.
Against the oracle; tolerance: that of TBS_ALGO_FP64."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu


def check(mesh, jac, n=4):
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    h = s.sweep(n)
    U = s.solution()
    s.close()
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, n, threads=4)
    assert np.all(np.abs(h - r["hist"]) <= 1e-12 * r["hist"][0])
    assert np.linalg.norm(U - r["U"]) <= 1e-12 * np.linalg.norm(r["U"])


@pytest.mark.parametrize("nvar", [2, 3, 5, 8, 10, 13, 16])
@pytest.mark.parametrize("lens", [list(range(1, 14)), [15, 16, 17, 18, 31, 32, 33, 34]])
def test_line_lengths(nvar, lens):
    mesh = ragged_mesh(lens, seed=nvar, nvar=nvar)
    check(mesh, Jacobian.generate(mesh, 10.0, nvar))


# lines per SM and length choose the form: many long lines (one warp), few
# lines too long for shared memory (copy warp alone)
@pytest.mark.parametrize("nvar,L,K", [(4, 900, 130), (7, 900, 40), (16, 4, 1700), (12, 800, 11)])
def test_forms(nvar, L, K):
    mesh = Mesh.structured(L, K, nvar=nvar)
    check(mesh, Jacobian.generate(mesh, 10.0, 3), 2)


def test_failed_check_goes_on():
    """A lagged factorization: the check fails and the sweeps go on from the
    true residual, until the new system's solution is reached (1e-9)."""
    mesh = Mesh.structured(20, 24, nvar=5)
    jac = Jacobian.generate(mesh, 9.0, 5)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    rng = np.random.default_rng(1)
    new = [a * (1.0 + 1e-3 * rng.uniform(-1, 1, a.size)) for a in (jac.jacD, jac.jacO1, jac.jacO2)]
    s.update_values(*new)
    s.solve(1e-11, 200)
    assert s.solve_check()[2] >= 1
    r = oracle.lij(mesh, *new, jac.rhs, 40, threads=4)
    assert np.linalg.norm(s.solution() - r["U"]) <= 1e-9 * np.linalg.norm(r["U"])
    s.close()
