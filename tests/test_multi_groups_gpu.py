"""The multi-RHS residual's thread groups and final sums.

A thread works on three right-hand sides, so the group that is not full repeats
its last one (1..8 right-hand sides, and fewer as rows retire); a cell has 0 to
4 cross-line blocks; the norm adds the tiles' sums 480 at a time and the rest
160 at a time (8, 60 and 750 tiles).  Every row is the single solve's, bit for
bit: each row's operations and their order are those of that solve.
"""
import numpy as np
import pytest

from meshes import point_mesh, ragged_mesh
from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu

MESHES = {
    "tiles-750": lambda: Mesh.structured(60, 200),
    "tiles-60": lambda: Mesh.structured(24, 40),
    "points": lambda: point_mesh(Mesh.structured(11, 13)),
    "ragged": lambda: ragged_mesh([5, 1, 7, 3, 3, 8, 13, 2, 9, 40], seed=4),
}


@pytest.mark.parametrize("nrhs", [1, 2, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("name", list(MESHES))
def test_rows(name, nrhs):
    mesh = MESHES[name]()
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(Jacobian.generate(mesh, 6.0, 7))
    s.factor(ALGO_FP64)
    try:
        rng = np.random.default_rng(nrhs)
        rhs = rng.uniform(-1, 1, (nrhs, 9 * mesh.nelem))
        # a row already smooth under the sweeps retires later than the others
        s.set_rhs(rhs[0])
        s.sweep(3)
        rhs[nrhs // 2] = s.residual()
        U, sweeps, hist = s.solve_multi(rhs, 1e-11, 60)
        for r in range(nrhs):
            s.set_rhs(rhs[r])
            n, h = s.solve(1e-11, 60)
            assert sweeps[r] == n
            np.testing.assert_array_equal(hist[r], h)
            np.testing.assert_array_equal(U[r], s.solution())
    finally:
        s.close()
