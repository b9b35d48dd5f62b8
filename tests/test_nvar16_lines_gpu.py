"""Block size 16 with more lines than have room for their vectors in shared
memory: chunks of four cells and a copy warp.  Lines of every length around
multiples of the chunk, against the oracle; tolerance: that of
TBS_ALGO_FP64."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_FP64, Jacobian, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [list(range(1, 14)) * 58, [15, 16, 17, 18, 19, 20, 31, 32, 33, 34] * 46])
def test_line_lengths(lens):
    mesh = ragged_mesh(lens, seed=len(lens), nvar=16)
    jac = Jacobian.generate(mesh, 10.0, 3)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    h = s.sweep(3)
    U = s.solution()
    s.close()
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, 3, threads=4)
    assert np.all(np.abs(h - r["hist"]) <= 1e-12 * r["hist"][0])
    assert np.linalg.norm(U - r["U"]) <= 1e-12 * np.linalg.norm(r["U"])
