"""The line solve at the edges of its chunks, against the oracle.

Lines of every length around multiples of the copy chunk (8 cells a chain,
two chains a line) and of the write-back group (4 cells), in one ragged mesh:
chains that end inside a chunk, chains of different chunk counts, lines
shorter than a group.  Tolerance: that of TBS_ALGO_FP64 (1e-12 of the initial
residual per sweep, 1e-12 relative in U)."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_FP64, Jacobian, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [list(range(1, 20)), list(range(28, 41)), [63, 64, 65, 66, 3, 127, 128, 129, 130]])
def test_line_lengths(lens):
    mesh = ragged_mesh(lens, seed=len(lens))
    jac = Jacobian.generate(mesh, 9.0, 3)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    h = s.sweep(6)
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, 6)
    assert np.all(np.abs(h - r["hist"]) <= 1e-12 * r["hist"][0])
    assert np.linalg.norm(s.solution() - r["U"]) <= 1e-12 * np.linalg.norm(r["U"])
    s.close()
