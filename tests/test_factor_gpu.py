"""The line factorization's two launch forms (few lines: one CTA per line;
more than two lines per SM: one CTA per three lines) and their edges: line
counts that are no multiple of three, chains of different lengths in one CTA,
lines of one and two cells, pivots outside the reciprocal's usual range, zero
pivots.  Against the oracle; tolerance: that of TBS_ALGO_FP64 (1e-12 of the
initial residual per sweep, 1e-12 relative in U), which does not depend on
the scale of the system."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver, TbsError

pytestmark = pytest.mark.gpu

MESHES = {
    "few_ragged": lambda: ragged_mesh([1, 2, 3, 9, 17, 30, 2, 1], seed=5),
    "many": lambda: Mesh.structured(301, 10),
    "many_ragged": lambda: ragged_mesh([1 + (7 * k) % 13 for k in range(302)], seed=6),
    "most": lambda: Mesh.structured(890, 5),
}


def check(mesh, jac, n=5):
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


@pytest.mark.parametrize("name", list(MESHES))
def test_forms(name):
    mesh = MESHES[name]()
    check(mesh, Jacobian.generate(mesh, 9.0, 4))


@pytest.mark.parametrize("name", ["few_ragged", "many"])
@pytest.mark.parametrize("scale", [2.0 ** -1010, 2.0 ** 1005])
def test_extreme_pivots(name, scale):
    """Blocks scaled by a power of two (exact): pivots beyond 2^-1000 and
    2^1000, whose reciprocals the general pass computes.  U scales by 1/scale,
    so rhs is scaled too and the solution stays of order one."""
    mesh = MESHES[name]()
    jac = Jacobian.generate(mesh, 9.0, 4)
    for a in (jac.jacD, jac.jacO1, jac.jacO2, jac.rhs):
        a *= scale
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    s.sweep(1)
    U = s.solution()
    s.close()
    for a in (jac.jacD, jac.jacO1, jac.jacO2, jac.rhs):
        a /= scale
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, 1)
    assert np.linalg.norm(U - r["U"]) <= 1e-12 * np.linalg.norm(r["U"])


@pytest.mark.parametrize("name", ["few_ragged", "many"])
def test_zero_pivot_is_refused(name):
    mesh = MESHES[name]()
    jac = Jacobian.generate(mesh, 9.0, 4)
    # the first cell of a line with a top chain (longer than 4 cells): its first pivot is its first diagonal entry
    e = int(mesh.lines[mesh.linepoint[int(np.argmax(mesh.linesize))]])
    jac.jacD.reshape(-1, 81)[e, 0] = 0.0
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    with pytest.raises(TbsError):
        s.factor(ALGO_FP64)
    s.close()
