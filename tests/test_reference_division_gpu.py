"""TBS_ALGO_REFERENCE at block size 9 forms its quotients from reciprocals
(correctly rounded) and leaves numerators and divisors outside the range
where that holds to the general division.  Bit for bit against the oracle:
zero numerators, blocks scaled far up and down (powers of two), cells that
mix both in one line, line lengths around the copy job of four cells."""
import numpy as np
import pytest

import oracle
from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_REFERENCE, Jacobian, Mesh, Solver, TbsError

pytestmark = pytest.mark.gpu


def check(mesh, jac, n=3):
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_REFERENCE)
    s.sweep(n)
    r = oracle.lij(mesh, jac.jacD, jac.jacO1, jac.jacO2, jac.rhs, n, threads=4)
    np.testing.assert_array_equal(s.solution(), r["U"])
    np.testing.assert_array_equal(s.residual(), r["R"])
    np.testing.assert_array_equal(s.update(), r["dU"])
    s.close()


@pytest.mark.parametrize("lens", [[1, 2, 3, 4, 5, 6, 7, 8, 9, 10], [12, 13, 16, 17, 33]])
def test_line_lengths(lens):
    mesh = ragged_mesh(lens, seed=3)
    check(mesh, Jacobian.generate(mesh, 9.0, 5))


@pytest.mark.parametrize("scale", [2.0 ** -520, 2.0 ** -420, 2.0 ** 430, 2.0 ** 510])
def test_scaled_blocks(scale):
    mesh = Mesh.structured(5, 23)
    jac = Jacobian.generate(mesh, 9.0, 6)
    for a in (jac.jacD, jac.jacO1, jac.jacO2):
        a *= scale
    check(mesh, jac, 1)


def test_zero_and_scaled_rows():
    mesh = Mesh.structured(6, 21)
    jac = Jacobian.generate(mesh, 9.0, 7)
    rng = np.random.default_rng(0)
    rhs = jac.rhs.reshape(-1, 9)
    rhs[rng.random(rhs.shape) < 0.3] = 0.0
    rhs[::5] *= 2.0 ** -450
    rhs[2::5] *= 2.0 ** 420
    check(mesh, jac, 1)


def test_zero_pivot_is_refused():
    mesh = Mesh.structured(3, 12)
    jac = Jacobian.generate(mesh, 9.0, 8)
    jac.jacD.reshape(-1, 81)[int(mesh.lines[0]), 0] = 0.0
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    with pytest.raises(TbsError):
        s.factor(ALGO_REFERENCE)
    s.close()
