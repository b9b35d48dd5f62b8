"""Roundings of the FP64 line solve.  A step's dot product is three partial
sums, so at most ceil(nvar / 3) + 1 roundings, of half an ulp each, stand
between a product and the result.  With unit diagonal blocks and in-line
blocks whose entries lie just under half an ulp of the vector, each of those
roundings loses what it can: a sum in one or two chains exceeds the bound."""
import numpy as np
import pytest

from triblocksolve_b200 import ALGO_FP64, Batch, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -52
G = 0.49 * ULP


def system(L, K, nvar):
    mesh = Mesh.structured(L, K, nvar=nvar)
    jac = Jacobian.generate(mesh, 9.0, 1)
    nb = nvar * nvar
    for a in (jac.jacD, jac.jacO1, jac.jacO2):
        a[:] = 0.0
    jac.jacD.reshape(-1, nb)[:, :: nvar + 1] = 1.0
    inline = mesh.lineface[mesh.lineface >= 0]
    jac.jacO1.reshape(-1, nb)[inline] = -G
    jac.jacO2.reshape(-1, nb)[inline] = -G
    jac.rhs[:] = -1.0
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    # x = 1 + G nvar (neighbours on the line), to first order in G
    faces = np.zeros(mesh.nelem)
    for e in mesh.fc.reshape(-1, 2)[inline]:
        faces[e] += 1
    return s, (nvar * G * faces / ULP).repeat(nvar)


def check(U, want_ulps, nvar):
    err = np.abs((U - 1.0) / ULP - want_ulps)
    bound = 2 * 0.5 * (-(-nvar // 3) + 1)  # a forward and a backward step
    assert err.max() <= bound, (err.max(), bound)


@pytest.mark.parametrize("nvar", [2, 4, 5, 9, 12, 16])
@pytest.mark.parametrize("L, K", [(3, 40), (300, 37)])
def test_sweep(nvar, L, K):
    s, want = system(L, K, nvar)
    s.sweep(1)
    check(s.solution(), want, nvar)
    s.close()


def test_solve_batch_and_multi():
    s, want = system(20, 45, 9)
    s.solve(1e-30, 1)
    check(s.solution(), want, 9)
    U, _, _ = s.solve_multi(np.full((3, want.size), -1.0), 1e-30, 1)
    for u in np.asarray(U).reshape(3, -1):
        check(u, want, 9)
    t, want_t = system(7, 60, 9)
    Batch([s, t]).solve(1e-30, 1)
    check(s.solution(), want, 9)
    check(t.solution(), want_t, 9)
    s.close()
    t.close()
