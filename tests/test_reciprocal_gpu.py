"""The factorizations' reciprocals and the reference order's quotients, which
are formed by Newton's iteration and Markstein's last step, against IEEE
division, bit for bit.  The systems are block diagonal, so that a sweep
returns them alone: with J = diag(d) the FP64 update is -(1/d) rhs, the
reference-order update (-rhs)/d, and a block with the entry (1, 0) set has
1/d_0 as a factor of its LU.  Divisors: significands at random, all ones (the
exception of Markstein's theorem) and next to a power of two, exponents over
the whole range and at the edges of the fast path's."""
import numpy as np
import pytest

from triblocksolve_b200 import ALGO_FP64, ALGO_REFERENCE, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu

ONES = 2.0 - 2.0 ** -52  # every bit of the significand set


def divisors(n, lo, hi, edges, rng):
    sig = 1.0 + rng.random(n)
    kind = rng.integers(0, 6, n)
    sig[kind == 0] = ONES
    sig[kind == 1] = 1.0 + 2.0 ** -52
    sig[kind == 2] = 1.0
    e = rng.integers(lo, hi + 1, n)
    at = rng.random(n) < 0.1
    e[at] = rng.choice(edges, int(at.sum()))
    return np.ldexp(sig, e) * rng.choice([-1.0, 1.0], n)


def system(mesh, d, rhs):
    jac = Jacobian.generate(mesh, 9.0, 1)
    jac.jacO1[:] = 0.0
    jac.jacO2[:] = 0.0
    D = jac.jacD.reshape(-1, 81)  # (i, j) at i + 9 j
    D[:] = 0.0
    D[:, ::10] = d.reshape(-1, 9)
    jac.rhs[:] = rhs.reshape(-1)
    return jac


def first_update(mesh, jac, algo):
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(algo)
    s.sweep(1)
    dU = s.update()
    s.close()
    return dU


# lines: one CTA per line, three lines a CTA; single cells and longer chains
@pytest.mark.parametrize("L, K", [(40, 60), (301, 8), (50, 1)])
# the fast path's range, and mostly beyond it (2^-1000 .. 2^1000)
@pytest.mark.parametrize("lo, hi, edges", [(-998, 998, [-999, 999]), (-1020, 1020, [-1001, -1000, -999, 999, 1000, 1001])])
def test_factor_reciprocals(L, K, lo, hi, edges):
    mesh = Mesh.structured(L, K)
    rng = np.random.default_rng(L * K)
    d = divisors(9 * mesh.nelem, lo, hi, edges, rng)
    rhs = rng.choice([-1.0, 1.0], d.size)
    got = first_update(mesh, system(mesh, d, rhs), ALGO_FP64)
    np.testing.assert_array_equal(got, -rhs * (1.0 / d))


@pytest.mark.parametrize("L, K", [(40, 60), (50, 1)])
@pytest.mark.parametrize("lo, hi, edges", [(-498, 498, [-499, 499]), (-508, 508, [-501, -500, -499, 499, 500, 501])])
def test_reference_quotients(L, K, lo, hi, edges):
    mesh = Mesh.structured(L, K)
    rng = np.random.default_rng(L + K)
    d = divisors(9 * mesh.nelem, lo, hi, edges, rng)
    rhs = divisors(9 * mesh.nelem, -398, 398, [-401, -400, -399, 399, 400, 401], rng)
    rhs[rng.random(rhs.size) < 0.1] = 0.0
    got = first_update(mesh, system(mesh, d, rhs), ALGO_REFERENCE)
    np.testing.assert_array_equal(got, -rhs / d)


def test_reference_pivot_reciprocals():
    mesh = Mesh.structured(40, 60)
    rng = np.random.default_rng(3)
    d = np.ones((mesh.nelem, 9))
    d[:, 0] = divisors(mesh.nelem, -498, 498, [-501, -500, -499, 499, 500, 501], rng)
    rhs = np.zeros((mesh.nelem, 9))
    rhs[:, 0] = -1.0
    jac = system(mesh, d, rhs)
    jac.jacD.reshape(-1, 81)[:, 1] = 1.0
    got = first_update(mesh, jac, ALGO_REFERENCE).reshape(-1, 9)
    np.testing.assert_array_equal(got[:, 0], 1.0 / d[:, 0])
    np.testing.assert_array_equal(got[:, 1], -(1.0 / d[:, 0]))
