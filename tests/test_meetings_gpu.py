"""The waits of the launches whose CTAs meet (solves of few lines, GMRES's
orthogonalization), made to run out: one CTA stays away, the others give up
after a short budget.  The call reports it, GMRES stops at the step it happened
in, and the next calls give what they gave before, bit for bit."""
import numpy as np
import pytest

from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver, TbsError
from triblocksolve_b200 import _native as N

pytestmark = pytest.mark.gpu

BUDGET = 1 << 20  # cycles, about half a millisecond


def solver(L, K):
    mesh = Mesh.structured(L, K)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(Jacobian.generate(mesh, 4.0, 2))
    s.factor(ALGO_FP64)
    return s


def meetings(s, absent, budget):
    N.check(N.lib.tbs_selftest_meetings(s.ctx, absent, budget), s.ctx)


def fails(call):
    with pytest.raises(TbsError) as e:
        call()
    assert e.value.code == N.TBS_ERR_CUDA
    assert "time budget" in str(e.value)


# CTAs 0 and L - 1 have lines, the last ones only tiles; more tiles than one a CTA
@pytest.mark.parametrize("L, K, absent", [(60, 64, 0), (60, 64, 59), (60, 64, 60), (4, 30, 3), (130, 150, 100)])
def test_solve(L, K, absent):
    s = solver(L, K)
    n, h = s.solve(1e-10, 100)
    U = s.solution()
    for _ in range(2):
        meetings(s, absent, BUDGET)
        fails(lambda: s.solve(1e-10, 100))
        fails(lambda: s.solve(1e-10, 100))
        meetings(s, -1, 0)
        n2, h2 = s.solve(1e-10, 100)
        assert n2 == n
        np.testing.assert_array_equal(h2, h)
        np.testing.assert_array_equal(s.solution(), U)
    s.close()


@pytest.mark.parametrize("absent", [0, 5])
def test_gmres(absent):
    s = solver(40, 33)
    n, h = s.gmres(1e-10, 20)
    U = s.solution()
    for _ in range(2):
        meetings(s, absent, BUDGET)
        s.profile(True)
        s.profile_reset()
        fails(lambda: s.gmres(1e-10, 20))
        assert s.profile_read()["kr_orth"][0] == 1
        s.profile(False)
        meetings(s, -1, 0)
        n2, h2 = s.gmres(1e-10, 20)
        assert n2 == n
        np.testing.assert_array_equal(h2, h)
        np.testing.assert_array_equal(s.solution(), U)
    s.close()
