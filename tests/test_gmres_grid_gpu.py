"""GMRES's orthogonalization is one cooperative launch, so all its CTAs have
to be resident: a device (or a part of one) that holds fewer than the blocks
the vectors are dealt to gets fewer CTAs, with the same results bit for bit."""
import numpy as np
import pytest

from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver
from triblocksolve_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L, K", [(9, 14), (301, 40)])
def test_fewer_ctas(L, K):
    mesh = Mesh.structured(L, K)
    jac = Jacobian.generate(mesh, 3.0, 3)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(jac)
    s.factor(ALGO_FP64)
    n, h = s.gmres(1e-10, 12, 1, 30)
    U = s.solution()
    for ctas in (1, 7, 148, 295, 100000, 0):
        N.check(N.lib.tbs_selftest_orth_ctas(s.ctx, ctas), s.ctx)
        n2, h2 = s.gmres(1e-10, 12, 1, 30)
        assert n2 == n
        np.testing.assert_array_equal(h2, h)
        np.testing.assert_array_equal(s.solution(), U)
    s.close()
