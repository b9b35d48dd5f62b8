"""tbs_resid_timer where all the sweeps of a solve are one launch: a record per
sweep, of the part of the sweep from the end of the longest line's solve to the
end of the last tile, whichever CTA has the longest line."""
import time

import pytest

from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [Mesh.structured(60, 64), ragged_mesh([3, 400, 7, 1, 90], seed=2),
                                  ragged_mesh([500, 2, 60], seed=3)])
def test_a_record_per_sweep(mesh):
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(Jacobian.generate(mesh, 9.0, 3))
    s.factor(ALGO_FP64)
    s.solve(1e-10, 100)
    s.resid_timer(reset=True)
    t = time.perf_counter()
    sweeps = sum(s.solve(1e-10, 100)[0] for _ in range(5))
    wall_us = 1e6 * (time.perf_counter() - t)
    us, n = s.resid_timer(reset=True)
    assert n == sweeps
    assert 0.0 < us < wall_us
    assert s.resid_timer() == (0.0, 0)
    s.close()
