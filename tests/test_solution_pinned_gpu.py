"""Solutions into pinned memory: the reordering stores there itself; into
pageable memory it goes through a device vector.  The same words either way, at
any 8-byte offset, and none beyond."""
import numpy as np
import pytest
import torch

from meshes import ragged_mesh
from triblocksolve_b200 import ALGO_FP64, ALGO_MIXED, ALGO_REFERENCE, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo, nvar", [(ALGO_FP64, 9), (ALGO_MIXED, 9), (ALGO_REFERENCE, 9), (ALGO_FP64, 5)])
@pytest.mark.parametrize("lens", [[1], [5, 1, 7, 3, 3, 8, 13, 2, 9], [96] * 41])
def test_pinned(algo, nvar, lens):
    mesh = ragged_mesh(lens, seed=4, nvar=nvar)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(Jacobian.generate(mesh, 9.0, 3))
    s.factor(algo)
    try:
        s.sweep(2)
        n = nvar * mesh.nelem
        want = s.solution()
        assert np.count_nonzero(want) > 0
        for off in (0, 1, 2):
            buf = torch.full((n + 4,), -7.0, dtype=torch.float64, pin_memory=True).numpy()
            s.solution(buf[off : off + n])
            np.testing.assert_array_equal(buf[off : off + n], want)
            assert (buf[:off] == -7.0).all() and (buf[off + n :] == -7.0).all()
    finally:
        s.close()
