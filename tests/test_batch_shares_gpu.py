"""How a batch deals its residual tiles to CTAs, and the schedule it picks.

A CTA takes full waves of 8 consecutive tiles and an equal share of the tiles
left over, counted over the systems still active.  Edges: fewer tiles than
CTAs, more than 32 systems (the prefix sums go by 32), systems that stop early,
a full wave and a remainder, systems of one tile between large ones.  Every
member's sweeps, norms and solution are the single solve's, bit for bit (each
tile's arithmetic and the norm's order do not depend on who runs it).
"""
import numpy as np
import pytest

from triblocksolve_b200 import ALGO_FP64, Batch, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu

CASES = {
    "one-tile": [(1, 1, 9.0)],
    "few": [(7, 11, 9.0), (1, 16, 9.0), (3, 5, 4.0)],
    "40-systems": [(1 + i % 9, 1 + (7 * i) % 23, 3.5 + (i % 5)) for i in range(40)],
    "wave-and-rest": [(2, 3, 9.0), (330, 300, 9.0), (1, 1, 4.0), (90, 200, 5.0), (5, 9, 9.0)],
}


@pytest.mark.parametrize("name", list(CASES))
def test_shares(name):
    solvers = []
    for i, (nl, nk, shift) in enumerate(CASES[name]):
        mesh = Mesh.structured(nl, nk)
        s = Solver(0)
        s.set_mesh(mesh)
        s.set_jacobian(Jacobian.generate(mesh, shift, i))
        s.factor(ALGO_FP64)
        solvers.append(s)
    batch = Batch(solvers)
    try:
        sweeps, hist = batch.solve(1e-11, 60)
        got = [s.solution() for s in solvers]
        for k, s in enumerate(solvers):
            n, h = s.solve(1e-11, 60)
            assert n == sweeps[k]
            np.testing.assert_array_equal(hist[k][: n + 1], h)
            np.testing.assert_array_equal(got[k], s.solution())
    finally:
        batch.close()
        for s in solvers:
            s.close()


@pytest.mark.parametrize("nl, nk, n, want", [(8, 64, 2, (4, 3, 2)), (150, 40, 8, (5, 3, 2)), (150, 40, 16, (8, 2, 1))])
def test_default_schedule(nl, nk, n, want):
    """Cells per SM over the longest line (148 SMs: 0.1, 8.1, 16.2) pick it; a
    set schedule replaces it, from one warp a line unless that was set."""
    mesh = Mesh.structured(nl, nk)
    jac = Jacobian.generate(mesh, 9.0, 1)
    solvers = []
    for _ in range(n):
        s = Solver(0)
        s.set_mesh(mesh)
        s.set_jacobian(jac)
        s.factor(ALGO_FP64)
        solvers.append(s)
    batch = Batch(solvers)
    try:
        assert batch.schedule()[:2] + (batch.warps_per_line(),) == want
        first = batch.solve(1e-11, 60)
        batch.set_schedule(8, 2, 0)
        assert batch.schedule() == (8, 2, 0) and batch.warps_per_line() == 1
        second = batch.solve(1e-11, 60)
        np.testing.assert_array_equal(first[0], second[0])
        for a, b in zip(first[1], second[1]):
            np.testing.assert_array_equal(a, b)
    finally:
        batch.close()
        for s in solvers:
            s.close()


@pytest.mark.parametrize("limit", [3, 60, 70000])
def test_history_rows(limit):
    """States and norms come back in one launch while the rows take at most
    1 MiB (two rows of 70001 norms: 1.07 MiB, copied one by one); rows shorter
    than the solve (3 sweeps) end at the limit."""
    solvers = []
    for i, (nl, nk, shift) in enumerate([(9, 31, 9.0), (4, 17, 4.0)]):
        mesh = Mesh.structured(nl, nk)
        s = Solver(0)
        s.set_mesh(mesh)
        s.set_jacobian(Jacobian.generate(mesh, shift, i))
        s.factor(ALGO_FP64)
        solvers.append(s)
    batch = Batch(solvers)
    try:
        for _ in range(2):
            sweeps, hist = batch.solve(1e-11, limit)
            got = [s.solution() for s in solvers]
            for k, s in enumerate(solvers):
                n, h = s.solve(1e-11, limit)
                assert n == sweeps[k]
                np.testing.assert_array_equal(hist[k][: n + 1], h)
                np.testing.assert_array_equal(got[k], s.solution())
    finally:
        batch.close()
        for s in solvers:
            s.close()
