"""Which solves are one launch of all sweeps, and its grid: not those of long
lines with much work for each SM; one to four neighbours off the line, even
and odd numbers of tiles.  On both sides of each edge the solve equals the one
with a launch per kernel, bit for bit."""
import numpy as np
import pytest

from triblocksolve_b200 import ALGO_FP64, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu


def columns(Li, Lj, K):
    """Lines (i, j) of K cells, each cell beside those of (i + 1, j) and (i, j + 1)."""
    at = np.arange(Li * Lj * K).reshape(Li, Lj, K)
    pairs = [(at[:, :, :-1], at[:, :, 1:]), (at[:, :-1], at[:, 1:]), (at[:-1], at[1:])]
    a = np.concatenate([p[0].ravel() for p in pairs])
    b = np.concatenate([p[1].ravel() for p in pairs])
    N, F = at.size, a.size
    ef = -np.ones((N, 6), np.int64)
    who = np.concatenate([a, b])
    order = np.argsort(who, kind="stable")
    first = np.searchsorted(who[order], np.arange(N))
    ef[who[order], np.arange(2 * F) - first[who[order]]] = order % F
    lineface = np.full(N, -7, np.int64)
    n = pairs[0][0].size
    lineface[b[:n]] = np.arange(n)
    return Mesh.from_arrays(9, epoint=np.arange(0, 6 * N + 1, 6), ef=ef.reshape(-1),
                            fc=np.stack([a, b], 1).reshape(-1), linesize=np.full(Li * Lj, K),
                            linepoint=np.arange(Li * Lj + 1) * K, lines=np.arange(N), lineface=lineface)


MESHES = {
    "one neighbour": lambda: Mesh.structured(2, 700),
    "odd tiles": lambda: Mesh.structured(11, 133),
    "two a CTA": lambda: Mesh.structured(60, 64),
    "three neighbours": lambda: columns(13, 2, 41),
    "four neighbours": lambda: columns(9, 7, 30),
    "long lines": lambda: Mesh.structured(60, 600),
    "long lines, too much": lambda: Mesh.structured(64, 640),
}


@pytest.mark.parametrize("name", list(MESHES))
def test_equals_a_launch_per_kernel(name):
    mesh = MESHES[name]()
    mesh.validate()
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(Jacobian.generate(mesh, 9.0, 2))
    s.factor(ALGO_FP64)
    n, h = s.solve(1e-10, 100)
    U, check = s.solution(), s.solve_check()
    assert h[-1] <= 1e-10 * h[0]
    s.profile(True)
    n2, h2 = s.solve(1e-10, 100)
    s.profile(False)
    assert n2 == n and s.solve_check() == check
    np.testing.assert_array_equal(h2, h)
    np.testing.assert_array_equal(s.solution(), U)
    s.close()
