"""Launches whose CTAs wait for one another (solves of few lines, GMRES) from
several threads at once and beside other streams' work: every result equals
the one the context gives alone, bit for bit."""
import threading

import numpy as np
import pytest

from triblocksolve_b200 import ALGO_FP64, ALGO_MIXED, Batch, Jacobian, Mesh, Solver

pytestmark = pytest.mark.gpu


def solver(L, K, algo=ALGO_FP64, seed=1):
    mesh = Mesh.structured(L, K)
    s = Solver(0)
    s.set_mesh(mesh)
    s.set_jacobian(Jacobian.generate(mesh, 9.0, seed))
    s.factor(algo)
    return s


def solve(s):
    n, h = s.solve(1e-10, 50)
    return n, np.asarray(h), s.solution()


def gmres(s):
    n, h = s.gmres(1e-10, 12)
    return n, np.asarray(h), s.solution()


def multi(s):
    rhs = np.random.default_rng(3).uniform(-1, 1, (5, 9 * s.nelem))
    U, n, h = s.solve_multi(rhs, 1e-10, 50)
    return n.tolist(), np.concatenate(h), U.copy()


def same(a, b):
    assert a[0] == b[0]
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[2], b[2])


def together(jobs, reps=12):
    """jobs: (context, call) pairs, a thread each, all at the same time."""
    want = [call(s) for s, call in jobs]
    got = [[] for _ in jobs]
    errors = []
    start = threading.Barrier(len(jobs))

    def run(k):
        try:
            start.wait()
            for _ in range(reps):
                got[k].append(jobs[k][1](jobs[k][0]))
        except Exception as e:  # the assertion below shows it
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w, g in zip(want, got):
        for x in g:
            same(w, x)


# grids that fit beside each other, that do not, and that fill the device
@pytest.mark.parametrize("sizes", [[(20, 24)] * 4, [(60, 64)] * 6, [(290, 40)] * 3, [(60, 64), (296, 30), (7, 500), (150, 20)]])
def test_small_solves(sizes):
    S = [solver(L, K, seed=k) for k, (L, K) in enumerate(sizes)]
    together([(s, solve) for s in S])
    for s in S:
        s.close()


def test_mixed_work():
    """Small solves and GMRES beside launches that fill the device."""
    S = [solver(60, 64), solver(40, 33, seed=2), solver(301, 200, seed=3), solver(500, 60, ALGO_MIXED, 4),
         solver(120, 90, seed=5)]
    together([(S[0], solve), (S[1], gmres), (S[2], gmres), (S[3], solve), (S[4], multi)])
    for s in S:
        s.close()


def test_beside_a_batch():
    S = [solver(60, 64), solver(33, 40, seed=2)]
    members = [solver(50 + 17 * k, 40 + 9 * k, seed=k) for k in range(5)]
    batch = Batch(members)

    def run(b):
        n, h = b.solve(1e-10, 50)
        return n.tolist(), np.concatenate(h), np.concatenate([m.solution() for m in members])

    together([(S[0], solve), (S[1], gmres), (batch, run)])
    batch.close()
    for s in S + members:
        s.close()
