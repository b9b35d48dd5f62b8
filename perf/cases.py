"""The work that a program has the solver do, through its public entry points.

A case is a kind of call and the system it is made on:

  kind "solve"  a factored system: ``Solver.solve`` to a tolerance, the solution read back into pinned
                host memory (what ``triblock.exe`` and the benchmark time); ``new_rhs``: ``set_rhs`` first
  kind "step"   one step of a time-marching caller: a new Jacobian (on the device), factorization,
                solve, solution
  kind "multi"  ``solve_multi_device``: several right-hand sides of one factored system
  kind "batch"  ``Batch.solve`` over independent systems of uneven sizes
  kind "gmres"  line-preconditioned restarted GMRES

on a structured mesh of ``L`` lines of ``K`` cells, or (``mesh`` "ragged") lines of ``kmin`` .. ``K`` cells
whose cells, faces and lines are numbered in random order.  Values are those of the synthetic systems of
the tests and the benchmark: diagonal blocks U(-1, 1) + shift I, face blocks 0.1 U(-1, 1), rhs U(-1, 1).
"""
import functools
import math

import numpy as np
import torch

import triblocksolve_b200 as tbs

ALGO = {"fp64": tbs.ALGO_FP64, "mixed": tbs.ALGO_MIXED, "reference": tbs.ALGO_REFERENCE, "pij": tbs.ALGO_PIJ}


def listed():
    return [
        # the reference's smallest data set (ex05), a new right-hand side each call: launches and latency
        _case("solve-60x64", L=60, K=64, shift=9.0, tol=1e-12, new_rhs=True),
        # an unstructured mesh as a flow solver hands it over: uneven lines, arbitrary numbering
        _case("solve-ragged", mesh="ragged", L=181, kmin=37, K=301, shift=9.0, tol=1e-10, new_rhs=True),
        # the reference's published middle size
        _case("solve-360x384", L=360, K=384, shift=9.0, tol=1e-12),
        # the headline configuration, the reference's largest published size
        _case("solve-1200x1280", L=1200, K=1280, shift=4.0, tol=1e-10),
        # the mixed-precision form where the benchmark quotes it
        _case("mixed-600x640", algo="mixed", L=600, K=640, shift=4.0, tol=1e-10),
        # a time step: new block values, factorization and solve, at two sizes
        _case("step-120x128", kind="step", L=120, K=128, shift=9.0, tol=1e-10),
        _case("step-600x640", kind="step", L=600, K=640, shift=4.0, tol=1e-10),
        # the reference's own operation order (bit-exact drop-in), factorization and sweeps
        _case("reference-360x384", kind="step", algo="reference", L=360, K=384, shift=9.0, tol=1e-10),
        # several right-hand sides of one system
        _case("multi8-360x384", kind="multi", L=360, K=384, shift=9.0, tol=1e-12, nrhs=8),
        # independent uneven systems in one launch sequence
        _case("batch-12", kind="batch", nsys=12, L=300, K=320, shift=9.0, tol=1e-10),
        # a smaller block (5 equations, one of the reference's resizeBlockSize sizes)
        _case("nvar5-600x640", nvar=5, L=600, K=640, shift=4.0, tol=1e-10),
        # the Krylov caller of the line sweep, on an odd mesh
        _case("gmres-301x257", kind="gmres", L=301, K=257, shift=4.0, tol=1e-10, restart=30),
    ]


def _case(name, kind="solve", algo="fp64", mesh="structured", nvar=9, **more):
    return {"name": name, "kind": kind, "algo": algo, "mesh": mesh, "nvar": nvar, **more}


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["solve", "solve", "solve", "mixed", "step", "step", "reference", "multi", "batch", "nvar",
                       "gmres", "pij"])
    ragged = what in ("solve", "step", "multi") and rng.random() < 0.35
    top = {"reference": 400, "batch": 400, "multi": 600, "gmres": 600, "step": 800}.get(what, 1100)
    L, K = size(20, top), size(24, top)
    tol = rng.choice([1e-8, 1e-10, 1e-12]) if what != "mixed" else 1e-10
    c = {"kind": "solve", "algo": "fp64", "mesh": "ragged" if ragged else "structured", "nvar": 9, "L": L, "K": K,
         "shift": rng.choice([4.0, 9.0]) if L * K < 200000 else 4.0, "tol": tol}
    if ragged:
        c["kmin"] = max(1, int(K * rng.uniform(0.05, 0.9)))
    if what == "solve":
        c["new_rhs"] = rng.random() < 0.5
    elif what in ("mixed", "pij"):
        c["algo"] = what
    elif what == "reference":
        c.update(kind="step", algo="reference")
    elif what == "multi":
        c.update(kind="multi", nrhs=rng.randint(2, 8))
    elif what == "batch":
        c.update(kind="batch", nsys=rng.randint(3, 16), shift=9.0)
    elif what == "nvar":
        c["nvar"] = rng.choice([4, 5, 7, 12])
        if c["nvar"] > 9:
            c["shift"] = 9.0
    elif what == "gmres":
        c.update(kind="gmres", restart=rng.choice([10, 30]), shift=4.0)
    else:
        c["kind"] = what
    return c


# ------------------------------------------------------------------ meshes

@functools.lru_cache(maxsize=4)
def _structured(L, K, nvar):
    return tbs.Mesh.structured(L, K, nvar=nvar)


def _ragged(lens, rng, nvar):
    """Lines of lens[l] cells, cell k of a line beside cell k of the next; cells, faces, face sides and
    lines in random order, every cell with four entries in ``ef`` (negative: a boundary)."""
    lens = np.asarray(lens, np.int64)
    L, N = lens.size, int(lens.sum())
    first = np.concatenate([[0], np.cumsum(lens)])
    line = np.repeat(np.arange(L), lens)
    k = np.arange(N) - first[line]
    inner = np.flatnonzero(k + 1 < lens[line])  # cells with a successor on their line
    up = np.flatnonzero((line + 1 < L) & (k < lens[np.minimum(line + 1, L - 1)]))
    a = np.concatenate([inner, up])
    b = np.concatenate([inner + 1, first[line[up] + 1] + k[up]])
    elem = rng.permutation(N)
    F = a.size
    fid = rng.permutation(F)
    swap = rng.random(F) < 0.5
    fc = np.empty((F, 2), np.int64)
    fc[fid, 0] = np.where(swap, elem[b], elem[a])
    fc[fid, 1] = np.where(swap, elem[a], elem[b])
    ef = -np.ones((N, 4), np.int64)
    who = np.concatenate([fc[:, 0], fc[:, 1]])
    order = np.argsort(who, kind="stable")
    start = np.searchsorted(who[order], np.arange(N))
    ef[who[order], np.arange(2 * F) - start[who[order]]] = order % F
    ef = np.take_along_axis(ef, np.argsort(rng.random((N, 4)), axis=1), axis=1)
    face_to_next = np.full(N, -7, np.int64)  # of the cell that comes second
    face_to_next[inner + 1] = fid[: inner.size]
    lorder = rng.permutation(L)
    cells = np.concatenate([np.arange(first[l], first[l + 1]) for l in lorder])
    return tbs.Mesh.from_arrays(
        nvar, epoint=np.arange(0, 4 * N + 1, 4), ef=ef.reshape(-1), fc=fc.reshape(-1), linesize=lens[lorder],
        linepoint=np.concatenate([[0], np.cumsum(lens[lorder])]), lines=elem[cells], lineface=face_to_next[cells])


def _meshes(case, seed):
    """The case's meshes (one, or one per system of a batch)."""
    rng = np.random.default_rng([seed, 77])
    L, K, nvar = case["L"], case["K"], case["nvar"]
    if case["kind"] == "batch":
        # the sizes are part of the case: the same for every seed, spread evenly on a logarithmic scale
        n = case["nsys"]
        at = [((i * 7) % n + 0.5) / n for i in range(n)]
        return [_structured(max(8, int(16 * (L / 16) ** at[i])), max(8, int(16 * (K / 16) ** at[(i * 5 + 3) % n])), nvar)
                for i in range(n)]
    if case["mesh"] == "ragged":
        return [_ragged(np.random.default_rng([L, K, case["kmin"]]).integers(case["kmin"], K + 1, L), rng, nvar)]
    return [_structured(L, K, nvar)]


def _values(case, mesh, seed, part=0):
    """jacD, jacO1, jacO2 (blocks column-major) and rhs on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + part)
    nv, ne, nf = mesh.nvar, mesh.nelem, mesh.nintface

    def uniform(n, scale):
        return torch.rand(n, dtype=torch.float64, device="cuda", generator=g).mul_(2 * scale).sub_(scale)

    D = uniform(ne * nv * nv, 1.0)
    D.view(ne, nv, nv).diagonal(dim1=1, dim2=2).add_(case["shift"])
    return D, uniform(nf * nv * nv, 0.1), uniform(nf * nv * nv, 0.1), uniform(ne * nv * case.get("nrhs", 1), 1.0)


# ----------------------------------------------------------------- the work

def prepare(case, seed):
    solvers, outs, values = [], [], []
    algo = ALGO[case["algo"]]
    for part, mesh in enumerate(_meshes(case, seed)):
        v = _values(case, mesh, seed, part)
        torch.cuda.synchronize()
        s = tbs.Solver(0)
        s.set_mesh(mesh)
        s.set_jacobian_device(*(x.data_ptr() for x in v))
        s.factor(algo)
        if case["algo"] == "mixed":
            s.set_inner_sweeps(5)
        solvers.append(s)
        outs.append(torch.empty(mesh.nelem * mesh.nvar, dtype=torch.float64, pin_memory=True).numpy())
        values.append(v)
    state = {"case": case, "solvers": solvers, "outs": outs}
    if case["kind"] == "step":
        state["values"] = values
    elif case["kind"] == "multi":
        state["rhs"] = values[0][3]
        state["U"] = torch.empty_like(state["rhs"])
    elif case["kind"] == "batch":
        state["batch"] = tbs.Batch(solvers)
    elif case.get("new_rhs"):
        state["rhs"] = values[0][3].cpu().pin_memory().numpy()
    return state


def run(state):
    case = state["case"]
    s, out, kind, tol = state["solvers"][0], state["outs"][0], case["kind"], case["tol"]
    if kind == "multi":
        sweeps, hist = s.solve_multi_device(state["rhs"].data_ptr(), state["U"].data_ptr(), case["nrhs"], tol, 200)
        return {"U": state["U"], "sweeps": sweeps, "hist": [_norms(h) for h in hist]}
    if kind == "batch":
        sweeps, hist = state["batch"].solve(tol, 200)
        return {"U": [q.solution(o) for q, o in zip(state["solvers"], state["outs"])], "sweeps": sweeps,
                "hist": [_norms(h) for h in hist]}
    if kind == "gmres":
        steps, hist = s.gmres(tol, case["restart"])
        return {"U": s.solution(out), "steps": steps, "hist": _norms(hist)}
    if kind == "step":
        s.set_jacobian_device(*(x.data_ptr() for x in state["values"][0]))
        s.factor(ALGO[case["algo"]])
    elif "rhs" in state:
        s.set_rhs(state["rhs"])
    sweeps, hist = s.solve(tol, 200)
    return {"U": s.solution(out), "sweeps": sweeps, "hist": _norms(hist)}


def _norms(hist):
    """The residual norms, as many for every input (the sweeps differ): zeros follow the last one."""
    h = np.zeros(301)
    h[: len(hist)] = hist
    return h


def work(case):
    """Every sweep needs each of the system's blocks (the diagonal and two of every face) once, and the
    residual's neighbours; a factorization reads the blocks, and writes the cells' three line blocks."""
    nv, nrhs = case["nvar"], case.get("nrhs", 1)
    total = {"bytes": 0.0, "flops": 0.0}
    for mesh in _meshes(case, 0):
        ne, nf = mesh.nelem, mesh.nintface
        blocks = ne + 2 * nf
        rate = {9.0: 1.5, 4.0: 1.1}[case["shift"]]  # decimal digits a line sweep gains
        if case["algo"] == "pij":
            rate *= 0.7
        sweeps = math.ceil(-math.log10(case["tol"]) / rate)
        word = 4 if case["algo"] == "mixed" else 8
        total["bytes"] += sweeps * (blocks * nv * nv * word + ne * nv * 8 * 4 * nrhs)
        total["flops"] += sweeps * blocks * 2 * nv * nv * nrhs
        if case["kind"] == "step":
            total["bytes"] += (blocks + 3 * ne) * nv * nv * 8
            total["flops"] += ne * 2 * nv ** 3 * 4
    return total


# ----------------------------------------------- the same results, in torch

class _System:
    """R = rhs + J U and the exact solve of the lines' block-tridiagonal part, lines side by side."""

    def __init__(self, mesh, D, O1, O2, points):
        nv, ne, nf = mesh.nvar, mesh.nelem, mesh.nintface

        def gpu(a):
            return torch.from_numpy(np.ascontiguousarray(a, np.int64)).cuda()

        self.D, self.O1, self.O2 = (x.view(-1, nv, nv).transpose(1, 2) for x in (D, O1, O2))
        self.fc = gpu(mesh.fc).view(nf, 2)
        size, first = mesh.linesize.astype(np.int64), mesh.linepoint[:-1].astype(np.int64)
        lines, lineface = mesh.lines, mesh.lineface
        if points:  # every cell its own line
            size, first, lines = np.ones(ne, np.int64), np.arange(ne), np.arange(ne)
        self.at, self.inv, self.A, self.gam = [], [], [], []
        by = np.argsort(-size, kind="stable")
        size, first = size[by], first[by]
        for k in range(int(size[0])):
            on = first[: int(np.count_nonzero(size > k))] + k
            e = gpu(lines[on])
            W = self.D[e]
            if k:
                f = gpu(lineface[on])
                second = (self.fc[f, 0] == e).view(-1, 1, 1)
                A, C = torch.where(second, self.O2[f], self.O1[f]), torch.where(second, self.O1[f], self.O2[f])
                self.gam.append(self.inv[-1][: e.numel()] @ C)
                W = W - A @ self.gam[-1]
                self.A.append(A)
            self.at.append(e)
            self.inv.append(torch.linalg.inv(W))

    def residual(self, rhs, U):
        R = rhs + torch.bmm(self.D, U.unsqueeze(2)).squeeze(2)
        R.index_add_(0, self.fc[:, 0], torch.bmm(self.O2, U[self.fc[:, 1]].unsqueeze(2)).squeeze(2))
        return R.index_add_(0, self.fc[:, 1], torch.bmm(self.O1, U[self.fc[:, 0]].unsqueeze(2)).squeeze(2))

    def update(self, R):
        ys = []
        for k, e in enumerate(self.at):
            b = -R[e].unsqueeze(2)
            if k:
                b = b - torch.bmm(self.A[k - 1], ys[-1][: e.numel()])
            ys.append(torch.bmm(self.inv[k], b))
        dU = torch.empty_like(R)
        for k in range(len(ys) - 1, -1, -1):
            if k + 1 < len(ys):
                n = ys[k + 1].shape[0]
                ys[k][:n] -= torch.bmm(self.gam[k], ys[k + 1])
            dU[self.at[k]] = ys[k].squeeze(2)
        return dU

    def iterate(self, rhs, tol, sweeps):
        U, R = torch.zeros_like(rhs), rhs
        hist = [float(R.norm())]
        while hist[-1] > tol * hist[0] and len(hist) <= sweeps:
            U = U + self.update(R)
            R = self.residual(rhs, U)
            hist.append(float(R.norm()))
        return U.reshape(-1), np.array(hist)


def exact(case, seed):
    Us, hists = [], []
    # the iterates of the line sweep where the path is that iteration; the solution itself (to 64 bits)
    # where the path only has to reach the tolerance
    solution = case["algo"] == "mixed" or case["kind"] == "gmres"
    for part, mesh in enumerate(_meshes(case, seed)):
        D, O1, O2, rhs = _values(case, mesh, seed, part)
        S = _System(mesh, D, O1, O2, case["algo"] == "pij")
        for r in rhs.view(case.get("nrhs", 1), mesh.nelem, mesh.nvar):
            U, hist = S.iterate(r, 1e-15 if solution else case["tol"], 30 if solution else 200)
            Us.append(U)
            hists.append(None if solution else _norms(hist))
        del S
    if case["kind"] == "batch":
        return {"U": [u.cpu().numpy() for u in Us], "sweeps": None, "hist": hists}
    if case["kind"] == "multi":
        return {"U": torch.cat(Us), "sweeps": None, "hist": hists}
    return {"U": Us[0].cpu().numpy(), "hist": hists[0]}
