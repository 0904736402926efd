"""The V-cycle of the AMG-BiCGSTAB solvers against a NumPy restatement.

One BiCGSTAB iteration from zero applies the V-cycle twice; its solution is
compared with the same iteration in NumPy, FP64, on the hierarchy and the
coarse matrices that the library reports.  FP64 V-cycle: both sides do the
same few hundred operations per value, so they agree to about 1e-13 of the
solution; 1e-11 is asked for.  FP32 V-cycle: unit roundoff 6e-8 on values of
the preconditioned vectors, a few dozen operations deep: 1e-4 is asked for."""
import ctypes as C

import numpy as np
import pytest

from flowsolversourcecode_b200 import case as cs
from flowsolversourcecode_b200 import mesh as fm

pytestmark = pytest.mark.gpu

OMEGA0, OMEGA, ALPHA = 0.8, 0.9, 1.8


def _dense(ac, nbr, anb):
    n = ac.shape[0]
    A = np.zeros((n, n))
    A[np.arange(n), np.arange(n)] = ac
    for j in range(nbr.shape[0]):
        ok = nbr[j] >= 0
        np.add.at(A, (np.nonzero(ok)[0], nbr[j][ok]), anb[j][ok])
    return A


def _matvec(ac, nbr, anb, x):
    y = ac * x
    for j in range(nbr.shape[0]):
        ok = nbr[j] >= 0
        y[ok] += anb[j][ok] * x[nbr[j][ok]]
    return y


class Hierarchy:
    def __init__(self, s, ac, anb, gs):
        info = s.mg_info()
        self.lc = info["prec_coarsest"]
        assert info["direct"]
        con = s.connectivity()
        self.lev = [(ac, con["cn"].reshape(s.W, s.N), anb.reshape(s.W, s.N))]
        self.par = []
        for l in range(self.lc):
            n = info["sizes"][l]
            p = np.zeros(n, np.int32)
            assert s.lib.fs_mg_parents(s.ctx, l, p.ctypes.data_as(C.POINTER(C.c_int32)), n) == 0
            self.par.append(p)
            m = s.mg_coarse_matrix(l + 1)
            nc, w = info["sizes"][l + 1], info["widths"][l + 1]
            nbr = m["nbr"].reshape(w, nc).copy()
            nbr[np.arange(w)[:, None] >= m["n_nbr"][None, :]] = -1
            self.lev.append((m["ac"], nbr, m["anb"].reshape(w, nc)))
        A = _dense(*self.lev[self.lc])
        if np.all(np.abs(A.sum(axis=1)) <= 1e-9 * np.abs(np.diag(A))):   # pure Neumann: the last unknown is pinned
            A[-1] = 0.0
            A[-1, -1] = 1.0
            self.inv = np.linalg.inv(A)
            self.inv[:, -1] = 0.0
        else:
            self.inv = np.linalg.inv(A)
        self.gs = gs
        self.color = self._colours(*self.lev[0]) if gs else None

    @staticmethod
    def _colours(ac, nbr, anb):
        col = np.full(ac.shape[0], -1)
        for i in range(ac.shape[0]):
            used = {col[k] for k in nbr[:, i] if k >= 0}
            c = 0
            while c in used:
                c += 1
            col[i] = c
        return col

    def cycle(self, l, b):
        if l == self.lc:
            return self.inv @ b
        ac, nbr, anb = self.lev[l]
        om = OMEGA0 if l == 0 else OMEGA
        smooth = self.gs and l == 0

        def sweep(x, colours):
            for c in colours:
                r = b - (_matvec(ac, nbr, anb, x) - ac * x)
                x = np.where(self.color == c, r / ac, x)
            return x

        nc = self.color.max() + 1 if smooth else 0
        x = sweep(np.zeros_like(b), range(nc)) if smooth else om * b / ac
        r = b - _matvec(ac, nbr, anb, x)
        bc = np.bincount(self.par[l], weights=r, minlength=self.lev[l + 1][0].shape[0])
        x = x + ALPHA * self.cycle(l + 1, bc)[self.par[l]]
        if smooth:
            return sweep(x, range(nc - 1, -1, -1))
        return x + om * (b - _matvec(ac, nbr, anb, x)) / ac


def _shuffled(mesh, seed):
    """The same mesh with its cells renumbered at random (faces back in
    upper-triangular order): neighbour offsets without a pattern."""
    rng = np.random.default_rng(seed)
    p = rng.permutation(mesh.n_cells).astype(np.int32)
    F = mesh.n_internal
    nodes = mesh.face_nodes.reshape(-1, 4).copy()
    own, nbr = p[mesh.owner], p[mesh.neighbour]
    swap = own[:F] > nbr
    nodes[:F][swap] = nodes[:F][swap][:, ::-1]
    own[:F], nbr = np.minimum(own[:F], nbr), np.maximum(own[:F], nbr)
    order = np.concatenate([np.lexsort((nbr, own[:F])), np.arange(F, mesh.n_faces)])
    return fm.PolyMesh(mesh.points, mesh.face_ptr, np.ascontiguousarray(nodes[order].ravel()), own[order],
                       nbr[order[:F]], mesh.patch_names, mesh.patch_start, mesh.patch_size)


# one coarse level; two; several; a 2-D mesh; more rows per level than a CTA's
# shared array of residuals holds and rows shared between threads and lanes
@pytest.mark.parametrize("dims", [(7, 6, 5), (13, 11, 9), (57, 43, 1), (41, 37, 23), (71, 67, 64)])
@pytest.mark.parametrize("solver", ["amg_bicgs", "amg32_bicgs", "amg32gs_bicgs"])
@pytest.mark.parametrize("neumann", [True, False])
def test_one_iteration_matches_numpy(dims, solver, neumann):
    if dims[0] > 60 and (solver == "amg32gs_bicgs" or neumann):
        pytest.skip("the largest mesh runs once per precision")
    _one_iteration(fm.box_mesh(*dims), solver, neumann)


# cells numbered without a pattern (the index table), at a size whose rows are
# shared between lanes and one with a thread per row
@pytest.mark.parametrize("dims", [(13, 11, 9), (45, 43, 40)])
@pytest.mark.parametrize("solver", ["amg_bicgs", "amg32_bicgs", "amg32gs_bicgs"])
def test_one_iteration_matches_numpy_shuffled(dims, solver):
    _one_iteration(_shuffled(fm.box_mesh(*dims), 5), solver, False)


def _one_iteration(mesh, solver, neumann):
    from flowsolversourcecode_b200.solver import Solver
    _, case = cs.cavity(4, krylov_tol=1e-14, krylov_maxit=1)
    s = Solver(mesh, case)
    rng = np.random.default_rng(3)
    con = s.connectivity()
    cn, cf = con["cn"].reshape(s.W, s.N), con["cf"].reshape(s.W, s.N)
    face = rng.uniform(0.5, 1.5, s.F)
    anb = np.where(cn >= 0, -face[np.minimum(cf, s.F - 1)], 0.0)
    ac = -anb.sum(axis=0)
    if not neumann:
        ac = ac + rng.uniform(0.0, 0.2, s.N)
    b = rng.standard_normal(s.N)
    x, it = s.solve_system(ac, anb.ravel(), b, solver=solver)
    assert it == 1
    h = Hierarchy(s, ac, anb.ravel(), solver == "amg32gs_bicgs")
    if neumann:
        b = b - b.mean()
    y = h.cycle(0, b)
    v = _matvec(*h.lev[0], y)
    alpha = (b @ b) / (b @ v)
    q = b - alpha * v
    z = h.cycle(0, q)
    t = _matvec(*h.lev[0], z)
    ref = alpha * y + (t @ q) / (t @ t) * z
    err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
    assert err < (1e-11 if solver == "amg_bicgs" else 1e-4), err
    s.close()
