"""The general V-cycle of the AMG-BiCGSTAB solvers (more than one sweep a leg, or
no level small enough for the dense inverse) against a NumPy restatement.

One BiCGSTAB iteration from zero, as in test_vcycle.py, on the hierarchy and the
coarse matrices that the library reports.  FP64 V-cycle: at most twenty sweeps of
a few dozen operations each per value, rounding about 1e-13 of the solution;
1e-11 is asked for.  FP32 V-cycle: unit roundoff 6e-8, the same depth, damped by
every sweep: 1e-4 is asked for."""
import ctypes as C

import numpy as np
import pytest

from flowsolversourcecode_b200 import case as cs
from flowsolversourcecode_b200 import mesh as fm
from test_vcycle import ALPHA, OMEGA, OMEGA0, _dense, _matvec

pytestmark = pytest.mark.gpu

COARSE_SWEEPS = 20


def _levels(s, ac, anb):
    info = s.mg_info()
    lev, par = [(ac, s.connectivity()["cn"].reshape(s.W, s.N), anb.reshape(s.W, s.N))], []
    for l in range(info["prec_coarsest"]):
        n, nc, w = info["sizes"][l], info["sizes"][l + 1], info["widths"][l + 1]
        p = np.zeros(n, np.int32)
        assert s.lib.fs_mg_parents(s.ctx, l, p.ctypes.data_as(C.POINTER(C.c_int32)), n) == 0
        par.append(p)
        m = s.mg_coarse_matrix(l + 1)
        nbr = m["nbr"].reshape(w, nc).copy()
        nbr[np.arange(w)[:, None] >= m["n_nbr"][None, :]] = -1
        lev.append((m["ac"], nbr, m["anb"].reshape(w, nc)))
    return lev, par, np.linalg.inv(_dense(*lev[-1])) if info["direct"] else None


def _cycle(lev, par, inv, sweeps, l, b):
    if l == len(lev) - 1 and inv is not None:
        return inv @ b
    ac = lev[l][0]
    om = OMEGA0 if l == 0 else OMEGA

    def jacobi(x, n):
        for _ in range(n):
            x = x + om * (b - _matvec(*lev[l], x)) / ac
        return x

    x = om * b / ac
    if l == len(lev) - 1:   # a hierarchy of level 0 alone takes its pre-sweeps too
        return jacobi(x, COARSE_SWEEPS - 1 + (sweeps - 1 if l == 0 else 0))
    x = jacobi(x, sweeps - 1)
    bc = np.bincount(par[l], weights=b - _matvec(*lev[l], x), minlength=lev[l + 1][0].shape[0])
    return jacobi(x + ALPHA * _cycle(lev, par, inv, sweeps, l + 1, bc)[par[l]], sweeps)


@pytest.mark.parametrize("solver", ["amg_bicgs", "amg32_bicgs"])
@pytest.mark.parametrize("dims", [(13, 11, 9), (41, 37, 23)])
@pytest.mark.parametrize("case_kw", [dict(mg_pre=2), dict(mg_max_levels=2), dict(mg_max_levels=2, mg_pre=2),
                                     dict(mg_max_levels=1), dict(mg_max_levels=1, mg_pre=2)])
def test_one_iteration_matches_numpy(dims, solver, case_kw):
    from flowsolversourcecode_b200.solver import Solver
    _, case = cs.cavity(4, krylov_tol=1e-14, krylov_maxit=1, **case_kw)
    s = Solver(fm.box_mesh(*dims), case)
    rng = np.random.default_rng(3)
    con = s.connectivity()
    cn, cf = con["cn"].reshape(s.W, s.N), con["cf"].reshape(s.W, s.N)
    face = rng.uniform(0.5, 1.5, s.F)
    anb = np.where(cn >= 0, -face[np.minimum(cf, s.F - 1)], 0.0)
    ac = -anb.sum(axis=0) + rng.uniform(0.0, 0.2, s.N)
    b = rng.standard_normal(s.N)
    x, it = s.solve_system(ac, anb.ravel(), b, solver=solver)
    assert it == 1
    lev, par, inv = _levels(s, ac, anb)
    sweeps = case_kw.get("mg_pre", 1)
    y = _cycle(lev, par, inv, sweeps, 0, b)
    v = _matvec(*lev[0], y)
    alpha = (b @ b) / (b @ v)
    q = b - alpha * v
    z = _cycle(lev, par, inv, sweeps, 0, q)
    t = _matvec(*lev[0], z)
    ref = alpha * y + (t @ q) / (t @ t) * z
    err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
    assert err < (1e-11 if solver == "amg_bicgs" else 1e-4), err
    s.close()
