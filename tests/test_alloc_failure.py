"""Device memory that cannot be had while a solver builds its tables on first
use: the call reports it, nothing half built is taken up by the next one, and no
later launch is blamed for it.  Every allocation of the part is refused in turn
(on the host: fs_test_alloc_failure)."""
import numpy as np
import pytest

from flowsolversourcecode_b200 import case as cs
from flowsolversourcecode_b200 import mesh as fm

pytestmark = pytest.mark.gpu


def _solver(**kw):
    from flowsolversourcecode_b200.solver import Solver
    _, case = cs.cavity(4, krylov_tol=1e-8, krylov_maxit=50, **kw)
    return Solver(fm.box_mesh(11, 10, 9), case)


@pytest.mark.parametrize("kw,solver,least", [
    ({}, "amg_bicgs", 12), ({}, "amg32_bicgs", 16), ({}, "amg32gs_bicgs", 16), (dict(mg_pre=2), "amg32_bicgs", 30),
    ({}, "amg", 30), ({}, "ilu", 10), ({}, "pbcg", 13)])
def test_every_refused_allocation_is_reported_and_undone(kw, solver, least):
    from flowsolversourcecode_b200 import _lib as L
    t = _solver(**kw)
    rng = np.random.default_rng(1)
    con = t.connectivity()
    cn, cf = con["cn"].reshape(t.W, t.N), con["cf"].reshape(t.W, t.N)
    face = rng.uniform(0.5, 1.5, t.F)
    anb = np.where(cn >= 0, -face[np.minimum(cf, t.F - 1)], 0.0)
    a = -anb.sum(axis=0) + rng.uniform(0.0, 0.2, t.N), anb.ravel(), rng.standard_normal(t.N)
    sor, _ = t.solve_system(*a, solver="sor")
    ref, ref_it = t.solve_system(*a, rrf=1e-8, solver=solver)
    t.close()
    for k in range(1, 400):
        s = _solver(**kw)
        assert s.lib.fs_test_alloc_failure(s.ctx, k) == 0
        refused = False
        try:
            s.solve_system(*a, rrf=1e-8, solver=solver)
        except L.FsError as e:
            assert e.status == L.FS_E_CUDA
            refused = True
        assert s.lib.fs_test_alloc_failure(s.ctx, 0) == 0
        if refused:
            y, _ = s.solve_system(*a, solver="sor")
            assert np.array_equal(y, sor)
            x, it = s.solve_system(*a, rrf=1e-8, solver=solver)
            assert it == ref_it and np.array_equal(x, ref), k
        s.close()
        if not refused:
            break
    assert k > least      # the last count asked for was past the last allocation
