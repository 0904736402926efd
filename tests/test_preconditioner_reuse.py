"""pc_refresh: which solves may take over a preconditioner built earlier.

With two smoothing sweeps the Gauss-Seidel form keeps its coarse matrices and
dense inverse in the V-cycle's layout and the Jacobi form in mesh order; a solve
by the one must not take over what only the other has built."""
import numpy as np
import pytest

from flowsolversourcecode_b200 import case as cs
from flowsolversourcecode_b200 import mesh as fm

pytestmark = pytest.mark.gpu


def _solver(**kw):
    from flowsolversourcecode_b200.solver import Solver
    _, case = cs.cavity(4, krylov_tol=1e-8, krylov_maxit=100, **kw)
    return Solver(fm.box_mesh(21, 19, 17), case)


def _system(s, seed):
    rng = np.random.default_rng(seed)
    con = s.connectivity()
    cn, cf = con["cn"].reshape(s.W, s.N), con["cf"].reshape(s.W, s.N)
    face = rng.uniform(0.5, 1.5, s.F)
    anb = np.where(cn >= 0, -face[np.minimum(cf, s.F - 1)], 0.0)
    return -anb.sum(axis=0) + rng.uniform(0.0, 0.2, s.N), anb.ravel(), rng.standard_normal(s.N)


@pytest.mark.parametrize("first,second", [("amg32gs_bicgs", "amg32_bicgs"), ("amg32_bicgs", "amg32gs_bicgs"),
                                          ("amg32gs_bicgs", "amg_bicgs")])
def test_a_solve_of_another_form_builds_its_own(first, second):
    kw = dict(pc_refresh=4, mg_pre=2)
    s, t = _solver(**kw), _solver(**kw)
    a, b = _system(s, 1), _system(s, 2)
    s.solve_system(*a, solver=first)
    # on a handle that solved nothing before, the second form builds everything:
    # the same operations, so the same bits
    x, it = s.solve_system(*b, solver=second)
    ref, ref_it = t.solve_system(*b, solver=second)
    assert it == ref_it and np.array_equal(x, ref)
    # and back: the first form's preconditioner is not left over from system a
    x, it = s.solve_system(*b, solver=first)
    u = _solver(**kw)
    ref, ref_it = u.solve_system(*b, solver=first)
    assert it == ref_it and np.array_equal(x, ref)
    for q in (s, t, u):
        q.close()
