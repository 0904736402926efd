"""Every call that hands results to the host reports a bounded device wait that
gave up, once, and the next solve is a normal one again.  The waits are made to
run out on the host's word (fs_test_wait_timeout: barriers wait for a CTA that
does not take part); nothing faults or hangs."""
import numpy as np
import pytest

from flowsolversourcecode_b200 import case as cs

pytestmark = pytest.mark.gpu


def _solver():
    from flowsolversourcecode_b200.solver import Solver
    mesh, case = cs.cavity(12, nz=12, solver_cont="amg_bicgs", krylov_tol=1e-8, krylov_maxit=50)
    return Solver(mesh, case)


def _system(s):
    rng = np.random.default_rng(7)
    con = s.connectivity()
    cn, cf = con["cn"].reshape(s.W, s.N), con["cf"].reshape(s.W, s.N)
    face = rng.uniform(0.5, 1.5, s.F)
    anb = np.where(cn >= 0, -face[np.minimum(cf, s.F - 1)], 0.0)
    return -anb.sum(axis=0) + rng.uniform(0.0, 0.2, s.N), anb.ravel(), rng.standard_normal(s.N)


def _times_out(call):
    from flowsolversourcecode_b200 import _lib as L
    with pytest.raises(L.FsError) as e:
        call()
    assert e.value.status == L.FS_E_TIMEOUT


@pytest.mark.parametrize("solver", ["amg_bicgs", "amg32_bicgs", "amg32gs_bicgs"])
def test_solve_system_reports_and_recovers(solver):
    s, t = _solver(), _solver()
    a = _system(s)
    assert s.lib.fs_test_wait_timeout(s.ctx, 1) == 0
    _times_out(lambda: s.solve_system(*a, solver=solver))
    assert s.lib.fs_test_wait_timeout(s.ctx, 0) == 0
    x, it = s.solve_system(*a, solver=solver)
    ref, ref_it = t.solve_system(*a, solver=solver)
    assert it == ref_it and np.array_equal(x, ref)
    s.close()
    t.close()


@pytest.mark.parametrize("read", ["get", "sync", "residuals"])
def test_solve_equation_reports_where_its_result_is_read(read):
    s = _solver()
    a = _system(s)
    for k, v in zip(("ac", "anb", "bc"), a):
        s.set(k, v)
    assert s.lib.fs_test_wait_timeout(s.ctx, 1) == 0
    s.SolveEquation("pressc", 1e-8, 50, "amg_bicgs")
    assert s.lib.fs_test_wait_timeout(s.ctx, 0) == 0
    calls = {"get": lambda: s.get("pc"), "sync": s.sync, "residuals": s.PrintConvergenceHistory}
    _times_out(calls[read])
    calls["get"]()                       # reported once
    s.set("pc", np.zeros(s.N))
    s.SolveEquation("pressc", 1e-8, 50, "amg_bicgs")
    x = s.get("pc")
    ref, _ = s.solve_system(*a, solver="amg_bicgs")
    assert np.array_equal(x, ref)
    s.close()


@pytest.mark.parametrize("batched", [False, True])
def test_ensemble_run_reports(batched):
    from flowsolversourcecode_b200 import ensemble as E
    specs = [E.CaseSpec(10, 1.0, 400.0), E.CaseSpec(12, 0.7, 150.0)]
    ens = E.Ensemble([E.build_case(q) for q in specs])
    c = ens.solvers[1]
    assert c.lib.fs_test_wait_timeout(c.ctx, -1) == 0      # in the graph, not in the iterations before it
    _times_out(lambda: ens.run(iters=2, launches=1, batched=batched))
    assert c.lib.fs_test_wait_timeout(c.ctx, 0) == 0
    ens.close()
    ens = E.Ensemble([E.build_case(q) for q in specs])
    assert np.all(np.isfinite(ens.run(iters=2, launches=1, batched=batched)["source"]))
    ens.close()


def test_long_serial_work_is_not_a_timeout():
    """CTA 0 does every level of this mesh alone, here for seconds a cycle, while
    the other CTAs wait at a barrier: their limit follows the sweeps asked for."""
    from flowsolversourcecode_b200 import mesh as fm
    from flowsolversourcecode_b200.solver import Solver
    _, case = cs.cavity(4, mg_post=40000, mg_max_cycles=1)
    s = Solver(fm.box_mesh(12, 12, 12), case)
    ac, anb, b = _system(s)
    x, it = s.solve_system(ac, anb, b, rrf=1e-300, solver="amg")
    assert it == 1
    cn = s.connectivity()["cn"].reshape(s.W, s.N)
    r = b - ac * x - np.where(cn >= 0, anb.reshape(s.W, s.N) * x[np.maximum(cn, 0)], 0.0).sum(axis=0)
    # so many sweeps leave rounding: a few units of 1e-16 times the row sums over |b|
    assert np.abs(r).max() < 1e-12 * np.abs(b).max()
    s.close()
