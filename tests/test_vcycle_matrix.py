"""The coarse matrices that the one-phase V-cycle works on: assembled from static
lists into a layout of their own, and equal bit for bit to those that
fs_mg_coarse_matrix gives (which tests/test_configs.py compares with the CPU
restatement): both sum every entry in the reference's order."""
import numpy as np
import pytest

from flowsolversourcecode_b200 import case as cs
from test_vcycle import _shuffled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("system", ["pc", "velx"])
def test_vcycle_matrices_equal_the_coarse_matrices(system, shuffled):
    from flowsolversourcecode_b200 import _lib as L
    from flowsolversourcecode_b200.solver import Solver
    mesh, case = cs.cavity(19, nz=16, jitter=0.2, seed=2, conv_scheme="sou", niter_start_hr=1, krylov_tol=1e-10,
                           krylov_maxit=300)
    s = Solver(_shuffled(mesh, 5) if shuffled else mesh, case)
    for _ in range(2):
        s.simple_iteration()
    s.set_iteration(3)
    if system == "pc":
        s.assemble_continuity()
    else:
        s.assemble_momentum(0)
    info = s.mg_info()
    assert info["direct"] and info["prec_coarsest"] >= 2
    for q in range(1, info["prec_coarsest"] + 1):
        n, w = info["sizes"][q], info["widths"][q]
        ref = s.mg_coarse_matrix(q)
        used = np.arange(w)[:, None] < ref["n_nbr"][None, :]
        for f32 in (0, 1):
            ac, anb = np.full(n, np.nan), np.full(n * w, np.nan)
            assert s.lib.fs_mg_vcycle_matrix(s.ctx, q, f32, L.dptr(ac), L.dptr(anb), n, w) == 0
            rac, ranb = ref["ac"], np.where(used, ref["anb"].reshape(w, n), 0.0)
            if f32:
                rac, ranb = rac.astype(np.float32).astype(float), ranb.astype(np.float32).astype(float)
            assert np.array_equal(ac, rac) and np.array_equal(anb.reshape(w, n), ranb), (q, f32)
    s.close()
