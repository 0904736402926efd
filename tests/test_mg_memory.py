"""Device memory that the first AMG-BiCGSTAB solve of a context adds to it.

The mesh-ordered levels in both precisions, which these solvers held before the
V-cycle had a layout of its own, took 273 bytes a cell on this mesh (112 of level
0, the rest coarse levels and the granularity of allocations).  The layout may
not take more, with or without row patterns of level 0, or the largest mesh that
fits the device shrinks: the mesh-ordered levels are allocated where a solver
works on them."""
import numpy as np
import pytest

from flowsolversourcecode_b200 import case as cs
from flowsolversourcecode_b200 import mesh as fm
from test_vcycle import _shuffled

pytestmark = pytest.mark.gpu

BYTES_PER_CELL = 273


@pytest.fixture(scope="module")
def meshes():
    m = fm.box_mesh(90, 83, 71)
    return {"rows": m, "shuffled": _shuffled(m, 5)}


@pytest.mark.parametrize("solver", ["amg_bicgs", "amg32_bicgs", "amg32gs_bicgs"])
@pytest.mark.parametrize("numbering", ["rows", "shuffled"])
def test_first_solve_takes_no_more_than_the_mesh_ordered_levels(meshes, numbering, solver):
    import torch
    from flowsolversourcecode_b200.solver import Solver
    _, case = cs.cavity(4, krylov_tol=1e-8, krylov_maxit=2)
    s = Solver(meshes[numbering], case)
    con = s.connectivity()
    anb = np.where(con["cn"] >= 0, -1.0, 0.0)
    ac = -anb.reshape(s.W, s.N).sum(axis=0) + 0.01
    s.sync()
    before = torch.cuda.mem_get_info()[0]
    s.solve_system(ac, anb, np.ones(s.N), solver=solver)
    assert before - torch.cuda.mem_get_info()[0] <= BYTES_PER_CELL * s.N
    s.close()
