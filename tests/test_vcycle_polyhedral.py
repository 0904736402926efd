"""The V-cycle on cells with more faces than a hexahedron, against the NumPy
restatement of test_vcycle.py: rows of level 0 with more slots than the six that
the row patterns give (bricks in a staggered bond: 8), than patterns take at all
(pairs of hexahedra with their faces kept apart: 10), and than the gradient
scratch holds of the FP32 cycle's matrix (blocks of four: 16 and a diagonal)."""
import numpy as np
import pytest

from flowsolversourcecode_b200 import mesh as fm
from test_vcycle import _one_iteration


def _outline(quads):
    """One polygon around coplanar quads that share edges."""
    edges = set()
    for q in quads:
        for a, b in zip(map(int, q), map(int, np.roll(q, -1))):
            if (b, a) in edges:
                edges.remove((b, a))
            else:
                edges.add((a, b))
    after = dict(edges)
    assert len(after) == len(edges)
    loop = [min(after)]
    while len(loop) < len(after):
        loop.append(after[loop[-1]])
    assert after[loop[-1]] == loop[0] and len(set(loop)) == len(loop)
    return loop


def _merged(dims, cell_of, join):
    """box_mesh(*dims) with its cells merged: cell_of(i, j, k) gives the new
    cell.  join: the faces between two cells, or of a cell on a patch, become one."""
    nx, ny, nz = dims
    m = fm.box_mesh(nx, ny, nz)
    c = np.arange(m.n_cells)
    new = np.array([cell_of(i, j, k) for i, j, k in zip(c % nx, c // nx % ny, c // (nx * ny))])
    _, new = np.unique(new, return_inverse=True)
    F = m.n_internal
    quads = m.face_nodes.reshape(-1, 4)
    groups = {}
    for f in range(m.n_faces):
        own = int(new[m.owner[f]])
        if f < F:
            nbr, patch, q = int(new[m.neighbour[f]]), -1, quads[f]
            if own == nbr:
                continue
            if own > nbr:
                own, nbr, q = nbr, own, q[::-1]
        else:
            nbr, q = -1, quads[f]
            patch = int(np.searchsorted(m.patch_start, f, side="right")) - 1
        axis = int(np.argmin(np.ptp(m.points[q], axis=0)))
        groups.setdefault((patch, own, nbr, axis if join else f), []).append(q)
    faces, owner, nbrs, size = [], [], [], [0] * len(m.patch_names)
    for (patch, own, nbr, _), qs in sorted(groups.items(), key=lambda kv: kv[0]):
        faces.append(_outline(qs) if len(qs) > 1 else [int(v) for v in qs[0]])
        owner.append(own)
        if patch < 0:
            nbrs.append(nbr)
        else:
            size[patch] += 1
    start = len(nbrs) + np.concatenate([[0], np.cumsum(size)[:-1]])
    return fm.PolyMesh(m.points, np.concatenate([[0], np.cumsum([len(f) for f in faces])]).astype(np.int32),
                       np.concatenate(faces).astype(np.int32), np.array(owner, np.int32), np.array(nbrs, np.int32),
                       m.patch_names, start.astype(np.int32), np.array(size, np.int32))


def _bricks():
    # rows of bricks two cells long, every other row shifted by a cell
    return _merged((16, 14, 10), lambda i, j, k: ((k * 14 + j) * 64) + (i + j % 2) // 2, True)


def _pairs():
    return _merged((14, 12, 20), lambda i, j, k: ((k // 2) * 12 + j) * 14 + i, False)


def _blocks():
    return _merged((14, 16, 20), lambda i, j, k: ((k // 2) * 8 + j // 2) * 14 + i, False)


MESHES = {"bricks": (_bricks, 8), "pairs": (_pairs, 10), "blocks": (_blocks, 16)}


def _slots(mesh):
    n = np.bincount(mesh.owner, minlength=mesh.n_cells)
    return int((n + np.bincount(mesh.neighbour, minlength=mesh.n_cells)).max())


@pytest.mark.parametrize("name", MESHES)
def test_meshes_have_the_slots_they_are_for(name):
    make, w = MESHES[name]
    assert _slots(make()) == w


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["amg_bicgs", "amg32_bicgs", "amg32gs_bicgs"])
@pytest.mark.parametrize("name", MESHES)
def test_one_iteration_matches_numpy_polyhedral(name, solver):
    _one_iteration(MESHES[name][0](), solver, False)
