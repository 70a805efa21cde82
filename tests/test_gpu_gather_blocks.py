"""The gather's block list at its edges: nodes in any order (element blocks
stored transposed), an element with a repeated node (two contributions of one
element to one block, one of them read transposed), nodes of no element, more
than six contributions to a block, a last warp that is not full, dofs left out
of the matrix.  FP64 and FS_MIXED values bitwise against a host sum of the
library's element matrices in assembly order, FS_MIXED_COMP within the bound
of its sums."""
import numpy as np
import pytest

import flexshell as F
import problems as PB
from test_gpu_gather_sums import _check

pytestmark = pytest.mark.gpu


def _femm(xyz, conn, fixed=None):
    dchi = F.NodalField(np.zeros((xyz.shape[0], 6)))
    for nodes, comp in fixed or []:
        dchi.setebc(nodes, comp)
    dchi.numberdofs()
    cls = F.FEMMShellQ4RS if conn.shape[1] == 4 else F.FEMMShellT3FF
    femm = cls(conn, 0.01, F.materials.MatDeforElastIso(2.0e11, 0.3, 7850.0))
    return femm, F.NodalField(xyz), dchi


@pytest.mark.parametrize("quads", [False, True])
@pytest.mark.parametrize("n", [1, 2, 5, 9])
def test_permuted_nodes_and_orphans(quads, n):
    xyz, conn, _, _ = PB.jittered_plate(n, quads, wavy=0.02, seed=n)
    rng = np.random.default_rng(n)
    nn = xyz.shape[0] + 3                     # three nodes of no element
    to = rng.permutation(nn)[:xyz.shape[0]]
    X = rng.normal(size=(nn, 3))
    X[to] = xyz
    c = to[conn - 1] + 1
    femm, geom0, dchi = _femm(X, c, [([c[0, 0]], 3), ([c[-1, 1]], 5), (c[0, 1:2], 1)])
    femm.associategeometry(geom0)
    _check(femm, geom0, dchi, c, dchi.nalldofs())
    _check(femm, geom0, dchi, c, dchi.nfreedofs)
    femm.close()


@pytest.mark.parametrize("repeat", [(2, 3), (0, 1), (3, 0)])
def test_quadrilaterals_with_a_repeated_node(repeat):
    xyz, conn, _, _ = PB.jittered_plate(3, True, wavy=0.0, seed=4)
    conn = conn.copy()
    conn[4, repeat[0]] = conn[4, repeat[1]]
    femm, geom0, dchi = _femm(xyz, conn)
    femm.associategeometry(geom0)
    nrm = np.zeros((xyz.shape[0], 3), order="F")
    nrm[:, 2] = 1.0
    femm.set_normals(nrm, np.ones(xyz.shape[0], np.uint8))
    assert np.isfinite(femm.element_matrices(geom0)).all()
    _check(femm, geom0, dchi, conn, dchi.nalldofs())
    femm.close()


@pytest.mark.parametrize("m", [3, 7, 8, 13, 40])
def test_fans(m):
    # m triangles around one node: m contributions to its own block
    ang = np.linspace(0, 2 * np.pi, m, endpoint=False)
    xyz = np.r_[np.c_[np.cos(ang), np.sin(ang), 0.05 * np.sin(2 * ang)], [[0.0, 0.0, 0.0]]]
    conn = np.array([[m + 1, 1 + k, 1 + (k + 1) % m] for k in range(m)])
    femm, geom0, dchi = _femm(xyz, conn, [([1], 2)])
    femm.associategeometry(geom0)
    _check(femm, geom0, dchi, conn, dchi.nalldofs())
    _check(femm, geom0, dchi, conn, dchi.nfreedofs)
    femm.close()
