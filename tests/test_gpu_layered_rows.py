"""Element matrices of the layered shells on the GPU (rows in the compact layout)
against the host build of the same rows in the dense one, at element counts
around the tiles, with two layups of which one couples membrane and bending."""
import numpy as np
import pytest

import flexshell as F
from flexshell import _abi
from hostcheck import hostmath as HC
import problems as PB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quads,avgk", [(False, 0), (False, 1), (True, 0)])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 33, 127, 129])
def test_against_the_host_rows(quads, avgk, n):
    xyz, conn, dof, nfree = PB.jittered_plate(9 if not quads else 12, quads, wavy=0.05, seed=n)
    conn = conn[:n]
    assert len(conn) == n
    c, s = np.cos(0.4), np.sin(0.4)
    cs = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1.0]])
    plies = [PB.cross_ply_groups((0, 90, 90, 0)), PB.cross_ply_groups((30, -45, 60))]
    groups = [F.laminate(p) for p in plies]
    groups[1].csmat[:] = list(cs.flatten(order="F"))
    eg = np.arange(n) % 2
    cls = F.FEMMShellQ4RSComp if quads else F.FEMMShellT3FFComp
    femm = cls(conn, [(g, np.flatnonzero(eg == k) + 1) for k, g in enumerate(groups[:min(n, 2)])])
    femm.transv_shear_formulation = avgk
    geom0 = F.NodalField(xyz)
    femm.associategeometry(geom0)
    et = _abi.FS_Q4RSCOMP if quads else _abi.FS_T3FFCOMP
    prm = _abi.make_params(np.eye(3), np.eye(2), 0.0, 0.0, quads=quads, transv_shear_formulation=avgk)
    tol = {F.FS_FP64: 1e-12, F.FS_MIXED: 2e-5, F.FS_MIXED_COMP: 2e-5}   # float rows: a few hundred 6e-8
    for precision in tol:
        G = femm.element_matrices(geom0, precision=precision)
        H = HC.element_matrices(et, precision, xyz, conn, femm._normals, femm._normal_valid, 0.0, prm, groups=groups,
                                egroup=eg)
        scale = np.abs(H).max(axis=(1, 2))
        assert (np.abs(G - H).max(axis=(1, 2)) <= tol[precision] * scale).all()
    femm.close()


@pytest.mark.parametrize("quads", [False, True])
def test_elements_beyond_the_fixed_point(quads):
    # FS_FP64: an element next to a double's limits or with no extent keeps the
    # products in double, among others that do not
    n, nen = 40, 4 if quads else 3
    rng = np.random.default_rng(8)
    base = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]] if quads else [[0, 0, 0], [1, 0, 0], [0, 1, 0]], float)
    X = base + rng.uniform(-0.1, 0.1, (n, nen, 3)) * [1, 1, 0.2]
    bad = [0, 17, 39]
    Y = X.copy()
    # (not smaller: squares of areas, which the double path forms too, lose digits)
    Y[0] *= 1e-70
    Y[17] = [0.5, 0.25, 0.0] if not quads else Y[17] * 1e-74
    Y[39] *= 1e70
    conn = np.arange(1, n * nen + 1).reshape(n, nen)
    group = F.laminate(PB.cross_ply_groups((30, -45, 60)))
    out = []
    for P in (X, Y):
        femm = (F.FEMMShellQ4RSComp if quads else F.FEMMShellT3FFComp)(conn, group)
        geom0 = F.NodalField(P.reshape(-1, 3))
        femm.associategeometry(geom0)
        out.append(femm.element_matrices(geom0))
        H = HC.element_matrices(_abi.FS_Q4RSCOMP if quads else _abi.FS_T3FFCOMP, F.FS_FP64, P.reshape(-1, 3), conn,
                                femm._normals, femm._normal_valid, 0.0,
                                _abi.make_params(np.eye(3), np.eye(2), 0.0, 0.0, quads=quads), groups=[group],
                                egroup=np.zeros(n))
        for e in range(n):
            assert np.array_equal(np.isfinite(out[-1][e]), np.isfinite(H[e]))
            # (a tiny element's largest entries are the rounding of its normals times 1e70)
            if np.isfinite(H[e]).all() and (P is X or e not in bad[:2]):
                assert np.abs(out[-1][e] - H[e]).max() <= 1e-12 * np.abs(H[e]).max()
        femm.close()
    rest = np.setdiff1d(np.arange(n), bad)
    assert np.array_equal(out[0][rest], out[1][rest])
